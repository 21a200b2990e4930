// Sparse MLA attention for calls of few tokens: a cluster of four blocks works on one token. The
// arithmetic is that of `attention_kernel`, operation for operation (a token's result does not
// depend on how many others are in the call); what is spread over the blocks is what does not
// depend on the order of the chunks.
//
//   1. Every block resolves the token and gathers up to three of its ten chunks (items r, r + 4 and
//      r + 8 for block r).
//   2. Q X^T of its own chunks, and their maxima per head, which go to all four blocks. Meanwhile it gathers, of
//      all chunks, the 128 features it will produce.
//   3. With all maxima known every block can follow the running reference through the chunks
//      (examples/sparse_attention/attention.py:398-490): it takes its own chunks' exponentials and sends
//      P and the partial sums to the other three (bulk copies).
//   4. O += P X over all chunks in order for its 128 features (M = 64, N = 128), normalise, store.
//
// Bound by latency. One token on one block takes 30 k cycles: 6 k until its first scores, 2 k per chunk, 3 k for
// the output pass. Here the chunks' first product and softmax run side by side, and the output pass is a
// quarter. Of the 15 k cycles that are left the token's resolution takes 2.9 k, gather, scores and maxima of up to
// three chunks 5.3 k, the first P 1 k, the second product, in the order of the chunks, 4.5 k (and a thousand more for
// every chunk at which a reference moves), output 1.3 k. Between calls of one token 8.8 us pass, of 16 tokens 9.2, of 33 tokens
// 11.2 (10.7, 11.0 and 12.9 before the issuing threads were elected and the softmax's way from maxima to P was cut short); 1.3 to 1.6 of
// them lie between the end of one launch and the first instruction of the next that may read. Eight blocks: 9.19 against 9.18 for one token,
// 10.3 against 9.3 for eight. P written to the other blocks by the softmax threads instead of bulk copies was slower by a fifth.
// Copies between blocks are of local shared memory; nothing multicasts.
//
// Tensor memory: columns 0-63, 128-191 and 384-447 the scores of the own chunks, 256-383 Q and 448-463 its
// metadata as in `attention_kernel`; once all scores are computed, 256-319 O (128 features).
#pragma once

#include "sparse_mla_tcgen05.cuh"

namespace sparse_mla {
namespace team {

using namespace sm100;
using namespace umma;

constexpr int kBlocks = 4;                       // of a cluster
constexpr int kOwnItems = 3;                     // chunks of a block, at most
constexpr int kSliceBytes = 2 * kBlockBytes;     // 64 rows x 128 features
static_assert(kOwnItems * kBlocks >= kMaxChunks && kFeatures == kBlocks * 128, "four blocks cover a token");

// Shared memory (bytes from the 1024-aligned base; the row list, token info and misc words lie where
// `attention_kernel` has them). The own chunks' tiles fill the ring's place. Once all blocks have
// computed their scores it holds eight slices (the last two chunks' come when the first two have been
// used) and, behind them, all P tiles and partial sums.
constexpr int kPBytes = kHeads * 128;
constexpr int kSumBytes = 2 * kHeads * 4;        // float[2 row halves][64 heads]
constexpr int kSliceSlots = 8;
constexpr int kTeamSlices = 0;
constexpr int kTeamP = kSliceSlots * kSliceBytes;
constexpr int kTeamSums = kTeamP + kMaxChunks * kPBytes;
constexpr int kTeamMaxima = kTeamSums + kMaxChunks * kSumBytes;  // float[10][64]
static_assert(kTeamMaxima + kMaxChunks * kHeads * 4 <= kSmemRows && kTeamMaxima >= kOwnItems * kTileBytes,
              "areas do not meet; maxima arrive while tiles are in use");
static_assert(kMaxChunks - kSliceSlots == 2, "two late slices");
static_assert(kTileBytes == kBlocks * kSliceBytes && kTeamSlices == kSmemKv && kSliceSlots == 2 * kBlocks, "slices of the first two own chunks lie in their tiles");
__host__ __device__ constexpr uint32_t score_columns(int own) { return own == 0 ? 0 : own == 1 ? 128 : 384; }
constexpr uint32_t kTeamO = kTmemQ;

enum TeamBar {
  kReady = 0, kQReady, kTile0, kTile1, kTile2, kScores0, kScores1, kScores2, kMaxima, kMaskReady, kPvDone, kRescaled, kOutput,
  kSlices0,                                   // of two chunks each
  kP0 = kSlices0 + kMaxChunks / 2,
  kSliceFree0 = kP0 + kMaxChunks, kSliceFree1,
  kTeamBarCount
};
static_assert(kTeamBarCount <= 32, "the barrier area holds 32 mbarriers");

template <int kFormat> constexpr uint32_t kIdescTeamPv = idesc_f16(64, 128, kFormat, 0, 1);  // issued as .ws

// The lazy running reference of one head through the chunks, from their maxima: `visit(item, reference,
// alpha)` for every chunk. The same comparisons as in `attention_kernel`, but where no head of the warp has a chunk behind
// the first that moves it, which is the rule, they are one: the highest of those chunks does not. (All maxima are loaded
// first: a chain of shared loads behind the slices' copies takes a thousand cycles.) Called by whole warps.
template <typename Visit>
__device__ __forceinline__ void follow_reference(const volatile float* maxima, float sink, int chunks, Visit visit) {
  float chunk_max[kMaxChunks];
#pragma unroll
  for (int i = 0; i < kMaxChunks; ++i) chunk_max[i] = maxima[i * kHeads];
  float reference = sink;
  const float first = move_reference(reference, chunk_max[0], true);
  visit(0, reference, first);
  float highest = -INFINITY;
#pragma unroll
  for (int i = 1; i < kMaxChunks; ++i) highest = fmaxf(highest, i < chunks ? chunk_max[i] : -INFINITY);
  const bool moves = __any_sync(0xffffffffu, highest - reference > kReferenceRoom);
  if (!moves) {
#pragma unroll
    for (int i = 1; i < kMaxChunks; ++i) visit(i, reference, 1.f);
    return;
  }
#pragma unroll
  for (int i = 1; i < kMaxChunks; ++i) {
    const float alpha = i < chunks ? move_reference(reference, chunk_max[i], false) : 1.f;
    visit(i, reference, alpha);
  }
}

// Phase A, producer warps: Q to tensor memory, the own chunks' tiles.
__device__ void team_gather(const Params& p, const Shared& sm, uint32_t tmem, int token, int rank) {
  const int tid = threadIdx.x - kFirstProducerWarp * 32, lane = tid & 31, warp = threadIdx.x >> 5;
  const int subpartition = warp & 3, part = (warp - kFirstProducerWarp) >> 2;
  volatile int* abort_flag = sm.abort_flag();
  uint32_t words[64];  // see producer_role
  load_q<0, kQLoads>(q_rows(p, token, subpartition, part, lane), words);
  if (!warp_wait(sm.bar(kReady), 0, abort_flag)) return;
  const int* rows = sm.rows(0);
  const TokenInfo* info = sm.info(0);
  const int chunks = info->chunks;
  for (int j = 0; j < kOwnItems; ++j) {
    const int item = rank + j * kBlocks;
    if (item >= chunks) break;
    gather_rows<0, 1>(p, rows, info->chunk[item], sm.base + kSmemKv + j * kTileBytes, tid);
    cp_async_arrive(sm.bar(kTile0 + j));
    if (j > 0) continue;
    const uint32_t q_tmem = tmem + kTmemQ + part * 64 + (uint32_t(subpartition * 32) << 16);
    store_q(q_tmem, words);
    if (part == 0) store_places(tmem + kTmemPlaces + (uint32_t(subpartition * 32) << 16), lane);
    tmem_wait_st();
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(sm.bar(kQReady));
  }
}

// Copies of `kItems` chunks' slices (as many of them as there are), this block's 128 features of their 64 rows, by
// `kThreadCount` threads: sixteen per row. All row numbers first: a round trip to shared memory per row would
// take as long as the copies.
template <int kItems, int kThreadCount>
__device__ __forceinline__ void gather_slices(const Params& p, const Shared& sm, int rank, int item, int chunks, int thread) {
  constexpr int kRows = kChunkRows / (kThreadCount / 16);
  const int unit = thread & 15;
  int chunk[kItems], row[kItems][kRows];
#pragma unroll
  for (int i = 0; i < kItems; ++i) chunk[i] = sm.info(0)->chunk[min(item + i, chunks - 1)];
#pragma unroll
  for (int i = 0; i < kItems; ++i)
#pragma unroll
    for (int k = 0; k < kRows; ++k) row[i][k] = sm.rows(0)[chunk[i] * kChunkRows + (thread >> 4) + k * (kThreadCount / 16)];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    if (item + i >= chunks) break;
    if (item + i < kSliceSlots && (item + i) % kBlocks == rank) continue;  // in place
    const char* cache = static_cast<const char*>(chunk[i] * kChunkRows < kWindow ? p.ori_kv : p.cmp_kv) + rank * 256 + unit * 16;
    const uint32_t slice = sm.base + kTeamSlices + (item + i) % kSliceSlots * kSliceBytes + (unit >> 3) * kBlockBytes;
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const int r = (thread >> 4) + k * (kThreadCount / 16);
      cp_async16(slice + r * 128 + (((unit & 7) ^ (r & 7)) << 4), cache + (size_t)max(row[i][k], 0) * kRowBytes, row[i][k] >= 0);
    }
  }
}

// Phase A, producer warps: the first eight chunks' slices. They fill the places of the own chunks' first two
// tiles, four each, which are free when these have been multiplied. A block's slice of its own chunk is there already: in the tile's order of
// features it lies just where the slice of that item has to be (one token 8.88 -> 8.80 us, 33 tokens 11.21 -> 11.11).
__device__ void team_early_slices(const Params& p, const Shared& sm, int rank) {
  const int tid = threadIdx.x - kFirstProducerWarp * 32;
  volatile int* abort_flag = sm.abort_flag();
  if (*abort_flag != 0) return;  // (the token may not be there)
  const int chunks = sm.info(0)->chunks;
  static_assert(kTileBytes == 4 * kSliceBytes && kSliceSlots == 8, "four slices to a tile");
#pragma unroll 1
  for (int item = 0; item < min(chunks, kSliceSlots); item += 2) {
    const int own = item / 4;
    if (item % 4 == 0 && rank + own * kBlocks < chunks && !warp_wait(sm.bar(kScores0 + own), 0, abort_flag)) return;
    gather_slices<2, kProducerThreads>(p, sm, rank, item, chunks, tid);
    cp_async_arrive(sm.bar(kSlices0 + item / 2));
  }
}

// Phase B, producer warps: four of them rescale O where a reference moves, the other four gather the last two
// slices.
__device__ void team_slices(const Params& p, const Shared& sm, uint32_t tmem, int rank) {
  const int tid = threadIdx.x - kFirstProducerWarp * 32, lane = tid & 31, warp = threadIdx.x >> 5;
  volatile int* abort_flag = sm.abort_flag();
  if (*abort_flag != 0) return;
  const int chunks = sm.info(0)->chunks;
  if (chunks == 0) return;
  if (warp >= kFirstProducerWarp + 4) {
    if (chunks <= kSliceSlots) return;
    for (int item = kSliceSlots; item < chunks; ++item) {
      if (!warp_wait(sm.bar(kSliceFree0 + item - kSliceSlots), 0, abort_flag)) return;
      gather_slices<1, 128>(p, sm, rank, item, chunks, tid - 128);
    }
    cp_async_arrive(sm.bar(kSlices0 + kSliceSlots / 2));
  } else {
    if (!warp_wait(sm.bar(kMaskReady), 0, abort_flag) || !warp_wait<true>(sm.bar(kMaxima), 0, abort_flag)) return;
    const int o_head = (warp & 1) * 32 + lane;  // lane l of tensor memory: head l % 64 (see softmax_role)
    const uint32_t o_addr = tmem + kTeamO + (uint32_t((warp & 3) * 32) << 16);
    const float sink = __ldg(p.sinks + o_head) * 1.4426950408889634f;
    uint32_t phase = 0;
    for (uint32_t left = *sm.rescale_mask(); left != 0; left &= left - 1) {
      const int item = __ffs(left) - 1;
      float factor = 1.f;
      follow_reference(sm.maxima(kTeamMaxima) + o_head, sink, chunks, [&](int i, float, float alpha) { if (i == item) factor = alpha; });
      if (!warp_wait(sm.bar(kPvDone), phase++ & 1, abort_flag)) return;
      tc_fence_after_sync();
#pragma unroll 1
      for (int c = 0; c < 64; c += 16) {
        uint32_t o[16];
        tmem_ld16(o_addr + c, o);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * factor);
        tmem_st16(o_addr + c, o);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(sm.bar(kRescaled));
    }
  }
}

// Phase B, one warp: the chunks after the first that move some head's reference.
__device__ void team_mask(const Shared& sm, float sink, float other_sink) {  // of heads lane, 32 + lane
  volatile int* abort_flag = sm.abort_flag();
  if (!warp_wait<true>(sm.bar(kMaxima), 0, abort_flag)) return;
  const int lane = threadIdx.x & 31, chunks = sm.info(0)->chunks;
  uint32_t moved = 0;
  auto note = [&](int i, float, float alpha) { moved |= uint32_t(i > 0 && alpha != 1.f) << i; };
  follow_reference(sm.maxima(kTeamMaxima) + lane, sink, chunks, note);
  follow_reference(sm.maxima(kTeamMaxima) + 32 + lane, other_sink, chunks, note);
  moved = __reduce_or_sync(0xffffffffu, moved);
  if (lane == 0) {
    *sm.rescale_mask() = moved;
    mbar_arrive(sm.bar(kMaskReady));
  }
}

// Phase A, one thread: the own chunks' scores.
template <int kFormat>
__device__ void team_qk(const Shared& sm, uint32_t tmem, int rank) {
  volatile int* abort_flag = sm.abort_flag();
  if (!mbar_wait(sm.bar(kReady), 0, abort_flag)) return;
  const int chunks = sm.info(0)->chunks;
  if (rank >= chunks || !mbar_wait(sm.bar(kQReady), 0, abort_flag)) return;
#pragma unroll
  for (int j = 0; j < kOwnItems; ++j) {
    if (rank + j * kBlocks >= chunks || !wait_for_copies(sm.bar(kTile0 + j), 0, abort_flag)) return;
    tc_fence_after_sync();
    issue_qk<kFormat>(sm, tmem, j, score_columns(j));
    mma_commit(sm.bar(kScores0 + j));
  }
}

template <int kFormat, int K, bool kFirst>
__device__ __forceinline__ void issue_team_pv(uint32_t tmem, uint64_t p_desc, uint64_t x_desc) {
  if constexpr (K < kChunkRows / 16) {
    mma_ws_ss_c<!(kFirst && K == 0)>(tmem + kTeamO, p_desc + ((K * 32) >> 4), x_desc + ((K * 2048) >> 4), kIdescTeamPv<kFormat>);
    issue_team_pv<kFormat, K + 1, kFirst>(tmem, p_desc, x_desc);
  }
}

// Phase B, one thread: O = P X over all chunks, this block's 128 features. Unrolled over the chunks, so that
// descriptors are constants off two addresses (in a loop one token 9.69 us against 8.83, 16 tokens 10.02 against 9.20; two
// chunks to a pass 9.14 and 9.46).
template <int kFormat>
__device__ void team_pv(const Shared& sm, uint32_t tmem) {
  volatile int* abort_flag = sm.abort_flag();
  if (!mbar_wait(sm.bar(kMaskReady), 0, abort_flag)) return;
  const int chunks = sm.info(0)->chunks;
  if (chunks == 0) return;
  const uint32_t rescale_mask = *sm.rescale_mask();
  uint32_t rescales = 0;
  const uint64_t p_first = smem_desc_sw128(sm.base + kTeamP, 16, 1024), x_first = smem_desc_sw128(sm.base + kTeamSlices, kBlockBytes, 1024);
#pragma unroll
  for (int i = 0; i < kMaxChunks; ++i) {
    if (i >= chunks) break;
    if ((i & 1) == 0 && !wait_for_copies(sm.bar(kSlices0 + i / 2), 0, abort_flag)) return;
    if (!mbar_wait<true>(sm.bar(kP0 + i), 0, abort_flag)) return;
    if (rescale_mask >> i & 1) {  // some head's reference moves here: O is rescaled first
      mma_commit(sm.bar(kPvDone));
      if (!mbar_wait(sm.bar(kRescaled), rescales++ & 1, abort_flag)) return;
    }
    tc_fence_after_sync();
    const uint64_t p_desc = p_first + uint32_t(i * (kPBytes >> 4));
    const uint64_t x_desc = x_first + uint32_t((i & (kSliceSlots - 1)) * (kSliceBytes >> 4));
    if (i == 0) issue_team_pv<kFormat, 0, true>(tmem, p_desc, x_desc);
    else issue_team_pv<kFormat, 0, false>(tmem, p_desc, x_desc);
    if (i + kSliceSlots < chunks) mma_commit(sm.bar(kSliceFree0 + i));
  }
  mma_commit(sm.bar(kOutput));
}

// Phase B, one thread: every own chunk's P and partial sums to the other blocks.
__device__ void team_send(const Shared& sm, int rank) {
  volatile int* abort_flag = sm.abort_flag();
  if (!mbar_wait(sm.bar(kReady), 0, abort_flag)) return;
  const int chunks = sm.info(0)->chunks;
  for (int item = rank; item < chunks; item += kBlocks) {
    if (!mbar_wait(sm.bar(kP0 + item), 0, abort_flag)) return;
    const uint32_t tile = sm.base + kTeamP + item * kPBytes, sums = sm.base + kTeamSums + item * kSumBytes;
    for (int other = 1; other < kBlocks; ++other) {
      const uint32_t to = uint32_t(rank + other) % kBlocks, bar = cluster_address(sm.bar(kP0 + item), to);
      bulk_copy_to_block(cluster_address(tile, to), tile, kPBytes, bar);
      bulk_copy_to_block(cluster_address(sums, to), sums, kSumBytes, bar);
    }
  }
}

// 32 bytes to global memory by one instruction, which covers whole sectors (one token 9.13 -> 9.01 us, 33 tokens 11.60 -> 11.56
// against two of 16), or by two where the output starts between sectors.
__device__ __forceinline__ void store_sector(char* to, const uint32_t (&words)[8], bool aligned) {
  if (aligned) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(to), "r"(words[0]), "r"(words[1]), "r"(words[2]),
                 "r"(words[3]), "r"(words[4]), "r"(words[5]), "r"(words[6]), "r"(words[7]) : "memory");
  } else {
    reinterpret_cast<uint4*>(to)[0] = make_uint4(words[0], words[1], words[2], words[3]);
    reinterpret_cast<uint4*>(to)[1] = make_uint4(words[4], words[5], words[6], words[7]);
  }
}

// A thread's scores of own chunk `own` (as in softmax_role): 32 rows of its head.
__device__ __forceinline__ void team_scores(uint32_t tmem, int own, unsigned live, float2 (&raw)[16]) {
  const uint32_t s_addr = tmem + score_columns(own) + (uint32_t((threadIdx.x >> 5) * 32) << 16);
  uint32_t low_a[16], low_b[16], high_a[16], high_b[16];
  tmem_ld16_halves<32>(s_addr, low_a);
  tmem_ld16_halves<32>(s_addr + 16, low_b);
  tmem_ld16_halves<32>(s_addr + kHalfLanes, high_a);
  tmem_ld16_halves<32>(s_addr + kHalfLanes + 16, high_b);
  tmem_wait_ld();
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    raw[e] = add_pair(make_float2(__uint_as_float(low_a[2 * e]), __uint_as_float(low_a[2 * e + 1])),
                      make_float2(__uint_as_float(high_a[2 * e]), __uint_as_float(high_a[2 * e + 1])));
    raw[8 + e] = add_pair(make_float2(__uint_as_float(low_b[2 * e]), __uint_as_float(low_b[2 * e + 1])),
                          make_float2(__uint_as_float(high_b[2 * e]), __uint_as_float(high_b[2 * e + 1])));
  }
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    if (!(live >> (2 * e) & 1u)) raw[e].x = -INFINITY;
    if (!(live >> (2 * e + 1) & 1u)) raw[e].y = -INFINITY;
  }
}

// Phase A, softmax warps: the own chunks' maxima to all blocks.
__device__ __forceinline__ void team_maxima(const Params& p, const Shared& sm, uint32_t tmem, int rank) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = lane >> 4, head = warp * 16 + (lane & 15);
  volatile int* abort_flag = sm.abort_flag();
  if (!warp_wait(sm.bar(kReady), 0, abort_flag)) return;
  const TokenInfo* info = sm.info(0);
  const int chunks = info->chunks;
  int own = 0;
  for (int item = rank; item < chunks; item += kBlocks, ++own) {
    if (!warp_wait(sm.bar(kScores0 + own), 0, abort_flag)) return;
    tc_fence_after_sync();
    float2 raw[16];
    team_scores(tmem, own, half ? info->live[item].y : info->live[item].x, raw);
    float own_max = -INFINITY, other_max = -INFINITY;
#pragma unroll
    for (int e = 0; e < 16; e += 2) {
      own_max = max3(own_max, raw[e].x, raw[e].y);
      other_max = max3(other_max, raw[e + 1].x, raw[e + 1].y);
    }
    own_max = fmaxf(own_max, other_max) * p.scale_log2;
    const float chunk_max = fmaxf(own_max, __shfl_xor_sync(0xffffffffu, own_max, 16));
    // Each of a head's two threads tells two blocks.
    const uint32_t at = sm.base + kTeamMaxima + (item * kHeads + head) * 4;
#pragma unroll
    for (int b = 0; b < kBlocks / 2; ++b) {
      const uint32_t to = half * (kBlocks / 2) + b;
      cluster_store_async(cluster_address(at, to), chunk_max, cluster_address(sm.bar(kMaxima), to));
    }
  }
  tc_fence_before_sync();
}

// Phase B, softmax warps: P of the own chunks, the denominators, the output. True: they have arrived at the cluster's last barrier.
template <int kFormat>
__device__ __forceinline__ bool team_softmax(const Params& p, const Shared& sm, uint32_t tmem, int token, int rank, float sink, float o_sink) {
  const bool aligned = (reinterpret_cast<uintptr_t>(p.out) & 31) == 0;  // (asked here: at the end it is waited for)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = lane >> 4, head = warp * 16 + (lane & 15);
  const int o_head = (warp & 1) * 32 + lane;  // see softmax_role
  const uint32_t o_addr = tmem + kTeamO + (uint32_t(warp * 32) << 16);
  volatile int* abort_flag = sm.abort_flag();
  const TokenInfo* info = sm.info(0);
  const int chunks = info->chunks;
  char* out = static_cast<char*>(p.out) + ((size_t)token * kHeads + o_head) * kRowBytes + rank * 256 + (warp >> 1) * 128;
  if (chunks == 0) {  // nothing visible: the output row is zero whatever the sink
    for (int u = 0; u < 8; ++u) *reinterpret_cast<uint4*>(out + u * 16) = make_uint4(0, 0, 0, 0);
    return false;
  }
  const volatile float* maxima = sm.maxima(kTeamMaxima);
  if (!warp_wait<true>(sm.bar(kMaxima), 0, abort_flag)) return false;  // all blocks' (and so all own scores have been read)
  // The references of all own chunks at once: followed for every chunk it took 200 cycles of the way from scores to P (16 tokens 9.37 -> 9.26 us).
  float references[kOwnItems] = {sink, sink, sink};
  follow_reference(maxima + head, sink, chunks, [&](int i, float reference, float) { if (i % kBlocks == rank) references[i / kBlocks] = reference; });
  tc_fence_after_sync();
  int own = 0;
  for (int item = rank; item < chunks; item += kBlocks, ++own) {
    const float run_max = own == 0 ? references[0] : own == 1 ? references[1] : references[2];  // (no array by a variable index)
    float2 prob[16];
    team_scores(tmem, own, half ? info->live[item].y : info->live[item].x, prob);
    const float2 scale = make_float2(p.scale_log2, p.scale_log2), reference = make_float2(-run_max, -run_max);
    float2 sum_a = make_float2(0.f, 0.f), sum_b = sum_a;  // four partial sums
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      prob[e] = fma_pair(prob[e], scale, reference);
      prob[e].x = exp2f(prob[e].x);
      prob[e].y = exp2f(prob[e].y);
      if (e & 1) sum_b = add_pair(sum_b, prob[e]); else sum_a = add_pair(sum_a, prob[e]);
    }
    unsigned char* tile = sm.ptr + kTeamP + item * kPBytes;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint4 v;
      v.x = pack_pair<kFormat>(prob[4 * u + 0].x, prob[4 * u + 0].y); v.y = pack_pair<kFormat>(prob[4 * u + 1].x, prob[4 * u + 1].y);
      v.z = pack_pair<kFormat>(prob[4 * u + 2].x, prob[4 * u + 2].y); v.w = pack_pair<kFormat>(prob[4 * u + 3].x, prob[4 * u + 3].y);
      *reinterpret_cast<uint4*>(tile + p_offset(head, half * 4 + u)) = v;
    }
    reinterpret_cast<float*>(sm.ptr + kTeamSums)[(item * 2 + half) * kHeads + head] = (sum_a.x + sum_a.y) + (sum_b.x + sum_b.y);
    fence_proxy_async();  // the PV and the copies to the other blocks read the tile through the async proxy
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(sm.bar(kP0 + item));
  }
  // The denominator: the two row halves' sums follow the reference, then add up (see softmax_role).
  // From here on the head of this thread is that of its accumulator lane.
  for (int i = 0; i < chunks; ++i)
    if (!warp_wait<true>(sm.bar(kP0 + i), 0, abort_flag)) return false;
  float low = 1.f, high = 0.f;  // the low half's share includes the sink's own weight
  follow_reference(maxima + o_head, o_sink, chunks, [&](int i, float, float alpha) {
    const volatile float* sums = reinterpret_cast<const volatile float*>(sm.ptr + kTeamSums + i * kSumBytes);
    if (i < chunks) {
      low = low * alpha + sums[o_head];
      high = high * alpha + sums[kHeads + o_head];
    }
  });
  const float inverse = 1.f / (low + high);
  // All that other blocks send is here. What they wait for at the cluster's last barrier is that, and not this block's output.
  cluster_arrive_relaxed();
  if (!warp_wait(sm.bar(kOutput), 0, abort_flag)) return true;
  tc_fence_after_sync();
  uint32_t o[64];
#pragma unroll
  for (int q = 0; q < 64; q += 16) tmem_ld16(o_addr + q, *reinterpret_cast<uint32_t(*)[16]>(&o[q]));
  tmem_wait_ld();
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    uint32_t words[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) words[e] = pack_pair<kFormat>(__uint_as_float(o[16 * u + 2 * e]) * inverse, __uint_as_float(o[16 * u + 2 * e + 1]) * inverse);
    store_sector(out + u * 32, words, aligned);
  }
  return true;
}

// Every thread passes the cluster's barrier twice: all blocks have started (their shared memory may be
// written); all copies have arrived (it may be given up). No role leaves before it has. The softmax warps, which wait for all
// copies, arrive the second time before the output. In between a block waits
// for what the others send: all maxima, with which all of them say too that their scores have been read (so that
// P may take the tiles' place; a barrier of the cluster there took 1.7 k cycles), and every chunk's P.
template <int kFormat>
__global__ void __launch_bounds__(kThreads, 1) team_kernel(const Params p) {
  extern __shared__ unsigned char smem_raw[];
  Shared sm;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw & 1023u)) & 1023u;
  sm.base = raw + pad;
  sm.ptr = smem_raw + pad;
  const int warp = threadIdx.x >> 5, rank = int(cluster_rank()), token = int(blockIdx.x) / kBlocks;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm.ptr + kSmemMisc);

  if (threadIdx.x < kTeamBarCount) {
    const int i = threadIdx.x;
    const bool a_chunk = i >= kP0 && i < kSliceFree0, mine = a_chunk && (i - kP0) % kBlocks == rank;
    const int count = i == kQReady ? kProducerWarps
                    : i == kSlices0 + kSliceSlots / 2 ? kProducerThreads / 2
                    : (i >= kTile0 && i <= kTile2) || (i >= kSlices0 && i < kP0) ? kProducerThreads
                    : mine || i == kRescaled ? kSoftmaxWarps : 1;
    mbar_init(sm.bar(i), count);
    mbar_fence_init();
    if (a_chunk && !mine) mbar_arrive_expect(sm.bar(i), kPBytes + kSumBytes);  // comes from the block that owns it
  }
  if (threadIdx.x == 0) { *sm.abort_flag() = 0; *sm.rescale_mask() = 0; }
  if (warp == kMmaWarp) { tmem_alloc(smem_u32(tmem_slot), kTmemColumns); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  prefetch_first(p, token);
  wait_for_predecessor();
  let_successor_start();
  cluster_wait();

  // Sinks (log2 domain), loaded early: of the thread's score head in the softmax warps, of heads lane and
  // 32 + lane in the others.
  const int lane = threadIdx.x & 31;
  const float sink = __ldg(p.sinks + (warp < kSoftmaxWarps ? warp * 16 + (lane & 15) : lane)) * 1.4426950408889634f;
  const float other_sink = __ldg(p.sinks + (warp < kSoftmaxWarps ? (warp & 1) * 32 : 32) + lane) * 1.4426950408889634f;
  bool arrived = false;
  if (warp == kResolverWarp) {
    publish_first_token<true>(p, sm, token, sm.bar(kReady));
    if (lane == 0) {
      mbar_arrive_expect(sm.bar(kMaxima), uint32_t(sm.info(0)->chunks * kHeads) * 4);
      team_send(sm, rank);
    }
  } else if (warp < kSoftmaxWarps) {
    publish_first_token<false>(p, sm, token, sm.bar(kReady));
    team_maxima(p, sm, tmem, rank);
    arrived = team_softmax<kFormat>(p, sm, tmem, token, rank, sink, other_sink);
  } else if (warp == kMmaWarp) {
    if (elect_one()) team_qk<kFormat>(sm, tmem, rank);
    __syncwarp();
    team_mask(sm, sink, other_sink);
  } else if (warp == kPvWarp) {
    if (elect_one()) team_pv<kFormat>(sm, tmem);
  } else {
    team_gather(p, sm, tmem, token, rank);
    team_early_slices(p, sm, rank);
    team_slices(p, sm, tmem, rank);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  }
  __syncwarp();
  // (A wait has given up: what is still on its way to or from this block gets time to arrive.)
  if (!arrived && *sm.abort_flag() != 0)
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  // What the last barrier is for is that the other blocks' copies to this one have arrived, which its waits have
  // seen, and that they have finished reading: nothing written here is read behind it, so nobody waits
  // for the output's way to memory (2.2 k cycles).
  tc_fence_before_sync();
  if (!arrived) cluster_arrive_relaxed();
  cluster_wait();
  __syncthreads();  // (the softmax warps come here from their last wait; the cluster's barrier they have passed before it)
  if (threadIdx.x == 0 && *sm.abort_flag() != 0) report(p, kStatusWaitExpired, blockIdx.x, 0);
  if (warp == kMmaWarp) tmem_dealloc(tmem, kTmemColumns);
}

inline cudaLaunchConfig_t team_config(cudaLaunchAttribute (&attributes)[2], int tokens, cudaStream_t stream) {
  attributes[0] = {};
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = kBlocks;
  attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
  attributes[1] = {};
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(unsigned(tokens * kBlocks));
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = kSmemBytes;
  config.stream = stream;
  config.attrs = attributes;
  config.numAttrs = 2;
  return config;
}

// How many tokens (clusters) the current device works on at a time; 0 if it cannot. Asked once per device
// (a word that everybody sets to the same value).
template <int kFormat>
inline int team_capacity(int device) {
  static int known[64] = {0};  // capacity + 1
  if (known[device] == 0) {
    cudaLaunchAttribute attributes[2];
    cudaLaunchConfig_t config = team_config(attributes, 1, nullptr);
    config.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(team_kernel<kFormat>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, team_kernel<kFormat>, &config) != cudaSuccess) {
      cudaGetLastError();  // not on this device, then; nothing has failed
      clusters = 0;
    }
    known[device] = clusters + 1;
  }
  return known[device] - 1;
}

// One cluster per token while all of them fit the device at once (33 on a B200); the persistent blocks
// beyond: a second round of clusters would take longer than they do.
template <int kFormat>
inline int launch(const Params& p, cudaStream_t stream, int multiprocessors) {
  int device = 0;
  const cudaError_t error = cudaGetDevice(&device);
  if (error != cudaSuccess) return int(error);
  if (device < 0 || device >= 64) return -1;
  if (p.tokens > team_capacity<kFormat>(device)) return umma::launch<kFormat>(p, stream, multiprocessors);
  cudaLaunchAttribute attributes[2];
  const cudaLaunchConfig_t config = team_config(attributes, p.tokens, stream);
  return int(cudaLaunchKernelEx(&config, team_kernel<kFormat>, p));
}

}  // namespace team
}  // namespace sparse_mla
