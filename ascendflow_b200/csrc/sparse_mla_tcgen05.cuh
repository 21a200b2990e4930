// Sparse MLA attention on the Blackwell tensor path: tcgen05.mma with operands and accumulators
// in tensor memory, warp-specialised and software-pipelined. BF16 or FP16 storage (template
// parameter kFormat), FP32 accumulation.
//
// One persistent block per SM owns one query token at a time (64 heads x 512 features) and
// walks the token's live 64-row chunks (window rows first, then the compressed ranks in list
// order, as the reference does: examples/sparse_attention/attention.py:42-64, 147-207). The
// chunks of all the block's tokens form one stream; the issue order is QK(c + 1), PV(c).
//
//   resolver warp    resolves slot -> physical row (`resolve_slots`) up to two tokens ahead.
//   producer warps   gather the token's rows with 16-byte cp.async into a three-stage ring of
//                    128-byte-swizzled shared tiles (a row is fetched once and serves as K and
//                    V), and move the token's Q from global to tensor memory through registers.
//   MMA warps        one thread issues S = Q X^T (Q from tensor memory, X K-major from the tile)
//                    and another O += P X (P from a shared tile, X MN-major from the same tile; issued
//                    as tcgen05.mma.ws so that M = 64 does not halve the rate).
//   softmax warps    tcgen05.ld S, joint online softmax with the per-head sink
//                    (examples/sparse_attention/attention.py:398-490: one maximum and one
//                    denominator over window, compressed rows and sink; P rounded to the storage
//                    type before PV, denominator from unrounded FP32), P to shared memory, O
//                    rescaled only when the running maximum moved by more than 2^15, final
//                    normalisation and store (after the next token's first chunk).
//
// Tensor memory (512 columns x 128 lanes):
//   columns   0-255  O: two weight-stationary M = 64, N = 256 accumulators (columns 0-127: features
//                    0-255, columns 128-255: features 256-511). Lane l holds head l % 64 and,
//                    of each accumulator, features 128 (l / 64) .. + 127.
//   columns 256-383  Q as 16-bit pairs: lanes 0-15 of every warp's 32 hold the even pairs of 16 heads
//                    (features 4 c and 4 c + 1 in column c), lanes 16-31 the odd pairs of the same heads.
//   columns 384-447  the score buffer of the QK product (see `issue_qk`): the partial scores of a
//                    lane's pairs.
//   columns 448-463  which pairs a lane holds, as the sparse product's metadata (written once).
// Thread (lane & 15) + 16 * half of softmax warp w works on head 16 w + (lane & 15) and rows 32 half .. + 31 of
// the chunk; it loads both partial scores of each.
//
// Every wait on an mbarrier is bounded (tcgen05_ptx.cuh): on expiry the block records
// kStatusWaitExpired, all roles leave their loops, tensor memory is released, the kernel returns. The softmax warps' named
// barrier is passed by all four of them or by none (`softmax_role`).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "sparse_mla_common.cuh"
#include "tcgen05_ptx.cuh"

namespace sparse_mla {
namespace umma {

using namespace sm100;

constexpr int kSoftmaxWarps = 4;
constexpr int kProducerWarps = 8;
constexpr int kMmaWarp = kSoftmaxWarps;                     // warp index 4
constexpr int kResolverWarp = kSoftmaxWarps + 1;            // warp index 5
constexpr int kFirstProducerWarp = kSoftmaxWarps + 2;
constexpr int kPvWarp = kFirstProducerWarp + kProducerWarps;  // warp index 14
constexpr int kThreads = 32 * (kSoftmaxWarps + 3 + kProducerWarps);
constexpr int kProducerThreads = 32 * kProducerWarps;

constexpr int kChunkRows = 64;
constexpr int kMaxChunks = kSlots / kChunkRows;             // 10
constexpr int kStages = 3;
constexpr int kBlockBytes = kChunkRows * 128;               // one 64-feature block of a tile: 8 KiB
constexpr int kTileBytes = 8 * kBlockBytes;                 // 64 rows x 512 features: 64 KiB

// Shared memory map (bytes from a 1024-aligned base).
constexpr int kSmemKv = 0;
// Two P tiles (64 heads x 64 rows, 8 KiB) for the chunks in turn and, per softmax warp, 2 KiB of epilogue staging
// (16 x 128-byte rows; 16 more in the P tile that is not in use then). All 1024-byte aligned like the tiles, because
// the swizzle is a function of the address.
constexpr int kSmemP = kSmemKv + kStages * kTileBytes;
constexpr int kPTileBytes = kHeads * 128;
constexpr int kSmemStore = kSmemP + 2 * kPTileBytes;
constexpr int kSmemRows = kSmemStore + kSoftmaxWarps * 2048;   // int[2][640]
constexpr int kSmemInfo = kSmemRows + 2 * kSlots * 4;       // TokenInfo[2]
constexpr int kSmemBars = kSmemInfo + 2 * 128;              // mbarriers
constexpr int kSmemMisc = kSmemBars + 32 * 8;               // tmem slot, abort flag
// Per-head factors handed between the softmax warps (float[2][64] each, double-buffered): a
// thread works out the softmax of one head but reads the accumulator of another (see below).
constexpr int kSmemAlpha = kSmemMisc + 64;
constexpr int kSmemInverse = kSmemAlpha + 2 * kHeads * 4;
constexpr int kSmemEnd = kSmemInverse + 2 * kHeads * 4;
constexpr int kSmemBytes = kSmemEnd + 1024;  // + slack for the 1024-byte alignment

constexpr uint32_t kTmemColumns = 512;
constexpr uint32_t kTmemO = 0;
constexpr uint32_t kTmemQ = 256;
constexpr uint32_t kTmemS = 384;                             // one 64-column score buffer
constexpr uint32_t kTmemPlaces = 448;                        // which features a lane of Q holds (see `issue_qk`)
constexpr uint32_t kTmemOHalf = 128;                         // columns of one 256-feature accumulator
constexpr uint32_t kHalfLanes = 16u << 16;                   // lane offset of lanes 16-31 (the odd pairs) in a tensor-memory address

struct TokenInfo {
  int token;
  int chunks;                 // live chunks of this token
  uint2 live[kMaxChunks];     // per live chunk, in order: live bits of its rows 0-31 and 32-63
  unsigned char chunk[kMaxChunks];
};
static_assert(sizeof(TokenInfo) <= 128, "the info area holds two 128-byte entries");

enum Bar {
  kTokenReady0 = 0, kTokenReady1, kTokenDone0, kTokenDone1, kQFull, kQFree,
  kKvFree0, kKvFree1, kKvFree2, kKvFree3, kKvFree4, kKvFree5,  // halves of the ring stages
  kSFull0, kSFull1, kPFull0, kPFull1, kOFree,
  kKvFull0, kKvFull1, kKvFull2, kOutReady, kInfoRead0, kInfoRead1, kBarCount
};
static_assert(kBarCount <= 32, "the barrier area holds 32 mbarriers");

// Storage formats of kind::f16 instructions: 0 = IEEE half, 1 = BF16.
template <int kFormat> constexpr uint32_t kIdescQK = idesc_f16(128, kChunkRows, kFormat, 0, 0) | kSparseA;
template <int kFormat> constexpr uint32_t kIdescPV = idesc_f16(64, 256, kFormat, 0, 1);  // issued as .ws

// Byte offset of 16-byte unit `unit` (0..63) of row `row` in a K-major 128-byte-swizzled tile
// of 64 rows: eight 64-feature blocks of [64 rows x 128 bytes].
__device__ __forceinline__ uint32_t swizzled(int row, int unit) {
  return (unit >> 3) * kBlockBytes + row * 128 + (((unit & 7) ^ (row & 7)) << 4);
}

// A P tile (64 heads x 64 rows of 16-bit probabilities, K-major, 128-byte swizzle: one
// 128-byte row per head): byte offset of 16-byte unit `unit` (0..7) of head `head`.
__device__ __forceinline__ uint32_t p_offset(int head, int unit) {
  return head * 128 + ((unit ^ (head & 7)) << 4);
}

struct Shared {
  uint32_t base;        // shared-space address of the 1024-aligned region
  unsigned char* ptr;   // generic pointer to the same
  __device__ __forceinline__ uint32_t bar(int which) const { return base + kSmemBars + which * 8; }
  __device__ __forceinline__ int* rows(int buffer) const {
    return reinterpret_cast<int*>(ptr + kSmemRows) + buffer * kSlots;
  }
  __device__ __forceinline__ TokenInfo* info(int buffer) const {
    return reinterpret_cast<TokenInfo*>(ptr + kSmemInfo + buffer * 128);
  }
  __device__ __forceinline__ volatile int* abort_flag() const {
    return reinterpret_cast<volatile int*>(ptr + kSmemMisc + 4);
  }
  __device__ __forceinline__ volatile uint32_t* rescale_mask() const {  // (team kernel)
    return reinterpret_cast<volatile uint32_t*>(ptr + kSmemMisc + 8);
  }
  __device__ __forceinline__ volatile int* first_negative() const {  // one per softmax warp
    return reinterpret_cast<volatile int*>(ptr + kSmemMisc + 16);
  }
  __device__ __forceinline__ const volatile float* maxima(int offset) const {  // (team kernel)
    return reinterpret_cast<const volatile float*>(ptr + offset);
  }
};

// The tokens of one persistent block, in order. Blocks take `token_group` consecutive tokens per round, so
// that a block's successive tokens share most of their window rows in L2 while different blocks read
// different windows at any one time. The last round, which is not full, is dealt in groups as small as it
// takes: 1493 tokens on 148 blocks in twos would be 12 for some, dealt singly in the end they are 11 at most.
// Every role of a block walks the same sequence.
struct TokenWalk {
  const Params& p;
  unsigned round, at, end;  // first token of the round; of it, the block's next token and the end of its group
  __device__ __forceinline__ explicit TokenWalk(const Params& params) : p(params), round(0) { enter(); }
  __device__ __forceinline__ unsigned stride() const { return gridDim.x * unsigned(p.token_group); }
  __device__ __forceinline__ void enter() {
    const unsigned group = round < unsigned(p.whole_rounds) ? p.token_group : p.last_group;
    at = round + blockIdx.x * group;  // (below 2^31 + 2^31)
    end = min(at + group, unsigned(p.tokens));
  }
  __device__ __forceinline__ int next() {  // next token of this block, or -1 when done
    if (at >= end) {
      if (round >= unsigned(p.whole_rounds)) return -1;
      round += stride();
      enter();
      if (at >= end) return -1;
    }
    return int(at++);
  }
  __device__ __forceinline__ int peek() const { TokenWalk copy = *this; return copy.next(); }
  static __device__ __forceinline__ int count(const Params& p) {  // how many tokens next() hands out in all
    const unsigned whole = unsigned(p.whole_rounds), rest = unsigned(p.tokens) - whole, mine = blockIdx.x * unsigned(p.last_group);
    return int(whole / gridDim.x + (rest <= mine ? 0 : min(rest - mine, unsigned(p.last_group))));
  }
};

// A wait whose outcome is uniform across the calling warp (all 32 lanes must call it).
template <bool kCluster = false>
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait<kCluster>(bar, parity, abort_flag));
}

// ---- producer warps ---------------------------------------------------------------------------

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool live) {
  // A masked slot is zero-filled (source size 0) so the tile never holds non-finite leftovers.
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(live ? 16 : 0));
}

// Arrive on `bar` once all cp.async copies this thread has issued so far have completed. The
// arrival counts towards the barrier's expected count (no pending-count increment).
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}

// Warp-cooperative form of `token_geometry`. A cold block starts with this chain of dependent
// loads on its critical path (700 cycles and more each), so the request search probes 32 positions
// of cu_seqlens_q per step, and in its last step (the only one for up to 32 requests) every lane
// loads all scalars of its candidate along with the probe.
__device__ __forceinline__ TokenGeometry token_geometry_warp(const Params& p, int token, int lane) {
  const int requested = __ldg(p.topk_len + token);
  int lo = 0, hi = p.batches;  // invariant: cu[lo] <= token < cu[hi]
  while (hi - lo > 32) {
    const int step = (hi - lo + 31) >> 5;
    const int probe = lo + lane * step;
    const bool below = probe < hi && __ldg(p.cu + probe) <= token;
    const unsigned mask = __ballot_sync(0xffffffffu, below) | 1u;  // a token before cu[0] counts to the first request
    lo += (31 - __clz(mask)) * step;
    hi = min(hi, lo + step);
  }
  const int mine = min(lo + lane, hi - 1);
  const int my_begin = __ldg(p.cu + mine), my_end = __ldg(p.cu + mine + 1);
  const int my_length = __ldg(p.seq_ori + mine), my_available = __ldg(p.seq_cmp + mine), my_residual = __ldg(p.residual + mine);
  const int found = 31 - __clz(__ballot_sync(0xffffffffu, lo + lane < hi && my_begin <= token) | 1u);
  const int begin = __shfl_sync(0xffffffffu, my_begin, found), end = __shfl_sync(0xffffffffu, my_end, found);
  const int length = __shfl_sync(0xffffffffu, my_length, found), available = __shfl_sync(0xffffffffu, my_available, found);
  const int residual = __shfl_sync(0xffffffffu, my_residual, found);
  const int count = end - begin, offset = token - begin;
  TokenGeometry g;
  g.batch = lo + found;
  g.right = max(0, length - count + offset + 1);
  g.visible = min(kWindow, g.right);
  if (requested > 0) g.visible = min(g.visible, requested);
  g.cutoff = max(0, available * p.ratio + residual - count + offset + 1) / p.ratio;
  g.bound = min(min(kTopK, available), g.cutoff);
  return g;
}

// ---- slot -> physical row -----------------------------------------------------------------------
// The selection of the reference's oracle (benchmarks/attention/sparse_reference.py:107-124) and
// of its device routines (examples/sparse_attention/gather.py:39-60, 87-131): window slot s is
// position right - visible + s of the raw cache; compressed rank r is kept when r < min(TOPK,
// C, cutoff), no entry before it is negative and its index is below the cutoff; a kept entry
// goes through the request's block table. A warp resolves kWindowSteps x 32 slots of the window (all of it or
// none) and kListSteps x 32 ranks of the list from `first_rank` on; lane l returns the l-th of every 32 in
// `resolved` (the physical cache row, or -1): neighbouring slots of a sorted list have neighbouring pages, so that
// a load of the table touches few sectors. `others_end` tells, given the rank of the first negative entry among the
// warp's own (kTopK when it has none), that among the other warps' ranks of the list.
//
// Everybody resolves through this one routine: one warp for all of a token (`resolve_token_warp`), five warps for
// the first token of a block (`resolve_first_part`), and the index-set export (`resolve_rows_kernel`) in the form
// that gathers the token, so that the exported set is the gathered set.
template <int kWindowSteps, int kListSteps, typename OthersEnd>
__device__ __forceinline__ void resolve_slots(const Params& p, int token, int lane, int first_rank, OthersEnd others_end, int (&resolved)[kWindowSteps + kListSteps]) {
  constexpr int kSteps = kWindowSteps + kListSteps;
  static_assert(kWindowSteps == 0 || kWindowSteps * 32 == kWindow, "a window is not split");
  // The index list does not depend on the geometry: its loads go out first.
  const int32_t* list = p.indices + (size_t)token * kTopK + first_rank + lane;
  int place[kSteps];  // position in the raw cache, or entry of the list
#pragma unroll
  for (int i = kWindowSteps; i < kSteps; ++i) place[i] = __ldg(list + (i - kWindowSteps) * 32);
  const TokenGeometry g = token_geometry_warp(p, token, lane);
  int first = kTopK;
#pragma unroll
  for (int i = kSteps - 1; i >= kWindowSteps; --i)
    if (place[i] < 0) first = first_rank + (i - kWindowSteps) * 32 + lane;
  const int own_end = kListSteps == 0 ? kTopK : __reduce_min_sync(0xffffffffu, first);
  const int cmp_shift = p.cmp_page == 64 ? 6 : 7;  // cmp_page is 64 or 128: shift and mask instead of a run-time division
  // Two passes so that all block-table loads are in flight together (a branch or vote between
  // them would serialise dependent round trips to memory): columns and loads, rows.
  const int first_position = g.right - g.visible + lane;
  const int rank_end = min(g.bound, own_end);
  const int32_t* ori_table = p.ori_table + (size_t)g.batch * p.pages;
  const int32_t* cmp_table = p.cmp_table + (size_t)g.batch * p.pages;
  int column[kSteps];  // -1: not live
#pragma unroll
  for (int i = 0; i < kSteps; ++i) {
    const bool window = i < kWindowSteps;
    const int rank = first_rank + (i - kWindowSteps) * 32 + lane;
    if (window) place[i] = first_position + i * 32;
    const bool live = window ? i * 32 + lane < g.visible : rank < rank_end && place[i] < g.cutoff;
    column[i] = live ? place[i] >> (window ? kPageShift : cmp_shift) : -1;
    resolved[i] = __ldg((window ? ori_table : cmp_table) + min(unsigned(column[i]), unsigned(p.pages - 1)));  // the page, for now
  }
  const int end = kListSteps == 0 ? kTopK : others_end(own_end);
  bool bad = false;
#pragma unroll
  for (int i = 0; i < kSteps; ++i) {
    const bool window = i < kWindowSteps;
    const int blocks = window ? p.ori_blocks : p.cmp_blocks, shift = window ? kPageShift : cmp_shift;
    const bool live = column[i] >= 0 && (window || first_rank + (i - kWindowSteps) * 32 + lane < end);
    const bool legal = column[i] < p.pages && (unsigned)resolved[i] < (unsigned)blocks;
    bad |= live && !legal;
    resolved[i] = live && legal ? (resolved[i] << shift) + (place[i] & ((1 << shift) - 1)) : -1;
  }
  if (bad) report(p, kStatusBadPage, token, lane);
}

// All slots of a token by one warp: slot 32 i + lane in resolved[i].
__device__ __forceinline__ void resolve_token_warp(const Params& p, int token, int lane, int (&resolved)[kSlots / 32]) {
  resolve_slots<kWindow / 32, kTopK / 32>(p, token, lane, 0, [](int) { return kTopK; }, resolved);
}

// A token by five warps: the window by one, a quarter of the list by each of warps 0 to 3, which tell each other through
// `first_negative` (one word each) and named barrier 1 where the list ends.
constexpr int kFirstParts = 4;
constexpr int kFirstSlots = kWindow / 32;  // per lane
static_assert(kTopK == kFirstParts * kWindow, "five parts of 128 slots");
template <bool window>
__device__ __forceinline__ void resolve_first_part(const Params& p, int token, volatile int* first_negative, int (&resolved)[kFirstSlots]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  resolve_slots<window ? kFirstSlots : 0, window ? 0 : kFirstSlots>(p, token, lane, window ? 0 : warp * kWindow, [&](int own) {
    if (lane == 0) first_negative[warp] = own;
    named_barrier_sync(1, kFirstParts * 32);
    int all = first_negative[0];
#pragma unroll
    for (int w = 1; w < kFirstParts; ++w) all = min(all, first_negative[w]);
    return all;
  }, resolved);
}

// The gathered index set of every token, written out, every token resolved as in a call of this many: the first token
// of each of its `firsts` blocks (clusters take a token each, persistent blocks `token_group` in the first round) by
// the five warps of a block here, the others by a warp each.
constexpr int kExportWarps = kFirstParts + 1;
__global__ void resolve_rows_kernel(const Params p, int firsts, int32_t* out) {
  __shared__ int first_negative[kFirstParts];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (int(blockIdx.x) < firsts) {
    const int token = int(blockIdx.x) * p.token_group, part = warp == kFirstParts ? 0 : warp + 1;
    int resolved[kFirstSlots];
    if (warp == kFirstParts) resolve_first_part<true>(p, token, first_negative, resolved);
    else resolve_first_part<false>(p, token, first_negative, resolved);
#pragma unroll
    for (int i = 0; i < kFirstSlots; ++i) out[(size_t)token * kSlots + part * kWindow + i * 32 + lane] = resolved[i];
    return;
  }
  const unsigned warps = (gridDim.x - firsts) * kExportWarps;
  for (unsigned token = (blockIdx.x - firsts) * kExportWarps + warp; token < unsigned(p.tokens); token += warps) {
    if (token % p.token_group == 0 && token / p.token_group < unsigned(firsts)) continue;
    int resolved[kSlots / 32];
    resolve_token_warp(p, int(token), lane, resolved);
#pragma unroll
    for (int i = 0; i < kSlots / 32; ++i) out[(size_t)token * kSlots + i * 32 + lane] = resolved[i];
  }
}

// Resolve the 640 slots of a token into row buffer `buffer` and list its live chunks (one warp).
__device__ __forceinline__ void publish_token(const Params& p, const Shared& sm, int token, int buffer, int lane) {
  int* rows = sm.rows(buffer);
  TokenInfo* info = sm.info(buffer);
  int resolved[kSlots / 32];
  resolve_token_warp(p, token, lane, resolved);
  unsigned live_chunks = 0;  // bit c set: chunk c holds a live slot (same in all lanes)
  unsigned mine = 0;         // lane l: live bits of slots 32 l ..
#pragma unroll
  for (int i = 0; i < kSlots / 32; ++i) {
    rows[i * 32 + lane] = resolved[i];
    const unsigned live = __ballot_sync(0xffffffffu, resolved[i] >= 0);
    if (live != 0) live_chunks |= 1u << (i * 32 / kChunkRows);
    if (lane == i) mine = live;
  }
  const int chunk = lane >> 1;     // two lanes per chunk (no bit beyond kMaxChunks - 1 is set)
  if (live_chunks >> chunk & 1) {
    const int item = __popc(live_chunks & ((1u << chunk) - 1));
    reinterpret_cast<unsigned*>(&info->live[item])[lane & 1] = mine;
    info->chunk[item] = (unsigned char)chunk;
  }
  if (lane == 0) {
    info->token = token;
    info->chunks = __popc(live_chunks);
  }
}

// The first token of a block, resolved by five warps together: the softmax warps, which have nothing else to
// do yet, take a quarter of the list each and the resolver warp the window, four slots per lane instead of
// twenty. Nothing of the token can start before, and one warp took 6.7 k of the 26 k cycles of a one-token
// call for it, now 3.5 k (the queue for loads and shared memory, which Q's loads stand in too, is most of
// it: with its instructions fetched beforehand it was hardly faster). 64 x 6 tokens at 128K 64.5 -> 62.0 us, 256
// tokens at 4K 31.1 -> 30.4. The rows and chunks are those of `publish_token`. One instantiation per kind of
// warp, each inside its role: a common one in front of the roles cost the loops behind it 3 %.
constexpr int kFirstThreads = (kFirstParts + 1) * 32;
static_assert(kFirstParts == kSoftmaxWarps, "warps 0 to 3 are the softmax warps");
template <bool window>
__device__ __forceinline__ void publish_first_token(const Params& p, const Shared& sm, int token, uint32_t ready_bar) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  TokenInfo* info = sm.info(0);
  const int part = window ? 0 : warp + 1;
  int* rows = sm.rows(0) + part * kWindow + lane;
  int resolved[kFirstSlots];
  resolve_first_part<window>(p, token, sm.first_negative(), resolved);
  unsigned mask[kFirstSlots];
#pragma unroll
  for (int i = 0; i < kFirstSlots; ++i) {
    rows[i * 32] = resolved[i];
    mask[i] = __ballot_sync(0xffffffffu, resolved[i] >= 0);
  }
  if (lane < 2) info->live[part * 2 + lane] = lane == 0 ? make_uint2(mask[0], mask[1]) : make_uint2(mask[2], mask[3]);
  if (!window) {
    named_barrier_arrive(2, kFirstThreads);
    return;
  }
  named_barrier_sync(2, kFirstThreads);
  // The live chunks, in order.
  const uint2 live = lane < kMaxChunks ? info->live[lane] : make_uint2(0, 0);
  const unsigned live_chunks = __ballot_sync(0xffffffffu, (live.x | live.y) != 0);
  if (live_chunks >> lane & 1) {
    const int item = __popc(live_chunks & ((1u << lane) - 1));
    info->live[item] = live;
    info->chunk[item] = (unsigned char)lane;
  }
  if (lane == 0) {
    info->token = token;
    info->chunks = __popc(live_chunks);
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(ready_bar);
}

// What a block reads first, for its first token, asked for on the way to L2 (and its pages'
// translations with it) while the kernel before is still running: L2 sees what that kernel writes,
// so nothing stale is read later.
__device__ __forceinline__ void prefetch_first(const Params& p, int token) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == kResolverWarp) {
    if (lane < 16) prefetch_l2(p.indices + (size_t)token * kTopK + lane * 32);
    else if (lane == 16) prefetch_l2(p.topk_len + token);
    else if (lane == 17) prefetch_l2(p.cu);
    else if (lane == 18) prefetch_l2(p.seq_ori);
    else if (lane == 19) prefetch_l2(p.seq_cmp);
    else if (lane == 20) prefetch_l2(p.residual);
    else if (lane == 21) prefetch_l2(p.ori_table);
    else if (lane == 22) prefetch_l2(p.cmp_table);
    else if (lane == 23) prefetch_l2(p.sinks);
  } else if (warp >= kFirstProducerWarp && warp < kPvWarp) {
    const char* q = static_cast<const char*>(p.q) + (size_t)token * kHeads * kRowBytes + (threadIdx.x - kFirstProducerWarp * 32) * 256;
    prefetch_l2(q);
    prefetch_l2(q + 128);
  }
}

// ---- resolver warp ----------------------------------------------------------------------------
// Runs ahead of everybody else: for each token of this block after the first it resolves the 640 slots into row
// buffer `token_count & 1`, lists the live chunks and publishes both.
__device__ void resolver_role(const Params& p, const Shared& sm) {
  const int lane = threadIdx.x & 31;
  volatile int* abort_flag = sm.abort_flag();
  uint32_t token_count = 0;
  TokenWalk walk(p);
  walk.next();  // the first token: `publish_first_token`
  ++token_count;
  for (int token = walk.next(); token >= 0; token = walk.next(), ++token_count) {
    const int buffer = token_count & 1;
    // The buffer is free once the softmax warps have finished the token that used it two tokens
    // ago. (Barriers that one role may pass without the others keeping up exist once per buffer:
    // a phase parity can only tell two consecutive phases apart.)
    // ... and once the MMA thread and the producer warps have read its chunk count: for a token
    // with nothing to do the softmax warps finish without waiting for anybody, and a role that
    // fell two publications behind could not tell them apart by parity.
    if (token_count >= 2 &&
        (!warp_wait(sm.bar(kTokenDone0 + buffer), ((token_count >> 1) & 1) ^ 1, abort_flag) ||
         !warp_wait(sm.bar(kInfoRead0 + buffer), ((token_count >> 1) & 1) ^ 1, abort_flag))) return;
    publish_token(p, sm, token, buffer, lane);
    __syncwarp();
    if (lane == 0) mbar_arrive(sm.bar(kTokenReady0 + buffer));
  }
}

// Q on its way to tensor memory: every thread of a producer warp loads 16 bytes of rows t / 4 and t / 4 + 8 of
// the warp's 16 heads in each of eight 64-byte segments. The 16-lane stores put the even words (two heads' each)
// to the low lanes and the odd words to the high lanes as they are: no exchange between lanes. (Loads of
// whole lines with 96 shuffles for a transpose and 32 for the split took 450 instructions more per thread and
// token, and their queue is the one that everybody's shared memory accesses stand in: prefill of 8K tokens
// 920 -> 900 us, 256 tokens at 4K 32.7 -> 31.0. 32-byte loads, which need no shuffles either if both lanes of a head
// load the same or the tile's units are permuted, were slower: 918, and 1600 as copies then split sectors.)
constexpr int kQLoads = 16;
__device__ __forceinline__ const char* q_rows(const Params& p, int token, int subpartition, int part, int lane) {
  return static_cast<const char*>(p.q) + ((size_t)token * kHeads + subpartition * 16 + (lane >> 2)) * kRowBytes + part * 512 + (lane & 3) * 16;
}
template <int kFirst, int kCount>
__device__ __forceinline__ void load_q(const char* rows, uint32_t (&words)[64]) {
#pragma unroll
  for (int k = kFirst; k < kFirst + kCount; ++k) {  // segment k / 2, row (k & 1) * 8
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(rows + (k >> 1) * 64 + (k & 1) * 8 * kRowBytes));
    words[4 * k + 0] = v.x; words[4 * k + 1] = v.y; words[4 * k + 2] = v.z; words[4 * k + 3] = v.w;
  }
}

// 64 columns of Q to tensor memory.
__device__ __forceinline__ void store_q(uint32_t q_tmem, const uint32_t (&words)[64]) {
#pragma unroll
  for (int half = 0; half < 2; ++half)
#pragma unroll
    for (int quad = 0; quad < 2; ++quad) {  // four segments: 32 columns
      uint32_t columns[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) columns[c] = words[32 * quad + 2 * c + half];
      tmem_st_16x256b(q_tmem + half * kHalfLanes + quad * 32, columns);
    }
}

// The metadata of the sparse QK product: of every four features a lane of Q holds numbers 0 and 1 (low
// lanes) or 2 and 3 (high lanes), two bits per number. The two entries of a word belong to two heads
// eight apart, whose lanes hold the same numbers: a lane's words are all alike. (Four columns are
// read at most; a store is sixteen wide.)
__device__ __forceinline__ void store_places(uint32_t places_tmem, int lane) {
  uint32_t columns[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) columns[e] = lane & 16 ? 0xeeeeeeeeu : 0x44444444u;
  tmem_st16(places_tmem, columns);
}

// Copies of a chunk's rows into a tile, all 64 or one half of them, by the 256 producer threads. A row is taken by eight threads, 128
// bytes at a time: two rows and their addresses to a thread. (Sixteen threads with 256 bytes at a time make as many requests, but four rows
// to a thread: 62.3 million instructions of a warp for 2072 tokens against 58.6; loops over the launch alone, one token 9.09 -> 8.97 us, 256 tokens at 4K 28.3 -> 27.6.)
template <int kHalf, int kHalves>
__device__ __forceinline__ void gather_rows(const Params& p, const int* rows, int chunk, uint32_t tile, int tid) {
  constexpr int kAtOnce = kProducerThreads / 8, kRows = kChunkRows / kAtOnce / kHalves;  // rows side by side; of a thread
  const int sub = tid & 7;  // eight threads per row: 128 bytes at a time
  const char* base = static_cast<const char*>(chunk * kChunkRows < kWindow ? p.ori_kv : p.cmp_kv) + sub * 16;
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    const int r = (tid >> 3) + (kHalf * kRows + k) * kAtOnce, row = rows[chunk * kChunkRows + r];
    const char* source = base + (size_t)max(row, 0) * kRowBytes;
    const uint32_t target = tile + swizzled(r, sub);
#pragma unroll
    for (int q = 0; q < 8; ++q) cp_async16(target + q * kBlockBytes, source + q * 128, row >= 0);
  }
}

__device__ void producer_role(const Params& p, const Shared& sm, uint32_t tmem) {
  const int tid = threadIdx.x - kFirstProducerWarp * 32;
  const int lane = tid & 31;
  volatile int* abort_flag = sm.abort_flag();
  // Q goes from global memory to tensor memory through registers, never through the ring. A warp
  // reaches the 32 tensor-memory lanes of subpartition (warp index % 4): two producer warps
  // share each subpartition and take 64 columns (512 bytes of every row) each. Lane l of a
  // subpartition holds head 16 * subpartition + (l & 15), its even 32-bit words (l < 16) or its odd ones.
  const int warp = threadIdx.x >> 5;
  const int subpartition = warp & 3, part = (warp - kFirstProducerWarp) >> 2;
  const uint32_t q_tmem = tmem + kTmemQ + part * 64 + (uint32_t(subpartition * 32) << 16);
  // Ring bookkeeping: the halves of stage s are free again once the PV of the tile it held has used them
  // (kKvFree0 + 2 s and + 1, committed by the MMA thread). A tile is announced without anybody waiting
  // for it: every producer thread attaches the completion of its own copies to the stage's
  // full barrier (cp.async.mbarrier.arrive), so the threads never block on data in flight and
  // the warps need not stay in step with each other.
  uint32_t ring = 0;  // tiles placed so far (all tokens)
  uint32_t token_count = 0, q_loads = 0;
  // Q staging registers: `words` holds (part of) the Q slice of `staged_token`, a quarter more with every step.
  constexpr int kQSteps = 4;
  constexpr int kQFirstItem = 2;  // the first two tiles of a token are issued without delay
  uint32_t words[64];
  int q_step = kQSteps;
  const char* q = nullptr;
  auto q_advance = [&]() {
    switch (q_step) {
      case 0: load_q<0, 4>(q, words); break;
      case 1: load_q<4, 4>(q, words); break;
      case 2: load_q<8, 4>(q, words); break;
      default: load_q<12, 4>(q, words); break;
    }
    ++q_step;
  };
  TokenWalk walk(p);
  // The first token's Q does not depend on the resolver: its loads go out while the token is
  // being resolved (a block that only gets a few tokens spends a good part of its time here).
  int staged_token = walk.peek();
  if (staged_token >= 0) load_q<0, kQLoads>(q_rows(p, staged_token, subpartition, part, lane), words);
  for (int token = walk.next(); token >= 0; token = walk.next(), ++token_count) {
    if (!warp_wait(sm.bar(kTokenReady0 + (token_count & 1)), (token_count >> 1) & 1, abort_flag)) return;
    const int* rows = sm.rows(token_count & 1);
    const TokenInfo* info = sm.info(token_count & 1);
    const int chunks = info->chunks;
    // (for a working token this is said behind the first tile, off the token's critical path)
    if (chunks == 0 && lane == 0) mbar_arrive(sm.bar(kInfoRead0 + (token_count & 1)));
    for (int item = 0; item < chunks; ++item, ++ring) {
      const uint32_t stage = ring % kStages, use = ring / kStages;
      const uint32_t tile = sm.base + kSmemKv + stage * kTileBytes;
      const int chunk = info->chunk[item];
      if (use > 0 && !warp_wait(sm.bar(kKvFree0 + 2 * stage), (use - 1) & 1, abort_flag)) return;
      gather_rows<0, 2>(p, rows, chunk, tile, tid);
      if (use > 0 && !warp_wait(sm.bar(kKvFree0 + 2 * stage + 1), (use - 1) & 1, abort_flag)) return;
      gather_rows<1, 2>(p, rows, chunk, tile, tid);
      cp_async_arrive(sm.bar(kKvFull0 + stage));
      if (item == 0 && lane == 0) mbar_arrive(sm.bar(kInfoRead0 + (token_count & 1)));
      if (item == 0) {
        // The token's Q, right behind its first tile. Its registers were filled while the
        // previous token's tiles were being issued, unless this is the block's first working
        // token or the walk skipped an empty one. The wait (the previous working token's last
        // QK has read the old Q) cannot depend on this thread: all its tiles have been issued.
        if (staged_token != token) { q = q_rows(p, token, subpartition, part, lane); q_step = 0; }
        while (q_step < kQSteps) q_advance();
        if (q_loads > 0 && !warp_wait(sm.bar(kQFree), (q_loads - 1) & 1, abort_flag)) return;
        tc_fence_after_sync();
        store_q(q_tmem, words);
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(sm.bar(kQFull));
        ++q_loads;
        staged_token = walk.peek();  // start on the next token's Q
        q = q_rows(p, max(staged_token, 0), subpartition, part, lane);
        q_step = staged_token >= 0 ? 0 : kQSteps;
      } else if (item >= kQFirstItem && q_step < kQSteps) {
        q_advance();  // one slice of the next token's Q per tile, so that it never comes as a burst
      }
    }
  }
}

// Wait for copies announced by `cp_async_arrive`, then make them visible to the async proxy. cp.async writes
// through the generic proxy and the barrier orders it for generic readers only; the tensor core reads
// operands through the async proxy. The copying threads cannot fence (they do not wait for their
// copies), so the thread that issues the product does: one instruction per tile.
__device__ __forceinline__ bool wait_for_copies(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (!mbar_wait(bar, parity, abort_flag)) return false;
  fence_proxy_async();
  return true;
}

// ---- MMA warp (one thread) --------------------------------------------------------------------

// Compile-time unrolled issue loops: every operand offset and accumulate flag is an immediate,
// so the issuing thread spends a couple of instructions per MMA and stays ahead of the pipe.
constexpr int kQkSteps = kFeatures / 32;
template <int kFormat, int K = 0>
__device__ __forceinline__ void issue_qk_steps(uint32_t s_tmem, uint32_t q_tmem, uint64_t x_desc, uint32_t places_tmem) {
  if constexpr (K < kQkSteps) {
    constexpr uint32_t offset = (K >> 1) * kBlockBytes + (K & 1) * 64;
    mma_sparse_ts_c<K != 0>(s_tmem, q_tmem + K * 8, x_desc + (offset >> 4), places_tmem, kIdescQK<kFormat>);
    issue_qk_steps<kFormat, K + 1>(s_tmem, q_tmem, x_desc, places_tmem);
  }
}

// S = Q X^T for one 64-row tile. 64 heads fill half of the M = 128 operand rows (tensor-memory lanes)
// that the pipe's full rate wants, so the features of a head are split between two lanes: lanes 0-15 of
// every subpartition hold the even pairs of features of 16 heads, lanes 16-31 the odd pairs. Either
// is a 2:4 sparse row, two of every four neighbours, and the sparse product multiplies just those: 16
// instructions M = 128, N = 64, K = 32 give every lane the partial scores of its pairs, no product is
// wasted, and the tile is read once.
//
// Bound by the 44 cycles that an instruction takes at least: 704 cycles per tile. Dense, with the low
// and the high half of the features stacked along M and along N (M = 128, N = 128, K = 16; two of
// the four quadrants thrown away) it was 1030 cycles and twice the multiplications, which the board's power
// limit turned into a lower clock; M = 64 without stacking takes 1420.
template <int kFormat>
__device__ __forceinline__ void issue_qk(const Shared& sm, uint32_t tmem, int stage, uint32_t scores = kTmemS) {
  const uint64_t x_desc = smem_desc_sw128(sm.base + kSmemKv + stage * kTileBytes, 16, 1024);
  issue_qk_steps<kFormat>(tmem + scores, tmem + kTmemQ, x_desc, tmem + kTmemPlaces);
}

constexpr int kPvSteps = 2 * (kChunkRows / 16);
template <int kFormat, int I, int kEnd, bool kFirst>
__device__ __forceinline__ void issue_pv_steps(uint32_t o_tmem, uint64_t p_desc, uint64_t x_desc) {
  if constexpr (I < kEnd) {
    constexpr int h = I % 2, k = I / 2;
    constexpr uint32_t offset = h * 4 * kBlockBytes + k * 2048;
    mma_ws_ss_c<!(kFirst && k == 0)>(o_tmem + h * kTmemOHalf, p_desc + ((k * 32) >> 4), x_desc + (offset >> 4), kIdescPV<kFormat>);
    issue_pv_steps<kFormat, I + 1, kEnd, kFirst>(o_tmem, p_desc, x_desc);
  }
}

// O += P X for one 64-row tile as two weight-stationary M = 64, N = 256 products (features 0-255
// and 256-511): with 64 heads a plain M = 64 instruction would leave half of the pipe idle.
// A = P from shared memory (one 128-byte row per head, 32 bytes per K = 16 step); B = X with
// features contiguous: 64-feature blocks kBlockBytes apart, 8-row groups 1024 bytes apart.
//
// The tile's rows are used up in order, both products of 16 rows after each other, and its first half is
// given back when it has been: a tile stays in the ring from its copies' issue to the end of its PV, through QK, softmax and
// PV, and the next tile of the stage can be 320 cycles on its way by that end. Two per cent of decode (128 x 6 and 64 x 6), of prefill
// of 8K tokens and of 23 mixed requests. (Quarters: 2 and 1 % of decode, nothing of prefill: what a wait and its commit
// cost is what they bring.)
template <int kFormat>
__device__ __forceinline__ void issue_pv(const Shared& sm, uint32_t tmem, int stage, int p_tile, bool accumulate) {
  const uint64_t x_desc = smem_desc_sw128(sm.base + kSmemKv + stage * kTileBytes, kBlockBytes, 1024);
  const uint64_t p_desc = smem_desc_sw128(sm.base + kSmemP + p_tile * kPTileBytes, 16, 1024);
  if (accumulate) issue_pv_steps<kFormat, 0, kPvSteps / 2, false>(tmem + kTmemO, p_desc, x_desc);
  else issue_pv_steps<kFormat, 0, kPvSteps / 2, true>(tmem + kTmemO, p_desc, x_desc);
  mma_commit(sm.bar(kKvFree0 + 2 * stage));
  issue_pv_steps<kFormat, kPvSteps / 2, kPvSteps, false>(tmem + kTmemO, p_desc, x_desc);
  mma_commit(sm.bar(kKvFree0 + 2 * stage + 1));
}

// Two issuing threads in two warps, one per product. Each follows its own data: the QK thread
// goes on as soon as a tile has landed and the score buffer is free, the PV thread as soon as a P
// is complete. The tensor pipe executes what arrives in the order it arrives, so the
// non-MMA instructions of one thread (barrier waits, commits, fences: a hundred cycles and more
// each, far beyond what the pipe's short queue covers) run while the other thread's product
// executes. Both walk the same token and chunk sequence as everybody else.

// S = Q X^T: chunk c of the block's chunk stream uses ring stage c % kStages and score barrier c % 2 (the buffer is one;
// two barriers tell phases two chunks apart from each other).
template <int kFormat>
__device__ void qk_role(const Params& p, const Shared& sm, uint32_t tmem) {
  volatile int* abort_flag = sm.abort_flag();
  uint32_t chunk_count = 0, working_tokens = 0;
  const uint32_t my_tokens = uint32_t(TokenWalk::count(p));  // closed form: no walk on this thread
  for (uint32_t token_count = 0; token_count < my_tokens; ++token_count) {
    if (!mbar_wait(sm.bar(kTokenReady0 + (token_count & 1)), (token_count >> 1) & 1, abort_flag)) return;
    const int chunks = sm.info(token_count & 1)->chunks;
    if (chunks == 0) {
      mbar_arrive(sm.bar(kInfoRead0 + (token_count & 1)));
      continue;
    }
    // the token's Q is in tensor memory
    if (!mbar_wait(sm.bar(kQFull), working_tokens & 1, abort_flag)) return;
    for (int i = 0; i < chunks; ++i, ++chunk_count) {
      const uint32_t stage = chunk_count % kStages;
      // One barrier says both that the tile has landed and that the single score buffer is free
      // (the softmax warps have read the previous chunk out of it).
      if (!wait_for_copies(sm.bar(kKvFull0 + stage), (chunk_count / kStages) & 1, abort_flag)) return;
      tc_fence_after_sync();
      issue_qk<kFormat>(sm, tmem, stage);
      mma_commit(sm.bar(kSFull0 + (chunk_count & 1)));
      if (i + 1 == chunks) mma_commit(sm.bar(kQFree));  // the last QK that reads this token's Q
      if (i == 0) mbar_arrive(sm.bar(kInfoRead0 + (token_count & 1)));  // chunk count read (see resolver)
    }
    ++working_tokens;
  }
}

// O += P X (O = P X for a token's first chunk, once the previous token's O has been read out).
template <int kFormat>
__device__ void pv_role(const Params& p, const Shared& sm, uint32_t tmem) {
  volatile int* abort_flag = sm.abort_flag();
  uint32_t chunk_count = 0, working_tokens = 0;
  const uint32_t my_tokens = uint32_t(TokenWalk::count(p));
  for (uint32_t token_count = 0; token_count < my_tokens; ++token_count) {
    if (!mbar_wait(sm.bar(kTokenReady0 + (token_count & 1)), (token_count >> 1) & 1, abort_flag)) return;
    const int chunks = sm.info(token_count & 1)->chunks;
    mbar_arrive(sm.bar(kInfoRead0 + (token_count & 1)));
    if (chunks == 0) continue;
    for (int i = 0; i < chunks; ++i, ++chunk_count) {
      const uint32_t stage = chunk_count % kStages;
      const int p_tile = chunk_count & 1;
      if (!mbar_wait(sm.bar(kPFull0 + p_tile), (chunk_count >> 1) & 1, abort_flag)) return;
      if (i == 0 && !mbar_wait(sm.bar(kOFree), (working_tokens & 1) ^ 1, abort_flag)) return;
      tc_fence_after_sync();
      issue_pv<kFormat>(sm, tmem, stage, p_tile, i != 0);
      mma_commit(sm.bar(kSFull0 + p_tile));  // the P tile is free: half of what the softmax warps wait for at chunk c + 2
      if (i + 1 == chunks) mma_commit(sm.bar(kOutReady));  // O is complete
    }
    ++working_tokens;
  }
}

// ---- softmax / correction / epilogue warps ----------------------------------------------------

template <int kFormat>
__device__ __forceinline__ uint32_t pack_pair(float a, float b) {  // two FP32 -> two storage words
  if constexpr (kFormat == 1) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}

__device__ __forceinline__ float max3(float a, float b, float c) {  // one instruction on sm_100
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// The running reference of a head (log2 domain; it starts at the sink) moves when a chunk's maximum exceeds it by more
// than kReferenceRoom, and then to kReferenceStep below that maximum. All terms of a head share the reference, which
// cancels in the final division; what it decides is how often the accumulator is rescaled (everybody waits for it) and
// which probabilities fit the storage type. Probabilities reach 2^15 (IEEE half ends below 2^16). Sums are FP32 and reach as much
// further: 640 rows stay finite up to values of 1.6e31 in a bf16 cache (2e33 with a room of 8). A reference
// that moved at 2^8 already, up to the maximum, rescaled in a tenth of all chunks where sinks are N(0, 1); now it takes a sink
// seven standard deviations down. The step back keeps the reference at or below that one's in every chunk: the room is at
// least a step wider, so whatever was a normal number in half still is. Four per cent of 8 x 2 tokens, one of one
// token, of 23 mixed requests and of prefill.
//
// With a token's first chunk, where there is nothing to rescale, it moves down to a whole number of binades below the maximum
// (by less than one): the probability of the chunk's best row is then a power of two and not rounded. The error against
// 64 bits, relative by the 2-norm: 2.14e-3 in bf16 and 2.67e-4 in half for N(0, 1) inputs (2.15e-3 and 2.70e-4 without the step and
// a room of 8), 7 to 10 % less than without it for scores three times as wide, 1 to 2 % less for six times. Beyond kReferenceAligned
// binades that row weighs nothing. Returns the factor of what has been accumulated.
constexpr float kReferenceRoom = 15.f, kReferenceStep = 8.f, kReferenceAligned = 64.f;
__device__ __forceinline__ float move_reference(float& reference, float chunk_max, bool first) {
  const float above = chunk_max - reference;
  float moved;
  if (above > kReferenceRoom) moved = chunk_max - kReferenceStep;
  else if (first && above > -kReferenceAligned) moved = chunk_max - ceilf(above);
  else return 1.f;
  const float alpha = exp2f(reference - moved);
  reference = moved;
  return alpha;
}

// Two FP32 additions / multiply-adds in one instruction.
__device__ __forceinline__ float2 add_pair(float2 a, float2 b) {
  float2 d;
  asm("add.rn.ftz.f32x2 %0, %1, %2;\n"
      : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
  return d;
}
__device__ __forceinline__ float2 fma_pair(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;\n"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)), "l"(reinterpret_cast<uint64_t&>(c)));
  return d;
}

// What paces the kernel. Inside of a token a chunk takes 1.75 k cycles: the instructions of QK and PV follow each other without a gap
// and take about 900 cycles each (704 and 640 by themselves): their operands, 144 KiB, and the copies that write 64 KiB beside
// them share the ports of one shared memory. From scores to P handed over these warps need 1.35 k; nothing that is known a
// chunk earlier is fetched late, and additions go two to an instruction. Between two tokens lie 4 to 5 k cycles more, for
// which no product runs: the output leaves the SM at 32 bytes per cycle (2.05 k for 64 KiB, by stores or bulk copies alike), and
// the conversion to 16 bits in front of it takes 1.7 k.
//
// A second P tile takes the wait for the previous PV out of the chain, and flags by a named barrier a word in shared memory and a
// wait: five per cent of 100 and of 256 tokens, two of 1000, one of prefill of 8K.
//
// Calls one after the other through the Python entry points take 822 us for prefill of 8K tokens at 32K (842 with sixteen threads to a gathered row and
// issuing threads that were not elected, in turn on one board), 163 for 23 mixed requests (167), 29.9 for 256 tokens at 4K (31.0); decode
// 128 x 6 at 128K 115 either way. The first two and the last are at the board's power limit (990 to 1000 W; 1.47 to 1.60 GHz while they run, by the board: three
// per cent of time between two of them), where energy decides more than cycles.
template <int kFormat>
__device__ void softmax_role(const Params& p, const Shared& sm, uint32_t tmem) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = lane >> 4;
  const int head = warp * 16 + (lane & 15);
  const uint32_t lane_base = uint32_t(warp * 32) << 16;
  volatile int* abort_flag = sm.abort_flag();
  const float sink = __ldg(p.sinks + head) * 1.4426950408889634f;  // log2 domain
  uint32_t chunk_count = 0, token_count = 0;
  // The accumulator's layout is that of the weight-stationary PV (lane = head for lanes 0-63, the
  // same heads again for lanes 64-127 with the next 128 features), not that of the scores: this
  // thread reads O of head `o_head`, features o_feature .. + 127 of each 256-feature half.
  const int o_head = (warp & 1) * 32 + lane, o_feature = (warp >> 1) * 128;
  float* alpha_exchange = reinterpret_cast<float*>(sm.ptr + kSmemAlpha);
  float* inverse_exchange = reinterpret_cast<float*>(sm.ptr + kSmemInverse);
  __nv_bfloat16* out_base = static_cast<__nv_bfloat16*>(p.out);
  const uint32_t s_addr = tmem + kTmemS + lane_base;

  store_places(tmem + kTmemPlaces + lane_base, lane);
  tmem_wait_st();
  tc_fence_before_sync();
  __syncwarp();
  // The score buffer starts out free (first chunk, stage 0), and the metadata is in place.
  if (lane == 0) mbar_arrive(sm.bar(kKvFull0));
  // What the four warps tell each other goes through a named barrier: P for chunk c needs no wait but that for the scores (its
  // barrier counts the end of PV c - 2, which read the same P tile), and a barrier that counts flags costs
  // less than the round trips to shared memory, behind the producers' copies, that an mbarrier and a word would be.
  // Nobody may be left waiting at it. A warp whose wait gives up says so the next time they meet, and all four leave
  // behind that. It counts with all its threads, one whose references move with one thread.
  bool failed = false;
  constexpr uint32_t kGivenUp = 32;
  auto meet = [&](bool flag) { return named_barrier_count(3, 32 * kSoftmaxWarps, failed || (flag && lane == 0)); };

  // A finished token waits for its epilogue until the first chunk of the next working token has
  // been through the softmax, so that the MMA thread has a P to go on with while O is written out.
  uint32_t outputs = 0;         // epilogues so far
  int done_token = -1;          // token whose O is complete (or about to be) and not yet stored
  uint32_t done_count = 0;      // its index in this block's walk

  // O / denominator -> 16-bit -> global for `done_token`: 64 columns per pass, tensor memory ->
  // registers -> a swizzled per-warp staging tile -> global, so that every store instruction
  // writes four complete 128-byte lines.
  // `chunks_before`: chunks of the stream whose PV precedes. Everybody's reciprocal denominators are there (a reduction lies between).
  auto epilogue = [&](uint32_t chunks_before) {
    if (!warp_wait(sm.bar(kOutReady), outputs & 1, abort_flag)) { failed = true; return; }
    ++outputs;
    tc_fence_after_sync();
    const float inverse = inverse_exchange[(done_count & 1) * kHeads + o_head];
    // Rows 0-15 of the staging tile lie in the warp's own 2 KiB, rows 16-31 where its own heads' rows of the unused P tile are.
    unsigned char* staging_low = sm.ptr + kSmemStore + warp * 2048;
    unsigned char* staging_high = sm.ptr + kSmemP + ((chunks_before & 1) ^ 1) * kPTileBytes + warp * 2048;
    unsigned char* staging_row = (half ? staging_high : staging_low) + (lane & 15) * 128;
    __nv_bfloat16* token_out = out_base + (size_t)done_token * kHeads * kFeatures;
    uint32_t o[64];  // loaded a pass ahead
#pragma unroll
    for (int q = 0; q < 64; q += 16) tmem_ld16(tmem + kTmemO + q + lane_base, *reinterpret_cast<uint32_t(*)[16]>(&o[q]));
#pragma unroll 1
    for (int c = 0; c < 256; c += 64) {
      tmem_wait_ld();
      if (c == 192) {  // O has been read completely: the next token's first PV may overwrite it
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(sm.bar(kOFree));
      }
#pragma unroll
      for (int unit = 0; unit < 8; ++unit) {
        uint4 v;
        v.x = pack_pair<kFormat>(__uint_as_float(o[unit * 8 + 0]) * inverse, __uint_as_float(o[unit * 8 + 1]) * inverse);
        v.y = pack_pair<kFormat>(__uint_as_float(o[unit * 8 + 2]) * inverse, __uint_as_float(o[unit * 8 + 3]) * inverse);
        v.z = pack_pair<kFormat>(__uint_as_float(o[unit * 8 + 4]) * inverse, __uint_as_float(o[unit * 8 + 5]) * inverse);
        v.w = pack_pair<kFormat>(__uint_as_float(o[unit * 8 + 6]) * inverse, __uint_as_float(o[unit * 8 + 7]) * inverse);
        *reinterpret_cast<uint4*>(staging_row + ((unit ^ (lane & 7)) << 4)) = v;
      }
      if (c < 192) {
#pragma unroll
        for (int q = 0; q < 64; q += 16) tmem_ld16(tmem + kTmemO + c + 64 + q + lane_base, *reinterpret_cast<uint32_t(*)[16]>(&o[q]));
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = i * 4 + (lane >> 3), unit = lane & 7;  // staging row = owning lane
        const uint4 v = *reinterpret_cast<const uint4*>((i < 4 ? staging_low : staging_high) + (row & 15) * 128 + ((unit ^ (row & 7)) << 4));
        // accumulator columns 0-127: features 0-255 (this warp's 128 of them), 128-255: 256-511
        __nv_bfloat16* dst = token_out + (size_t)((warp & 1) * 32 + row) * kFeatures + (c >> 7) * 256 + o_feature + (c & 127) + unit * 8;
        __stcs(reinterpret_cast<uint4*>(dst), v);  // written once, read by nobody here
      }
      __syncwarp();
    }
    if (lane == 0) mbar_arrive(sm.bar(kTokenDone0 + (done_count & 1)));
    done_token = -1;
  };

  TokenWalk walk(p);
  for (int token = walk.next();; token = walk.next(), ++token_count) {
    const TokenInfo* info = sm.info(token_count & 1);
    int chunks = 0;
    if (token >= 0) {
      if (!warp_wait(sm.bar(kTokenReady0 + (token_count & 1)), (token_count >> 1) & 1, abort_flag)) { failed = true; break; }
      chunks = info->chunks;
    }
    if (chunks == 0) {
      // No chunk to put the finished token's output behind. (And the resolver needs the finished token's row buffer
      // back before it can publish the token after this one: no point in holding its epilogue any longer.)
      if (done_token >= 0) {
        if (meet(false) != 0) return;
        epilogue(chunk_count);
      }
      if (token < 0) break;
      // nothing visible: the output row is zero whatever the sink
      __nv_bfloat16* out = out_base + ((size_t)token * kHeads + head) * kFeatures + half * 256;
      for (int i = 0; i < 256; i += 8) *reinterpret_cast<uint4*>(out + i) = make_uint4(0, 0, 0, 0);
      __syncwarp();
      if (lane == 0) mbar_arrive(sm.bar(kTokenDone0 + (token_count & 1)));
      continue;
    }
    // `run_sum` is this lane's share of the denominator; the low lane's share includes the
    // sink's own weight exp2(sink - run_max) = 1.
    float run_max = sink, run_sum = half ? 0.f : 1.f;
    uint2 next_live = info->live[0];
    for (int i = 0; i < chunks; ++i, ++chunk_count) {
      const unsigned live_lo = next_live.x, live_hi = next_live.y;
      next_live = info->live[min(i + 1, kMaxChunks - 1)];  // a chunk ahead: shared loads queue behind the producers' copies

      if (!warp_wait(sm.bar(kSFull0 + (chunk_count & 1)), (chunk_count >> 1) & 1, abort_flag)) { failed = true; meet(true); return; }
      tc_fence_after_sync();
      // Of a head's two lanes the low one (0-15) holds the scores' sums over the even pairs of features, the
      // high one (16-31) those over the odd pairs. The two threads of a head share the softmax work: the low
      // thread owns tile rows 0-31, the high thread rows 32-63. Both partial scores of a row come
      // straight to the thread that owns it: a load over the 16 low lanes gives threads 0-15
      // columns j and threads 16-31 columns 32 + j of the even pairs' sums; a load over the 16 high
      // lanes gives them the same columns of the odd pairs' sums. No exchange between lanes.
      const unsigned live = half ? live_hi : live_lo;
      const bool all_live = (live_lo & live_hi) == 0xffffffffu;  // the usual case: nothing to mask
      float2 raw[16];  // unscaled scores: the scale goes into the exponent's FMA
      {
        uint32_t low_a[16], low_b[16], high_a[16], high_b[16];
        tmem_ld16_halves<32>(s_addr, low_a);                       // rows 0-15 | 32-47, even pairs
        tmem_ld16_halves<32>(s_addr + 16, low_b);                  // rows 16-31 | 48-63
        tmem_ld16_halves<32>(s_addr + kHalfLanes, high_a);         // the same rows, odd pairs
        tmem_ld16_halves<32>(s_addr + kHalfLanes + 16, high_b);
        tmem_wait_ld();
        // The scores are in registers: the next QK may overwrite the buffer. Its tile's full
        // barrier counts this as well as the copies.
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(sm.bar(kKvFull0 + (chunk_count + 1) % kStages));
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          raw[e] = add_pair(make_float2(__uint_as_float(low_a[2 * e]), __uint_as_float(low_a[2 * e + 1])),
                            make_float2(__uint_as_float(high_a[2 * e]), __uint_as_float(high_a[2 * e + 1])));
          raw[8 + e] = add_pair(make_float2(__uint_as_float(low_b[2 * e]), __uint_as_float(low_b[2 * e + 1])),
                                make_float2(__uint_as_float(high_b[2 * e]), __uint_as_float(high_b[2 * e + 1])));
        }
      }
      if (!all_live) {
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          if (!(live >> (2 * e) & 1u)) raw[e].x = -INFINITY;
          if (!(live >> (2 * e + 1) & 1u)) raw[e].y = -INFINITY;
        }
      }
      float partial_max[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        partial_max[k] = max3(raw[4 * k].x, raw[4 * k].y, raw[4 * k + 1].x);
        partial_max[k] = max3(partial_max[k], raw[4 * k + 1].y, raw[4 * k + 2].x);
        partial_max[k] = max3(partial_max[k], raw[4 * k + 2].y, raw[4 * k + 3].x);
        partial_max[k] = fmaxf(partial_max[k], raw[4 * k + 3].y);
      }
      const float own_max = fmaxf(fmaxf(partial_max[0], partial_max[1]), fmaxf(partial_max[2], partial_max[3])) * p.scale_log2;  // scale > 0
      // `move_reference` says when the running reference moves. Behind the first chunk it usually does not, so the
      // two lanes of a head exchange their maxima only in the rare case: a shuffle waits in the same queue as
      // the producers' copies, a vote does not.
      float alpha = 1.f;
      const bool look = __any_sync(0xffffffffu, own_max - run_max > (i == 0 ? -kReferenceAligned : kReferenceRoom));
      if (look) alpha = move_reference(run_max, fmaxf(own_max, __shfl_xor_sync(0xffffffffu, own_max, 16)), i == 0);
      const bool moves = look && i > 0;  // some head's, and O holds earlier chunks
      // The factor of a head is known to the threads that have its scores; the head's accumulator rows are in other threads' lanes.
      // It goes along with every chunk: written only where some reference moves, behind the meeting and with another one for itself, it made
      // chunks that rescale slower (4000 tokens whose scores rise by twelve binades from chunk to chunk 474 -> 456 us without; prefill
      // of 8K tokens, which hardly rescales, 832 -> 818, 23 mixed requests 163.8 -> 162.0).
      float* factors = alpha_exchange + (chunk_count & 1) * kHeads;
      if (half == 0) factors[head] = alpha;
      // P to shared memory, one 128-byte row per head; this lane writes its 32 rows (64 bytes).
      const float2 scale = make_float2(p.scale_log2, p.scale_log2), reference = make_float2(-run_max, -run_max);
      float2 sum_a = make_float2(0.f, 0.f), sum_b = sum_a;  // four partial sums
      unsigned char* p_tile = sm.ptr + kSmemP + (chunk_count & 1) * kPTileBytes;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        uint32_t words[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const int e = 4 * u + w;
          float2 prob = fma_pair(raw[e], scale, reference);
          prob.x = exp2f(prob.x);
          prob.y = exp2f(prob.y);
          if (e & 1) sum_b = add_pair(sum_b, prob); else sum_a = add_pair(sum_a, prob);
          words[w] = pack_pair<kFormat>(prob.x, prob.y);
        }
        *reinterpret_cast<uint4*>(p_tile + p_offset(head, half * 4 + u)) = make_uint4(words[0], words[1], words[2], words[3]);
      }
      run_sum = run_sum * alpha + ((sum_a.x + sum_a.y) + (sum_b.x + sum_b.y));
      const uint32_t met = meet(moves);
      if (met >= kGivenUp) return;
      if (met != 0) {
        const float o_alpha = factors[o_head];
        // PV c - 1 has ended when its tile's second half is free. A parity tells that phase from the one before only, the end of
        // PV c - 4, which is long past: the producers waited for it before they brought tile c - 1 into the stage.
        if (!warp_wait(sm.bar(kKvFree0 + 2 * ((chunk_count - 1) % kStages) + 1), ((chunk_count - 1) / kStages) & 1, abort_flag)) failed = true;
        tc_fence_after_sync();
        // 32 columns at a time: a round trip to tensor memory each (in 16s the pass took 1500 cycles).
#pragma unroll 1
        for (int c = 0; c < 256; c += 32) {
          uint32_t o[32];
          tmem_ld16(tmem + kTmemO + c + lane_base, *reinterpret_cast<uint32_t(*)[16]>(&o[0]));
          tmem_ld16(tmem + kTmemO + c + 16 + lane_base, *reinterpret_cast<uint32_t(*)[16]>(&o[16]));
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * o_alpha);
          tmem_st16(tmem + kTmemO + c + lane_base, *reinterpret_cast<uint32_t(*)[16]>(&o[0]));
          tmem_st16(tmem + kTmemO + c + 16 + lane_base, *reinterpret_cast<uint32_t(*)[16]>(&o[16]));
        }
        tmem_wait_st();
      }
      fence_proxy_async();  // the PV reads the tile through the async proxy
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(sm.bar(kPFull0 + (chunk_count & 1)));
      // The previous token's output, now that the MMA thread has this token's first P to go on with.
      if (done_token >= 0) epilogue(chunk_count);
    }
    done_token = token;
    done_count = token_count;
    // Hand the reciprocal denominators over now; the epilogue picks them up a chunk later.
    const float own_inverse = 1.f / (run_sum + __shfl_xor_sync(0xffffffffu, run_sum, 16));
    if (half == 0) inverse_exchange[(done_count & 1) * kHeads + head] = own_inverse;
  }
  meet(false);  // with a warp that has given up since the last time
}

// ---- kernel and launch ------------------------------------------------------------------------

template <int kFormat>
__global__ void __launch_bounds__(kThreads, 1) attention_kernel(const Params p) {
  extern __shared__ unsigned char smem_raw[];
  Shared sm;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw & 1023u)) & 1023u;
  sm.base = raw + pad;
  sm.ptr = smem_raw + pad;
  const int warp = threadIdx.x >> 5;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm.ptr + kSmemMisc);

  if (threadIdx.x == 0) {
    const int P = kProducerWarps, S = kSoftmaxWarps, T = kProducerThreads;
    const int counts[kBarCount] = {1, 1, S, S, P, 1, 1, 1, 1, 1, 1, 1, 2, 2, S, S, S, T + S, T + S, T + S, 1, P + 2, P + 2};
    for (int i = 0; i < kBarCount; ++i) mbar_init(sm.bar(i), counts[i]);
    mbar_fence_init();
    mbar_arrive(sm.bar(kSFull0));  // the P tiles start out free
    mbar_arrive(sm.bar(kSFull1));
    *sm.abort_flag() = 0;
  }
  if (warp == kMmaWarp) { tmem_alloc(smem_u32(tmem_slot), kTmemColumns); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  // Up to here nothing has touched global memory: a block's start, and the launch itself, overlap
  // the end of the kernel before.
  const int first = TokenWalk(p).next();  // (there is one: no more blocks than tokens)
  prefetch_first(p, first);
  wait_for_predecessor();
  let_successor_start();

  if (warp < kSoftmaxWarps) {
    publish_first_token<false>(p, sm, first, sm.bar(kTokenReady0));
    softmax_role<kFormat>(p, sm, tmem);
  } else if (warp == kMmaWarp) {
    if (elect_one()) qk_role<kFormat>(p, sm, tmem);
    __syncwarp();
  } else if (warp == kPvWarp) {
    if (elect_one()) pv_role<kFormat>(p, sm, tmem);
    __syncwarp();
  } else if (warp == kResolverWarp) {
    publish_first_token<true>(p, sm, first, sm.bar(kTokenReady0));
    resolver_role(p, sm);
  } else {
    producer_role(p, sm, tmem);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  }

  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *sm.abort_flag() != 0) report(p, kStatusWaitExpired, blockIdx.x, 0);
  if (warp == kMmaWarp) tmem_dealloc(tmem, kTmemColumns);
}

// How a call's tokens are dealt to the persistent blocks (see `TokenWalk`).
inline int persistent_blocks(const Params& p, int multiprocessors) { return p.tokens < multiprocessors ? p.tokens : multiprocessors; }
inline void deal_tokens(Params& p, int grid) {
  const int per_block = p.tokens / (grid * 4);
  p.token_group = per_block < 1 ? 1 : (per_block > 8 ? 8 : per_block);
  const int rest = p.tokens % (grid * p.token_group);
  p.whole_rounds = p.tokens - rest;
  p.last_group = (rest + grid - 1) / grid;
}

template <int kFormat>
inline int launch(const Params& p, cudaStream_t stream, int multiprocessors) {
  static bool configured[64] = {false};
  int device = 0;
  cudaError_t error = cudaGetDevice(&device);
  if (error != cudaSuccess) return int(error);
  if (device < 0 || device >= 64) return -1;
  if (!configured[device]) {
    error = cudaFuncSetAttribute(attention_kernel<kFormat>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (error != cudaSuccess) return int(error);
    configured[device] = true;
  }
  const int grid = persistent_blocks(p, multiprocessors);
  Params launch_params = p;
  deal_tokens(launch_params, grid);
  return int(launch_overlapped(attention_kernel<kFormat>, grid, kThreads, kSmemBytes, stream, launch_params));
}

}  // namespace umma
}  // namespace sparse_mla
