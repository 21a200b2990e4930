// The two steps next to the attention operator whose output format the operator fixes: choosing
// each query token's TopK compressed rows from index scores (the producer of
// `cmp_sparse_indices`), and appending a call's new raw rows to the paged cache (the producer
// of `ori_kv`). The reference leaves both to its caller (docs/operators/sparse-mla.md:8,
// 263-266: "indexer, compressor, projections and cache writes are provided by the caller"), so
// there is no reference implementation to match: the contracts below are derived from what the
// operator reads (docs/operators/sparse-mla.md:62-87) and pinned by this repository's oracle.
// Both are byte/integer work bound by memory traffic.

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/sparse_mla.h"
#include "sparse_mla_common.cuh"
#include "tcgen05_ptx.cuh"

namespace sparse_mla {
namespace {

// Monotone map of an FP32 value, given by its bits, to an unsigned key: larger value, larger key. NaNs lie beyond the infinities,
// on the side that their sign says. (Scores are loaded as words where their keys are wanted: comparing the key of
// a float, the compiler may compare the floats, and NaNs come out wrong.)
__device__ __forceinline__ uint32_t score_key(uint32_t bits) {
  return (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
}

__device__ __forceinline__ uint32_t key_score(uint32_t key) {  // its inverse
  return (key & 0x80000000u) ? key ^ 0x80000000u : ~key;
}

struct SelectParams {
  const float* scores;       // [T, span]
  const int32_t* cu;         // [B + 1]
  const int32_t* seq_cmp;    // [B]
  const int32_t* residual;   // [B]
  int32_t* out;              // [T, 512]
  int32_t batches, tokens, ratio;
  bool one_wave;             // no more rows than blocks of 256 threads run at once
  int64_t span;
};

// A token's request and what is known about it, found by a whole warp: 32 probes of cu_seqlens_q per
// step, so that 128 requests take two dependent loads and not seven. kAhead: in the last step (the only
// one for up to 32 requests) every lane loads its candidate's scalars with the probe, which saves one
// more (append + selection + attention of 16 requests 35.8 -> 35.1 us); calls of many rows do not wait
// for it and are 0.5 % faster without.
struct Request {
  int index, begin, count;  // its row in the tables; its first token and how many it has
  int first, second;        // its entries in the two arrays given
};
template <bool kAhead>
__device__ __forceinline__ Request request_of(const int32_t* cu, int batches, int token, int lane, const int32_t* first, const int32_t* second) {
  int lo = 0, hi = batches;  // invariant: cu[lo] <= token < cu[hi]
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) >> 5;
    const int probe = lo + lane * step;
    const bool ahead = kAhead && step == 1;
    int begin = INT32_MAX, end = 0, a = 0, b = 0;
    if (probe < hi) {
      begin = __ldg(cu + probe);
      if (ahead) { end = __ldg(cu + probe + 1); a = __ldg(first + probe); b = __ldg(second + probe); }
    }
    const int winner = 31 - __clz(__ballot_sync(0xffffffffu, begin <= token) | 1u);  // a token before cu[0] counts to the first request
    lo += winner * step;
    if (ahead) {
      begin = __shfl_sync(0xffffffffu, begin, winner);
      return {lo, begin, __shfl_sync(0xffffffffu, end, winner) - begin, __shfl_sync(0xffffffffu, a, winner), __shfl_sync(0xffffffffu, b, winner)};
    }
    hi = min(hi, lo + step);
  }
  const int begin = __ldg(cu + lo);
  return {lo, begin, __ldg(cu + lo + 1) - begin, __ldg(first + lo), __ldg(second + lo)};
}

// Completed compressed rows a token may see: min(C, cutoff), with the attention operator's
// cutoff = max(0, C R + r - n + j + 1) / R (examples/sparse_attention/attention.py:339-341).
// Called by whole warps.
template <bool kAhead>
__device__ __forceinline__ int visible_compressed_rows(const SelectParams& p, int token, int lane) {
  const Request request = request_of<kAhead>(p.cu, p.batches, token, lane, p.seq_cmp, p.residual);
  const int available = request.first;
  const int completed = available * p.ratio + request.second;
  return min(available, max(0, completed - request.count + (token - request.begin) + 1) / p.ratio);
}

// Four consecutive scores and their keys (one 16-byte load); `span` is a multiple of four, so every row
// starts on a 16-byte boundary and a load may run past `end` but never past the row.
__device__ __forceinline__ uint4 load_keys(const float* row, unsigned i, unsigned end, uint32_t (&key)[4], bool (&valid)[4]) {
  uint4 v = make_uint4(0, 0, 0, 0);
  if (i < end) v = __ldg(reinterpret_cast<const uint4*>(row + i));
  key[0] = score_key(v.x); key[1] = score_key(v.y); key[2] = score_key(v.z); key[3] = score_key(v.w);
#pragma unroll
  for (int e = 0; e < 4; ++e) valid[e] = i + e < end;
  return v;
}

constexpr int kSelectBins = 256;
constexpr int kHalfCapacity = 2560;  // of the list of 256 threads
// The longest row. Loops over a row reach up to one of their steps past its end and count unsigned.
constexpr int kMostSpan = INT32_MAX - 8192;

// Shared memory of one selecting block. kWindow: row positions covered by the bitmap of winners at a time.
template <int kThreads, int kCapacity, int kWindowSize>
struct SelectShared {
  static constexpr int kWindow = kWindowSize;
  uint2 list[kCapacity];               // candidates: row position, score
  __align__(16) unsigned bitmap[kWindow / 32];
  __align__(16) unsigned short place[kWindow / 32];  // winners before each word of the bitmap
  __align__(16) unsigned histogram[kSelectBins];
  unsigned warp_sum[2][kThreads / 32];
  unsigned count, low, high;           // candidates listed; extremes of what is being binned
  unsigned bin, before, in_bin;        // result of find_bin
  unsigned few_count;                  // entries in `few`
  bool mass;                           // many scores of the sample equal the key below the floor
  unsigned long long few[32], limit;   // the threshold bin's entries; the last winner
};

// Start `bytes` (a multiple of 16) at a 16-byte aligned address on their way to L2.
__device__ __forceinline__ void prefetch_l2(const void* at, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(at), "r"(bytes));
}

// Inclusive prefix sum over a warp.
__device__ __forceinline__ unsigned warp_scan(unsigned value, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned up = __shfl_up_sync(0xffffffffu, value, d);
    if (lane >= d) value += up;
  }
  return value;
}

// The bin in which the running count over the histogram reaches `wanted`, what lies before it and
// what it holds. If the whole histogram holds fewer, s.bin is kSelectBins and s.before what it holds. Clears
// the histogram.
// One warp does it, eight bins per lane. Called by the whole block after a barrier; ends with one.
template <typename Shared>
__device__ __forceinline__ void find_bin(Shared& s, unsigned wanted) {
  if (threadIdx.x < 32) {
    static_assert(kSelectBins == 8 * 32, "eight bins per lane");
    uint4* bins = reinterpret_cast<uint4*>(&s.histogram[threadIdx.x * 8]);
    const uint4 a = bins[0], b = bins[1];
    bins[0] = bins[1] = make_uint4(0, 0, 0, 0);
    const unsigned count[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    unsigned mine = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) mine += count[i];
    unsigned before = warp_scan(mine, threadIdx.x) - mine;
    const bool here = before < wanted && wanted <= before + mine;
    if (!__any_sync(0xffffffffu, here) && threadIdx.x == 31) { s.bin = kSelectBins; s.before = before + mine; }
    if (here) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (before < wanted && wanted <= before + count[i]) { s.bin = threadIdx.x * 8 + i; s.before = before; s.in_bin = count[i]; }
        before += count[i];
      }
    }
  }
  __syncthreads();
}

// Every candidate above `threshold`, and the first `equal_taken` of those equal to it, in index order; TopK of
// them at most. Returns how many equal ones there were up to the last winner. Sixteen scores side by
// side per thread and step, one barrier per step. Called by the whole block after a barrier.
template <int kThreads, typename Shared>
__device__ __noinline__ unsigned write_winners(Shared& s, const float* row, unsigned end, int32_t* list, unsigned threshold, unsigned equal_taken) {
  constexpr int kPerThread = 16;
  static_assert(kPerThread * kThreads < 65536, "two counts to a word");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned greater = 0, equal = 0;  // before this step
  for (unsigned first = 0, buffer = 0; first < end && greater + min(equal, equal_taken) < kTopK; first += kPerThread * kThreads, buffer ^= 1) {
    const unsigned mine = first + threadIdx.x * kPerThread;
    unsigned is_greater = 0, is_equal = 0;
#pragma unroll
    for (int h = 0; h < kPerThread; h += 4) {
      uint32_t key[4];
      bool valid[4];
      load_keys(row, mine + h, end, key, valid);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        is_greater |= unsigned(valid[e] && key[e] > threshold) << (h + e);
        is_equal |= unsigned(valid[e] && key[e] == threshold) << (h + e);
      }
    }
    const unsigned counts = unsigned(__popc(is_greater)) | unsigned(__popc(is_equal)) << 16;
    const unsigned scan = warp_scan(counts, lane);
    if (lane == 31) s.warp_sum[buffer][warp] = scan;
    __syncthreads();  // (the other buffer is read until everybody has come here)
    unsigned before = scan - counts, total = 0;
    for (int w = 0; w < kThreads / 32; ++w) {
      const unsigned sum = s.warp_sum[buffer][w];
      if (w < warp) before += sum;
      total += sum;
    }
    unsigned greater_before = greater + (before & 0xffffu), equal_before = equal + (before >> 16);
    for (unsigned left = is_greater | is_equal; left != 0; left &= left - 1) {
      const int bit = __ffs(left) - 1;
      const unsigned at = greater_before + min(equal_before, equal_taken);
      const bool above = is_greater >> bit & 1;
      if ((above || equal_before < equal_taken) && at < kTopK) list[at] = int32_t(mine + bit);
      if (above) ++greater_before; else ++equal_before;
    }
    greater += total & 0xffffu;
    equal += total >> 16;
  }
  return equal;
}

// For rows that the sample said too little about: a key that at least TopK candidates reach and at most
// `most`. Or, where so many are equal that there is none, the threshold itself (`equal` of the candidates
// equal to it are winners).
//
// Histograms over the whole row, 256 bins between `lower` and `upper`, then inside the bin that the
// `wanted`-th highest key up to `upper` lies in. Keys above `upper` are TopK - wanted winners; or, if
// `open`, any number of candidates (a sample's maximum is no maximum). One pass is the rule: scores that
// fool the sample are few in the bins. Called by the whole block after a barrier.
struct Floor {
  unsigned key, equal;
};
template <int kThreads, typename Shared>
__device__ __noinline__ Floor find_floor(Shared& s, const float* row, unsigned end, unsigned most, unsigned lower, unsigned upper, unsigned wanted, bool open) {
  const int lane = threadIdx.x & 31;
  // Six passes at most: the open range, four digits of one that holds the threshold, one that turns out not to.
  // (Scores that change meanwhile have no TopK best, but must not keep the block.)
  for (int pass = 0; pass < 8; ++pass) {
    const int shift = max(0, 24 - __clz(int(upper - lower)));
    for (unsigned first = threadIdx.x * 4; first < end + threadIdx.x * 4; first += 16 * kThreads) {
      uint32_t key[4][4];
      bool valid[4][4];
#pragma unroll
      for (int h = 0; h < 4; ++h) load_keys(row, first + h * 4 * kThreads, end, key[h], valid[h]);
#pragma unroll
      for (int h = 0; h < 4; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool counted = valid[h][e] && key[h][e] >= lower && (open || key[h][e] <= upper);
          if (!__any_sync(0xffffffffu, counted)) continue;
          // Lanes that fall into the same bin (most of them, among equal scores) add once.
          const unsigned bin = counted ? (upper - min(key[h][e], upper)) >> shift : kSelectBins;
          const unsigned peers = __match_any_sync(0xffffffffu, bin);
          if (counted && lane == __ffs(peers) - 1) atomicAdd(&s.histogram[bin], unsigned(__popc(peers)));
        }
    }
    __syncthreads();
    find_bin(s, wanted);
    if (s.bin == kSelectBins) {  // everything here is a winner, and more below
      wanted -= s.before;
      upper = lower - 1;
      lower = 0;
      open = false;
      continue;
    }
    const unsigned depth = ((s.bin + 1) << shift) - 1;
    const unsigned bottom = depth >= upper - lower ? lower : upper - depth;
    const bool beyond = open && s.bin == 0;  // the bin goes on above `upper`
    if (kTopK - wanted + s.before + s.in_bin <= most) return {bottom, 0};
    if (shift == 0 && !beyond) return {bottom, wanted - s.before};
    upper = beyond ? 0xffffffffu : upper - (s.bin << shift);
    lower = bottom;
    wanted -= s.before;
    open = false;
  }
  return {lower, wanted};
}

// Additions to and ors into words of shared memory where a predicate says so: one instruction, no branch around it.
__device__ __forceinline__ void shared_add_if(bool wanted, uint32_t address) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %0, 0;\n@p red.shared.add.u32 [%1], 1;\n}\n" ::"r"(uint32_t(wanted)), "r"(address) : "memory");
}
__device__ __forceinline__ void shared_or_if(bool wanted, uint32_t address, unsigned bits) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %0, 0;\n@p red.shared.or.b32 [%1], %2;\n}\n" ::"r"(uint32_t(wanted)), "r"(address), "r"(bits) : "memory");
}
// Four bytes on their way to shared memory; `cp.async.wait_all` waits for them.
__device__ __forceinline__ void copy_word(uint32_t to, const float* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(to), "l"(from) : "memory");
}

// The TopK best of the `listed` entries (not more than there is room for), written in index order. False, and nothing
// written, if fewer than TopK of them reach the floor. Called by the whole block after a barrier.
//
// Every instruction here is executed for each of the eight or nine hundred entries of every row, and rows are
// bound by what is issued, or wait for it: scores become keys once, behind the first digit an entry is compared with two keys, a
// winner is known by its bit when it looks for its place, and loops have no ends to look for and no branches. 8192 rows of 12-16 K scores 118 ->
// 110 us (93.5 -> 86.5 million instructions of a warp), of 4 K 85 -> 76, 1500 x 10 K 28.9 -> 25.8, 2000 x 20 K 40.4 -> 35.8, 16 x 16 K 6.85 -> 6.45.
template <int kThreads, int kCapacity, bool kKeysApart, typename Shared>
__device__ __forceinline__ bool select_from_list(Shared& s, unsigned end, int listed, unsigned floor_key, int32_t* list) {
  constexpr int kWindow = Shared::kWindow;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // ---- the TopK best of the list ----------------------------------------------------------------
  // Ordered by (distance of the key from the highest, row position): smaller is better, all
  // distinct. First the distance, then (more than 32 equal scores at the threshold) the position.
  // "The highest" is the sample's, and what lies above it counts as distance 0, until the
  // threshold turns out to lie there.
  unsigned top = s.high, bottom = floor_key;
  bool exact = false;
  auto find_extremes = [&](bool scores) {
    unsigned low = 0xffffffffu, high = 0;
    for (int i = threadIdx.x; i < listed; i += kThreads) {
      unsigned key = s.list[i].y;
      if (scores) s.list[i].y = key = score_key(key);
      low = min(low, key);
      high = max(high, key);
    }
    low = __reduce_min_sync(0xffffffffu, low);
    high = __reduce_max_sync(0xffffffffu, high);
    if (lane == 0) { atomicMin(&s.low, low); atomicMax(&s.high, high); }
    __syncthreads();
    top = s.high;
    bottom = s.low;
    exact = true;
  };
  const bool sampled = floor_key != 0;
  // The list is filled up to whole rounds of the block: no loop over it looks for its end. The filling's position is one that no row has (it is in
  // no window and not before `end`), its key is 0: it reaches no sampled floor, which is at least 1, and lies above no key.
  const int rounds = (listed + kThreads - 1) / kThreads;
  static_assert(kCapacity % kThreads == 0, "whole rounds fit");
  if (listed + int(threadIdx.x) < rounds * kThreads) s.list[listed + threadIdx.x] = make_uint2(0xffffffffu, kKeysApart || sampled ? 0xffffffffu : 0u);
  const uint32_t histogram = sm100::smem_u32(s.histogram);
  // Rows listed whole have nothing counted yet: their keys are made on the way to the extremes (600 x 600 scores 9.45 -> 8.9 us, 888 x 600 10.9 ->
  // 10.2, 8192 x 600 59.6 -> 56.8). kKeysApart: in the loop of the others, and gone through again.
  if (kKeysApart || sampled) {
    const int shift = max(0, 24 - __clz(int(top - bottom)));
    __syncthreads();
#pragma unroll 4
    for (int r = 0; r < rounds; ++r) {
      uint2& entry = s.list[r * kThreads + threadIdx.x];
      const unsigned key = score_key(entry.y);
      entry.y = key;
      shared_add_if(sampled && key >= floor_key, histogram + ((top - min(key, top)) >> shift) * 4);
    }
  }
  if (!sampled) find_extremes(!kKeysApart);  // of the entries that this thread has made keys, or makes keys now
  int above = 32 - __clz(int(top - bottom)), shift = max(0, above - 8);  // bits of the distance; bits below the digit
  bool counted = sampled;  // the present digit
  unsigned wanted = kTopK;
  unsigned prefix = 0;  // leading bits found so far
  unsigned ties = 0xffffffffu;  // distance of the threshold, once the position decides
  while (true) {
    if (!counted)
      for (int i = threadIdx.x; i < listed; i += kThreads) {
        const uint2 entry = s.list[i];
        const unsigned distance = top - min(entry.y, top), value = ties == 0xffffffffu ? distance : entry.x;
        if ((unsigned long long)value >> above == prefix && (ties == 0xffffffffu || distance == ties) && entry.y >= floor_key)
          atomicAdd(&s.histogram[value >> shift & (kSelectBins - 1)], 1u);
      }
    counted = false;
    __syncthreads();
    find_bin(s, wanted);
    if (s.bin == kSelectBins) {  // the rest are NaNs with a sign: scores again for who looks next
      for (int i = threadIdx.x; i < listed; i += kThreads) s.list[i].y = key_score(s.list[i].y);
      __syncthreads();
      return false;
    }
    prefix = prefix << (above - shift) | s.bin;
    if (prefix == 0 && !exact && ties == 0xffffffffu) {
      find_extremes(false);
      above = 32 - __clz(int(top - bottom));
      shift = max(0, above - 8);
      continue;
    }
    wanted -= s.before;
    if (s.in_bin <= 32) break;
    above = shift;
    if (shift == 0) {  // (positions are distinct: only for the distance)
      ties = prefix;
      prefix = 0;
      above = 32 - __clz(int(end - 1));
    }
    shift = max(0, above - 8);
  }

  // ---- winners in index order ---------------------------------------------------------------------
  // A bitmap of winning positions and the number of winners before each of its words: every winner
  // finds its place in the output by itself. What lies before the threshold's bin has won; the bin's entries go side by side, and one
  // warp finds the wanted-th smallest of them, the last winner.
  static_assert(uint64_t(kMostSpan) + kWindow <= UINT32_MAX, "unsigned positions");
  const uint32_t bitmap = sm100::smem_u32(s.bitmap);
  auto win_if = [&](bool wins, unsigned position) { shared_or_if(wins && position < kWindow, bitmap + (position >> 5) * 4, 1u << (position & 31)); };
  auto compare = [&](uint2 entry) { s.few[atomicAdd(&s.few_count, 1u)] = (unsigned long long)~entry.y << 32 | entry.x; };
  if (ties == 0xffffffffu) {
    // Keys above `before` lie before the bin (whatever lies above the sample's highest among them), keys from `within` on in it. A bin that
    // reaches down to key 0 (rows listed whole, with masks or NaNs that have a sign at the threshold) has the filling's key in it, which a
    // real entry may have too: there it is the position that tells them apart.
    const unsigned before = top - (prefix << shift), depth = prefix << shift | ((1u << shift) - 1);
    const unsigned within = max(floor_key, top - min(depth, top));
#pragma unroll 4
    for (int r = 0; r < rounds; ++r) {
      const uint2 entry = s.list[r * kThreads + threadIdx.x];
      win_if(entry.y > before, entry.x);
      if (entry.y <= before && entry.y >= within && entry.x < end) compare(entry);
    }
  } else {
    const unsigned tie = top - ties;
    for (int i = threadIdx.x; i < listed; i += kThreads) {
      const uint2 entry = s.list[i];
      win_if(entry.y > tie || (entry.y == tie && entry.x >> shift < prefix), entry.x);
      if (entry.y == tie && entry.x >> shift == prefix) compare(entry);
    }
  }
  __syncthreads();
  if (warp == 0) {
    const int few = int(s.few_count);  // 32 at most
    const unsigned long long mine = lane < few ? s.few[lane] : ~0ull;
    unsigned smaller = 0;
    if constexpr (kThreads >= 256) {
      // Eight at a time (the room behind them was filled with what is smaller than nothing): their reads wait together, where one after
      // the other each took the loop's test and a load's time. 768 rows of 64 K 42.8 -> 42.3 us, of 32 K 26.2 -> 25.7. Blocks of 128
      // threads, of which others run meanwhile, lost by the longer code (8192 rows 109.8 -> 110.3).
#pragma unroll
      for (int first = 0; first < 32; first += 8) {
        if (first >= few) break;
#pragma unroll
        for (int i = first; i < first + 8; ++i) smaller += s.few[i] < mine;
      }
    } else {
      for (int i = 0; i < few; ++i) smaller += s.few[i] < mine;
    }
    if (lane < few && smaller < wanted) {
      win_if(true, unsigned(mine));
      if (smaller + 1 == wanted) s.limit = mine;
    }
  }
  __syncthreads();
  unsigned written = 0;
  constexpr int kWords = kWindow / 32 > 4 * kThreads ? 8 : 4;  // of the bitmap, per thread: threads beyond it have none
  static_assert(kWindow / 32 <= kWords * kThreads, "the threads' words cover the window");
  for (unsigned window = 0; window < end; window += kWindow) {
    if (window > 0) {
      for (int i = threadIdx.x; i < kWindow / 32; i += kThreads) s.bitmap[i] = 0;
      __syncthreads();
      const unsigned long long limit = s.limit;
      for (int i = threadIdx.x; i < listed; i += kThreads) {
        const uint2 entry = s.list[i];
        win_if(((unsigned long long)~entry.y << 32 | entry.x) <= limit, entry.x - window);
      }
      __syncthreads();
    }
    const int words = int(min(end - window, unsigned(kWindow)) + 31) / 32, first = threadIdx.x * kWords;
    unsigned counts[kWords], mine = 0;
#pragma unroll
    for (int q = 0; q < kWords; q += 4) {
      uint4 quad = make_uint4(0, 0, 0, 0);
      if (first + q < words) quad = *reinterpret_cast<const uint4*>(&s.bitmap[first + q]);
      counts[q] = __popc(quad.x); counts[q + 1] = __popc(quad.y); counts[q + 2] = __popc(quad.z); counts[q + 3] = __popc(quad.w);
      mine += counts[q] + counts[q + 1] + counts[q + 2] + counts[q + 3];
    }
    const unsigned scan = warp_scan(mine, lane);
    if (lane == 31) s.warp_sum[0][warp] = scan;
    __syncthreads();
    unsigned at = written + scan - mine;
    for (int w = 0; w < kThreads / 32; ++w) {
      if (w < warp) at += s.warp_sum[0][w];
      written += s.warp_sum[0][w];
    }
    if (first < words) {
      unsigned packed[kWords / 2];  // a count is at most 512: two to a word
#pragma unroll
      for (int q = 0; q < kWords / 2; ++q) {
        packed[q] = at | (at + counts[2 * q]) << 16;
        at += counts[2 * q] + counts[2 * q + 1];
      }
#pragma unroll
      for (int q = 0; q < kWords / 2; q += 2) *reinterpret_cast<uint2*>(&s.place[first + 2 * q]) = make_uint2(packed[q], packed[q + 1]);
    }
    __syncthreads();
#pragma unroll 4
    for (int r = 0; r < rounds; ++r) {
      const unsigned position = s.list[r * kThreads + threadIdx.x].x, index = position - window, at = min(index, unsigned(kWindow - 1)) >> 5;
      const unsigned word = s.bitmap[at], bit = 1u << (index & 31);
      if ((word & bit) && index < kWindow) list[s.place[at] + __popc(word & (bit - 1))] = position;
    }
    if (end - window > kWindow) __syncthreads();  // the bitmap and the sums are free again
  }
  return true;
}

// In blocks of 128 threads a function: within 48 registers the pass over the row spills beside it (8192 x 12-16 K scores 121 us inlined,
// 115 called, rows of one constant 112.5 and 106.8). Larger blocks have it inline (768 x 64 K 37.6, called 39.0).
template <int kThreads, int kCapacity, typename Shared>
__device__ __noinline__ bool select_from_list_apart(Shared& s, unsigned end, int listed, unsigned floor_key, int32_t* list) {
  return select_from_list<kThreads, kCapacity, false>(s, end, listed, floor_key, list);
}
template <int kThreads, int kCapacity, bool kKeysApart = false, typename Shared>
__device__ __forceinline__ bool select_listed(Shared& s, unsigned end, int listed, unsigned floor_key, int32_t* list) {
  if constexpr (kThreads == 128) return select_from_list_apart<kThreads, kCapacity>(s, end, listed, floor_key, list);
  else return select_from_list<kThreads, kCapacity, kKeysApart>(s, end, listed, floor_key, list);
}

// Lists what reaches the floor, by keys. For 128 threads: with 48 registers the loop in `select_by_keys` spills and waits for every
// load, which took rows of zeros (8192 x 16 K, whose floor is subnormal) from 130 to 143 us when ten blocks came to share an SM.
// The scores' order in place of their bits, a look at the highest of sixteen first, and 16 KiB on their way to L2: 111. (With 256
// threads and 40 registers the whole kernel is slower for it, usual rows of 768 x 65536 scores 38.1 -> 43.2.)
template <int kThreads, int kCapacity, typename Shared>
__device__ __forceinline__ void list_by_order(Shared& s, const float* row, unsigned end, unsigned floor_key) {
  constexpr unsigned kStep = 16 * kThreads, kAhead = kStep > 4096 ? kStep : 4096;
  const auto order = [](uint32_t bits) { return int(bits ^ (uint32_t(int(bits) >> 31) & 0x7fffffffu)); };  // its own inverse
  const int least = int(floor_key ^ 0x80000000u);
  for (unsigned first = threadIdx.x * 4; first < end + threadIdx.x * 4; first += kStep) {
    if (threadIdx.x == 0 && first + kAhead < end) prefetch_l2(row + first + kAhead, 4u * min((end - first - kAhead + 3u) & ~3u, kStep));
    int v[16];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const unsigned i = first + h * 4 * kThreads;
      const uint4 w = i < end ? __ldcs(reinterpret_cast<const uint4*>(row + i)) : make_uint4(0, 0, 0, 0);
      v[4 * h] = order(w.x); v[4 * h + 1] = order(w.y); v[4 * h + 2] = order(w.z); v[4 * h + 3] = order(w.w);
    }
    int best = v[0];
#pragma unroll
    for (int e = 1; e < 16; ++e) best = max(best, v[e]);
    if (best < least) continue;
    unsigned hits = 0;
#pragma unroll
    for (int e = 0; e < 16; ++e) hits |= unsigned(v[e] >= least) << e;
    if (first + 12 * kThreads + 3 >= end) {  // the last step: drop what lies past the end
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const unsigned i = first + h * 4 * kThreads, left = i < end ? min(end - i, 4u) : 0u;
        hits &= ~((15u << left & 15u) << (4 * h));
      }
      if (hits == 0) continue;
    }
    unsigned at = atomicAdd(&s.count, unsigned(__popc(hits)));
    if (at + unsigned(__popc(hits)) > kCapacity) continue;
#pragma unroll
    for (int e = 0; e < 16; ++e)
      if (hits >> e & 1) s.list[at++] = make_uint2(first + (e >> 2) * 4 * kThreads + (e & 3), unsigned(order(unsigned(v[e]))));
  }
}

// What is left of `topk_select_kernel` where the list of what reaches the floor is too short or too long, or has not
// been made (`listed`), since the floor is zero, subnormal, infinite or a NaN. All by keys, and not inline: the
// usual row's instructions stay together.
template <int kThreads, int kCapacity, typename Shared>
__device__ __noinline__ void select_by_keys(Shared& s, const float* row, unsigned end, int32_t* list, unsigned floor_key, bool listed) {
  bool fits = false;  // the floor has been found to
  while (true) {
    if (!listed) {
      if constexpr (kThreads == 128) {
        list_by_order<kThreads, kCapacity>(s, row, end, floor_key);
      } else {
        for (unsigned first = threadIdx.x * 4; first < end + threadIdx.x * 4; first += 16 * kThreads) {
          uint32_t key[4][4];
          bool valid[4][4];
          uint4 v[4];
#pragma unroll
          for (int h = 0; h < 4; ++h) v[h] = load_keys(row, first + h * 4 * kThreads, end, key[h], valid[h]);
          unsigned hits = 0;
#pragma unroll
          for (int e = 0; e < 16; ++e) hits |= unsigned(valid[e >> 2][e & 3] && key[e >> 2][e & 3] >= floor_key) << e;
          if (hits == 0) continue;
          unsigned at = atomicAdd(&s.count, unsigned(__popc(hits)));
          if (at + unsigned(__popc(hits)) > kCapacity) continue;
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const unsigned values[4] = {v[h].x, v[h].y, v[h].z, v[h].w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (hits >> (4 * h + e) & 1) s.list[at++] = make_uint2(first + h * 4 * kThreads + e, values[e]);
          }
        }
      }
      __syncthreads();
      const unsigned count = s.count;
      if (count >= kTopK && count <= kCapacity && select_listed<kThreads, kCapacity>(s, end, int(count), floor_key, list)) return;
      if (fits) return;  // the scores have changed since they were counted
    }
    Floor found;
    const unsigned count = s.count;
    if (count > kCapacity) {
      found = find_floor<kThreads>(s, row, end, kCapacity, floor_key, max(s.high, floor_key), kTopK, true);
    } else {
      unsigned reached = 0;  // of the list, without NaNs
      for (unsigned i = threadIdx.x; i < count; i += kThreads) reached += score_key(s.list[i].y) >= floor_key;
      reached = __reduce_add_sync(0xffffffffu, reached);
      if ((threadIdx.x & 31) == 0) atomicAdd(&s.few_count, reached);
      __syncthreads();
      unsigned missing = kTopK - s.few_count, upper = floor_key - 1, lower = min(s.low, upper);
      if (s.mass) {
        const unsigned equal = write_winners<kThreads>(s, row, end, list, upper, missing);
        if (equal >= missing) return;
        missing -= equal;
        --upper;
        lower = 0;
      }
      found = find_floor<kThreads>(s, row, end, kCapacity, lower, upper, missing, false);
    }
    if (found.equal != 0) {
      write_winners<kThreads>(s, row, end, list, found.key, found.equal);
      return;
    }
    floor_key = found.key;
    fits = true;
    listed = false;
    __syncthreads();
    if (threadIdx.x == 0) s.count = s.few_count = 0;
    __syncthreads();
  }
}

template <int kCount>
struct Loads {
  static constexpr int value = kCount;
};

// One block per query token. Candidates are compressed rows [0, min(available, cutoff)): the rows
// the attention kernel would accept for this token. The min(TopK, candidates) highest scores win,
// ties going to the lower index; winners are written in ascending index order, the rest of the 512
// entries is -1.
//
// Bound by memory for long rows (768 x 65536 scores: 44 us as called, 70 % of the copy bandwidth; the radix
// select that read the row five times took 335 us) and by what is issued, instructions and shared memory's accesses, for many
// short ones (8192 x 12-16 K: 110 us, 4.3 TB/s; issue slots 69 %; before 1003 us). The row is streamed once. A strided sample (one or
// two thousand scores in 128-byte pieces) gives a floor that about twice TopK scores lie above; the
// stream lists what reaches the floor (two instructions per score, next to nothing listed), and the exact selection runs on
// that short list in shared memory: a histogram of the keys' distances from the highest, 256
// bins, normally once; the few entries of the threshold's bin are ranked by comparison; a bitmap
// of winning positions gives the output order. The list holds every score that reaches the
// floor, so the result is exact whenever the list has at least TopK entries and did not
// overflow. Otherwise the row is gone through again, by keys (`select_by_keys`):
//   many equal scores  (zeros behind a ReLU, masks) show in the sample as a floor that many samples are
//                      equal to. What lies above it is listed; if that is too little, one more pass in index
//                      order takes the first of the equal ones (`write_winners`).
//   a sample that      (scores that change slowly along the row) is set right by `find_floor`, and the
//   says too little    row streamed once more with a floor that is known to fit.
// 768 x 65536 scores, against the radix select that read every row five times: constant 373 -> 55 us, zeros 383
// -> 80, all but 300 masked 360 -> 142, correlated over 64 positions 326 -> 192 (a fifth of the rows);
// 100 rows of the latter 114 -> 80. With that select as the way out they took 461, 433, 457, 283 and 127.
template <int kThreads, int kCapacity, int kMostQuads, int kInFlight, int kWindowSize, int kShortRow, bool kCopyScores>
__device__ __forceinline__ void select_row(const SelectParams& p, unsigned char* shared, const float* row, int candidates, int32_t* list) {
  using Shared = SelectShared<kThreads, kCapacity, kWindowSize>;
  constexpr int kWindow = Shared::kWindow;
  Shared& s = *reinterpret_cast<Shared*>(shared);
  const int lane = threadIdx.x & 31;
  for (int i = threadIdx.x * 4; i < min(candidates + 31, kWindow) / 32; i += kThreads * 4)
    *reinterpret_cast<uint4*>(&s.bitmap[i]) = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < kSelectBins; i += kThreads) s.histogram[i] = 0;
  if (kThreads >= 256 && threadIdx.x < 32) s.few[threadIdx.x] = ~0ull;  // smaller than none: select_from_list reads in rounds
  if (threadIdx.x == 0) { s.count = s.few_count = 0; s.mass = false; s.low = 0xffffffffu; s.high = 0; s.bin = kSelectBins; }
  __syncthreads();

  // kInFlight: 16-byte loads in flight per thread of the pass over the row (four for rows of up to kShortRow scores)
  static_assert(kInFlight <= 8, "a word of signs");
  constexpr unsigned kHead = kInFlight * 4 * kThreads > 4096 ? kInFlight * 4 * kThreads : 4096;
  const unsigned end = unsigned(candidates);  // unsigned: a step may reach past INT32_MAX

  // ---- floor ----------------------------------------------------------------------------------
  unsigned floor_key = 0;  // short rows: everything is listed
  constexpr int kListed = 4 * kThreads > 1024 ? 4 * kThreads : 1024;  // (listing 8 K scores costs more than sampling them)
  static_assert(kListed <= kCapacity, "the whole row fits the list");
  if (candidates > kListed) {
    // An eighth of the row, or kMostQuads 16-byte quads per thread: eight threads share a 128-byte
    // segment, and the segments lie at equal distances.
    constexpr int kSegments = kThreads / 8;
    // Where more quads than these are for long rows only, short ones step over them (8192 x 4 K scores 76 -> 73 us).
    constexpr int kFewQuads = 2;
    // Larger blocks have more quads for rows beyond this many (see the launch): a buffer is as wide as the longest context (in one of 128 K scores
    // 888 x 64 K 40.3 -> 38.8 us, 600 x 96 K 46.1 -> 45.1).
    constexpr int kLargeSampleRow = 98304;
    const int most = kThreads >= 256 && candidates <= kLargeSampleRow ? min(kMostQuads, kFewQuads) : kMostQuads;
    const int quads = max(1, min(most, candidates / (32 * kThreads))), sampled = quads * kThreads;
    const unsigned step = (unsigned(candidates) >> 2) / unsigned(quads * kSegments);  // at least eight quads
    uint4 v[kMostQuads];
#pragma unroll
    for (int q = 0; q < kMostQuads; ++q)
      if (q < quads) v[q] = __ldg(reinterpret_cast<const uint4*>(row) + (q * kSegments + (threadIdx.x >> 3)) * step + (threadIdx.x & 7));
    // The row's head on its way to L2 behind the sample, while the floor is found. Not where all rows of a call start at once and are not
    // long: the heads of those that are first stand in front of the others' samples (800 x 8 K 14.26 -> 13.60 us, 500 x 16 K 13.86 -> 13.38, 888 x
    // 18000 19.4 -> 18.9, 300 x 16 K 11.6 -> 11.3; but 300 x 3000 8.03 -> 8.12, 300 x 18000 with little L1 12.7 -> 13.2, 1200 x 16 K 25.6 -> 26.9).
    constexpr bool kMayWait = kThreads == 256 && kWindow <= 24576;
    if (threadIdx.x == 0 && !(kMayWait && p.one_wave && end > kHead / 4 * 3)) prefetch_l2(row, 4u * min((end + 3u) & ~3u, kHead));
    uint32_t key[4 * kMostQuads] = {};
#pragma unroll
    for (int q = 0; q < kMostQuads; ++q) {
      if (q == kFewQuads && quads <= kFewQuads) break;
      key[4 * q + 0] = q < quads ? score_key(v[q].x) : 0; key[4 * q + 1] = q < quads ? score_key(v[q].y) : 0;
      key[4 * q + 2] = q < quads ? score_key(v[q].z) : 0; key[4 * q + 3] = q < quads ? score_key(v[q].w) : 0;
    }
    // Samples expected among the TopK best, and five standard deviations of that count on top: of
    // independent scores, the floor lies below the TopK-th best in all but a few rows in a million. (A piece of
    // neighbours that are alike is one draw and not 32: such rows miss more often, see `select_by_keys`.)
    const float expected = float(kTopK) * float(4 * sampled) / float(candidates);
    unsigned wanted = unsigned(expected + 5.f * sqrtf(expected) + 2.f);
    // Only the sample's upper end matters: its maximum, and the lowest of the maxima of G groups, above
    // which lie about four G samples: G = all threads, or a quarter of them where that is enough.
    unsigned best = 0;
#pragma unroll
    for (int e = 0; e < 4 * kMostQuads; ++e) {
      if (e == 4 * kFewQuads && quads <= kFewQuads) break;
      best = max(best, key[e]);
    }
    if (wanted <= unsigned(kThreads / 4)) {
      best = max(best, __shfl_xor_sync(0xffffffffu, best, 1));
      best = max(best, __shfl_xor_sync(0xffffffffu, best, 2));
    }
    const unsigned warp_low = __reduce_min_sync(0xffffffffu, best), warp_high = __reduce_max_sync(0xffffffffu, best);
    if (lane == 0) { atomicMin(&s.low, warp_low); atomicMax(&s.high, warp_high); }
    __syncthreads();
    unsigned lower = s.low, upper = s.high, above = 0;  // (samples above `upper`)
    while (true) {  // normally once; again inside a bin that holds too many (a sample of both signs, say)
      const int shift = max(0, 24 - __clz(int(upper - lower)));  // 256 bins over [lower, upper]
#pragma unroll
      for (int e = 0; e < 4 * kMostQuads; ++e) {
        if (e == 4 * kFewQuads && quads <= kFewQuads) break;
        if (key[e] >= lower && key[e] <= upper) atomicAdd(&s.histogram[(upper - key[e]) >> shift], 1u);
      }
      __syncthreads();
      find_bin(s, wanted);
      if (s.bin == kSelectBins) break;  // fewer samples than wanted: all of them
      const unsigned depth = ((s.bin + 1) << shift) - 1;
      lower = depth >= upper - lower ? lower : upper - depth;
      if (s.in_bin <= 32) break;
      if (shift == 0) {  // many are equal to the floor: what lies above it, unless all of them are likely to fit
        above += s.before + s.in_bin;
        if (float(above) * float(candidates) > 0.8f * kCapacity * float(4 * sampled) && lower != 0xffffffffu) {
          ++lower;
          if (threadIdx.x == 0) s.mass = true;
        }
        break;
      }
      upper -= s.bin << shift;
      wanted -= s.before;
      above += s.before;
    }
    floor_key = lower;
  }

  // ---- one pass over the row --------------------------------------------------------------------
  // Scores that reach the floor are listed in any order, by the sign of score - floor: two instructions per
  // score. That is no less exact than the keys but for NaNs, which are listed whatever their sign (those with one
  // have the lowest keys of all and do not count), and for subnormals, which are flushed.
  const unsigned floor_bits = floor_key == 0 ? 0xff800000u : floor_key & 0x80000000u ? floor_key ^ 0x80000000u : ~floor_key;
  const unsigned exponent = floor_bits & 0x7f800000u;
  const bool normal = floor_key == 0 || (exponent != 0 && exponent != 0x7f800000u);
  const float floor_value = __uint_as_float(floor_bits);
  if (normal) {
    // What lies further on is on its way to L2 meanwhile, 16 KiB with 128 and 256 threads, a step with more: a block's own loads are
    // not in flight while it looks at what they brought (768 x 65536 scores, 256 threads: 51.1 -> 45.0 us, 1800 x 65536:
    // 105 -> 89; 12 and 32 KiB: 46.1, and 64 KiB at the row's head alone, 51.1. 512 threads with eight loads, 16 and 100 x 64 K:
    // no difference between 16, 32 and 64 KiB).
    auto list_row = [&](auto loads) {
      constexpr int kLoads = decltype(loads)::value;
      constexpr unsigned kStep = kLoads * 4 * kThreads, kAhead = kStep > 4096 ? kStep : 4096;
      for (unsigned base = 0; base < end; base += kStep) {
        const unsigned first = base + threadIdx.x * 4;
        if (threadIdx.x == 0 && first + kAhead < end) prefetch_l2(row + first + kAhead, 4u * min((end - first - kAhead + 3u) & ~3u, kStep));
        // Large blocks wait for the last step's copies (below) before they load on, and not only behind the pass: calls that fill the memory lost by these (148 x 200 K scores 33.0 -> 32.1 us, 148 x 300 K 46.5 -> 44.2, 300 x 300 K 113 -> 109.5; 1 x 200 K 20.1 -> 20.3).
        if constexpr (kThreads == 1024 && kCopyScores) asm volatile("cp.async.wait_all;\n" ::: "memory");
        uint4 v[kLoads];
#pragma unroll
        for (int h = 0; h < kLoads; ++h) {
          const unsigned i = first + h * kThreads * 4;
          v[h] = i < end ? __ldcs(reinterpret_cast<const uint4*>(row + i)) : make_uint4(0, 0, 0, 0);
        }
        // The sign of score - floor, shifted in: bit 31 - (4 h + e) is clear where the score reaches it.
        unsigned below = 0;
#pragma unroll
        for (int h = 0; h < kLoads; ++h) {
          below = __funnelshift_l(__float_as_uint(__uint_as_float(v[h].x) - floor_value), below, 1);
          below = __funnelshift_l(__float_as_uint(__uint_as_float(v[h].y) - floor_value), below, 1);
          below = __funnelshift_l(__float_as_uint(__uint_as_float(v[h].z) - floor_value), below, 1);
          below = __funnelshift_l(__float_as_uint(__uint_as_float(v[h].w) - floor_value), below, 1);
        }
        unsigned hits = ~below << (32 - 4 * kLoads);
        if (first + (kLoads - 1) * kThreads * 4 + 3 >= end) {  // the last step: drop what lies past the end
#pragma unroll
          for (int h = 0; h < kLoads; ++h) {
            const unsigned i = first + h * kThreads * 4, left = i < end ? min(end - i, 4u) : 0u;
            hits &= ~((15u >> left) << (28 - 4 * h));
          }
        }
        if (hits == 0) continue;
        unsigned at = atomicAdd(&s.count, unsigned(__popc(hits)));
        if (at + unsigned(__popc(hits)) > kCapacity) continue;  // noticed below: s.count says so
        // Few rows wait for what is issued for them, all of a step's scores as candidates for a place: a loop over the hits, which
        // copies the scores from where the load has just put them (16 x 16 K scores 6.56 -> 6.44 us, 100 x 64 K 10.7 -> 9.2). With many
        // rows these copies wait for L2, or for memory where it has been given up (8192 x 12-16 K 116 -> 145, 768 x 64 K 38 -> 56, 600 x 200 K 113 -> 117).
        if constexpr (kCopyScores) {
          do {
            const unsigned which = __clz(hits), position = first + (which >> 2) * 4 * kThreads + (which & 3);
            s.list[at].x = position;
            copy_word(sm100::smem_u32(&s.list[at].y), row + position);
            ++at;
            hits &= 0x7fffffffu >> which;
          } while (hits != 0);
        } else {
#pragma unroll
          for (int h = 0; h < kLoads; ++h) {
            const unsigned values[4] = {v[h].x, v[h].y, v[h].z, v[h].w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (hits >> (31 - 4 * h - e) & 1) s.list[at++] = make_uint2(first + h * kThreads * 4 + e, values[e]);
          }
        }
      }
    };
    if (kShortRow > 0 && end <= unsigned(kShortRow)) list_row(Loads<4>{});
    else list_row(Loads<kInFlight>{});
    if constexpr (kCopyScores) asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    const int listed = int(s.count);
    // (With the keys of whole rows made apart the pass over long rows is slower in this one form: 768 x 64 K 41.8 -> 43.0 us, 2000 x 64 K 90.6 -> 96.2.)
    constexpr bool kKeysApart = kThreads == 256 && kWindow == 65536 && kMostQuads == 2;
    if (listed >= kTopK && listed <= kCapacity) {
      if (select_listed<kThreads, kCapacity, kKeysApart>(s, end, listed, floor_key, list)) return;
    }
  }
  select_by_keys<kThreads, kCapacity>(s, row, end, list, floor_key, normal);
}

// kHalfRow: rows of up to so many scores are left to the first half of the block, which does as a block of its size.
template <int kThreads, int kCapacity, int kBlocks, int kMostQuads, int kInFlight, int kWindowSize, int kShortRow, bool kCopyScores, int kHalfRow>
__global__ void __launch_bounds__(kThreads, kBlocks) topk_select_kernel(const SelectParams p) {
  extern __shared__ __align__(16) unsigned char select_smem[];
  const int token = blockIdx.x;
  sm100::wait_for_predecessor();
  // Many rows: blocks of the next launch come when these end. Waiting beside them they take the slots
  // of SMs that got fewer rows, and so spread their own unevenly (600 x 16 K: 19.3 against 16.4 us; two rows per SM and less, 149 of 600 to 64 K
  // scores 10.9 / 10.3).
  constexpr bool kFewRows = kThreads >= 512 && kHalfRow == 0;
  if constexpr (kFewRows) sm100::let_successor_start();
  const int candidates = int(min((int64_t)visible_compressed_rows<kFewRows>(p, token, threadIdx.x & 31), p.span));
  int32_t* list = p.out + (size_t)token * kTopK;
  const float* row = p.scores + (size_t)token * p.span;
  if (candidates <= kTopK) {
    for (int i = threadIdx.x; i < kTopK; i += kThreads) list[i] = i < candidates ? i : -1;
    return;
  }
  if constexpr (kHalfRow > 0) {
    if (candidates <= kHalfRow) {
      // (Barriers of the block are of the threads that have not left.)
      if (threadIdx.x < kThreads / 2) select_row<kThreads / 2, kHalfCapacity, 2, 4, kHalfRow, 0, false>(p, select_smem, row, candidates, list);
      return;
    }
  }
  select_row<kThreads, kCapacity, kMostQuads, kInFlight, kWindowSize, kShortRow, kCopyScores>(p, select_smem, row, candidates, list);
}

// One warp per new row: token j of n of request b goes to logical position L_b - n + j of the raw
// cache (L_b includes this call's tokens, as `seqused_ori_kv` does for the attention operator),
// i.e. to row `position % rows_per_page` of page `table[b][position / rows_per_page]`.
__global__ void cache_append_kernel(const char* new_rows, char* cache, const int32_t* table, const int32_t* cu,
                                    const int32_t* lengths, int batches, int tokens, int pages, int blocks,
                                    int page_rows, int32_t* status, volatile int32_t* flag) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  sm100::wait_for_predecessor();
  sm100::let_successor_start();
  for (int token = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; token < tokens; token += warps) {
    // (the row itself is loaded meanwhile)
    const uint4* source = reinterpret_cast<const uint4*>(new_rows + (size_t)token * kRowBytes);
    const uint4 low = __ldg(source + lane), high = __ldg(source + lane + 32);
    const Request request = request_of<true>(cu, batches, token, lane, lengths, lengths);
    const int position = request.first - request.count + (token - request.begin);
    const int column = position / page_rows;
    const int page = position >= 0 && column < pages ? __ldg(table + (size_t)request.index * pages + column) : -1;
    if (position < 0 || (unsigned)page >= (unsigned)blocks) {  // nowhere to put it: reported, not written
      if (lane == 0 && atomicCAS(status, kStatusOk, kStatusBadPage) == kStatusOk) {
        status[1] = token;
        status[2] = position;
        if (flag != nullptr) *flag = 1;
      }
      continue;
    }
    uint4* target = reinterpret_cast<uint4*>(cache + ((size_t)page * page_rows + position % page_rows) * kRowBytes);
    target[lane] = low;
    target[lane + 32] = high;
  }
}

template <int kThreads, int kCapacity, int kBlocks, int kMostQuads, int kInFlight = 4, int kWindow = (kThreads >= 256 ? 65536 : 256 * kThreads), int kShortRow = 0,
          bool kCopyScores = (kThreads >= 512), int kHalfRow = 0>
int launch_select(const SelectParams& p, cudaStream_t stream) {
  auto* kernel = topk_select_kernel<kThreads, kCapacity, kBlocks, kMostQuads, kInFlight, kWindow, kShortRow, kCopyScores, kHalfRow>;
  constexpr int bytes = int(sizeof(SelectShared<kThreads, kCapacity, kWindow>));
  static_assert(kHalfRow == 0 || sizeof(SelectShared<kThreads / 2, kHalfCapacity, kHalfRow>) <= bytes, "the half's fits");
  // A per-device setting: plain words written with the same value by whoever gets there first.
  static bool configured[64] = {false};
  int device = 0;
  if (cudaError_t error = cudaGetDevice(&device)) return int(error);
  if (device < 0 || device >= 64) return -1;
  if (!configured[device]) {
    if (cudaError_t error = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)) return int(error);
    configured[device] = true;
  }
  return int(sm100::launch_overlapped(kernel, p.tokens, kThreads, bytes, stream, p));
}

}  // namespace
}  // namespace sparse_mla

using namespace sparse_mla;

extern "C" {

int launch_sparse_mla_topk_indices(void* stream, void* arg_scores, void* arg_cu_seqlens_q, void* arg_seqused_cmp_kv,
                                   void* arg_cmp_residual_kv, void* arg_cmp_sparse_indices, int64_t B, int64_t T,
                                   int64_t SPAN, int64_t CMP_PAGE) {
  if (B <= 0 || T <= 0 || SPAN <= 0 || B > INT32_MAX || T > INT32_MAX || SPAN > kMostSpan || SPAN % 4 != 0) return -1;
  if (CMP_PAGE != 64 && CMP_PAGE != 128) return -1;
  SelectParams p = {};
  p.scores = static_cast<const float*>(arg_scores);
  p.cu = static_cast<const int32_t*>(arg_cu_seqlens_q);
  p.seq_cmp = static_cast<const int32_t*>(arg_seqused_cmp_kv);
  p.residual = static_cast<const int32_t*>(arg_cmp_residual_kv);
  p.out = static_cast<int32_t*>(arg_cmp_sparse_indices);
  p.batches = int32_t(B); p.tokens = int32_t(T); p.ratio = int32_t(kPage / CMP_PAGE);
  p.span = SPAN;
  int device = 0, multiprocessors = 148;
  if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&multiprocessors, cudaDevAttrMultiProcessorCount, device);
  p.one_wave = T <= int64_t(multiprocessors) * 6;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // T x N below are T rows of N scores, in a buffer as wide unless its width is given; us per call, scores from memory, these kernels unless said otherwise.
  //
  // Rows so long that a smaller block's sample says too little: 1024 threads (1024 / 512: 16 x 1 M 89 / 318, 300 x 1 M 330 / 599, 148 x 300 K 44.3 / 46.7, 16 x 200 K
  // 23.4 / 26.8), for more rows than SMs only beyond 256 K: two blocks of 512 threads to an SM are better before that (300 x 200 K 81.2 / 71.9, 600 x 200 K 137 /
  // 114) and where the buffer is wide but the rows are not (2000 x 2000 in 140000 107 / 57). What loses by it: 600 x 300 K 186 / 162, 16 x 6000 in 140000 8.7 / 6.9.
  //
  // No more rows than SMs: a row's latency counts, 512 threads (1024 / 512 / 256: 16 x 16 K 8.1 / 6.7 / 7.6, 148 x 64 K 13.8 / 12.8 / 17.5, 148 x 128 K 21.4 / 19.8 / 30.0; what
  // loses: 16 x 8 K 8.7 / 6.9 / 6.6, 16 x 2000 8.0 / 7.3 / 6.2), with eight loads in flight per thread for rows of more than three steps of
  // four. The kernel looks at the row for that: a buffer is as wide as the longest context (four / eight in a buffer of 64 K, 16 x 64 K 9.7 / 8.8, 30000 7.9 / 7.6, 24000
  // 7.4 / 7.5, 4096 6.8 / 7.0). Two such blocks run on an SM: up to twice as
  // many rows in buffers beyond 32 K, where rows of up to 16 K scores are left to half of their block, since what is shorter waits for sixteen
  // warps' barriers and not for memory (296 rows in a buffer of 64 K, eight warps / sixteen / sixteen or half of them: 64 K scores 19.9 / 19.0 / 18.6, 32000
  // 13.1 / 12.4 / 11.9, 17000 10.9 / 10.8 / 10.1, 8000 8.3 / 9.5 / 8.5, 2000 7.3 / 10.1 / 7.3, 600 6.8 / 8.0 / 6.5, 600 to 64 K 17.0 / 12.8 / 12.2; in a
  // buffer of 32772 the last 12.4 / 10.9 / 10.9).
  //
  // More rows: small blocks, several to an SM, whose phases overlap. Four warps per row from twelve rows per SM on (four / eight, 8192 x 12 K 103 / 124, 4096 x 8 K 47.7 /
  // 57.8, 2000 x 4 K 22.5 / 26.6, 4096 x 32 K 97.5 / 102). Fewer rows too would be faster with four (1184 x 8 K 16.0 / 21.2, 1500 x 4 K 19.1 / 20.7), but not where scores
  // correlate: the list misses more often the smaller the sample is (1184 x 8 K 40.0 / 35.5, 1500 x 16 K 79 / 64, 888 x 16 K 69 / 55; beyond the line as well, 1776 x 16 K
  // 83 / 69, 4096 x 16 K 124 / 114).
  // Of these, rows of up to 16 K scores (a bitmap of one window) run ten blocks of 48 registers per SM with four loads in flight, or eight blocks with eight loads (ten /
  // eight). Up to 10 K ten: 8192 x 2000 63.2 / 72.0, 8192 x 4 K 73.3 / 76.3, 4096 x 8 K 47.7 / 47.6, 4096 x 10 K 51.8 / 53.6. Beyond, ten where they make fewer waves: 2450 x
  // 12 K 36.1 / 36.6, 4096 of 600 to 16 K 44.4 / 46.7, but 4096 x 16 K 65.1 / 63.0, 7400 x 16 K 108 / 106, 8192 of 12 to 16 K 109.8 / 107.8; where they do not, eight: 1776 x
  // 12 K 31.3 / 27.2, 3300 x 16 K 55.5 / 51.1. With as many waves eight are better from 5 K on by now (1776 x 2000 18.5 / 19.2, 1776 x 4 K 21.3 / 20.8, 1800 of 7.5
  // to 10 K 30.2 / 26.6, 3000 x 8 K 38.7 / 36.1): the line at 10 K is that of a slower ranking. Longer rows are streaming for the most part: eight blocks, eight
  // loads (against ten, with that ranking: 4096 x 17408: 74.3 / 76.9, 2000 x 20 K: 39.2 / 43.9, 4096 x 32 K: 107.4 / 112.8). Eleven blocks leave a list of 1536
  // entries, which rows that correlate overflow (8192 x 16 K of zeros 130 -> 164).
  if (SPAN > 262144 || (SPAN > 131072 && T <= multiprocessors)) return launch_select<1024, 8192, 1, 2>(p, s);
  if (T <= multiprocessors && SPAN <= 24576) return launch_select<512, 4096, 2, 2>(p, s);
  if (SPAN <= 131072 && T <= multiprocessors) return launch_select<512, 4096, 2, 2, 8, 65536, 24576>(p, s);
  if (SPAN <= 131072 && T <= int64_t(multiprocessors) * 2 && SPAN > 32768) return launch_select<512, 4096, 2, 2, 8, 65536, 24576, true, 16384>(p, s);
  if (SPAN > 131072)
    return T <= int64_t(multiprocessors) * 2 ? launch_select<512, 4096, 2, 2>(p, s) : launch_select<512, 4096, 2, 2, 4, 65536, 0, false>(p, s);
  const bool fewer_waves = (T - 1) / (multiprocessors * 10) < (T - 1) / (multiprocessors * 8);
  if (T >= int64_t(multiprocessors) * 12 && SPAN <= 32768)
    return SPAN <= (fewer_waves ? 16384 : 10240) ? launch_select<128, 2048, 10, 4, 4, 16384>(p, s) : launch_select<128, 2048, 8, 4, 8>(p, s);
  // A bitmap no larger than the row: what shared memory it does not take holds scores that are read again (860 x 16 K 18.8 ->
  // 17.2, such rows that correlate 54.5 -> 53.2; blocks of 512 threads: no change).
  if (SPAN <= 16384) return launch_select<256, 2560, 6, 2, 4, 16384>(p, s);
  // The same beyond, where three more such steps lie: six blocks with a bitmap of 24 K leave 92 KiB of L1 on an SM, of 32 and 48 K 60, of 64 K
  // 28, and the sample's 48 KiB are read again in the pass (64 K / the smaller one: 600 x 18000 17.8 / 16.2, 888 x 24000 23.0 / 20.9, 1200
  // x 18000 30.7 / 28.1, 300 x 20000 12.2 / 12.0). The steps to 32 and 48 K are taken where the last wave is at least half full (600 x 30000
  // 23.2 / 21.1, 888 x 32768 26.2 / 25.1, 1750 x 30000 50.2 / 46.8, 600 x 45000 28.5 / 25.2, 888 x 48 K 35.0 / 33.6; where it is not, 300 x
  // 32768 14.8 / 15.2, 1200 x 32768 35.5 / 35.7, 1000 x 48 K 43.3 / 45.0).
  // A smaller one for longer rows, in several rounds: 500 x 50000 27.5 / 26.2, but 300 x 64 K 21.8 / 24.4.
  if (SPAN <= 24576) return launch_select<256, 2560, 6, 2, 4, 24576>(p, s);
  if (SPAN <= 49152 && (T - 1) % (int64_t(multiprocessors) * 6) >= int64_t(multiprocessors) * 3)
    return SPAN <= 32768 ? launch_select<256, 2560, 6, 2, 4, 32768>(p, s) : launch_select<256, 2560, 6, 2, 4, 49152>(p, s);
  // Of 128 K scores a sample of 2048 leaves some fifteen hundred in the list, give or take three hundred, and room for 2560: every few
  // thousand rows one is gone through again, which the call waits for. Twice the sample (scores from memory): 768 x 128 K 80.9 us where it was 166,
  // 888: 85 / 168, 1500: 136 / 223. Calls without such a row pay up to two per cent for it (600 x 128 K 65.3 / 64.2);
  // with one they take 80 us more. Rows of up to 98304 scores have the smaller sample.
  return SPAN > 98304 ? launch_select<256, 2560, 6, 4>(p, s) : launch_select<256, 2560, 6, 2>(p, s);
}

int launch_sparse_mla_cache_append_flagged(void* stream, void* arg_new_rows, void* arg_cache, void* arg_block_table,
                                           void* arg_cu_seqlens_q, void* arg_seqused_kv, void* status_words, void* flag,
                                           int64_t B, int64_t T, int64_t PAGES, int64_t BLOCKS, int64_t PAGE_ROWS) {
  if (B <= 0 || T <= 0 || PAGES <= 0 || BLOCKS < 0 || status_words == nullptr) return -1;
  if (PAGE_ROWS != 64 && PAGE_ROWS != 128) return -1;
  if (B > INT32_MAX || T > INT32_MAX || PAGES > INT32_MAX || BLOCKS > INT32_MAX / kPage) return -1;
  const int64_t blocks = (T + 7) / 8;  // eight warps = eight rows per block
  return int(sm100::launch_overlapped(cache_append_kernel, int(blocks), 256, 0, static_cast<cudaStream_t>(stream),
                                      static_cast<const char*>(arg_new_rows), static_cast<char*>(arg_cache), static_cast<const int32_t*>(arg_block_table),
                                      static_cast<const int32_t*>(arg_cu_seqlens_q), static_cast<const int32_t*>(arg_seqused_kv), int(B), int(T), int(PAGES),
                                      int(BLOCKS), int(PAGE_ROWS), static_cast<int32_t*>(status_words), static_cast<volatile int32_t*>(flag)));
}

int launch_sparse_mla_cache_append(void* stream, void* arg_new_rows, void* arg_cache, void* arg_block_table,
                                   void* arg_cu_seqlens_q, void* arg_seqused_kv, void* npu_workspace, int64_t B,
                                   int64_t T, int64_t PAGES, int64_t BLOCKS, int64_t PAGE_ROWS) {
  if (npu_workspace == nullptr || B <= 0 || T <= 0) return -1;
  if (int status = int(cudaMemsetAsync(npu_workspace, 0, kWorkspaceBytes, static_cast<cudaStream_t>(stream)))) return status;
  return launch_sparse_mla_cache_append_flagged(stream, arg_new_rows, arg_cache, arg_block_table, arg_cu_seqlens_q, arg_seqused_kv,
                                                static_cast<char*>(npu_workspace) + kWorkspaceStatusOffset, nullptr, B, T, PAGES,
                                                BLOCKS, PAGE_ROWS);
}

}  // extern "C"
