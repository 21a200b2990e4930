// One block of the index selection on the CPU: `topk_select_kernel` and the rule that chooses its form, taken from the
// kernel's source (select.inc), with a fiber for every thread, threads of a warp that meet at its votes, shuffles and reductions, and
// shared memory of just the block's size behind which nothing may change. stdin, for each call: rows of the launch, width of the
// buffer, rows that are looked at, and for each of those its length and the bits of its scores. stdout: 512 indices for each, or a
// line that says what went wrong.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <type_traits>
#include <vector>
#include <ucontext.h>

#define __device__
#define __global__
#define __shared__
#define __noinline__ __attribute__((noinline))
#define __forceinline__ inline
#define __align__(n) __attribute__((aligned(n)))
#define __launch_bounds__(...)

struct uint2 { uint32_t x, y; };
struct uint4 { uint32_t x, y, z, w; };
inline uint2 make_uint2(uint32_t x, uint32_t y) { return {x, y}; }
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }
struct Index { unsigned x; } threadIdx, blockIdx;

// ---- the block's threads ------------------------------------------------------------------------
struct Meeting { uint32_t value[2][32]; int arrived; unsigned generation; } warps[32];
int block_threads, block_arrived;
unsigned block_generation;
ucontext_t scheduler, fibers[1024];
std::vector<char> stacks(1024 * size_t(32768));
bool finished[1024];
std::function<void()> body;

inline void yield() {
  const unsigned thread = threadIdx.x;
  swapcontext(&fibers[thread], &scheduler);
  threadIdx.x = thread;
}
void enter() {
  body();
  finished[threadIdx.x] = true;
  if (block_arrived == --block_threads && block_arrived > 0) { block_arrived = 0; ++block_generation; }  // barriers are of those who have not left
  swapcontext(&fibers[threadIdx.x], &scheduler);
}
inline void __syncthreads() {
  const unsigned generation = block_generation;
  if (++block_arrived == block_threads) { block_arrived = 0; ++block_generation; }
  while (block_generation == generation) yield();
}
// The values of all lanes of the warp.
inline const uint32_t* meet(uint32_t mine) {
  Meeting& warp = warps[threadIdx.x >> 5];
  const unsigned generation = warp.generation;
  warp.value[generation & 1][threadIdx.x & 31] = mine;
  if (++warp.arrived == 32) { warp.arrived = 0; ++warp.generation; }
  while (warp.generation == generation) yield();
  return warp.value[generation & 1];
}
inline bool run_block(int threads) {  // false: somebody waits for ever
  block_threads = threads;
  block_arrived = 0;
  memset(warps, 0, sizeof(warps));
  for (int t = 0; t < threads; ++t) {
    finished[t] = false;
    getcontext(&fibers[t]);
    fibers[t].uc_stack.ss_sp = &stacks[t * size_t(32768)];
    fibers[t].uc_stack.ss_size = 32768;
    fibers[t].uc_link = nullptr;
    makecontext(&fibers[t], enter, 0);
  }
  for (int round = 0; round < 1000000; ++round) {
    bool left = false;
    for (int t = 0; t < threads; ++t)
      if (!finished[t]) { threadIdx.x = t; swapcontext(&scheduler, &fibers[t]); left = true; }
    if (!left) return true;
  }
  return false;
}

// ---- what the kernel calls ------------------------------------------------------------------------
template <typename A, typename B> inline std::common_type_t<A, B> min(A a, B b) { using T = std::common_type_t<A, B>; return T(a) < T(b) ? T(a) : T(b); }
template <typename A, typename B> inline std::common_type_t<A, B> max(A a, B b) { using T = std::common_type_t<A, B>; return T(a) < T(b) ? T(b) : T(a); }
inline int __clz(int v) { return v == 0 ? 32 : __builtin_clz(unsigned(v)); }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(unsigned v) { return __builtin_ffs(int(v)); }
inline float __uint_as_float(uint32_t v) { float f; memcpy(&f, &v, 4); return f; }
inline uint32_t __float_as_uint(float f) { uint32_t v; memcpy(&v, &f, 4); return f != f ? 0x7fffffff : v; }  // the GPU's arithmetic has one NaN
inline uint32_t __funnelshift_l(uint32_t low, uint32_t high, int by) { return high << by | low >> (32 - by); }
template <typename T> inline T __ldg(const T* p) { return *p; }
template <typename T> inline T __ldcs(const T* p) { return *p; }
inline uint32_t __ballot_sync(uint32_t, bool v) { const uint32_t* all = meet(v); uint32_t b = 0; for (int l = 0; l < 32; ++l) b |= all[l] << l; return b; }
inline bool __any_sync(uint32_t m, bool v) { return __ballot_sync(m, v) != 0; }
template <typename T> inline T __shfl_sync(uint32_t, T v, int lane) { return T(meet(uint32_t(v))[lane & 31]); }
template <typename T> inline T __shfl_up_sync(uint32_t, T v, int by) { const int lane = threadIdx.x & 31; return T(meet(uint32_t(v))[lane < by ? lane : lane - by]); }
template <typename T> inline T __shfl_xor_sync(uint32_t, T v, int by) { const int lane = threadIdx.x & 31; return T(meet(uint32_t(v))[lane ^ by]); }
inline uint32_t __reduce_min_sync(uint32_t, uint32_t v) { const uint32_t* all = meet(v); return *std::min_element(all, all + 32); }
inline uint32_t __reduce_max_sync(uint32_t, uint32_t v) { const uint32_t* all = meet(v); return *std::max_element(all, all + 32); }
inline uint32_t __reduce_add_sync(uint32_t, uint32_t v) { const uint32_t* all = meet(v); uint32_t s = 0; for (int l = 0; l < 32; ++l) s += all[l]; return s; }
inline uint32_t __match_any_sync(uint32_t, uint32_t v) { const uint32_t* all = meet(v); uint32_t b = 0; for (int l = 0; l < 32; ++l) b |= uint32_t(all[l] == v) << l; return b; }
inline unsigned atomicAdd(unsigned* at, unsigned v) { const unsigned old = *at; *at += v; return old; }
inline unsigned atomicMin(unsigned* at, unsigned v) { const unsigned old = *at; *at = min(old, v); return old; }
inline unsigned atomicMax(unsigned* at, unsigned v) { const unsigned old = *at; *at = max(old, v); return old; }

typedef void* cudaStream_t;
typedef int cudaError_t;
constexpr int cudaSuccess = 0, cudaDevAttrMultiProcessorCount = 0;
inline int cudaGetDevice(int* device) { return *device = 0; }
inline int cudaDeviceGetAttribute(int* value, int, int) { *value = 148; return 0; }

namespace sparse_mla {
constexpr int kTopK = 512, kPage = 128;
namespace {
constexpr size_t kBehind = 1 << 16;  // watched bytes behind the block's shared memory
alignas(16) unsigned char select_smem[(227 << 10) + kBehind];
}  // namespace
namespace sm100 {
inline void wait_for_predecessor() {}
inline void let_successor_start() {}
inline uint32_t smem_u32(const void* at) { return uint32_t(static_cast<const unsigned char*>(at) - select_smem); }
}  // namespace sm100
namespace {
inline uint32_t& shared_word(uint32_t address) { return *reinterpret_cast<uint32_t*>(select_smem + address); }
inline void shared_add_if(bool wanted, uint32_t address) { if (wanted) ++shared_word(address); }
inline void shared_or_if(bool wanted, uint32_t address, unsigned bits) { if (wanted) shared_word(address) |= bits; }
inline void copy_word(uint32_t to, const float* from) { memcpy(&shared_word(to), from, 4); }
inline void wait_for_words() {}
inline void prefetch_l2(const void*, unsigned) {}

struct SelectParams;
template <int kThreads, int kCapacity, int kBlocks, int kMostQuads, int kInFlight = 4, int kWindow = (kThreads >= 256 ? 65536 : 256 * kThreads), int kShortRow = 0,
          bool kCopyScores = (kThreads >= 512), int kHalfRow = 0>
int launch_select(const SelectParams& p, cudaStream_t);

#include "select.inc"

const char* fault;
int looked_at;
template <int kThreads, int kCapacity, int kBlocks, int kMostQuads, int kInFlight, int kWindow, int kShortRow, bool kCopyScores, int kHalfRow>
int launch_select(const SelectParams& p, cudaStream_t) {
  constexpr size_t bytes = sizeof(SelectShared<kThreads, kCapacity, kWindow>);
  static_assert(bytes <= 227 << 10, "a block's shared memory");
  for (int token = 0; token < looked_at && fault == nullptr; ++token) {
    memset(select_smem, 0xa5, sizeof(select_smem));
    blockIdx.x = unsigned(token);
    body = [&] { topk_select_kernel<kThreads, kCapacity, kBlocks, kMostQuads, kInFlight, kWindow, kShortRow, kCopyScores, kHalfRow>(p); };
    if (!run_block(kThreads)) fault = "a thread waits for ever";
    for (size_t i = bytes; i < sizeof(select_smem); ++i)
      if (select_smem[i] != 0xa5) { fault = "written behind the block's shared memory"; break; }
  }
  return 0;
}
}  // namespace
}  // namespace sparse_mla

int main() {
  using namespace sparse_mla;
  int32_t head[3];
  while (fread(head, 4, 3, stdin) == 3) {
    const int64_t rows = head[0], span = head[1];
    looked_at = head[2];
    std::vector<int32_t> cu(rows + 1), seq(rows, 0), residual(rows, 0), out(size_t(looked_at) * kTopK, -77);
    for (int64_t i = 0; i <= rows; ++i) cu[i] = int32_t(i);
    std::vector<uint4> scores(size_t(looked_at) * span / 4);
    if (fread(seq.data(), 4, looked_at, stdin) != size_t(looked_at) || fread(scores.data(), 16, scores.size(), stdin) != scores.size()) return 1;
    const int status = launch_sparse_mla_topk_indices(nullptr, scores.data(), cu.data(), seq.data(), residual.data(), out.data(), rows, rows, span, 128);
    if (status != 0 || fault != nullptr) { fprintf(stderr, "%s\n", fault != nullptr ? fault : "refused"); return 1; }
    fwrite(out.data(), 4, out.size(), stdout);
  }
}
