// The softmax warps' control flow on the CPU: `softmax_role`, taken from the kernel's source (role.inc), with one thread
// for a warp, data that nobody looks at, and waits that give up where a run says so. The named barrier has no limit: whoever
// would be left behind at it is what this looks for. stdin: runs as lines
//   mode tokens chunks... rescale-mask warp wait     (mode 0: this wait of this warp gives up; 1: and every later one of anybody;
// 2: as 0, and later ones by the toss of a coin). Prints "ok", or "left behind" for the first run in which not all four leave.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <iostream>
#include <mutex>
#include <random>
#include <thread>
#include <vector>

#define __device__
#define __forceinline__ inline
using std::min;
struct uint2 { uint32_t x, y; };
struct float2 { float x, y; };
struct uint4 { uint32_t x, y, z, w; };
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }
inline float2 make_float2(float x, float y) { return {x, y}; }
struct Index { unsigned x; };
thread_local Index threadIdx;
using __nv_bfloat16 = uint16_t;

constexpr int kSoftmaxWarps = 4, kHeads = 64, kFeatures = 512, kMaxChunks = 10, kStages = 3, kPTileBytes = kHeads * 128;
constexpr int kTmemS = 0, kTmemO = 0, kTmemPlaces = 0, kHalfLanes = 0;
constexpr int kSmemP = 0, kSmemStore = 2 * kPTileBytes, kSmemAlpha = kSmemStore + 4 * 2048, kSmemInverse = kSmemAlpha + 256, kSmemEnd = kSmemInverse + 512;
struct Params { const float* sinks; void* out; float scale_log2; int tokens; };
struct TokenInfo { int chunks; uint2 live[kMaxChunks]; };

struct Run { int mode; std::vector<int> chunks; uint32_t rescale; int warp, wait; } run;
std::vector<TokenInfo> infos;
int abort_word;
alignas(16) unsigned char shared_bytes[kSmemEnd];

struct Barrier {  // like the hardware's: arrivals of any warps, four to a generation
  int arrived = 0, generation = 0;
  uint32_t count = 0, result = 0;
} barriers[4];
std::mutex mutex;
std::condition_variable changed;
bool stuck;
struct LeftBehind {};
template <typename Flag>
inline uint32_t named_barrier_count(int id, int threads, Flag flag) {  // flag: of a lane
  std::unique_lock<std::mutex> lock(mutex);
  Barrier& b = barriers[id];
  for (int lane = 0; lane < 32; ++lane) b.count += flag(lane);
  const int generation = b.generation;
  if (++b.arrived == threads / 32) {
    b.result = b.count;
    b.arrived = 0;
    b.count = 0;
    ++b.generation;
    changed.notify_all();
    return b.result;
  }
  if (!changed.wait_for(lock, std::chrono::seconds(3), [&] { return b.generation != generation || stuck; }) || stuck) {
    stuck = true;
    changed.notify_all();
    throw LeftBehind();
  }
  return b.result;
}

thread_local int waits;
thread_local std::minstd_rand coin;
thread_local int chunk_of_warp;
inline bool warp_wait(uint32_t, uint32_t, volatile int*) {
  const bool mine = int(threadIdx.x >> 5) == run.warp && waits++ == run.wait;
  std::lock_guard<std::mutex> lock(mutex);
  if (mine) abort_word = 1;
  return !mine && !(abort_word && (run.mode == 1 || (run.mode == 2 && coin() % 3 == 0)));
}

inline void mbar_arrive(uint32_t) {}
inline void store_places(uint32_t, int) {}
inline void tmem_wait_st() {}
inline void tmem_wait_ld() {}
inline void tc_fence_before_sync() {}
inline void tc_fence_after_sync() {}
inline void fence_proxy_async() {}
inline void __syncwarp() {}
inline bool __any_sync(unsigned, bool) { return true; }
inline float __shfl_xor_sync(unsigned, float value, int) { return value; }
inline float __ldg(const float* at) { return *at; }
inline void __stcs(uint4*, uint4) {}
inline float __uint_as_float(uint32_t) { return 1.f; }
inline uint32_t __float_as_uint(float) { return 0; }
inline void tmem_ld16(uint32_t, uint32_t (&)[16]) {}
inline void tmem_st16(uint32_t, uint32_t (&)[16]) {}
template <int kColumns> inline void tmem_ld16_halves(uint32_t, uint32_t (&)[16]) {}
template <int kFormat> inline uint32_t pack_pair(float, float) { return 0; }
inline float max3(float a, float, float) { return a; }
inline float2 add_pair(float2 a, float2) { return a; }
inline float2 fma_pair(float2 a, float2, float2) { return a; }
inline uint32_t p_offset(int head, int unit) { return head * 128 + unit * 16; }
constexpr float kReferenceRoom = 15.f, kReferenceAligned = 64.f;
// One warp's heads move their reference in a chunk, by its bit and in turn.
inline float move_reference(float&, float, bool) {
  const int chunk = chunk_of_warp++;
  return (run.rescale >> (chunk & 31) & 1) && chunk % kSoftmaxWarps == int(threadIdx.x >> 5) ? 0.5f : 1.f;
}

struct Shared {
  unsigned char* ptr = shared_bytes;
  uint32_t bar(int which) const { return which; }
  TokenInfo* info(int buffer) const;
  volatile int* abort_flag() const { return &abort_word; }
};
thread_local int tokens_walked;  // next() has run this often
inline TokenInfo* Shared::info(int) const { return &infos[min(std::max(tokens_walked - 1, 0), int(infos.size()) - 1)]; }
struct TokenWalk {
  int at = 0, tokens;
  explicit TokenWalk(const Params& p) : tokens(p.tokens) {}
  int next() { ++tokens_walked; return at < tokens ? at++ : -1; }
};

#include "role.inc"

int main() {
  std::vector<float> sinks(kHeads, 0.f);
  int tokens;
  for (int number = 0; std::cin >> run.mode >> tokens; ++number) {
    run.chunks.resize(tokens);
    for (int& chunks : run.chunks) std::cin >> chunks;
    std::cin >> run.rescale >> run.warp >> run.wait;
    infos.assign(std::max(tokens, 1), TokenInfo{});
    for (int t = 0; t < tokens; ++t) {
      infos[t].chunks = run.chunks[t];
      for (auto& live : infos[t].live) live = {0xffffffffu, 0xffffffffu};
    }
    abort_word = 0;
    for (auto& b : barriers) b = Barrier();
    std::vector<uint16_t> out(size_t(std::max(tokens, 1)) * kHeads * kFeatures + 8);
    void* aligned = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(out.data()) + 15) & ~uintptr_t(15));
    const Params p = {sinks.data(), aligned, 1.f, tokens};
    std::vector<std::thread> warps;
    for (int w = 0; w < kSoftmaxWarps; ++w)
      warps.emplace_back([&, w] {
        threadIdx.x = w * 32;
        waits = chunk_of_warp = tokens_walked = 0;
        coin.seed(number * 4 + w + 1);
        try { softmax_role<0>(p, Shared(), 0); } catch (LeftBehind&) {}
      });
    for (auto& warp : warps) warp.join();
    for (const auto& b : barriers) stuck |= b.arrived != 0;  // somebody arrived whom nobody waits for
    if (stuck) {
      std::printf("left behind: mode %d warp %d wait %d rescale %x chunks", run.mode, run.warp, run.wait, run.rescale);
      for (int chunks : run.chunks) std::printf(" %d", chunks);
      std::printf("\n");
      return 1;
    }
  }
  std::printf("ok\n");
}
