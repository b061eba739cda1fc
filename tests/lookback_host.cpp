// The two-level look-back (massively_b200/csrc/lookback_group.cuh) on the host: one thread per
// lane, and every warp vote or shuffle a meeting of all 32 lanes.  A lane that does not come to a
// meeting leaves the others waiting there, as it would on the device; here they give up after a
// second and the run fails.  Lane l sees a published word only on its (l % 3 + 1)-th read of it:
// the memory model lets the lanes of a warp disagree for a while.
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#define __device__
#define __forceinline__ inline

namespace mb {

constexpr uint32_t kFlagNone = 0, kFlagAgg = 1, kFlagIncl = 2;
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr uint32_t MB_DEV_ERR_LOOKBACK = 1;

struct Stuck {};

struct Warp {
  std::mutex m;
  std::condition_variable cv;
  uint64_t in[32], out[32];
  int arrived = 0;
  uint64_t round = 0;
  bool stuck = false;

  // Every lane brings a word and gets all 32.
  void meet(int lane, uint64_t v, uint64_t (&all)[32]) {
    std::unique_lock<std::mutex> lock(m);
    in[lane] = v;
    const uint64_t r = round;
    if (++arrived == 32) {
      memcpy(out, in, sizeof(in));
      arrived = 0;
      ++round;
      cv.notify_all();
    } else if (!cv.wait_for(lock, std::chrono::seconds(1),
                            [&] { return stuck || round != r; }) || round == r) {
      stuck = true;
      cv.notify_all();
      throw Stuck{};
    }
    memcpy(all, out, sizeof(out));
  }
};

static Warp* g_warp;
static thread_local int t_lane;
static thread_local std::map<const void*, int> t_reads;  // reads of each word by this lane

inline uint32_t lane_id() { return (uint32_t)t_lane; }
inline uint32_t ballot(bool b) {
  uint64_t all[32];
  g_warp->meet(t_lane, b, all);
  uint32_t m = 0;
  for (int i = 0; i < 32; ++i) m |= (uint32_t)(all[i] != 0) << i;
  return m;
}
#define __ballot_sync(mask, p) mb::ballot(p)
#define __any_sync(mask, p) (mb::ballot(p) != 0)
#define __all_sync(mask, p) (mb::ballot(p) == mb::kFull)
#define __ffs(x) __builtin_ffs((int)(x))
#define __syncwarp() (void)mb::ballot(true)
inline void __nanosleep(unsigned) { std::this_thread::yield(); }

template <class T>
T shfl_idx(T v, int src) {
  uint64_t all[32], w = 0;
  memcpy(&w, &v, sizeof(T));
  g_warp->meet(t_lane, w, all);
  memcpy(&v, &all[src & 31], sizeof(T));
  return v;
}
template <class T>
T shfl_up(T v, int d) {
  uint64_t all[32], w = 0;
  memcpy(&w, &v, sizeof(T));
  g_warp->meet(t_lane, w, all);
  memcpy(&v, &all[t_lane >= d ? t_lane - d : t_lane], sizeof(T));
  return v;
}

static std::mutex g_mem;
inline bool seen(const void* p) { return ++t_reads[p] > t_lane % 3; }
inline uint64_t ld_relaxed_u64(const uint64_t* p) {
  std::lock_guard<std::mutex> lock(g_mem);
  return seen(p) ? *p : 0;
}
inline uint32_t ld_acquire_u32(const uint32_t* p) {
  std::lock_guard<std::mutex> lock(g_mem);
  return seen(p) ? *p : 0;
}
template <class T>
T ld_relaxed_any(const T* p) {
  std::lock_guard<std::mutex> lock(g_mem);
  return *p;
}
inline void st_relaxed_u64(uint64_t* p, uint64_t v) {
  std::lock_guard<std::mutex> lock(g_mem);
  *p = v;
}
inline void st_release_u32(uint32_t* p, uint32_t v) {
  std::lock_guard<std::mutex> lock(g_mem);
  *p = v;
}
template <class T>
void st_relaxed_any(T* p, const T& v) {
  std::lock_guard<std::mutex> lock(g_mem);
  *p = v;
}

template <class T>
struct StatePack {
  static uint64_t pack(uint32_t flag, const T& v) { return (uint64_t)flag << 32 | (uint32_t)v; }
  static uint32_t unpack(uint64_t w, T& v) {
    v = (T)(uint32_t)w;
    return (uint32_t)(w >> 32);
  }
};

struct DevErr {
  uint32_t* status;
  uint32_t* abort;
};
static bool g_raised = false;
inline void raise_device_error(DevErr, uint32_t) { g_raised = true; }
struct SpinGuard {
  explicit SpinGuard(const uint32_t*) {}
  bool expired() { return false; }
};

}  // namespace mb

#include "lookback_group.cuh"

namespace mb {

// Published state of a chain of tiles, each lane late by its own count.
template <class T>
struct Slot {
  std::vector<uint64_t> word;  // 0: not published, else value + 1
  explicit Slot(size_t n) : word(n, 0) {}
  bool peek(uint64_t i, T& v) const {
    std::lock_guard<std::mutex> lock(g_mem);
    if (!seen(&word[i]) || word[i] == 0) return false;
    v = (T)(word[i] - 1);
    return true;
  }
  void publish(uint64_t i, const T& v) const {
    std::lock_guard<std::mutex> lock(g_mem);
    const_cast<uint64_t&>(word[i]) = (uint64_t)v + 1;
  }
};
template <class T>
struct Chain {
  Slot<T> tile, gagg, gincl;
  uint32_t peek(uint64_t i, T& v) const { return tile.peek(i, v) ? kFlagAgg : kFlagNone; }
};

// Runs the look-back of tiles 1 .. tiles - 1 one after another; tile i's aggregate is i + 1.
template <class T>
int run(uint64_t tiles) {
  const auto add = [](T a, T b) { return (T)(a + b); };
  Chain<T> st{Slot<T>(tiles), Slot<T>(tiles / 32 + 1), Slot<T>(tiles / 32 + 1)};
  std::vector<char> mem(GroupLines<T>::bytes(tiles) + 128, 0);
  char* base = mem.data() + (128 - (uintptr_t)mem.data() % 128);
  const GroupLines<T> lines{base};
  T want = 0;
  for (uint64_t t = 0; t < tiles; ++t) {
    st.tile.publish(t, (T)(t + 1));
    if (t > 0) {
      Warp warp;
      g_warp = &warp;
      T got[32] = {};
      std::vector<std::thread> lanes;
      for (int l = 0; l < 32; ++l)
        lanes.emplace_back([&, l] {
          t_lane = l;
          try {
            got[l] = lookback_two_level<T>(st, lines, t, add, DevErr{nullptr, nullptr}, (T)0);
          } catch (const Stuck&) {
          }
        });
      for (auto& x : lanes) x.join();
      if (warp.stuck || warp.arrived != 0) {
        printf("tile %llu: some lanes wait for others that have left\n", (unsigned long long)t);
        return 1;
      }
      for (int l = 0; l < 32; ++l)
        if (got[l] != want || g_raised) {
          printf("tile %llu lane %d: %llu, not %llu\n", (unsigned long long)t, l,
                 (unsigned long long)got[l], (unsigned long long)want);
          return 1;
        }
    }
    want = add(want, (T)(t + 1));
  }
  return 0;
}

}  // namespace mb

int main() {
  // two groups and the first tiles of a third: every branch, with the flag beside the value
  // (4 bytes) and apart from it (8 bytes)
  if (mb::run<uint32_t>(70) || mb::run<uint64_t>(70)) return 1;
  puts("ok");
  return 0;
}
