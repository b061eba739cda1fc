// lookback_group.cuh -- the two-level look-back of the streaming kernels.
//
// About 900 tiles of 32 KB are in flight at a time, and at the full rate 100
// of them finish per microsecond.  A look-back that walks 32 predecessors per
// L2 round trip (lookback.cuh) from each tile to the nearest inclusive prefix
// needs many dependent round trips: with the look-back taken out, the scan of
// 2^30 u32 took 1.24 ms instead of 1.95 ms.  What limits the alternatives is
// how often one L2 line is polled: reading 256 predecessors per round trip
// took 2.24 ms, and a two-level scheme in which every tile polls the same
// group words 6.3 ms.  Here no line has more than about 32 pollers:
//
//   * tiles form groups of 32; a tile reads the aggregates of its group's
//     earlier tiles, and the group's last tile also publishes the group's
//     aggregate A(g);
//   * the group's first tile, whose look-back has nothing else to do, finds
//     the group's exclusive prefix P(g) from the 32 groups before it (the
//     nearest P(h) and A(h) .. A(g - 1)) and publishes it for the other first
//     tiles and, on a line of the group's own, for the group's tiles.
//
// The exclusive prefix of tile 32 g + r is P(g) op H(r - 1), H the inclusive
// scan of the group's aggregates.  Scan of 2^30 u32: 1.82 ms, of 2^28 f32 0.466
// ms (0.53 ms).  The association is fixed (a shuffle tree inside a group, a
// left fold over groups), so floats give the same bits whatever the timing;
// operands keep their order, so operators need not commute.  Tiles publish
// their aggregate alone.
#pragma once

#include "lookback.cuh"

namespace mb {

// Between two polls of one warp (1.81 -> 1.80 ms for the scan above).
constexpr unsigned kPollSleepNs = 100;

// Group prefixes as the group's own tiles read them: one 128-byte line each,
// so that a line is polled by 32 warps and not by every tile in flight.
template <class T>
struct GroupLines {
  char* base;

  static size_t bytes(uint64_t tiles) { return (tiles / 32 + 1) * 128; }
  __device__ __forceinline__ void publish(uint64_t g, const T& v) const {
    char* line = base + g * 128;
    if constexpr (sizeof(T) == 4) {
      st_relaxed_u64((uint64_t*)line, StatePack<T>::pack(kFlagIncl, v));
    } else {
      st_relaxed_any((T*)line, v);
      st_release_u32((uint32_t*)(line + 64), 1u);
    }
  }
  __device__ __forceinline__ bool peek(uint64_t g, T& v) const {
    const char* line = base + g * 128;
    if constexpr (sizeof(T) == 4) {
      return StatePack<T>::unpack(ld_relaxed_u64((const uint64_t*)line), v) != kFlagNone;
    } else {
      if (ld_acquire_u32((const uint32_t*)(line + 64)) == 0) return false;
      v = ld_relaxed_any((const T*)line);
      return true;
    }
  }
};

// Exclusive prefix of `tile` (tile >= 1), by one full warp; valid in every
// lane.  The tile's own aggregate must be published by other warps, or before
// the call (the last tile of a group reads it back with the others').  On a
// wait that expires, records the error and returns `fallback`.
template <class T, class OpT, class State>
__device__ __forceinline__ T lookback_two_level(const State& st, const GroupLines<T>& lines,
                                                uint64_t tile, const OpT& op, DevErr err,
                                                T fallback) {
  const int lane = (int)lane_id();
  SpinGuard guard(err.abort);
  const int64_t g = (int64_t)(tile >> 5);
  const int r = (int)(tile & 31);
  if (r == 0) {
    // The group's first tile finds P(g) for all of its tiles: from the nearest
    // group h before it with P(h), and A(h) .. A(g - 1).
    const int64_t q = g - 1 - lane;
    T va = fallback, vp = fallback;
    while (true) {
      bool ha = false, hp = false;
      if (q >= 0) {
        ha = st.gagg.peek((uint64_t)q, va);
        hp = q == 0 || st.gincl.peek((uint64_t)q, vp);
      }
      const uint32_t mp = __ballot_sync(kFull, hp);
      const int hl = mp ? __ffs(mp) - 1 : 31;
      const uint32_t need = kFull >> (31 - hl);  // A of lanes 0 .. hl
      const uint32_t have = __ballot_sync(kFull, ha);
      if (mp && (have & need) == need) {
        T acc = shfl_idx(va, hl);
        if (g - 1 - hl > 0) acc = op(shfl_idx(vp, hl), acc);
        for (int k = hl - 1; k >= 0; --k) acc = op(acc, shfl_idx(va, k));
        if (lane == 0) {
          lines.publish((uint64_t)g, acc);
          st.gincl.publish((uint64_t)g, acc);
        }
        return acc;
      }
      __nanosleep(kPollSleepNs);
      if (__any_sync(kFull, guard.expired())) {
        raise_device_error(err, MB_DEV_ERR_LOOKBACK);
        return fallback;
      }
    }
  }
  // The tiles of the group before this one (and, for the last, itself).
  const int last = r == 31 ? 31 : r - 1;
  T v = fallback;
  while (true) {
    const uint32_t f = lane <= last ? st.peek((uint64_t)(g << 5) + lane, v) : kFlagAgg;
    if (!__any_sync(kFull, f == kFlagNone)) break;
    __nanosleep(kPollSleepNs);
    if (__any_sync(kFull, guard.expired())) {
      raise_device_error(err, MB_DEV_ERR_LOOKBACK);
      return fallback;
    }
  }
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const T y = shfl_up(v, d);
    if (lane >= d) v = op(y, v);
  }
  const T hs = shfl_idx(v, r - 1);
  if (r == 31) {
    const T a = shfl_idx(v, 31);
    if (lane == 0) st.gagg.publish((uint64_t)g, a);
  }
  if (g == 0) return hs;
  // Every lane polls the same word, but two lanes' loads may still see
  // different values for a while: the exit is voted.
  T acc = fallback;
  while (true) {
    const bool seen = lines.peek((uint64_t)g, acc);
    if (__all_sync(kFull, seen)) break;
    __nanosleep(kPollSleepNs);
    if (__any_sync(kFull, guard.expired())) {
      raise_device_error(err, MB_DEV_ERR_LOOKBACK);
      return fallback;
    }
  }
  return op(acc, hs);
}

}  // namespace mb
