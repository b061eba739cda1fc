// merge.cu -- merge-path merge / merge_by_key and the multiset set
// operations.
//
// Merge (massively/src/core/merge.rs:24-1230: a merge-path control kernel of
// 64 threads x 4 items writing a permutation, then a separate apply pass for
// the payload) becomes two kernels: the merge-path splits of all tile
// boundaries, then the tiles.  Plain keys alone take the warp-window kernel.
// With payloads, lazy inputs, and floats under LESS / GREATER, each thread
// finds its own split in shared memory and merges kItems outputs serially (an
// odd count, so the threads' strided accesses fall in distinct banks).  Ties
// take the left element first (vector.rs:493-513 of massively's oracle: the
// right element is taken only when strictly less).
//
// Set operations (massively/src/core/set.rs:14-401) keep massively's
// occurrence-rank rule: the k-th copy of a value in one input is kept by
// intersection when the other input holds more than k copies, by difference
// when it holds at most k; union is the merge of the left input with the
// right input's extra copies.  Intersection and difference of plain columns
// look each left item's partner up on the right (warp-window kernel); union
// and the other inputs take one pass over the merged runs.  Kept items are
// compacted behind a look-back and the result count stays on the device.

#include <algorithm>

#include "bulk.cuh"
#include "common.cuh"
#include "dispatch.cuh"
#include "lookback_group.cuh"

namespace mb {

namespace {

constexpr int kThreads = 256;
constexpr int kItems = 9;  // odd: conflict-free strided shared-memory access
constexpr int kTile = kThreads * kItems;
constexpr int kMaxPay = 12;

template <class T>
__device__ __forceinline__ bool cmp_less(int less, T a, T b) {
  switch (less) {
    case MB_GREATER: return b < a;
    case MB_TOTAL_LESS: return radix_enc<T>(a) < radix_enc<T>(b);
    default: return a < b;
  }
}

// The comparison with the predicate fixed at compile time (hot kernels).
template <class T, int LESS>
__device__ __forceinline__ bool cmp_ct(T a, T b) {
  if constexpr (LESS == MB_GREATER) return b < a;
  else if constexpr (LESS == MB_TOTAL_LESS) return radix_enc<T>(a) < radix_enc<T>(b);
  else return a < b;
}

// Element i of an input: a direct load for plain columns of type T, the
// lazy-view loader otherwise.
template <class T, bool PLAIN>
__device__ __forceinline__ T merge_load(const Src& s, uint64_t i) {
  if constexpr (PLAIN) return ((const T*)s.data)[i];
  else return src_load<T>(s, i);
}

// Number of left elements among the first d outputs of the stable merge.
template <class T, int LESS, bool PLAIN>
__device__ uint64_t merge_path(const Src& L, const Src& R, uint64_t nl, uint64_t nr, uint64_t d) {
  uint64_t lo = d > nr ? d - nr : 0;
  uint64_t hi = d < nl ? d : nl;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    const T l = merge_load<T, PLAIN>(L, mid);
    const T r = merge_load<T, PLAIN>(R, d - 1 - mid);
    if (!cmp_ct<T, LESS>(r, l)) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

struct Payload {
  int ncols;
  Src left[kMaxPay];
  Src right[kMaxPay];
  void* out[kMaxPay];
  int esize[kMaxPay];
};

__device__ __forceinline__ void st_raw_pay(void* p, uint64_t i, int esize, uint64_t bits) {
  switch (esize) {
    case 1: ((uint8_t*)p)[i] = (uint8_t)bits; break;
    case 2: ((uint16_t*)p)[i] = (uint16_t)bits; break;
    case 4: ((uint32_t*)p)[i] = (uint32_t)bits; break;
    default: ((uint64_t*)p)[i] = bits; break;
  }
}

constexpr uint32_t kFromRight = 0x80000000u;

// The merge-path split of every tile boundary, one thread per boundary (all
// binary searches in flight together rather than one dependent search at the
// start of each tile).
template <class T, int LESS, bool PLAIN>
__global__ void __launch_bounds__(kThreads)
    merge_splits_kernel(Src L, Src R, uint64_t tiles, uint64_t* __restrict__ splits) {
  const uint64_t nl = src_len(L), nr = src_len(R), n = nl + nr;
  for (uint64_t b = blockIdx.x * (uint64_t)kThreads + threadIdx.x; b <= tiles;
       b += (uint64_t)gridDim.x * kThreads)
    splits[b] = merge_path<T, LESS, PLAIN>(L, R, nl, nr, min(b * (uint64_t)kTile, n));
}

template <class T, int LESS, bool PLAIN>
__global__ void __launch_bounds__(kThreads)
    merge_kernel(Src L, Src R, void* out, int out_dtype, Payload pay,
                 uint32_t* count_dev, const uint64_t* __restrict__ splits) {
  __shared__ T s_keys[kTile];
  __shared__ T s_out[kTile];
  __shared__ uint32_t s_src[kTile];
  __shared__ uint64_t s_split[2];
  const uint64_t nl = src_len(L), nr = src_len(R), n = nl + nr;
  if (blockIdx.x == 0 && threadIdx.x == 0 && count_dev) *count_dev = (uint32_t)n;
  const uint64_t d0 = (uint64_t)blockIdx.x * kTile;
  if (d0 >= n) return;
  const uint64_t d1 = min(d0 + (uint64_t)kTile, n);
  if (threadIdx.x < 2) s_split[threadIdx.x] = splits[blockIdx.x + threadIdx.x];
  __syncthreads();
  const uint64_t i0 = s_split[0], i1 = s_split[1];
  const uint64_t j0 = d0 - i0, j1 = d1 - i1;
  const int la = (int)(i1 - i0), lb = (int)(j1 - j0);
  for (int t = threadIdx.x; t < la; t += kThreads) s_keys[t] = merge_load<T, PLAIN>(L, i0 + t);
  for (int t = threadIdx.x; t < lb; t += kThreads) s_keys[la + t] = merge_load<T, PLAIN>(R, j0 + t);
  __syncthreads();
  const int total = la + lb;
  const int dt = min((int)threadIdx.x * kItems, total);
  // Per-thread split inside the tile.
  int lo = dt > lb ? dt - lb : 0, hi = dt < la ? dt : la;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (!cmp_ct<T, LESS>(s_keys[la + dt - 1 - mid], s_keys[mid])) lo = mid + 1;
    else hi = mid;
  }
  // Serial merge with the two heads in registers: one shared-memory read per
  // output.
  int a = lo, b = dt - lo;
  T ka = a < la ? s_keys[a] : T(0);
  T kb = b < lb ? s_keys[la + b] : T(0);
  const bool pay_on = pay.ncols != 0;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    if (dt + k >= total) break;
    const bool take_left = b >= lb || (a < la && !cmp_ct<T, LESS>(kb, ka));
    s_out[dt + k] = take_left ? ka : kb;
    if (pay_on) s_src[dt + k] = take_left ? (uint32_t)a : (kFromRight | (uint32_t)b);
    if (take_left) {
      ++a;
      ka = a < la ? s_keys[a] : ka;
    } else {
      ++b;
      kb = b < lb ? s_keys[la + b] : kb;
    }
  }
  __syncthreads();
  const bool same_type = out_dtype == DTypeOf<T>::value;
  for (int t = threadIdx.x; t < total; t += kThreads) {
    if (out) {
      if (same_type) __stcs((T*)out + d0 + t, s_out[t]);
      else st_cast<T>(out_dtype, out, d0 + t, s_out[t]);
    }
    if (pay.ncols) {
      const uint32_t s = s_src[t];
      const bool right = s & kFromRight;
      const uint64_t idx = right ? j0 + (s & ~kFromRight) : i0 + s;
      for (int c = 0; c < pay.ncols; ++c) {
        const uint64_t bits = src_load_bits(right ? pay.right[c] : pay.left[c], idx);
        st_raw_pay(pay.out[c], d0 + t, pay.esize[c], bits);
      }
    }
  }
}

// ------------------------------------------------------ set operations --
//
// One pass over the stable merge M of the two inputs (ties: left first).
// Equivalent items (neither less than the other) form one run of M: its
// left copies, then its right copies.  With rs / re the run's first and
// one-past-last merged positions and lr the position of its first right
// copy (cl = lr - rs left copies, cr = re - lr right copies), massively's
// multiset rule (core/set.rs:18-46; the two-pointer walk of its oracle,
// verification/oracle/src/vector.rs:595-664) keeps, for the item at p:
//   intersection: a left copy with p - rs <  cr;
//   difference:   a left copy with p - rs >= cr;
//   union:        every left copy, and a right copy with p - lr >= cl.
// A tile of M (its merge-path split) merges its two slices in shared
// memory, finds every position's run with block-wide scans of the run heads
// and of the left / right positions, and takes the runs that cross its
// edges from the run of each boundary's item (four binary searches per
// boundary, for all boundaries at once before the tile kernel).  It counts
// the kept items, gets the count of all earlier tiles by a decoupled
// look-back, and writes the kept items in order; the total stays on the
// device.  The inputs must be sorted under a strict weak order (no NaN
// under LESS / GREATER; TOTAL_LESS orders every float).

struct SetRun {
  uint32_t lbl, ubl, lbr, ubr;  // the run's bounds in the left and in the right input
};

template <class T, int LESS>
__device__ __forceinline__ bool equiv_ct(T a, T b) {
  return !cmp_ct<T, LESS>(a, b) && !cmp_ct<T, LESS>(b, a);
}

// First index in [0, n) whose item is not less than v (UPPER: that v is
// less than).
template <class T, int LESS, bool PLAIN, bool UPPER>
__device__ uint64_t bound_of(const Src& s, uint64_t n, T v) {
  uint64_t lo = 0, hi = n;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    const T x = merge_load<T, PLAIN>(s, mid);
    const bool before = UPPER ? !cmp_ct<T, LESS>(v, x) : cmp_ct<T, LESS>(x, v);
    if (before) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Per tile boundary b: the merge-path split, the item at merged position
// b * kTile and the bounds of its run in both inputs.
template <class T, int LESS, bool PLAIN>
__global__ void __launch_bounds__(kThreads)
    set_bounds_kernel(Src L, Src R, uint64_t tiles, uint64_t* __restrict__ splits,
                      SetRun* __restrict__ runs, T* __restrict__ vals) {
  const uint64_t nl = src_len(L), nr = src_len(R), n = nl + nr;
  for (uint64_t b = blockIdx.x * (uint64_t)kThreads + threadIdx.x; b <= tiles;
       b += (uint64_t)gridDim.x * kThreads) {
    const uint64_t d = min(b * (uint64_t)kTile, n);
    const uint64_t i = merge_path<T, LESS, PLAIN>(L, R, nl, nr, d);
    splits[b] = i;
    if (d >= n) continue;
    const uint64_t j = d - i;
    const bool from_left =
        i < nl && (j >= nr || !cmp_ct<T, LESS>(merge_load<T, PLAIN>(R, j),
                                               merge_load<T, PLAIN>(L, i)));
    const T v = from_left ? merge_load<T, PLAIN>(L, i) : merge_load<T, PLAIN>(R, j);
    vals[b] = v;
    SetRun r;
    r.lbl = (uint32_t)bound_of<T, LESS, PLAIN, false>(L, nl, v);
    r.ubl = (uint32_t)bound_of<T, LESS, PLAIN, true>(L, nl, v);
    r.lbr = (uint32_t)bound_of<T, LESS, PLAIN, false>(R, nr, v);
    r.ubr = (uint32_t)bound_of<T, LESS, PLAIN, true>(R, nr, v);
    runs[b] = r;
  }
}

constexpr int kNone = 0x7FFFFFFF;

// Exclusive block-wide scans over the threads' chunk summaries: a running
// maximum of (a, b) from the left, and a running minimum of (c, d) from the
// right (each thread gets the extremes of the chunks before / after it).
__device__ __forceinline__ void set_block_scans(int& a, int& b, int& c, int& d, int* s_tmp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int W = kThreads / 32;
  int ia = a, ib = b, ic = c, id = d;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int oa = __shfl_up_sync(kFull, ia, off), ob = __shfl_up_sync(kFull, ib, off);
    const int oc = __shfl_down_sync(kFull, ic, off), od = __shfl_down_sync(kFull, id, off);
    if (lane >= off) { ia = max(ia, oa); ib = max(ib, ob); }
    if (lane + off < 32) { ic = min(ic, oc); id = min(id, od); }
  }
  if (lane == 31) { s_tmp[warp] = ia; s_tmp[W + warp] = ib; }
  if (lane == 0) { s_tmp[2 * W + warp] = ic; s_tmp[3 * W + warp] = id; }
  __syncthreads();
  int ca = -1, cb = -1, cc = kNone, cd = kNone;
  for (int w = 0; w < warp; ++w) { ca = max(ca, s_tmp[w]); cb = max(cb, s_tmp[W + w]); }
  for (int w = warp + 1; w < W; ++w) { cc = min(cc, s_tmp[2 * W + w]); cd = min(cd, s_tmp[3 * W + w]); }
  const int pa = __shfl_up_sync(kFull, ia, 1), pb = __shfl_up_sync(kFull, ib, 1);
  const int pc = __shfl_down_sync(kFull, ic, 1), pd = __shfl_down_sync(kFull, id, 1);
  a = lane > 0 ? max(ca, pa) : ca;
  b = lane > 0 ? max(cb, pb) : cb;
  c = lane < 31 ? min(cc, pc) : cc;
  d = lane < 31 ? min(cd, pd) : cd;
}

// MODE: 0 union, 1 intersection, 2 difference.
template <class T, int LESS, bool PLAIN>
__global__ void __launch_bounds__(kThreads, 4)
    set_tile_kernel(int MODE, Src L, Src R, void* out, int out_esize, uint32_t* count_dev,
                    const uint64_t* __restrict__ splits, const SetRun* __restrict__ runs,
                    const T* __restrict__ vals, uint32_t* counter, TileState<uint32_t, true> st,
                    DevErr err) {
  __shared__ T s_keys[kTile];
  __shared__ T s_out[kTile];
  __shared__ uint8_t s_right[kTile];
  __shared__ int s_tmp[4 * (kThreads / 32)];
  __shared__ uint32_t s_wcount[kThreads / 32];
  __shared__ uint32_t s_tile, s_excl, s_tile_kept;
  __shared__ uint64_t s_split[2];
  const uint64_t nl = src_len(L), nr = src_len(R), n = nl + nr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_tile = atomicAdd(counter, 1u);
  __syncthreads();
  const uint64_t tile = s_tile;
  const uint64_t d0 = tile * (uint64_t)kTile;
  if (d0 >= n) return;
  const uint64_t d1 = min(d0 + (uint64_t)kTile, n);
  if (tid < 2) s_split[tid] = splits[tile + tid];
  __syncthreads();
  const uint64_t i0 = s_split[0], i1 = s_split[1];
  const uint64_t j0 = d0 - i0, j1 = d1 - i1;
  const int la = (int)(i1 - i0), lb = (int)(j1 - j0);
  for (int t = tid; t < la; t += kThreads) s_keys[t] = merge_load<T, PLAIN>(L, i0 + t);
  for (int t = tid; t < lb; t += kThreads) s_keys[la + t] = merge_load<T, PLAIN>(R, j0 + t);
  __syncthreads();
  const int total = la + lb;
  const int dt = min(tid * kItems, total);
  {
    int lo = dt > lb ? dt - lb : 0, hi = dt < la ? dt : la;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (!cmp_ct<T, LESS>(s_keys[la + dt - 1 - mid], s_keys[mid])) lo = mid + 1;
      else hi = mid;
    }
    int a = lo, b = dt - lo;
    T ka = a < la ? s_keys[a] : T(0);
    T kb = b < lb ? s_keys[la + b] : T(0);
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      if (dt + k >= total) break;
      const bool take_left = b >= lb || (a < la && !cmp_ct<T, LESS>(kb, ka));
      s_out[dt + k] = take_left ? ka : kb;
      s_right[dt + k] = take_left ? 0 : 1;
      if (take_left) {
        ++a;
        ka = a < la ? s_keys[a] : ka;
      } else {
        ++b;
        kb = b < lb ? s_keys[la + b] : kb;
      }
    }
  }
  __syncthreads();

  // Chunk summaries: last head, last left position (forward); first head,
  // first right position (backward).  Position 0 is a head of the tile.
  const int cnt = min(kItems, total - dt);
  bool head[kItems], right[kItems];
  int lastH = -1, lastL = -1, firstH = kNone, firstR = kNone;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const int t = dt + k;
    head[k] = false;
    right[k] = false;
    if (k < cnt) {
      head[k] = t == 0 || !equiv_ct<T, LESS>(s_out[t - 1], s_out[t]);
      right[k] = s_right[t] != 0;
      if (head[k]) { lastH = t; if (firstH == kNone) firstH = t; }
      if (right[k]) { if (firstR == kNone) firstR = t; } else { lastL = t; }
    }
  }
  int eh = lastH, el = lastL, fh = firstH, fr = firstR;
  set_block_scans(eh, el, fh, fr, s_tmp);
  // rs / last left (at or before t) forward; re (head after t) / first right
  // (at or after t) backward -- tile positions.
  int rs[kItems], ll[kItems], re[kItems], rr[kItems];
  {
    int h = eh, l = el;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      if (k < cnt) {
        if (head[k]) h = dt + k;
        if (!right[k]) l = dt + k;
      }
      rs[k] = h;
      ll[k] = l;
    }
    int nh = fh, nrp = fr;
#pragma unroll
    for (int k = kItems - 1; k >= 0; --k) {
      re[k] = nh;
      if (k < cnt) {
        if (right[k]) nrp = dt + k;
        if (head[k]) nh = dt + k;
      }
      rr[k] = nrp;
    }
  }
  // Runs that cross the tile's edges: the first (when it started before
  // d0) from boundary `tile`, the last (when it goes on past d1) from
  // boundary `tile + 1`.
  const SetRun r0 = runs[tile];
  const uint64_t rs0 = (uint64_t)r0.lbl + r0.lbr;
  const bool first_open = rs0 < d0;
  bool last_open = false;
  SetRun r1{};
  if (d1 < n) {
    r1 = runs[tile + 1];
    last_open = equiv_ct<T, LESS>(s_out[total - 1], vals[tile + 1]);
  }
  // Tile position of the last run's head (every thread reads the same).
  __shared__ int s_last_rs;
  if (tid == 0) s_last_rs = -1;
  __syncthreads();
  if (cnt > 0 && dt + cnt == total) s_last_rs = rs[cnt - 1];
  __syncthreads();
  const int last_rs = s_last_rs;

  bool keep[kItems];
  uint32_t kept = 0;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    keep[k] = false;
    if (k >= cnt) continue;
    const bool use0 = first_open && rs[k] == 0;
    const bool use1 = !use0 && last_open && rs[k] == last_rs;
    bool kp;
    if (use0 || use1) {  // a run crossing the tile's edge: global positions
      const SetRun x = use0 ? r0 : r1;
      const uint64_t g = d0 + dt + k;
      const uint64_t grs = (uint64_t)x.lbl + x.lbr;
      const uint64_t cl = x.ubl - x.lbl, cr = x.ubr - x.lbr;
      if (!right[k]) {
        const uint64_t rank = g - grs;
        kp = MODE == 0 || (MODE == 1 ? rank < cr : rank >= cr);
      } else {
        kp = MODE == 0 && g - (grs + cl) >= cl;
      }
    } else {  // a run inside the tile: tile positions
      const int t = dt + k;
      const int e = re[k] == kNone ? total : re[k];
      if (!right[k]) {
        const int lr = min(rr[k] == kNone ? total : rr[k], e);
        const int rank = t - rs[k], cr = e - lr;
        kp = MODE == 0 || (MODE == 1 ? rank < cr : rank >= cr);
      } else {
        const int lr = max(ll[k] + 1, rs[k]);
        kp = MODE == 0 && t - lr >= lr - rs[k];
      }
    }
    keep[k] = kp;
    kept += kp ? 1u : 0u;
  }

  // Output offsets: warp and block prefix of the kept counts, then the
  // counts of all earlier tiles by the look-back.
  uint32_t incl = kept;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t o = __shfl_up_sync(kFull, incl, off);
    if (lane >= off) incl += o;
  }
  if (lane == 31) s_wcount[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t c = lane < kThreads / 32 ? s_wcount[lane] : 0u;
    const uint32_t agg = __reduce_add_sync(kFull, c);
    const Op<uint32_t, MB_OP_ADD> add{MB_OP_ADD};
    uint32_t excl = 0;
    if (tile == 0) {
      if (lane == 0) st.publish(0, kFlagIncl, agg);
    } else {
      if (lane == 0) st.publish(tile, kFlagAgg, agg);
      excl = lookback_exclusive<uint32_t, Op<uint32_t, MB_OP_ADD>, false>(st, tile, add, err, 0u);
      if (lane == 0) st.publish(tile, kFlagIncl, excl + agg);
    }
    if (lane == 0) {
      s_excl = excl;
      s_tile_kept = agg;
      if (d1 == n && count_dev) *count_dev = excl + agg;
    }
  }
  // The kept items, compacted in tile order into s_keys (free since the
  // merge), then written with consecutive threads on consecutive addresses.
  uint32_t lpos = incl - kept;
  for (int w = 0; w < warp; ++w) lpos += s_wcount[w];
#pragma unroll
  for (int k = 0; k < kItems; ++k)
    if (keep[k]) s_keys[lpos++] = s_out[dt + k];
  __syncthreads();
  const uint64_t base = s_excl;
  const uint32_t tile_kept = s_tile_kept;
  const uint64_t cap = MODE == 0 ? n : nl;
  for (uint32_t i = tid; i < tile_kept; i += kThreads) {
    if (base + i < cap) st_raw_pay(out, base + i, out_esize, to_bits64(s_keys[i]));
    else raise_device_error(err, MB_DEV_ERR_BOUNDS);  // only after a failed look-back
  }
}

// ------------------------------------------------- warp-window kernels --
//
// Plain columns of 4- and 8-byte elements whose order is that of unsigned
// words after a bijection (integers under any predicate, floats in the total
// order), and, for the set operations, floats under LESS / GREATER (-0 mapped
// to +0, which tie).  What bounded the thread-serial kernels below was
// instruction issue (merge 2 x 2^25 u32: 88% of issue slots, 103 warp
// instructions per 32 outputs; set_intersection 250): each thread searched
// its own split in shared memory and then took one dependent step per output.
// Here a warp takes a whole window of both inputs per step: the items of
// window A and of window B reversed, compared lane by lane, give the split of
// the next 32 x R outputs with one ballot per register (the merge-path
// predicate is monotone along the diagonal), so there is no search per
// thread and every shared-memory access is to consecutive words.  Merge of
// 100000007 and 150000001 u32: 788 -> 478 us (4.2 TB/s); set_intersection of
// 33554393 and 30000001: 825 -> 420 us with its count read back.

// Order- and equivalence-preserving map to unsigned words.  ENC: 0 integers
// (raw ^ flip), 1 floats under LESS / GREATER, 2 floats in the total order;
// `flip` holds the sign flip of signed integers and the inversion of GREATER.
template <class U, int ENC>
__device__ __forceinline__ U ord_of(U raw, U flip) {
  if constexpr (ENC == 0) {
    return raw ^ flip;
  } else {
    constexpr U sign = (U)1 << (sizeof(U) * 8 - 1);
    if constexpr (ENC == 1) {
      if (raw == sign) raw = 0;
    }
    return enc_bits<U, kEncFloat>(raw) ^ flip;
  }
}
// The raw bits of an ordered word (ENC 0 and 2 are bijections).
template <class U, int ENC>
__device__ __forceinline__ U ord_to_raw(U u, U flip) {
  u ^= flip;
  return ENC == 2 ? dec_bits<U, kEncFloat>(u) : u;
}

// The merge-path split of every tile boundary by groups of G lanes, G + 1
// sub-ranges per round.  Shorter lists take eight lanes: a 27-step binary search
// becomes nine rounds of independent loads, and the searches' latency is what
// the tile kernel waits for.  Longer ones take two (17 rounds): the probes are
// then mostly DRAM reads, and wide rounds make more of them.  The line lies
// between 64 and 80 M items of 4 bytes (merge 138.9 / 140.9 us with 8 / 2 lanes,
// then 171.7 / 170.7; 265 / 258 us at 128 M) and between 32 and 48 M items of 8
// (157.5 / 159.5, then 230.5 / 226.9; 301 / 295 us at 64 M), about twice the L2
// cache.  It goes by capacity, a device length is not known here; two lanes cost
// up to 5 us (16 M items of 4 bytes: 48.1 and 53.0 us).  Boundaries past the
// logical end are not computed.
constexpr uint64_t kSplitWideBytes = 1ull << 28;

template <class U, int ENC, int G>
__global__ void __launch_bounds__(kThreads)
    window_splits_kernel(Src L, Src R, uint32_t tile_items, uint64_t tiles, U flip,
                         uint32_t* __restrict__ splits) {
  const uint64_t nl = src_len(L), nr = src_len(R), n = nl + nr;
  const U* l = (const U*)L.data;
  const U* r = (const U*)R.data;
  const int lane = threadIdx.x & 31, sub = lane & (G - 1);
  const int shift = lane & ~(G - 1);
  constexpr uint32_t kAll = (1u << G) - 1u;
  const uint64_t b = (blockIdx.x * (uint64_t)kThreads + threadIdx.x) / G;
  // (a boundary of the last, partial tile is still wanted: b * tile < n + tile)
  const bool on = b <= tiles && b * tile_items < n + tile_items;
  const uint64_t d = on ? min(b * tile_items, n) : 0;
  uint64_t lo = d > nr ? d - nr : 0, hi = d < nl ? d : nl;
  while (__any_sync(kFull, lo < hi)) {
    const uint64_t step = (hi - lo + G) / (G + 1);
    const uint64_t mid = lo + (uint64_t)(sub + 1) * step - 1;
    bool before = false;  // the split lies after mid
    if (lo < hi && mid < hi)
      before = ord_of<U, ENC>(l[mid], flip) <= ord_of<U, ENC>(r[d - 1 - mid], flip);
    const uint32_t m = (__ballot_sync(kFull, before) >> shift) & kAll;
    if (lo < hi) {
      lo += (uint64_t)__popc(m) * step;
      if (m != kAll) hi = min(hi, lo + step - 1);
    }
  }
  if (on && sub == 0) splits[b] = (uint32_t)lo;
}

// The slices of one tile in shared memory: left items at [a_off, a_off + la),
// right items at [b_off, b_off + lb) of `buf`.
struct TileSlices {
  uint32_t i0, j0;  // global index of the first left / right item
  int la, lb, a_off, b_off;
};

template <class U>
__device__ __forceinline__ TileSlices tile_slices(uint64_t d0, uint64_t d1, uint32_t s0,
                                                  uint32_t s1) {
  constexpr int V = 16 / (int)sizeof(U);
  const int total = (int)(d1 - d0);
  TileSlices t;
  t.i0 = s0;
  t.j0 = (uint32_t)(d0 - s0);
  // (unsorted inputs can give splits that go back: still in bounds)
  t.la = s1 <= s0 ? 0 : (int)min(s1 - s0, (uint32_t)total);
  t.lb = total - t.la;
  t.a_off = (int)(t.i0 % V);
  t.b_off = (t.a_off + t.la + V - 1) / V * V + (int)(t.j0 % V);
  return t;
}

// Bulk-copies src[g0, g0 + len) to buf + off (off % V == g0 % V): whole
// 16-byte vectors inside the column by one cp.async.bulk issued by thread 0,
// whose bytes are returned for the barrier; the last items of a column whose
// length is no multiple of a vector are copied by the calling threads.
template <class U>
__device__ __forceinline__ uint32_t slice_bytes(uint32_t g0, int len, uint64_t n) {
  constexpr uint64_t V = 16 / sizeof(U);
  if (len == 0) return 0;
  const uint64_t lo = g0 / V * V;
  const uint64_t hi = min(((uint64_t)g0 + len + V - 1) / V * V, n / V * V);
  return hi > lo ? (uint32_t)((hi - lo) * sizeof(U)) : 0u;
}
template <class U>
__device__ __forceinline__ void slice_load(U* buf, int off, const U* src, uint32_t g0,
                                           uint32_t bytes, uint64_t* bar) {
  constexpr uint64_t V = 16 / sizeof(U);
  if (bytes) bulk_load(buf + off - (int)(g0 % V), src + g0 / V * V, bytes, bar);
}
template <class U>
__device__ __forceinline__ void slice_tail(U* buf, int off, const U* src, uint32_t g0, int len,
                                           uint64_t n, int tid) {
  constexpr uint64_t V = 16 / sizeof(U);
  const uint64_t g = n / V * V + tid;  // at most V - 1 items
  if (tid < (int)V && g >= g0 && g < (uint64_t)g0 + len) buf[off + (int)(g - g0)] = src[g];
}

// Fetches both slices into buf; all threads call it, the items are there
// after it returns (block barrier inside).  `phase`: the barrier's parity.
template <class U, int THREADS>
__device__ __forceinline__ void tile_fetch(U* buf, const TileSlices& t, const U* l, const U* r,
                                           uint64_t nl, uint64_t nr, bool aligned, uint64_t* bar,
                                           uint32_t phase, const DevErr& err) {
  const int tid = threadIdx.x;
  if (aligned) {
    if (tid == 0) {
      const uint32_t ba = slice_bytes<U>(t.i0, t.la, nl), bb = slice_bytes<U>(t.j0, t.lb, nr);
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(bar, ba + bb);
      slice_load<U>(buf, t.a_off, l, t.i0, ba, bar);
      slice_load<U>(buf, t.b_off, r, t.j0, bb, bar);
    }
    slice_tail<U>(buf, t.a_off, l, t.i0, t.la, nl, tid);
    slice_tail<U>(buf, t.b_off, r, t.j0, t.lb, nr, tid);
    if (!mbar_wait(bar, phase)) raise_device_error(err, MB_DEV_ERR_LOOKBACK);
  } else {
    for (int k = tid; k < t.la; k += THREADS) buf[t.a_off + k] = l[t.i0 + k];
    for (int k = tid; k < t.lb; k += THREADS) buf[t.b_off + k] = r[t.j0 + k];
  }
  __syncthreads();
}

// The split of diagonal d of a tile in shared memory, by one warp: 33
// sub-ranges per round, three rounds for any tile.
template <class U, int ENC>
__device__ __forceinline__ int warp_split(const U* a, int la, const U* b, int lb, int d, U flip) {
  const int lane = (int)lane_id();
  int lo = d > lb ? d - lb : 0, hi = d < la ? d : la;
  while (lo < hi) {  // warp-uniform
    const int step = (hi - lo + 32) / 33;
    const int mid = lo + (lane + 1) * step - 1;
    const bool before =
        mid < hi && ord_of<U, ENC>(a[mid], flip) <= ord_of<U, ENC>(b[d - 1 - mid], flip);
    const uint32_t m = __ballot_sync(kFull, before);
    lo += __popc(m) * step;
    if (m != kFull) hi = min(hi, lo + step - 1);
  }
  return lo;
}

// ---- merge: a tile per CTA, kMergeSeg outputs per warp, windows of 64 ----
//
// The window's 64 smallest items come out of the reversed comparison as a
// bitonic sequence and are sorted by one in-register and five shuffle steps.
// Equal words are equal items here, so which input a tied item came from
// cannot be seen.  A window past the end of a slice reads the largest word;
// should it be taken for an equal real item, the same values come out.
// 8 warps x 5.5 KB, five CTAs per SM: a tile pays its loads and the warps'
// splits once (16 / 28 / 32 / 44 KB tiles: 603 / 513 / 496 / 478 us).
constexpr int kMergeWarpBytes = 5632;

template <class U>
struct MergeCfg {
  static constexpr int SEG = kMergeWarpBytes / (int)sizeof(U);
  static constexpr int TILE = SEG * (kThreads / 32);
  static constexpr int BUF = TILE + 4 * (16 / (int)sizeof(U));
};

template <class U, int ENC>
__global__ void __launch_bounds__(kThreads)
    merge_window_kernel(Src L, Src R, U* __restrict__ out, U flip, bool aligned,
                        const uint32_t* __restrict__ splits, DevErr err) {
  using C = MergeCfg<U>;
  __shared__ __align__(16) U buf[C::BUF];
  __shared__ __align__(8) uint64_t bar;
  const uint64_t nl = src_len(L), nr = src_len(R), n = nl + nr;
  const uint64_t d0 = (uint64_t)blockIdx.x * C::TILE;
  if (d0 >= n) return;
  const uint64_t d1 = min(d0 + (uint64_t)C::TILE, n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(&bar, 1);
    mbar_init_fence();
  }
  const TileSlices t = tile_slices<U>(d0, d1, splits[blockIdx.x], splits[blockIdx.x + 1]);
  __syncthreads();
  tile_fetch<U, kThreads>(buf, t, (const U*)L.data, (const U*)R.data, nl, nr, aligned, &bar, 0,
                          err);
  const U* sa = buf + t.a_off;
  const U* sb = buf + t.b_off;
  const int total = t.la + t.lb;
  const int w0 = warp * C::SEG;
  if (w0 >= total) return;
  int a = warp_split<U, ENC>(sa, t.la, sb, t.lb, w0, flip);
  int b = w0 - a;
  const int w1 = min(w0 + C::SEG, total);
  constexpr U kMax = ~(U)0;
  U* o = out + d0;
  for (int d = w0; d < w1; d += 64) {
    const int ia = a + lane, ib = b + 31 - lane;
    const U a0 = ia < t.la ? ord_of<U, ENC>(sa[ia], flip) : kMax;
    const U a1 = ia + 32 < t.la ? ord_of<U, ENC>(sa[ia + 32], flip) : kMax;
    const U b1 = ib < t.lb ? ord_of<U, ENC>(sb[ib], flip) : kMax;
    const U b0 = ib + 32 < t.lb ? ord_of<U, ENC>(sb[ib + 32], flip) : kMax;
    const int ca = __popc(__ballot_sync(kFull, a0 <= b0)) + __popc(__ballot_sync(kFull, a1 <= b1));
    a += ca;
    b += 64 - ca;
    U x = min(a0, b0), y = min(a1, b1);
    const U lo = min(x, y);
    y = max(x, y);
    x = lo;
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
      const U ox = __shfl_xor_sync(kFull, x, s), oy = __shfl_xor_sync(kFull, y, s);
      const bool up = (lane & s) != 0;
      x = up ? max(x, ox) : min(x, ox);
      y = up ? max(y, oy) : min(y, oy);
    }
    if (d + lane < w1) __stcs(o + d + lane, ord_to_raw<U, ENC>(x, flip));
    if (d + 32 + lane < w1) __stcs(o + d + 32 + lane, ord_to_raw<U, ENC>(y, flip));
  }
}

// ---- intersection / difference: only the left items are wanted ----------
//
// The r-th copy (r from 0) of a value in the left input has a partner when
// the right input's r-th copy exists: right[lower_bound(right, v) + r] == v.
// Intersection keeps the items with a partner, difference the others.  A
// window of 32 left and 32 right items gives the split of the next 32 merged
// items; each left item taken in it finds its lower bound among the window's
// right items by five shuffles, its r from the run heads of the window
// (ballot) or the run start carried from the windows before, and its partner
// with one read of the right slice (global memory past the slice's end).  At
// the start of a warp's segment the run start is looked up in the 32 left
// items before it, and by a search when they are all equal.  Kept items are
// compacted over the warp's own left items, which no other warp reads, then
// written behind the count of all earlier tiles (decoupled look-back).
// CTAs take tiles from a ticket until none is left, so a capacity far above
// the device length costs no launch of empty blocks.
// 32 KB tiles, six CTAs per SM (16 / 24 / 32 / 44 KB: 422 / 381 / 371 / 374 us;
// 323 us without the look-back).
constexpr int kSetWarpBytes = 4096;

template <class U>
struct SetCfg {
  static constexpr int SEG = kSetWarpBytes / (int)sizeof(U);
  static constexpr int TILE = SEG * (kThreads / 32);
  static constexpr int BUF = TILE + 4 * (16 / (int)sizeof(U));
};

// First index in [0, hi] of the run of `v` that reaches index hi (ordered
// words of a sorted column), by one warp.
template <class U, int ENC>
__device__ uint32_t warp_run_start(const U* __restrict__ x, uint32_t hi, U v, U flip) {
  const uint32_t lane = lane_id();
  uint64_t lo = 0, top = hi;
  while (lo < top) {
    const uint64_t step = (top - lo + 32) / 33;
    const uint64_t mid = lo + (uint64_t)(lane + 1) * step - 1;
    const bool before = mid < top && ord_of<U, ENC>(x[mid], flip) < v;
    const uint32_t m = __ballot_sync(kFull, before);
    lo += (uint64_t)__popc(m) * step;
    if (m != kFull) top = min(top, lo + step - 1);
  }
  return (uint32_t)lo;
}

template <class U, int ENC>
__global__ void __launch_bounds__(kThreads, 6)
    set_window_kernel(bool difference, Src L, Src R, U* __restrict__ out, U flip, bool aligned,
                      uint32_t* count_dev, const uint32_t* __restrict__ splits, uint32_t* counter,
                      TileState<uint32_t, true> st, GroupLines<uint32_t> lines, DevErr err) {
  using C = SetCfg<U>;
  constexpr int W = kThreads / 32;
  __shared__ __align__(16) U buf[C::BUF];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t s_tile, s_excl;
  __shared__ int s_split[W + 1];
  __shared__ uint32_t s_kept[W];
  const uint64_t nl = src_len(L), nr = src_len(R), n = nl + nr;
  const U* lg = (const U*)L.data;
  const U* rg = (const U*)R.data;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr U kMax = ~(U)0;
  if (tid == 0) {
    mbar_init(&bar, 1);
    mbar_init_fence();
  }
  for (uint32_t phase = 0;; phase ^= 1) {
    if (tid == 0) s_tile = atomicAdd(counter, 1u);
    __syncthreads();
    const uint64_t tile = s_tile;
    const uint64_t d0 = tile * (uint64_t)C::TILE;
    if (d0 >= n) return;
    const uint64_t d1 = min(d0 + (uint64_t)C::TILE, n);
    const TileSlices t = tile_slices<U>(d0, d1, splits[tile], splits[tile + 1]);
    tile_fetch<U, kThreads>(buf, t, lg, rg, nl, nr, aligned, &bar, phase, err);
    U* sa = buf + t.a_off;
    const U* sb = buf + t.b_off;
    const int total = t.la + t.lb;
    const int w0 = min(warp * C::SEG, total);
    int a = warp_split<U, ENC>(sa, t.la, sb, t.lb, w0, flip);
    if (lane == 0) s_split[warp] = a;
    if (tid == 0) s_split[W] = t.la;
    __syncthreads();
    int b = w0 - a;
    const int a0 = a, a1 = s_split[warp + 1];
    int kept = 0;
    if (a < a1) {
      // run start of the segment's first left item
      uint32_t run = t.i0 + (uint32_t)a;
      U prev = ord_of<U, ENC>(sa[a], flip);
      bool cont = false;  // the first item continues a run
      {
        const bool in = run > (uint32_t)lane;
        const bool eq = in && ord_of<U, ENC>(lg[run - 1 - lane], flip) == prev;
        const uint32_t ne = __ballot_sync(kFull, !eq);
        if (ne) {
          const uint32_t back = (uint32_t)__ffs(ne) - 1u;
          cont = back > 0;
          run -= back;
        } else {
          cont = true;
          run = warp_run_start<U, ENC>(lg, run - 32, prev, flip);
        }
      }
      while (a < a1) {
        const bool va = a + lane < a1, vb = b + lane < t.lb;
        const U raw = va ? sa[a + lane] : U(0);
        const U ka = ord_of<U, ENC>(raw, flip);
        const U kb = vb ? ord_of<U, ENC>(sb[b + lane], flip) : kMax;
        const U rb = __shfl_xor_sync(kFull, kb, 31);
        const bool rv = b + 31 - lane < t.lb;
        const int ca = __popc(__ballot_sync(kFull, va && (!rv || ka <= rb)));
        // right items of the window below this left item (at most 31)
        int pos = 0;
#pragma unroll
        for (int s = 16; s >= 1; s >>= 1) {
          const U p = __shfl_sync(kFull, kb, pos + s - 1);
          if (p < ka) pos += s;
        }
        // run of this left item
        const U up = __shfl_up_sync(kFull, ka, 1);
        const bool head = lane == 0 ? !(cont && ka == prev) : ka != up;
        const uint32_t heads = __ballot_sync(kFull, head) & (kFull >> (31 - lane));
        const uint32_t me = t.i0 + (uint32_t)(a + lane);
        const uint32_t start = heads ? t.i0 + (uint32_t)(a + 31 - __clz(heads)) : run;
        // its partner on the right
        bool keep = false;
        if (lane < ca) {
          const uint64_t p = (uint64_t)(b + pos) + (me - start);  // in the right slice
          if (p < (uint64_t)t.lb)
            keep = ord_of<U, ENC>(sb[p], flip) == ka;
          else if (t.j0 + p < nr)
            keep = ord_of<U, ENC>(rg[t.j0 + p], flip) == ka;
          keep = keep != difference;
        }
        const uint32_t km = __ballot_sync(kFull, keep);
        if (keep) sa[a0 + kept + __popc(km & ((1u << lane) - 1u))] = raw;
        kept += __popc(km);
        if (ca > 0) {
          prev = __shfl_sync(kFull, ka, ca - 1);
          run = __shfl_sync(kFull, start, ca - 1);
          cont = true;
        }
        a += ca;
        b += 32 - ca;
      }
    }
    if (lane == 0) s_kept[warp] = (uint32_t)kept;
    __syncthreads();
    if (warp == 0) {
      const uint32_t agg = __reduce_add_sync(kFull, lane < W ? s_kept[lane] : 0u);
      const Op<uint32_t, MB_OP_ADD> add{MB_OP_ADD};
      uint32_t excl = 0;
      if (tile == 0) {
        if (lane == 0) st.publish(0, kFlagIncl, agg);
      } else {
        if (lane == 0) st.publish(tile, kFlagAgg, agg);
        excl = lookback_two_level<uint32_t>(st, lines, tile, add, err, 0u);
      }
      if (lane == 0) {
        s_excl = excl;
        if (d1 == n && count_dev) *count_dev = excl + agg;
      }
    }
    __syncthreads();
    uint64_t base = s_excl;
    for (int w = 0; w < warp; ++w) base += s_kept[w];
    for (int k = lane; k < kept; k += 32) {
      if (base + k < nl) out[base + k] = sa[a0 + k];
      else raise_device_error(err, MB_DEV_ERR_BOUNDS);  // only after a failed look-back
    }
    __syncthreads();  // buf, s_tile and s_split are free again
  }
}

// Whether the warp-window kernels take these inputs, and how they order them:
// plain 4- and 8-byte columns.  `ties`: items that tie must also be equal
// (merge writes whichever it meets), so floats only in the total order.
template <class T>
bool window_order(const mb_src& l, const mb_src& r, int less, bool ties, int& enc,
                  typename UnsignedOf<T>::type& flip) {
  using U = typename UnsignedOf<T>::type;
  const int ct = DTypeOf<T>::value;
  if (!src_plain(l, ct) || !src_plain(r, ct)) return false;
  constexpr U sign = (U)1 << (sizeof(U) * 8 - 1);
  flip = less == MB_GREATER ? ~(U)0 : (U)0;
  if constexpr (std::is_floating_point<T>::value) {
    if (ties && less != MB_TOTAL_LESS) return false;
    enc = less == MB_TOTAL_LESS ? 2 : 1;
  } else {
    enc = 0;
    if (std::is_signed<T>::value) flip ^= sign;
  }
  return true;
}

// Whether `out` shares memory with the column `in` (`bytes` of each).
inline bool overlaps(const void* out, const mb_src& in, uint64_t bytes) {
  const uintptr_t o = (uintptr_t)out, i = (uintptr_t)in.data;
  return o < i + bytes && i < o + bytes;
}

inline bool aligned16(const mb_src& l, const mb_src& r) {
  return (uintptr_t)l.data % 16 == 0 && (uintptr_t)r.data % 16 == 0;
}

template <class U, int ENC>
int window_splits(mb_executor* ex, const mb_src& l, const mb_src& r, uint32_t tile_items,
                  uint64_t tiles, U flip, uint32_t* splits) {
  const bool wide = (l.len + r.len) * sizeof(U) >= kSplitWideBytes;
  const uint64_t threads = (tiles + 1) * (wide ? 2 : 8);
  auto kern = wide ? window_splits_kernel<U, ENC, 2> : window_splits_kernel<U, ENC, 8>;
  kern<<<(unsigned)((threads + kThreads - 1) / kThreads), kThreads, 0, ex->stream>>>(
      to_src(l), to_src(r), tile_items, tiles, flip, splits);
  MB_CUDA(cudaGetLastError());
  return MB_OK;
}

template <class U, int ENC>
int merge_window(mb_executor* ex, const mb_src& l, const mb_src& r, U flip, void* out) {
  using C = MergeCfg<U>;
  const uint64_t tiles = (l.len + r.len + C::TILE - 1) / C::TILE;
  Scratch scratch;
  MB_TRY(scratch.alloc(ex, (tiles + 1) * sizeof(uint32_t)));
  uint32_t* splits = scratch.as<uint32_t>();
  MB_TRY((window_splits<U, ENC>(ex, l, r, C::TILE, tiles, flip, splits)));
  merge_window_kernel<U, ENC><<<(unsigned)tiles, kThreads, 0, ex->stream>>>(
      to_src(l), to_src(r), (U*)out, flip, aligned16(l, r), splits,
      DevErr{ex->status_dev, nullptr});
  MB_CUDA(cudaGetLastError());
  return MB_OK;
}

template <class U, int ENC>
int set_window(mb_executor* ex, const mb_src& l, const mb_src& r, bool difference, U flip,
               void* out, uint32_t* count_dev) {
  using C = SetCfg<U>;
  const uint64_t tiles = (l.len + r.len + C::TILE - 1) / C::TILE;
  const size_t state_b = TileState<uint32_t, true>::bytes(tiles);
  Scratch scratch;
  const size_t lines_b = GroupLines<uint32_t>::bytes(tiles);
  MB_TRY(scratch.alloc(ex, 256 + state_b + lines_b + (tiles + 1) * sizeof(uint32_t)));
  char* base = scratch.as<char>();
  MB_CUDA(cudaMemsetAsync(base, 0, 256 + state_b + lines_b, ex->stream));
  uint32_t* splits = (uint32_t*)(base + 256 + state_b + lines_b);
  MB_TRY((window_splits<U, ENC>(ex, l, r, C::TILE, tiles, flip, splits)));
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ex->device);
  const uint64_t grid = std::min<uint64_t>(tiles, (uint64_t)sms * 6);  // 6 CTAs per SM reside
  set_window_kernel<U, ENC><<<(unsigned)grid, kThreads, 0, ex->stream>>>(
      difference, to_src(l), to_src(r), (U*)out, flip, aligned16(l, r), count_dev, splits,
      (uint32_t*)base, TileState<uint32_t, true>::make(base + 256, tiles),
      GroupLines<uint32_t>{base + 256 + state_b}, DevErr{ex->status_dev, (uint32_t*)base + 1});
  MB_CUDA(cudaGetLastError());
  return MB_OK;
}

template <class T, int LESS, bool PLAIN>
int merge_launch(mb_executor* ex, const mb_src& l, const mb_src& r, void* out, int out_dtype,
                 const Payload& pay, uint32_t* count_dev) {
  const uint64_t cap = l.len + r.len;
  const uint64_t tiles = std::max<uint64_t>(1, (cap + kTile - 1) / kTile);
  Scratch splits;
  MB_TRY(splits.alloc(ex, (tiles + 1) * sizeof(uint64_t)));
  const uint64_t sblocks = std::min<uint64_t>((tiles + kThreads) / kThreads, 4096);
  merge_splits_kernel<T, LESS, PLAIN><<<(unsigned)sblocks, kThreads, 0, ex->stream>>>(
      to_src(l), to_src(r), tiles, splits.as<uint64_t>());
  MB_CUDA(cudaGetLastError());
  merge_kernel<T, LESS, PLAIN><<<(unsigned)tiles, kThreads, 0, ex->stream>>>(
      to_src(l), to_src(r), out, out_dtype, pay, count_dev, splits.as<uint64_t>());
  MB_CUDA(cudaGetLastError());
  return MB_OK;
}

template <class T, int LESS>
int merge_less(mb_executor* ex, const mb_src& l, const mb_src& r, void* out, int out_dtype,
               const Payload& pay, uint32_t* count_dev) {
  const int ct = DTypeOf<T>::value;
  if (src_plain(l, ct) && src_plain(r, ct))
    return merge_launch<T, LESS, true>(ex, l, r, out, out_dtype, pay, count_dev);
  return merge_launch<T, LESS, false>(ex, l, r, out, out_dtype, pay, count_dev);
}

template <class T>
int merge_run(mb_executor* ex, const mb_src& l, const mb_src& r, int less, void* out,
              int out_dtype, const Payload& pay, uint32_t* count_dev) {
  // Keys alone, element type kept: the warp-window kernel (floats under LESS
  // and GREATER, where -0 and +0 tie, need to know the side of each item).
  using U = typename UnsignedOf<T>::type;
  constexpr int kBijection = std::is_floating_point<T>::value ? 2 : 0;
  int enc = 0;
  U flip = 0;
  if (pay.ncols == 0 && !count_dev && out && out_dtype == DTypeOf<T>::value &&
      window_order<T>(l, r, less, true, enc, flip))
    return merge_window<U, kBijection>(ex, l, r, flip, out);
  switch (less) {
    case MB_GREATER: return merge_less<T, MB_GREATER>(ex, l, r, out, out_dtype, pay, count_dev);
    case MB_TOTAL_LESS:
      return merge_less<T, MB_TOTAL_LESS>(ex, l, r, out, out_dtype, pay, count_dev);
    default: return merge_less<T, MB_LESS>(ex, l, r, out, out_dtype, pay, count_dev);
  }
}

// Set operation over n = |l| + |r| > 0 merged items (mode 0 union, 1
// intersection, 2 difference); the kept count goes to count_dev.
template <class T, int LESS, bool PLAIN>
int set_launch(mb_executor* ex, const mb_src& l, const mb_src& r, int mode, const mb_col& out,
               uint32_t* count_dev) {
  const uint64_t n = l.len + r.len;
  const uint64_t tiles = (n + kTile - 1) / kTile;
  const size_t state_b = TileState<uint32_t, true>::bytes(tiles);
  const size_t splits_b = ((tiles + 1) * 8 + 255) / 256 * 256;
  const size_t runs_b = ((tiles + 1) * sizeof(SetRun) + 255) / 256 * 256;
  const size_t vals_b = ((tiles + 1) * sizeof(T) + 255) / 256 * 256;
  Scratch scratch;
  MB_TRY(scratch.alloc(ex, 256 + state_b + splits_b + runs_b + vals_b));
  char* base = scratch.as<char>();
  MB_CUDA(cudaMemsetAsync(base, 0, 256 + state_b, ex->stream));
  uint64_t* splits = (uint64_t*)(base + 256 + state_b);
  SetRun* runs = (SetRun*)(base + 256 + state_b + splits_b);
  T* vals = (T*)(base + 256 + state_b + splits_b + runs_b);
  const uint64_t sblocks = std::min<uint64_t>((tiles + kThreads) / kThreads, 4096);
  set_bounds_kernel<T, LESS, PLAIN><<<(unsigned)sblocks, kThreads, 0, ex->stream>>>(
      to_src(l), to_src(r), tiles, splits, runs, vals);
  MB_CUDA(cudaGetLastError());
  const DevErr err{ex->status_dev, (uint32_t*)base + 1};
  set_tile_kernel<T, LESS, PLAIN><<<(unsigned)tiles, kThreads, 0, ex->stream>>>(
      mode, to_src(l), to_src(r), out.data, (int)dtype_size(out.dtype), count_dev, splits, runs,
      vals,
      (uint32_t*)base, TileState<uint32_t, true>::make(base + 256, tiles), err);
  MB_CUDA(cudaGetLastError());
  return MB_OK;
}

template <class T>
int set_run(mb_executor* ex, const mb_src& l, const mb_src& r, int less, int mode,
            const mb_col& out, uint32_t* count_dev) {
  using U = typename UnsignedOf<T>::type;
  int enc = 0;
  U flip = 0;
  // (The window kernel looks up run starts in left items of earlier tiles, the
  // tile kernel reads only its own slice: an output over the left column is
  // its business.)
  if (mode != 0 && window_order<T>(l, r, less, false, enc, flip) &&
      !overlaps(out.data, l, l.len * sizeof(T))) {
    if constexpr (std::is_floating_point<T>::value) {
      if (enc == 1) return set_window<U, 1>(ex, l, r, mode == 2, flip, out.data, count_dev);
      return set_window<U, 2>(ex, l, r, mode == 2, flip, out.data, count_dev);
    } else {
      return set_window<U, 0>(ex, l, r, mode == 2, flip, out.data, count_dev);
    }
  }
  const int ct = DTypeOf<T>::value;
  const bool plain = src_plain(l, ct) && src_plain(r, ct);
#define MB_SET_LESS(LESSID)                                                              \
  return plain ? set_launch<T, LESSID, true>(ex, l, r, mode, out, count_dev)             \
               : set_launch<T, LESSID, false>(ex, l, r, mode, out, count_dev)
  switch (less) {
    case MB_GREATER: MB_SET_LESS(MB_GREATER);
    case MB_TOTAL_LESS: MB_SET_LESS(MB_TOTAL_LESS);
    default: MB_SET_LESS(MB_LESS);
  }
#undef MB_SET_LESS
}

int merge_dispatch(mb_executor* ex, const mb_src& l, const mb_src& r, int less, void* out,
                   int out_dtype, const Payload& pay, uint32_t* count_dev) {
  const int ct = compute_type(l.vtype);
  MB_DISPATCH_CTYPE(ct, merge_run, ex, l, r, less, out, out_dtype, pay, count_dev);
  return set_error(MB_ERR_LAUNCH, "unsupported element type");
}

int set_dispatch(mb_executor* ex, const mb_src& l, const mb_src& r, int less, int mode,
                 const mb_col& out, uint32_t* count_dev) {
  const int ct = compute_type(l.vtype);
  MB_DISPATCH_CTYPE(ct, set_run, ex, l, r, less, mode, out, count_dev);
  return set_error(MB_ERR_LAUNCH, "unsupported element type");
}

int check_pair(mb_executor* ex, const mb_src* l, const mb_src* r, int less) {
  MB_TRY(check_exec(ex));
  MB_TRY(check_src(ex, l, "left"));
  MB_TRY(check_src(ex, r, "right"));
  if (compute_type(l->vtype) != compute_type(r->vtype))
    return set_error(MB_ERR_LAUNCH, "left and right element types differ");
  if (less < MB_LESS || less > MB_TOTAL_LESS)
    return set_error(MB_ERR_LAUNCH, "takes LESS, GREATER or TOTAL_LESS");
  return MB_OK;
}

// Set operation: mode 1 intersection, 2 difference, 0 union.
int set_op(mb_executor* ex, const mb_src* l, const mb_src* r, int less, mb_col out,
           uint32_t* count_dev, uint32_t* count_host, int mode) {
  MB_TRY(check_pair(ex, l, r, less));
  MB_TRY(check_col(ex, out, "output"));
  const uint64_t need = mode == 0 ? l->len + r->len : l->len;
  if (out.len < need) return set_error(MB_ERR_OUTPUT_TOO_SHORT, "output is shorter than input", need, out.len);
  if (dtype_size(out.dtype) != dtype_size(l->vtype))
    return set_error(MB_ERR_LAUNCH, "output element type differs from the input's");
  MB_TRY(check_len_u32(l->len + r->len));
  Scratch cnt;
  if (!count_dev) {
    MB_TRY(cnt.alloc(ex, 16));
    count_dev = cnt.as<uint32_t>();
  }
  // Zero first: inputs whose device lengths are both 0 launch no tile that
  // writes the count.
  MB_CUDA(cudaMemsetAsync(count_dev, 0, 4, ex->stream));
  if (l->len + r->len > 0) MB_TRY(set_dispatch(ex, *l, *r, less, mode, out, count_dev));
  if (count_host) MB_TRY(read_u32(ex, count_dev, count_host));
  return MB_OK;
}

}  // namespace
}  // namespace mb

using namespace mb;

extern "C" {

int mb_merge(mb_executor* ex, const mb_src* left, const mb_src* right, int less, mb_col out) {
  MB_TRY(check_pair(ex, left, right, less));
  MB_TRY(check_col(ex, out, "output"));
  const uint64_t n = left->len + right->len;
  MB_TRY(check_len_u32(n));
  if (out.len < n) return set_error(MB_ERR_OUTPUT_TOO_SHORT, "output is shorter than input", n, out.len);
  if (compute_type(out.dtype) != compute_type(left->vtype))
    return set_error(MB_ERR_LAUNCH, "output element type differs from the input's");
  if (n == 0) return MB_OK;
  Payload none{};
  return merge_dispatch(ex, *left, *right, less, out.data, out.dtype, none, nullptr);
}

int mb_merge_by_key(mb_executor* ex, const mb_src* left_keys, const mb_src* left_values,
                    const mb_src* right_keys, const mb_src* right_values, int nvals, int less,
                    mb_col out_keys, const mb_col* out_values) {
  MB_TRY(check_pair(ex, left_keys, right_keys, less));
  if (nvals < 0 || nvals > kMaxPay) return set_error(MB_ERR_LAUNCH, "values take 0 to 12 columns");
  const uint64_t n = left_keys->len + right_keys->len;
  MB_TRY(check_len_u32(n));
  Payload pay{};
  pay.ncols = nvals;
  for (int c = 0; c < nvals; ++c) {
    MB_TRY(check_src(ex, &left_values[c], "left values"));
    MB_TRY(check_src(ex, &right_values[c], "right values"));
    MB_TRY(check_col(ex, out_values[c], "value output"));
    if (left_values[c].len != left_keys->len)
      return set_error(MB_ERR_LENGTH_MISMATCH, "input lengths differ", left_keys->len, left_values[c].len);
    if (right_values[c].len != right_keys->len)
      return set_error(MB_ERR_LENGTH_MISMATCH, "input lengths differ", right_keys->len, right_values[c].len);
    if (out_values[c].len < n)
      return set_error(MB_ERR_OUTPUT_TOO_SHORT, "output is shorter than input", n, out_values[c].len);
    pay.left[c] = to_src(left_values[c]);
    pay.right[c] = to_src(right_values[c]);
    pay.out[c] = out_values[c].data;
    pay.esize[c] = (int)dtype_size(left_values[c].vtype);
  }
  if (out_keys.data) {
    MB_TRY(check_col(ex, out_keys, "key output"));
    if (out_keys.len < n) return set_error(MB_ERR_OUTPUT_TOO_SHORT, "output is shorter than input", n, out_keys.len);
  }
  if (n == 0) return MB_OK;
  return merge_dispatch(ex, *left_keys, *right_keys, less, out_keys.data, out_keys.dtype, pay,
                        nullptr);
}

int mb_set_union(mb_executor* ex, const mb_src* left, const mb_src* right, int less, mb_col out,
                 uint32_t* count_dev, uint32_t* count_host) {
  return set_op(ex, left, right, less, out, count_dev, count_host, 0);
}

int mb_set_intersection(mb_executor* ex, const mb_src* left, const mb_src* right, int less,
                        mb_col out, uint32_t* count_dev, uint32_t* count_host) {
  return set_op(ex, left, right, less, out, count_dev, count_host, 1);
}

int mb_set_difference(mb_executor* ex, const mb_src* left, const mb_src* right, int less,
                      mb_col out, uint32_t* count_dev, uint32_t* count_host) {
  return set_op(ex, left, right, less, out, count_dev, count_host, 2);
}

}  // extern "C"
