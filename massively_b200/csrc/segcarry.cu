// segcarry.cu -- the carries of the tile-local segmented scans (segmented.cu).
//
// The tile kernel scans every tile as if it started a segment and leaves the
// fold of its last, open segment (part_tail).  What is missing are the items
// before each tile's first segment start: they belong to a segment that began
// in an earlier tile.  Their carry is a segmented scan, over the tiles, of
// (tile holds a start, part_tail):
//   1. seg_carry_blocks_kernel scans blocks of 1024 tiles (one tile per
//      thread, shuffles) and leaves each block's fold;
//   2. seg_carry_top_kernel, one block, scans those folds;
//   3. seg_carry_apply_kernel joins the two and applies the carry, one warp
//      per tile over the items that need it (a few dozen of a tile's 4096 for
//      ordinary segments), whole blocks for tiles that need much.
// One block walking all tiles with dependent loads took 45 us for 2^14 tiles
// and the fix-up, 16 unrolled run-time-typed rounds per tile whatever the
// tile needed, 112 us of the 308 us of a segmented scan of 2^26 f32 in 2^20
// segments.  Every association is fixed, so floats give the same bits from
// run to run.

#include <algorithm>

#include "common.cuh"
#include "lookback.cuh"

namespace mb {
namespace {

constexpr int kBlock = 1024;   // tiles per block of the first pass
constexpr int kApply = 256;    // threads of the apply pass: a warp per tile
constexpr int kLong = 512;     // items above which a tile takes the whole block
constexpr int kPerWarp = 4;    // loads in flight per lane

// Folds under the segmented operator: `start` says that a segment starts
// inside, v is the fold since the last start (or over all of it).
template <class V>
struct Fold {
  V v;
  bool start;
  bool any;  // not empty
};

template <class V>
__device__ __forceinline__ Fold<V> join(const Op<V, kOpDyn>& op, const Fold<V>& a,
                                        const Fold<V>& b) {
  if (!b.any) return a;
  if (!a.any || b.start) return Fold<V>{b.v, a.start || b.start, true};
  return Fold<V>{op(a.v, b.v), a.start, true};
}
template <class V>
__device__ __forceinline__ Fold<V> up(const Fold<V>& f, int d) {
  Fold<V> r;
  r.v = shfl_up(f.v, d);
  r.start = __shfl_up_sync(kFull, (int)f.start, d) != 0;
  r.any = __shfl_up_sync(kFull, (int)f.any, d) != 0;
  return r;
}

// Exclusive scan of one fold per thread over a block of kBlock threads; `all`
// gets the fold of everything.
template <class V>
__device__ __forceinline__ Fold<V> block_scan(const Op<V, kOpDyn>& op, Fold<V> x, Fold<V>& all) {
  __shared__ V s_v[32];
  __shared__ int s_f[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const Fold<V> y = up(x, d);
    if (lane >= d) x = join(op, y, x);
  }
  if (lane == 31) {
    s_v[warp] = x.v;
    s_f[warp] = (x.start ? 1 : 0) | (x.any ? 2 : 0);
  }
  __syncthreads();
  Fold<V> w{s_v[lane], (s_f[lane] & 1) != 0, (s_f[lane] & 2) != 0};
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const Fold<V> y = up(w, d);
    if (lane >= d) w = join(op, y, w);
  }
  all.v = shfl_idx(w.v, 31);
  all.start = __shfl_sync(kFull, (int)w.start, 31) != 0;
  all.any = __shfl_sync(kFull, (int)w.any, 31) != 0;
  // the warps before this one, then the lanes before this one
  Fold<V> before{shfl_idx(w.v, (warp + 31) & 31),
                 __shfl_sync(kFull, (int)w.start, (warp + 31) & 31) != 0,
                 __shfl_sync(kFull, (int)w.any, (warp + 31) & 31) != 0};
  if (warp == 0) before = Fold<V>{V(0), false, false};
  Fold<V> e = up(x, 1);
  if (lane == 0) e = Fold<V>{V(0), false, false};
  __syncthreads();  // s_v is free again
  return join(op, before, e);
}

struct CarryShape {
  const uint32_t* offsets;
  const uint32_t* tile_lb;  // first segment starting at or after each tile's begin
  uint64_t tiles, tile_items, cap;
  const uint32_t* n_dev;
};

__device__ __forceinline__ uint64_t shape_items(const CarryShape& s) {
  return s.n_dev ? min((uint64_t)*s.n_dev, s.cap) : s.cap;
}

// carry[t]: the fold of the block's tiles before t; flags[t]: whether it is
// complete (a segment starts in them); top / topf: the block's fold.
template <class V>
__global__ void __launch_bounds__(kBlock)
    seg_carry_blocks_kernel(CarryShape s, int opid, const V* __restrict__ part_tail,
                            V* __restrict__ carry, uint8_t* __restrict__ flags,
                            V* __restrict__ top, uint8_t* __restrict__ topf) {
  const Op<V, kOpDyn> op{opid};
  const uint64_t n = shape_items(s);
  const uint64_t t = blockIdx.x * (uint64_t)kBlock + threadIdx.x;
  Fold<V> x{V(0), false, false};
  if (t < s.tiles && t * s.tile_items < n) {
    const uint64_t te = min((t + 1) * s.tile_items, n);
    x = Fold<V>{part_tail[t], (uint64_t)s.offsets[s.tile_lb[t]] < te, true};
  }
  Fold<V> all;
  const Fold<V> e = block_scan(op, x, all);
  if (t < s.tiles) {
    carry[t] = e.v;
    flags[t] = (e.start ? 1 : 0) | (e.any ? 2 : 0);
  }
  if (threadIdx.x == 0) {
    // A single block has none before it: what the top kernel would leave.
    if (gridDim.x == 1) all = Fold<V>{V(0), false, false};
    top[blockIdx.x] = all.v;
    topf[blockIdx.x] = (all.start ? 1 : 0) | (all.any ? 2 : 0);
  }
}

// top / topf in place: the fold of the blocks before each one.
template <class V>
__global__ void __launch_bounds__(kBlock)
    seg_carry_top_kernel(uint64_t blocks, int opid, V* __restrict__ top,
                         uint8_t* __restrict__ topf) {
  const Op<V, kOpDyn> op{opid};
  Fold<V> run{V(0), false, false};
  for (uint64_t b0 = 0; b0 < blocks; b0 += kBlock) {
    const uint64_t b = b0 + threadIdx.x;
    Fold<V> x{V(0), false, false};
    if (b < blocks) x = Fold<V>{top[b], (topf[b] & 1) != 0, (topf[b] & 2) != 0};
    Fold<V> all;
    const Fold<V> e = join(op, run, block_scan(op, x, all));
    if (b < blocks) {
      top[b] = e.v;
      topf[b] = (e.start ? 1 : 0) | (e.any ? 2 : 0);
    }
    run = join(op, run, all);
  }
}

// `out` holds tile-local inclusive values.  Inclusive: carry op local;
// exclusive: init op (carry op local of the item before), init op carry for
// the tile's first item.  OUT: the output's element type (V for the wide
// types; narrow columns keep their own).
template <class V, class OUT, bool EXCL>
__device__ __forceinline__ void apply_items(const Op<V, kOpDyn>& op, V init, V c, OUT* out,
                                            uint64_t len, uint64_t start, uint64_t step, V prev) {
  // The calling warp (or block, in steps of `step`) reads every item before it
  // writes; `prev` is the old value before the warp's first item.
  const uint32_t lane = lane_id();
  for (uint64_t b = start; b < len; b += step) {
    V x[kPerWarp];
#pragma unroll
    for (int k = 0; k < kPerWarp; ++k) {
      const uint64_t i = b + k * 32 + lane;
      x[k] = i < len ? (V)out[i] : V(0);
    }
#pragma unroll
    for (int k = 0; k < kPerWarp; ++k) {
      const uint64_t i = b + k * 32 + lane;
      V v;
      if constexpr (EXCL) {
        V before = shfl_up(x[k], 1);
        if (lane == 0) before = prev;
        prev = shfl_idx(x[k], 31);
        v = op(init, i == 0 ? c : op(c, before));
      } else {
        v = op(c, x[k]);
      }
      if (i < len) out[i] = (OUT)v;
    }
  }
}

template <class V, class OUT, bool EXCL>
__global__ void __launch_bounds__(kApply)
    seg_carry_apply_kernel(CarryShape s, int opid, V init, const V* __restrict__ carry,
                           const uint8_t* __restrict__ flags, const V* __restrict__ top,
                           const uint8_t* __restrict__ topf, OUT* __restrict__ out) {
  const Op<V, kOpDyn> op{opid};
  constexpr int W = kApply / 32;
  __shared__ uint32_t s_len[W];
  __shared__ V s_carry[W];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t n = shape_items(s);
  const uint64_t t0 = 1 + blockIdx.x * (uint64_t)W;  // tile 0 starts with a segment
  const uint64_t t = t0 + warp;
  uint32_t len = 0;
  V c = V(0);
  if (t < s.tiles && t * s.tile_items < n) {
    const uint64_t tb = t * s.tile_items, te = min(tb + s.tile_items, n);
    len = (uint32_t)(min((uint64_t)s.offsets[s.tile_lb[t]], te) - tb);
    if (len) {
      const uint64_t b = t / kBlock;
      const Fold<V> e = join(
          op, Fold<V>{top[b], (topf[b] & 1) != 0, (topf[b] & 2) != 0},
          Fold<V>{carry[t], (flags[t] & 1) != 0, (flags[t] & 2) != 0});
      c = e.v;
      if (len <= (uint32_t)kLong)
        apply_items<V, OUT, EXCL>(op, init, c, out + tb, len, 0, 32 * kPerWarp, V(0));
    }
  }
  if (lane == 0) {
    s_len[warp] = len;
    s_carry[warp] = c;
  }
  __syncthreads();
  // Tiles with much to do: the whole block, each warp its own stretch.
  for (int w = 0; w < W; ++w) {
    const uint32_t l = s_len[w];
    if (l <= (uint32_t)kLong) continue;
    OUT* o = out + (t0 + w) * s.tile_items;
    const uint32_t stretch = (l + W * 32 * kPerWarp - 1) / (W * 32 * kPerWarp) * 32 * kPerWarp;
    const uint32_t from = min((uint32_t)warp * stretch, l), to = min(from + stretch, l);
    const V prev = EXCL && from > 0 ? (V)o[from - 1] : V(0);
    __syncthreads();  // the item before each stretch is read before it is written
    if (from < to)
      apply_items<V, OUT, EXCL>(op, init, s_carry[w], o, to, from, 32 * kPerWarp, prev);
  }
}

template <class V, class OUT>
int carry_apply(mb_executor* ex, const CarryShape& s, int op, int exclusive, V init,
                const V* carry, const uint8_t* flags, const V* top, const uint8_t* topf,
                void* out) {
  const unsigned g = (unsigned)((s.tiles - 1 + kApply / 32 - 1) / (kApply / 32));
  if (exclusive)
    seg_carry_apply_kernel<V, OUT, true>
        <<<g, kApply, 0, ex->stream>>>(s, op, init, carry, flags, top, topf, (OUT*)out);
  else
    seg_carry_apply_kernel<V, OUT, false>
        <<<g, kApply, 0, ex->stream>>>(s, op, init, carry, flags, top, topf, (OUT*)out);
  MB_CUDA(cudaGetLastError());
  return MB_OK;
}

template <class V>
int carry_run(mb_executor* ex, const CarryShape& s, int op, int exclusive, const void* init,
              const void* part_tail, void* out, int out_dtype) {
  if (s.tiles < 2) return MB_OK;
  const uint64_t blocks = (s.tiles + kBlock - 1) / kBlock;
  const size_t carry_b = (s.tiles * sizeof(V) + 255) / 256 * 256;
  const size_t top_b = (blocks * sizeof(V) + 255) / 256 * 256;
  const size_t flags_b = (s.tiles + 255) / 256 * 256;
  Scratch scratch;
  MB_TRY(scratch.alloc(ex, carry_b + top_b + flags_b + blocks));
  V* carry = scratch.as<V>();
  V* top = (V*)(scratch.as<char>() + carry_b);
  uint8_t* flags = (uint8_t*)(scratch.as<char>() + carry_b + top_b);
  uint8_t* topf = flags + flags_b;
  seg_carry_blocks_kernel<V><<<(unsigned)blocks, kBlock, 0, ex->stream>>>(
      s, op, (const V*)part_tail, carry, flags, top, topf);
  MB_CUDA(cudaGetLastError());
  if (blocks > 1) {
    seg_carry_top_kernel<V><<<1, kBlock, 0, ex->stream>>>(blocks, op, top, topf);
    MB_CUDA(cudaGetLastError());
  }
  V i;
  memcpy(&i, init, sizeof(V));
#define MB_CARRY_OUT(OUT) \
  return carry_apply<V, OUT>(ex, s, op, exclusive, i, carry, flags, top, topf, out)
  if constexpr (sizeof(V) == 4 && !std::is_floating_point<V>::value) {
    // narrow integers are computed in 32 bits and stored narrow
    switch (out_dtype) {
      case MB_U8: MB_CARRY_OUT(uint8_t);
      case MB_I8: MB_CARRY_OUT(int8_t);
      case MB_U16: MB_CARRY_OUT(uint16_t);
      case MB_I16: MB_CARRY_OUT(int16_t);
      default: break;
    }
  }
  MB_CARRY_OUT(V);
#undef MB_CARRY_OUT
}

}  // namespace

// Applies the carries of a tile-local segmented scan to `out` (compute type
// `ct`, output element type `out_dtype` of the same compute type).
int seg_scan_carries(mb_executor* ex, int ct, const uint32_t* offsets, const uint32_t* tile_lb,
                     uint64_t tiles, uint64_t tile_items, uint64_t cap, const uint32_t* n_dev,
                     int op, int exclusive, const void* init, const void* part_tail, void* out,
                     int out_dtype) {
  const CarryShape s{offsets, tile_lb, tiles, tile_items, cap, n_dev};
  switch (ct) {
    case MB_U32: return carry_run<uint32_t>(ex, s, op, exclusive, init, part_tail, out, out_dtype);
    case MB_I32: return carry_run<int32_t>(ex, s, op, exclusive, init, part_tail, out, out_dtype);
    case MB_U64: return carry_run<uint64_t>(ex, s, op, exclusive, init, part_tail, out, out_dtype);
    case MB_I64: return carry_run<int64_t>(ex, s, op, exclusive, init, part_tail, out, out_dtype);
    case MB_F32: return carry_run<float>(ex, s, op, exclusive, init, part_tail, out, out_dtype);
    case MB_F64: return carry_run<double>(ex, s, op, exclusive, init, part_tail, out, out_dtype);
    default: return set_error(MB_ERR_LAUNCH, "unsupported element type");
  }
}

}  // namespace mb
