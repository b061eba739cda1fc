// smallsort.cu -- radix sort of a column that fits one CTA's shared memory.
//
// The onesweep path (radix.cu) is a memset, a histogram, a plan and one
// launch per digit: seven launches for 32-bit keys and eleven for 64-bit ones,
// whatever the length.  A small request (a few thousand rows of a serving
// loop) spends its time between them: 72 us for 3001 u32 pairs, of which one
// tile's sorting is a few.  Here one CTA does the whole sort in one launch:
// the keys and a 16-bit row number stay in shared memory through a stable LSD
// sort of 8-bit digits (digits that all keys share are skipped), then keys are
// written and values of any width gathered by row number.  Ranking is the
// onesweep's lane-mask method.
//
// Taken up to kSmallSort items (1024 threads x 16 rounds for 4-byte keys, half
// of that for 8-byte ones, whose passes are twice as many).

#include <algorithm>

#include "common.cuh"

namespace mb {
namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kBins = 256;
constexpr unsigned kAll = 0xFFFFFFFFu;

template <class K, int ITEMS>
struct SmallSmem {
  K key[kThreads * ITEMS];
  uint16_t row[kThreads * ITEMS];
  uint32_t mask[kWarps][kBins + 1];  // peers of a round; slot kBins: no item
  uint32_t cnt[kWarps][kBins + 1];   // per-warp digit counts, then first positions
  uint32_t wsum[kBins / 32];
  K diff[kWarps];
};

template <class K>
__device__ __forceinline__ K small_enc(K raw, int enc) {
  if (enc == kEncFloat) return enc_bits<K, kEncFloat>(raw);
  return enc == kEncSigned ? enc_bits<K, kEncSigned>(raw) : raw;
}
template <class K>
__device__ __forceinline__ K small_dec(K u, int enc) {
  if (enc == kEncFloat) return dec_bits<K, kEncFloat>(u);
  return enc == kEncSigned ? dec_bits<K, kEncSigned>(u) : u;
}

template <class V, class K, int ITEMS>
__device__ __forceinline__ void small_gather(const SmallSmem<K, ITEMS>& sm, const V* in, V* out,
                                             uint32_t n) {
  // Every value is read before the first is written, so the output may be the
  // input column.
  V v[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const uint32_t i = k * kThreads + threadIdx.x;
    if (i < n) v[k] = in[sm.row[i]];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const uint32_t i = k * kThreads + threadIdx.x;
    if (i < n) out[i] = v[k];
  }
}

template <class K, int ITEMS>
__global__ void __launch_bounds__(kThreads, 1)
    small_sort_kernel(const K* in_k, K* out_k, const void* in_v, void* out_v, int vsize,
                      uint32_t n, const uint32_t* n_dev, int enc) {
  extern __shared__ __align__(16) unsigned char small_smem[];
  auto& sm = *reinterpret_cast<SmallSmem<K, ITEMS>*>(small_smem);
  if (n_dev && *n_dev < n) n = *n_dev;
  if (n == 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // Items of a round are consecutive and a warp's rounds follow each other, so
  // ranks in (warp, round, lane) order keep the input order.
  const uint32_t first = (uint32_t)warp * 32 * ITEMS + lane;
  const K ref = small_enc<K>(in_k[0], enc);
  K diff = 0;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const uint32_t i = first + k * 32;
    if (i < n) {
      const K u = small_enc<K>(in_k[i], enc);
      sm.key[i] = u;
      sm.row[i] = (uint16_t)i;
      diff |= u ^ ref;
    }
  }
  for (int d = lane; d <= kBins; d += 32) sm.mask[warp][d] = 0;
  {
    K w = (K)__reduce_or_sync(kAll, (uint32_t)diff);
    if constexpr (sizeof(K) == 8)
      w |= (K)__reduce_or_sync(kAll, (uint32_t)((uint64_t)diff >> 32)) << 32;
    if (lane == 0) sm.diff[warp] = w;
  }
  __syncthreads();
  diff = 0;
  for (int w = 0; w < kWarps; ++w) diff |= sm.diff[w];

  const uint32_t below = (1u << lane) - 1u;
  for (int shift = 0; shift < (int)sizeof(K) * 8; shift += 8) {
    if (((diff >> shift) & (kBins - 1)) == 0) continue;  // the same digit everywhere
    for (int d = lane; d <= kBins; d += 32) sm.cnt[warp][d] = 0;
    __syncwarp();
    uint32_t rd[ITEMS];  // digit << 16 | rank within the warp
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const uint32_t i = first + k * 32;
      const uint32_t d =
          i < n ? (uint32_t)(sm.key[i] >> shift) & (kBins - 1) : (uint32_t)kBins;
      atomicOr(&sm.mask[warp][d], 1u << lane);
      __syncwarp();
      const uint32_t peers = sm.mask[warp][d];
      __syncwarp();
      sm.mask[warp][d] = 0;
      uint32_t base = 0;
      if ((peers & below) == 0) {
        base = sm.cnt[warp][d];
        sm.cnt[warp][d] = base + __popc(peers);
      }
      base = __shfl_sync(kAll, base, __ffs(peers) - 1);
      rd[k] = (d << 16) | (base + __popc(peers & below));
      __syncwarp();
    }
    __syncthreads();
    // Thread d: exclusive positions of digit d over the warps, then over the
    // digits.
    uint32_t total = 0;
    if (tid < kBins) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const uint32_t c = sm.cnt[w][tid];
        sm.cnt[w][tid] = total;
        total += c;
      }
      uint32_t incl = total;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(kAll, incl, off);
        if (lane >= off) incl += o;
      }
      if (lane == 31) sm.wsum[warp] = incl;
      total = incl - total;
    }
    __syncthreads();
    if (tid < kBins) {
      for (int w = 0; w < warp; ++w) total += sm.wsum[w];
#pragma unroll
      for (int w = 0; w < kWarps; ++w) sm.cnt[w][tid] += total;
    }
    K key[ITEMS];
    uint32_t row[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const uint32_t i = first + k * 32;
      key[k] = i < n ? sm.key[i] : K(0);
      row[k] = i < n ? sm.row[i] : 0u;
    }
    __syncthreads();  // every key is in registers, the positions are final
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      if (first + k * 32 >= n) continue;
      const uint32_t pos = sm.cnt[warp][rd[k] >> 16] + (rd[k] & 0xFFFFu);
      sm.key[pos] = key[k];
      sm.row[pos] = (uint16_t)row[k];
    }
    __syncthreads();
  }

  // Values before keys: out_k may be the value column (in_k is not read again).
  if (vsize == 4)
    small_gather<uint32_t>(sm, (const uint32_t*)in_v, (uint32_t*)out_v, n);
  else if (vsize == 8)
    small_gather<uint64_t>(sm, (const uint64_t*)in_v, (uint64_t*)out_v, n);
  if (out_k)
    for (uint32_t i = tid; i < n; i += kThreads) out_k[i] = small_dec<K>(sm.key[i], enc);
}

template <class K, int ITEMS>
int small_launch(mb_executor* ex, const void* ik, const void* iv, void* ok, void* ov,
                 size_t vsize, uint64_t n, const uint32_t* n_dev, int enc) {
  auto kern = small_sort_kernel<K, ITEMS>;
  const size_t smem = sizeof(SmallSmem<K, ITEMS>);
  MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<1, kThreads, smem, ex->stream>>>((const K*)ik, (K*)ok, iv, ov, (int)vsize, (uint32_t)n,
                                          n_dev, enc);
  MB_CUDA(cudaGetLastError());
  return MB_OK;
}

template <class K>
int small_sized(mb_executor* ex, const void* ik, const void* iv, void* ok, void* ov, size_t vsize,
                uint64_t n, const uint32_t* n_dev, int enc) {
  if (n <= 1 * kThreads) return small_launch<K, 1>(ex, ik, iv, ok, ov, vsize, n, n_dev, enc);
  if (n <= 4 * kThreads) return small_launch<K, 4>(ex, ik, iv, ok, ov, vsize, n, n_dev, enc);
  return small_launch<K, (sizeof(K) == 4 ? 16 : 8)>(ex, ik, iv, ok, ov, vsize, n, n_dev, enc);
}

}  // namespace

// Items up to which one CTA sorts faster than the onesweep launches.
uint64_t small_sort_max(int kdt) { return (dtype_size(kdt) == 4 ? 16 : 8) * (uint64_t)kThreads; }

// radix_sort_plain (radix.cu) for n <= small_sort_max(kdt), vsize 0, 4 or 8.
int small_sort(mb_executor* ex, int kdt, const void* ik, const void* iv, void* ok, void* ov,
               size_t vsize, uint64_t n, const uint32_t* n_dev) {
  if (n == 0) return MB_OK;
  const int enc = dtype_is_float(kdt) ? kEncFloat : dtype_is_signed(kdt) ? kEncSigned : kEncUnsigned;
  if (dtype_size(kdt) == 4)
    return small_sized<uint32_t>(ex, ik, iv, ok, ov, vsize, n, n_dev, enc);
  return small_sized<uint64_t>(ex, ik, iv, ok, ov, vsize, n, n_dev, enc);
}

}  // namespace mb
