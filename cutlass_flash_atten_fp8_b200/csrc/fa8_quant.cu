// Amax quantisation fp16/bf16 -> e4m3: the step before the attention path in the reference's own
// pipeline (test.py:12-23 casts with torch, test.py:68-70), here so that a caller can go from
// half-precision Q/K/V to the FP8 operator without leaving the stream.
//
//   amax = max |x|,  y = e4m3(x * 448 / amax) round-to-nearest-even, saturating,  descale = amax / 448
//
// of one tensor, or (n_seg > 1) of n_seg equal, contiguous segments of it (one per head, say), each
// with its own amax and descale.  amax and descale are caller-provided device floats (outputs);
// nothing else is written.  Bound by memory: 2 bytes read and 1 written per element would do, but
// every element depends on the maximum of all.  Two forms:
//
//   segment_kernel   a segment per thread-block cluster, one launch: the maximum is exchanged through
//                    distributed shared memory, what a thread read first stays in its registers
//                    and the rest is read again while it is still in L2, so HBM sees 3 bytes per
//                    element.
//   amax_kernel +    longer segments: two passes over the tensor (5 bytes per element), the second last
//   cast_kernel      to first.  amax is cleared before by a memset and accumulated with atomicMax.
//
// A long lone tensor in one launch with a barrier over the whole grid is faster (8 MB 6.6 us, 32 MB 11.5, 128 MB 50) but
// starts only once all its CTAs fit the GPU at the same time: beside a kernel on another stream that keeps a
// single SM busy it waits for that kernel's end (64 MB beside one block of 20 ms: 18 ms), for ever if that
// kernel waits for this stream.  The two passes need no more than one free SM.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "fa8_kernel.h"
#include "ptx_sm100.cuh"

namespace fa8 {

namespace {

namespace cg = cooperative_groups;

// 16-byte vectors at the end of the first pass that are meant to stay in L2 for the second: the ones
// before them are read as streamed data, first to be replaced.  96 MB of a 256 MB tensor: 107.2 us; 64 MB
// 108.3, none 112.8 (the second pass forwards, neither marked as streamed: 116.4).
constexpr int64_t kKeep = 96ll << 16;
constexpr int kQuantThreads = 256;     // of the two-pass kernels
constexpr int kSegThreads = 512;       // most threads of a segment_kernel CTA
constexpr int kHold = 8;               // 16-byte vectors of a thread that stay in registers between the passes

template <bool kBf16>
__device__ __forceinline__ float2 unpack_pair(uint32_t w) {
  if (kBf16) {
    // bf16 -> fp32 is a 16-bit shift
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
  const __half2 h = *reinterpret_cast<const __half2*>(&w);
  return __half22float2(h);
}

// Running maximum of |x| over 16-byte vectors, kept as packed pairs of the source type (the
// maximum of a set of its numbers is one of them, so nothing is rounded).  max drops NaN inputs,
// so a NaN does not reach amax (it still casts to the fp8 NaN); an infinite input makes amax
// infinite, the scale 448/inf = 0 and every finite output 0 (inf * 0 = NaN for the infinite ones):
// inputs are expected to be finite.
template <bool kBf16>
struct AbsMax {
  uint32_t m[2] = {0u, 0u};
  __device__ __forceinline__ void pair(int k, uint32_t w) {
    w &= 0x7fff7fffu;
    if (kBf16) asm("max.bf16x2 %0, %0, %1;" : "+r"(m[k]) : "r"(w));
    else asm("max.f16x2 %0, %0, %1;" : "+r"(m[k]) : "r"(w));
  }
  __device__ __forceinline__ void take(const uint4& v) {
    pair(0, v.x); pair(1, v.y); pair(0, v.z); pair(1, v.w);
  }
  __device__ __forceinline__ float value() const {
    const float2 a = unpack_pair<kBf16>(m[0]), b = unpack_pair<kBf16>(m[1]);
    return fmaxf(fmaxf(a.x, a.y), fmaxf(b.x, b.y));
  }
};

// Maximum over the CTA, valid in every thread.
__device__ __forceinline__ float cta_max(float m) {
  __shared__ float part[kSegThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
  __syncthreads();
  for (int w = 0; w < (blockDim.x >> 5); ++w) m = fmaxf(m, part[w]);
  return m;
}

template <bool kBf16>
__device__ __forceinline__ uint2 cast8(const uint4& v, float scale) {
  const float2 f0 = unpack_pair<kBf16>(v.x), f1 = unpack_pair<kBf16>(v.y);
  const float2 f2 = unpack_pair<kBf16>(v.z), f3 = unpack_pair<kBf16>(v.w);
  uint2 o;
  o.x = cvt_e4m3x2(f0.x * scale, f0.y * scale) | (cvt_e4m3x2(f1.x * scale, f1.y * scale) << 16);
  o.y = cvt_e4m3x2(f2.x * scale, f2.y * scale) | (cvt_e4m3x2(f3.x * scale, f3.y * scale) << 16);
  return o;
}
__device__ __forceinline__ float scale_of(float amax) { return amax > 0.f ? 448.f / amax : 1.f; }
__device__ __forceinline__ float descale_of(float amax) { return amax > 0.f ? amax / 448.f : 1.f; }

// n_vec = 16-byte vectors of a segment; the n_tail elements behind them exist for a lone segment only.
// x and tail_in are not declared __restrict__: the launch ahead may still be writing them when this one
// starts, and const __restrict__ lets the compiler read them by the non-coherent path, ahead of the wait.
template <bool kBf16>
__global__ void __launch_bounds__(kSegThreads, 2) segment_kernel(const uint4* x, uint2* __restrict__ y,
                                                                 int64_t n_vec, const uint16_t* tail_in,
                                                                 uint8_t* __restrict__ tail_out, int n_tail, int csize,
                                                                 float* __restrict__ amax, float* __restrict__ descale) {
  __shared__ float peers[8];
  start_after_predecessor();
  const int seg = blockIdx.x / csize, rank = blockIdx.x - seg * csize;
  x += seg * n_vec;
  y += seg * n_vec;
  const int64_t stride = static_cast<int64_t>(csize) * blockDim.x;
  const int64_t i0 = static_cast<int64_t>(rank) * blockDim.x + threadIdx.x;
  uint4 hold[kHold];
  AbsMax<kBf16> mx;
  // A CTA may be written to by its peers once all of them run: told now, waited for below.
  if (csize > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
#pragma unroll
  for (int u = 0; u < kHold; ++u) {
    const int64_t i = i0 + u * stride;
    hold[u] = i < n_vec ? x[i] : make_uint4(0u, 0u, 0u, 0u);
  }
#pragma unroll
  for (int u = 0; u < kHold; ++u) mx.take(hold[u]);
  const int64_t first = i0 + kHold * stride;               // what does not fit the registers
#pragma unroll 4
  for (int64_t i = first; i < n_vec; i += stride) mx.take(x[i]);
  float tail = 0.f;
  const bool has_tail = rank == 0 && threadIdx.x < n_tail;
  if (has_tail) {
    const uint32_t w = tail_in[threadIdx.x];
    tail = unpack_pair<kBf16>(w).x;
    mx.pair(0, w);
  }
  float a = cta_max(mx.value());
  if (csize > 1) {
    // Every CTA leaves its maximum with all of them: after the one barrier only local memory is read.
    cg::cluster_group cluster = cg::this_cluster();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (threadIdx.x < csize) *cluster.map_shared_rank(&peers[rank], static_cast<int>(threadIdx.x)) = a;
    cluster.sync();
    for (int p = 0; p < csize; ++p) a = fmaxf(a, peers[p]);
  }
  if (rank == 0 && threadIdx.x == 0) {
    amax[seg] = a;
    if (descale != nullptr) descale[seg] = descale_of(a);
  }
  const float scale = scale_of(a);
  if (first < n_vec) {
    // last to first: what was read last is the nearest
#pragma unroll 4
    for (int64_t i = first + (n_vec - 1 - first) / stride * stride; i >= first; i -= stride)
      y[i] = cast8<kBf16>(x[i], scale);
  }
#pragma unroll
  for (int u = 0; u < kHold; ++u) {
    const int64_t i = i0 + u * stride;
    if (i < n_vec) y[i] = cast8<kBf16>(hold[u], scale);
  }
  if (has_tail) tail_out[threadIdx.x] = static_cast<uint8_t>(cvt_e4m3x2(tail * scale, 0.f) & 0xffu);
}

template <bool kBf16>
__global__ void __launch_bounds__(kQuantThreads, 8) amax_kernel(const uint4* __restrict__ x, int64_t n_vec,
                                                            const uint16_t* __restrict__ tail, int n_tail,
                                                            float* __restrict__ amax) {
  start_after_predecessor();
  let_successor_start();
  x += blockIdx.y * n_vec;
  amax += blockIdx.y;
  AbsMax<kBf16> mx;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t keep_from = n_vec - kKeep / gridDim.y;
  int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
#pragma unroll 4
  for (; i < keep_from; i += stride) mx.take(__ldcs(x + i));
#pragma unroll 4
  for (; i < n_vec; i += stride) mx.take(ld_global(x + i));
  if (blockIdx.x == 0 && threadIdx.x < n_tail) mx.pair(0, ld_global(tail + threadIdx.x));
  const float m = cta_max(mx.value());
  // non-negative floats order like their bit patterns
  if (threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned int*>(amax), __float_as_uint(m));
}

template <bool kBf16>
__global__ void __launch_bounds__(kQuantThreads, 8) cast_kernel(const uint4* __restrict__ x, uint2* __restrict__ y,
                                                            int64_t n_vec, const uint16_t* __restrict__ tail_in,
                                                            uint8_t* __restrict__ tail_out, int n_tail,
                                                            const float* amax, float* __restrict__ descale) {
  start_after_predecessor();
  x += blockIdx.y * n_vec;
  y += blockIdx.y * n_vec;
  const float a = ld_global(amax + blockIdx.y);           // written by amax_kernel, whose tail this kernel starts under
  const float scale = scale_of(a);
  if (blockIdx.x == 0 && threadIdx.x == 0 && descale != nullptr) descale[blockIdx.y] = descale_of(a);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
#pragma unroll 4
  for (int64_t i = n_vec - 1 - (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x); i >= 0; i -= stride)
    __stcs(y + i, cast8<kBf16>(__ldcs(x + i), scale));
  if (blockIdx.x == 0 && threadIdx.x < n_tail) {
    const float f = unpack_pair<kBf16>(tail_in[threadIdx.x]).x * scale;
    tail_out[threadIdx.x] = static_cast<uint8_t>(cvt_e4m3x2(f, 0.f) & 0xffu);
  }
}

template <bool kBf16>
cudaError_t launch_segments(const uint4* x, uint2* y, int64_t n_vec, const uint16_t* tail_in, uint8_t* tail_out, int n_tail,
                            int n_seg, float* amax, float* descale, cudaStream_t stream) {
  // as many CTAs as it takes to hold the segment in registers, at most a cluster of eight
  const int threads = n_vec <= 1024 ? 128 : kSegThreads;
  int csize = 1;
  while (csize < 8 && n_vec > static_cast<int64_t>(csize) * threads * kHold) csize *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(n_seg) * csize, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {overlap_attribute()};
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = csize;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = csize > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, &segment_kernel<kBf16>, x, y, n_vec, tail_in, tail_out, n_tail, csize, amax, descale);
}

template <bool kBf16>
cudaError_t launch_two_pass(const uint4* x, uint2* y, int64_t n_vec, const uint16_t* tail_in, uint8_t* tail_out, int n_tail,
                            int n_seg, float* amax, float* descale, int sms, cudaStream_t stream) {
  const int64_t want = (n_vec + kQuantThreads - 1) / kQuantThreads;
  const int64_t cap = (8ll * sms + n_seg - 1) / n_seg;      // about eight CTAs per SM in all
  const dim3 grid(static_cast<unsigned>(want < 1 ? 1 : (want > cap ? cap : want)), static_cast<unsigned>(n_seg), 1);
  cudaError_t e = cudaMemsetAsync(amax, 0, sizeof(float) * n_seg, stream);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kQuantThreads, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1] = {overlap_attribute()};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, &amax_kernel<kBf16>, x, n_vec, tail_in, n_tail, amax);
  if (e != cudaSuccess) return e;
  return cudaLaunchKernelEx(&cfg, &cast_kernel<kBf16>, x, y, n_vec, tail_in, tail_out, n_tail, static_cast<const float*>(amax),
                            descale);
}

// Which form (us, fp16, measured on segments of the given size):
//   up to 512 KB a cluster holds a segment in registers: 16 x 128 KB 8.3 two-pass, 4.3 by cluster;
//   up to 1.5 MB the second half is read again from L2, worth it when there are enough clusters to
//   fill the GPU: 128 x 1 MB 64 -> 55, 32 x 1 MB 20.2 -> 15.7, 16 x 1 MB 14.5 -> 12.5, but 4 x 2 MB 12.4 -> 17;
//   anything else: two passes.
template <bool kBf16>
cudaError_t launch_any(const uint4* x, uint2* y, int64_t n_vec, const uint16_t* tail_in, uint8_t* tail_out, int n_tail,
                       int n_seg, float* amax, float* descale, cudaStream_t stream) {
  if (n_vec <= 32 * 1024 || (n_vec <= 96 * 1024 && n_seg >= 12))
    return launch_segments<kBf16>(x, y, n_vec, tail_in, tail_out, n_tail, n_seg, amax, descale, stream);
  cudaError_t e = cudaSuccess;
  const int sms = current_sm_count(&e);
  if (sms <= 0) return e;
  return launch_two_pass<kBf16>(x, y, n_vec, tail_in, tail_out, n_tail, n_seg, amax, descale, sms, stream);
}

}  // namespace

cudaError_t launch_quantize(const void* src, bool bf16, void* dst, int64_t n, int n_seg, float* amax,
                            float* descale, cudaStream_t stream) {
  // n = elements per segment; segments other than a lone one are whole 16-byte vectors
  const int64_t n_vec = n / 8;
  const int n_tail = static_cast<int>(n - n_vec * 8);
  if (n_seg < 1 || n_seg > 65535 || (n_seg > 1 && n_tail != 0)) return cudaErrorInvalidValue;
  const uint4* x = static_cast<const uint4*>(src);
  uint2* y = static_cast<uint2*>(dst);
  const uint16_t* tail_in = static_cast<const uint16_t*>(src) + n_vec * 8;
  uint8_t* tail_out = static_cast<uint8_t*>(dst) + n_vec * 8;
  return bf16 ? launch_any<true>(x, y, n_vec, tail_in, tail_out, n_tail, n_seg, amax, descale, stream)
              : launch_any<false>(x, y, n_vec, tail_in, tail_out, n_tail, n_seg, amax, descale, stream);
}

}  // namespace fa8
