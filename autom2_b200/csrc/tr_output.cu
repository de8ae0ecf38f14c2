// Byte output of a reconstruction (--f2b) on the device.
//
// The reference maps its volume to bytes slab by slab on the GPU
// (TiltRec_cuda_y/recon_y.cu:164-181 with CufloatToByteKernel,
// basic.cu:442-475): for each slab of the volume it takes the slab's mean and
// standard deviation, folds them into exponentially averaged values
// (alpha 0.9, both starting at 0; the Z-layout drivers take the whole volume
// as one slab with its own statistics, alpha 0, TiltRec_cuda_z/recon_z.cu:
// 164-172), and maps every value of each complete group of four to
// (clamp((v - mean) / std, -10, 10) + 10) / 20 * 255, truncated to an
// unsigned byte.  Here the slab statistics are sums in FP64 over fixed
// partitions of each slab, added in a fixed order, so the bytes are the same
// from run to run; the mean is the float of sum / n, the deviation the float
// square root of the FP64 sum of the float squares of (v - mean), as the
// drop-in executables compute them on the host.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "tr_internal.cuh"

namespace trb {

// All three passes are bound by HBM: the volume is read three times, the bytes
// written once.  Four values per read, several reads in flight, each pass
// walking the volume against the one before it, so that it starts with what L2
// still holds.  1024 x 256 x 1024 voxels in 16 slabs: 2.05 -> 0.64 ms (floor 0.53).  Slabs and
// volumes that do not start on 16 bytes go value by value.

// Sum of a slab's parts, in a fixed order, by one warp (all lanes get it).
__device__ __forceinline__ double f2b_slab_sum(const double *part, int lane) {
  double a = 0.0;
#pragma unroll
  for (int b = 0; b < kF2bParts; b += 32) a += part[b + lane];
#pragma unroll
  for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}

// Per slab s and part b: the part's sum of x (PASS 0) or of the float
// (x - mean[s])^2 (PASS 1), in FP64.
// grid = (kF2bParts, nslabs), 256 threads.
template <int PASS>
__global__ void __launch_bounds__(256)
    f2b_partials_kernel(const float *__restrict__ v, size_t n, size_t slab,
                        const float *__restrict__ mean, double *__restrict__ part) {
  const int s = PASS ? gridDim.y - 1 - blockIdx.y : blockIdx.y;
  const int b = PASS ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const size_t s0 = (size_t)s * slab;
  const size_t len = min(slab, n - s0);
  const size_t per = ((len + kF2bParts - 1) / kF2bParts + 3) & ~(size_t)3;
  const size_t lo = min(len, (size_t)b * per), hi = min(len, lo + per);
  const float m = PASS ? mean[s] : 0.f;
  const float *p = v + s0;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  auto add = [&](double &a, float x) {
    if (PASS) {
      const float d = x - m;
      a += (double)(d * d);
    } else {
      a += (double)x;
    }
  };
  size_t i = lo;
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    const float4 *q = reinterpret_cast<const float4 *>(p);
    const size_t h4 = hi / 4;  // lo is a whole group
#pragma unroll 4
    for (size_t j = lo / 4 + threadIdx.x; j < h4; j += 256) {
      const float4 x = __ldg(q + j);
      add(acc[0], x.x);
      add(acc[1], x.y);
      add(acc[2], x.z);
      add(acc[3], x.w);
    }
    i = max(lo, h4 * 4);
  }
  for (i += threadIdx.x; i < hi; i += 256) add(acc[0], p[i]);
  __shared__ double red[256];
  red[threadIdx.x] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[(size_t)s * kF2bParts + b] = red[0];
}

// Each slab's mean, a warp per slab.
__global__ void __launch_bounds__(256)
    f2b_mean_kernel(const double *__restrict__ part, size_t n, size_t slab, int nslabs,
                    float *mean) {
  const int s = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (s >= nslabs) return;
  const double a = f2b_slab_sum(part + (size_t)s * kF2bParts, threadIdx.x & 31);
  if ((threadIdx.x & 31) == 0) mean[s] = (float)(a / (double)min(slab, n - (size_t)s * slab));
}

// Each slab's deviation, and the exponential averages over the slabs in order
// (g = alpha g + (1 - alpha) stat) into gm / gs.  One block: a warp per slab,
// then one thread over the slabs.
__global__ void __launch_bounds__(1024)
    f2b_slab_kernel(const double *__restrict__ part, size_t n, size_t slab, int nslabs,
                    const float *__restrict__ mean, float *sd, float *gm, float *gs, float alpha) {
  for (int s = threadIdx.x >> 5; s < nslabs; s += 32) {
    const size_t len = min(slab, n - (size_t)s * slab);
    const double a = f2b_slab_sum(part + (size_t)s * kF2bParts, threadIdx.x & 31);
    if ((threadIdx.x & 31) == 0) sd[s] = sqrtf((float)(a / (double)len));
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  float g_mean = 0.f, g_std = 0.f;
  for (int s = 0; s < nslabs; ++s) {
    g_mean = alpha * g_mean + (1.f - alpha) * mean[s];
    g_std = alpha * g_std + (1.f - alpha) * sd[s];
    gm[s] = g_mean;
    gs[s] = g_std;
  }
}

__device__ __forceinline__ unsigned char f2b_byte(float v, float m, float sd) {
  const float sf = 10.f;
  const float x = fmaxf(-sf, fminf(sf, (v - m) / sd));
  return (unsigned char)(((x + sf) / (2.0f * sf)) * 255.0f);
}

// The same byte without the divisions where the mapped value is clear of an
// integer: t = 12.75 (v - m)/sd + 127.5, k = 12.75/sd.  f2b_byte's expression is
// within 5.4e-5 of the exact value (its division's rounding on up to 127.5, three
// more on up to 255), t within 2.3e-5, so 1.5e-4 away from the nearest integer
// both truncate alike; else, and for anything not finite, f2b_byte itself.
__device__ __forceinline__ unsigned char f2b_fast(float v, float m, float sd, float k) {
  const float t = fmaxf(0.f, fminf(255.f, fmaf(v - m, k, 127.5f)));
  const float r = t + 12582912.f;  // 1.5 2^23: rounds to the nearest integer
  const float d = t - (r - 12582912.f);
  if (!(fabsf(d) > 1.5e-4f)) return f2b_byte(v, m, sd);
  return (unsigned char)((__float_as_int(r) & 0x1FF) - (d < 0.f ? 1 : 0));
}

// grid.y: slab.
__global__ void __launch_bounds__(256)
    f2b_map_kernel(const float *__restrict__ v, size_t n, size_t slab,
                   const float *__restrict__ gm, const float *__restrict__ gs,
                   unsigned char *__restrict__ out) {
  const size_t s0 = (size_t)blockIdx.y * slab;
  const size_t len = min(slab, n - s0), groups = len / 4;
  const float *p = v + s0;
  unsigned char *o = out + s0;
  const float m = gm[blockIdx.y], sd = gs[blockIdx.y], k = 12.75f / sd;
  const size_t first = blockIdx.x * 256 + threadIdx.x, step = (size_t)gridDim.x * 256;
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0 && (reinterpret_cast<uintptr_t>(o) & 3) == 0) {
    const float4 *q = reinterpret_cast<const float4 *>(p);
    for (size_t i = first; i < groups; i += 4 * step) {
      float4 x[4];
#pragma unroll
      for (int h = 0; h < 4; ++h)
        x[h] = i + h * step < groups ? __ldg(q + i + h * step) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int h = 0; h < 4; ++h)
        if (i + h * step < groups)
          reinterpret_cast<uchar4 *>(o)[i + h * step] =
              make_uchar4(f2b_fast(x[h].x, m, sd, k), f2b_fast(x[h].y, m, sd, k),
                          f2b_fast(x[h].z, m, sd, k), f2b_fast(x[h].w, m, sd, k));
    }
  } else {
    for (size_t i = first; i < groups * 4; i += step) o[i] = f2b_byte(p[i], m, sd);
  }
  // the values past the last complete group of four
  for (size_t i = groups * 4 + first; i < len; i += step) o[i] = 0;
}

cudaError_t launch_f2b(const float *vol, size_t n, size_t slab, float alpha, unsigned char *out,
                       double *part, float *stats, int nsm, cudaStream_t s) {
  const int nslabs = (int)((n + slab - 1) / slab);
  float *mean = stats, *sd = stats + nslabs, *gm = sd + nslabs, *gs = gm + nslabs;
  const dim3 pg(kF2bParts, nslabs);
  f2b_partials_kernel<0><<<pg, 256, 0, s>>>(vol, n, slab, mean, part);
  f2b_mean_kernel<<<(nslabs + 7) / 8, 256, 0, s>>>(part, n, slab, nslabs, mean);
  f2b_partials_kernel<1><<<pg, 256, 0, s>>>(vol, n, slab, mean, part);
  f2b_slab_kernel<<<1, 1024, 0, s>>>(part, n, slab, nslabs, mean, sd, gm, gs, alpha);
  const size_t want = std::max<size_t>(1, (size_t)nsm * 16 / nslabs);
  const size_t need = std::max<size_t>(1, (std::min(n, slab) / 4 + 255) / 256);
  f2b_map_kernel<<<dim3((unsigned)std::min(want, need), nslabs), 256, 0, s>>>(vol, n, slab, gm, gs,
                                                                            out);
  return cudaGetLastError();
}

}  // namespace trb
