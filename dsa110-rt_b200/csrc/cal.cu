// Per-(channel, pol, antenna) complex gain on split real/imag voltages
// (sm_100a): apply_cal_split of the reference (services/slow_corr_kernel.py:
// 417-423, 459-528):
//   out_re = re * g_re - im * g_im
//   out_im = re * g_im + im * g_re
// on the GEMM layout (nchan, ntimes, npol, npkt, nant), with the gains in the
// broadcast layout (cal_nchan, 1, npol, 1, nant), cal_nchan 1 or nchan.
//
// Rounding follows the reference's eager torch ops, one tensor op at a time:
//   float16: each product rounded to half (the float32 product of two halves
//            is exact), then the sum or difference of the two halves taken in
//            float32 and rounded to half (torch's half arithmetic computes in
//            float32 and stores half);
//   float32: each product and the sum rounded to float32, no fused
//            multiply-add.
// 16 bytes per access where every plane starts on that boundary.
#include "dsb_common.cuh"

#include <algorithm>

namespace {

int launch_status() { return cudaGetLastError() == cudaSuccess ? DSB_OK : DSB_E_CUDA; }

DSB_DEV __half cal_re_h(__half r, __half i, __half gr, __half gi) {
  const float a = __half2float(__hmul(r, gr)), b = __half2float(__hmul(i, gi));
  return __float2half_rn(a - b);
}
DSB_DEV __half cal_im_h(__half r, __half i, __half gr, __half gi) {
  const float a = __half2float(__hmul(r, gi)), b = __half2float(__hmul(i, gr));
  return __float2half_rn(a + b);
}
DSB_DEV float cal_re_f(float r, float i, float gr, float gi) {
  return __fsub_rn(__fmul_rn(r, gr), __fmul_rn(i, gi));
}
DSB_DEV float cal_im_f(float r, float i, float gr, float gi) {
  return __fadd_rn(__fmul_rn(r, gi), __fmul_rn(i, gr));
}

// element (ch, t, p, k, a) -> gain index (ch or 0, p, a)
DSB_DEV long long gain_index(long long e, int nant, int npkt, int npol, int ntimes, bool per_ch) {
  const long long a = e % nant;
  long long r = e / nant;
  r /= npkt;
  const long long p = r % npol;
  r /= npol;
  const long long ch = r / ntimes;
  return ((per_ch ? ch : 0) * npol + p) * nant + a;
}

// A CTA takes a segment of one (channel, t, pol) plane, 16 bytes of each part
// per thread and access, with the plane's gains in shared memory.  Bound by
// memory (both parts read and written once); dividing the
// 64-bit index of each pair five times to find its gain held it to 2.5 TB/s.
// Here the only division is one 32-bit remainder per 16 bytes:
// 972 -> 361 us for a native float16 page (2.4 GB moved, 6.7 TB/s).
constexpr int CAL_THREADS = 256, CAL_ITERS = 8, CAL_MAX_NANT = 2048;
template <typename T>
__global__ void __launch_bounds__(CAL_THREADS) cal_apply_kernel(
    const T* __restrict__ re, const T* __restrict__ im, const T* __restrict__ gre,
    const T* __restrict__ gim, int n_seg, int plane, int nant, int npol, int ntimes, int per_ch,
    T* __restrict__ ore, T* __restrict__ oim) {
  constexpr int V = 16 / sizeof(T);  // elements per access
  // gains of antenna i % nant, V - 1 past the last antenna too: a run of V
  // elements starting at any antenna reads V consecutive entries
  extern __shared__ __align__(16) uint8_t cal_smem[];
  T* s_gr = reinterpret_cast<T*>(cal_smem);
  T* s_gi = s_gr + (nant + 2 * V - 1) / V * V;
  const int seg = (int)(blockIdx.x % n_seg);
  const long long pl = blockIdx.x / n_seg;           // (ch, t, pol)
  const long long g0 = ((per_ch ? pl / ((long long)npol * ntimes) : 0) * npol + pl % npol) * nant;
  for (int i = threadIdx.x; i < nant + V - 1; i += CAL_THREADS) {
    s_gr[i] = gre[g0 + i % nant];
    s_gi[i] = gim[g0 + i % nant];
  }
  __syncthreads();
  const long long base = pl * plane;
  const int v0 = seg * (CAL_THREADS * CAL_ITERS) + (int)threadIdx.x, nv = plane / V;
#pragma unroll 4
  for (int it = 0; it < CAL_ITERS; ++it) {
    const int v = v0 + it * CAL_THREADS;
    if (v >= nv) break;
    const int a = (int)((unsigned)(v * V) % (unsigned)nant);
    const uint4 r4 = *reinterpret_cast<const uint4*>(re + base + (long long)v * V);
    const uint4 i4 = *reinterpret_cast<const uint4*>(im + base + (long long)v * V);
    const T* r = reinterpret_cast<const T*>(&r4);
    const T* i = reinterpret_cast<const T*>(&i4);
    uint4 or4, oi4;
    T* wr = reinterpret_cast<T*>(&or4);
    T* wi = reinterpret_cast<T*>(&oi4);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      if constexpr (sizeof(T) == 2) {
        wr[k] = cal_re_h(r[k], i[k], s_gr[a + k], s_gi[a + k]);
        wi[k] = cal_im_h(r[k], i[k], s_gr[a + k], s_gi[a + k]);
      } else {
        wr[k] = cal_re_f(r[k], i[k], s_gr[a + k], s_gi[a + k]);
        wi[k] = cal_im_f(r[k], i[k], s_gr[a + k], s_gi[a + k]);
      }
    }
    *reinterpret_cast<uint4*>(ore + base + (long long)v * V) = or4;
    *reinterpret_cast<uint4*>(oim + base + (long long)v * V) = oi4;
  }
}

// Any shape and alignment, one element per access.
template <typename T>
__global__ void __launch_bounds__(256) cal_apply_scalar_kernel(
    const T* __restrict__ re, const T* __restrict__ im, const T* __restrict__ gre,
    const T* __restrict__ gim, long long n, int nant, int npkt, int npol, int ntimes,
    int per_ch, T* __restrict__ ore, T* __restrict__ oim) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const long long gi = gain_index(e, nant, npkt, npol, ntimes, per_ch != 0);
    if constexpr (sizeof(T) == 2) {
      ore[e] = cal_re_h(re[e], im[e], gre[gi], gim[gi]);
      oim[e] = cal_im_h(re[e], im[e], gre[gi], gim[gi]);
    } else {
      ore[e] = cal_re_f(re[e], im[e], gre[gi], gim[gi]);
      oim[e] = cal_im_f(re[e], im[e], gre[gi], gim[gi]);
    }
  }
}

}  // namespace

extern "C" {

int dsb_cal_apply(const void* re, const void* im, const void* gain_re, const void* gain_im,
                  int dtype_f16, int nchan, int ntimes, int npol, int npkt, int nant,
                  int gain_nchan, void* out_re, void* out_im, cudaStream_t stream) {
  if (!re || !im || !gain_re || !gain_im || !out_re || !out_im || nchan <= 0 || ntimes <= 0 ||
      npol <= 0 || npkt <= 0 || nant <= 0 || (gain_nchan != 1 && gain_nchan != nchan))
    return DSB_E_ARG;
  const long long n = (long long)nchan * ntimes * npol * npkt * nant;
  const int per_ch = gain_nchan == nchan && nchan > 1;
  const size_t esz = dtype_f16 ? 2 : 4;
  const uintptr_t all_vec = reinterpret_cast<uintptr_t>(re) | reinterpret_cast<uintptr_t>(im) |
                            reinterpret_cast<uintptr_t>(out_re) |
                            reinterpret_cast<uintptr_t>(out_im);
  // whole 16-byte accesses in every plane, gains that fit shared memory, and
  // 32-bit offsets inside a plane
  const int V = (int)(16 / esz);
  const long long plane = (long long)npkt * nant;
  const long long n_seg = (plane / V + CAL_THREADS * CAL_ITERS - 1) / (CAL_THREADS * CAL_ITERS);
  const long long segs = n_seg * nchan * ntimes * npol;
  if (plane % V == 0 && all_vec % 16 == 0 && nant <= CAL_MAX_NANT && plane <= 0x7fffffff &&
      segs <= 0x7fffffff) {
    const size_t smem = (size_t)2 * ((nant + 2 * V - 1) / V * V) * esz;
    auto go = [&](auto t) {
      using T = decltype(t);
      cal_apply_kernel<T><<<(unsigned)segs, CAL_THREADS, smem, stream>>>(
          (const T*)re, (const T*)im, (const T*)gain_re, (const T*)gain_im, (int)n_seg, (int)plane,
          nant, npol, ntimes, per_ch, (T*)out_re, (T*)out_im);
    };
    if (dtype_f16) go(__half{});
    else go(float{});
    return launch_status();
  }
  const int blocks = (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 148 * 32));
  if (dtype_f16)
    cal_apply_scalar_kernel<__half><<<blocks, 256, 0, stream>>>(
        (const __half*)re, (const __half*)im, (const __half*)gain_re, (const __half*)gain_im, n,
        nant, npkt, npol, ntimes, per_ch, (__half*)out_re, (__half*)out_im);
  else
    cal_apply_scalar_kernel<float><<<blocks, 256, 0, stream>>>(
        (const float*)re, (const float*)im, (const float*)gain_re, (const float*)gain_im, n, nant,
        npkt, npol, ntimes, per_ch, (float*)out_re, (float*)out_im);
  return launch_status();
}

}  // extern "C"
