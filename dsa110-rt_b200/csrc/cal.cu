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
// Up to 16 bytes per access, as the planes' alignment allows.
#include "dsb_common.cuh"

#include <algorithm>
#include <type_traits>

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

// B bytes of elements per access: 16 where every plane starts on that
// boundary, else the widest power of two that does (planes of an odd number of
// elements: one).
template <int B> struct CalWord;
template <> struct CalWord<16> { using U = uint4; };
template <> struct CalWord<8> { using U = uint2; };
template <> struct CalWord<4> { using U = uint32_t; };
template <> struct CalWord<2> { using U = uint16_t; };

// The V elements of one access: parts at re, im (offset o), gains g(k).
template <typename T, int B, typename G>
DSB_DEV void cal_access(const T* __restrict__ re, const T* __restrict__ im, T* __restrict__ ore,
                        T* __restrict__ oim, long long o, G gain) {
  using U = typename CalWord<B>::U;
  constexpr int V = B / (int)sizeof(T);
  const U r4 = *reinterpret_cast<const U*>(re + o), i4 = *reinterpret_cast<const U*>(im + o);
  const T* r = reinterpret_cast<const T*>(&r4);
  const T* i = reinterpret_cast<const T*>(&i4);
  U or4, oi4;
  T* wr = reinterpret_cast<T*>(&or4);
  T* wi = reinterpret_cast<T*>(&oi4);
#pragma unroll
  for (int k = 0; k < V; ++k) {
    T gr, gi;
    gain(k, gr, gi);
    if constexpr (sizeof(T) == 2) {
      wr[k] = cal_re_h(r[k], i[k], gr, gi);
      wi[k] = cal_im_h(r[k], i[k], gr, gi);
    } else {
      wr[k] = cal_re_f(r[k], i[k], gr, gi);
      wi[k] = cal_im_f(r[k], i[k], gr, gi);
    }
  }
  *reinterpret_cast<U*>(ore + o) = or4;
  *reinterpret_cast<U*>(oim + o) = oi4;
}

// A CTA takes a segment of one (channel, t, pol) plane, one access of each
// part per thread and step, with the plane's gains in shared memory.  Bound by
// memory (both parts read and written once); dividing the
// 64-bit index of each pair five times to find its gain held it to 2.5 TB/s.
// Here the only division is one 32-bit remainder per access:
// 972 -> 361 us for a native float16 page (2.4 GB moved, 6.7 TB/s).
constexpr int CAL_THREADS = 256, CAL_ITERS = 8, CAL_MAX_SMEM = 48 * 1024;
template <typename T, int B>
__global__ void __launch_bounds__(CAL_THREADS) cal_apply_kernel(
    const T* __restrict__ re, const T* __restrict__ im, const T* __restrict__ gre,
    const T* __restrict__ gim, int n_seg, int plane, int nant, int npol, int ntimes, int per_ch,
    T* __restrict__ ore, T* __restrict__ oim) {
  constexpr int V = B / (int)sizeof(T);  // elements per access
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
    cal_access<T, B>(re, im, ore, oim, base + (long long)v * V, [&](int k, T& gr, T& gi) {
      gr = s_gr[a + k];
      gi = s_gi[a + k];
    });
  }
}

// Planes too short for a CTA of their own (1024 channels x one packet of 16
// antennas: 2.2 us, 8.2 us with a CTA per plane), or more antennas than the
// shared gains hold: accesses counted over all planes, gains from global
// memory.
template <typename T, int B>
__global__ void __launch_bounds__(CAL_THREADS) cal_apply_flat_kernel(
    const T* __restrict__ re, const T* __restrict__ im, const T* __restrict__ gre,
    const T* __restrict__ gim, long long n_acc, long long plane, int nant, int npol, int ntimes,
    int per_ch, T* __restrict__ ore, T* __restrict__ oim) {
  constexpr int V = B / (int)sizeof(T);
  const long long nv = plane / V;
  const bool narrow = n_acc <= 0xffffffffLL && plane <= 0x7fffffff;   // 32-bit divisions
  for (long long j = (long long)blockIdx.x * CAL_THREADS + threadIdx.x; j < n_acc;
       j += (long long)gridDim.x * CAL_THREADS) {
    const long long pl = narrow ? (unsigned)j / (unsigned)nv : j / nv;
    const long long e = (j - pl * nv) * V;
    int a = narrow ? (int)((unsigned)e % (unsigned)nant) : (int)(e % nant);
    const unsigned p = (unsigned)(pl % npol);
    const long long g0 = ((per_ch ? pl / ((long long)npol * ntimes) : 0) * npol + p) * nant;
    cal_access<T, B>(re, im, ore, oim, j * V, [&](int, T& gr, T& gi) {
      gr = gre[g0 + a];
      gi = gim[g0 + a];
      if (++a == nant) a = 0;
    });
  }
}

template <typename T, int B>
int launch_cal(const void* re, const void* im, const void* gre, const void* gim, long long plane,
               long long n_planes, int nant, int npol, int ntimes, int per_ch, void* ore, void* oim,
               cudaStream_t stream) {
  constexpr int V = B / (int)sizeof(T);
  const long long nv = plane / V;
  const long long n_seg = (nv + CAL_THREADS * CAL_ITERS - 1) / (CAL_THREADS * CAL_ITERS);
  const size_t smem = (size_t)2 * (((size_t)nant + 2 * V - 1) / V * V) * sizeof(T);
  if (nv >= CAL_THREADS && plane <= 0x7fffffff && smem <= CAL_MAX_SMEM &&
      n_seg * n_planes <= 0x7fffffffLL) {
    cal_apply_kernel<T, B><<<(unsigned)(n_seg * n_planes), CAL_THREADS, smem, stream>>>(
        (const T*)re, (const T*)im, (const T*)gre, (const T*)gim, (int)n_seg, (int)plane, nant, npol,
        ntimes, per_ch, (T*)ore, (T*)oim);
    return launch_status();
  }
  const long long n_acc = n_planes * nv;
  const unsigned blocks =
      (unsigned)std::min<long long>((n_acc + CAL_THREADS - 1) / CAL_THREADS, 148 * 32);
  cal_apply_flat_kernel<T, B><<<blocks, CAL_THREADS, 0, stream>>>(
      (const T*)re, (const T*)im, (const T*)gre, (const T*)gim, n_acc, plane, nant, npol, ntimes,
      per_ch, (T*)ore, (T*)oim);
  return launch_status();
}

}  // namespace

extern "C" {

int dsb_cal_apply(const void* re, const void* im, const void* gain_re, const void* gain_im,
                  int dtype_f16, int nchan, int ntimes, int npol, int npkt, int nant,
                  int gain_nchan, void* out_re, void* out_im, cudaStream_t stream) {
  if (!re || !im || !gain_re || !gain_im || !out_re || !out_im || nchan <= 0 || ntimes <= 0 ||
      npol <= 0 || npkt <= 0 || nant <= 0 || (gain_nchan != 1 && gain_nchan != nchan))
    return DSB_E_ARG;
  const long long plane = (long long)npkt * nant;
  const long long n_planes = (long long)nchan * ntimes * npol;
  const int per_ch = gain_nchan == nchan && nchan > 1;
  const uintptr_t esz = dtype_f16 ? 2 : 4;
  // the widest access that every plane of every array starts on
  const uintptr_t at = reinterpret_cast<uintptr_t>(re) | reinterpret_cast<uintptr_t>(im) |
                       reinterpret_cast<uintptr_t>(out_re) | reinterpret_cast<uintptr_t>(out_im) |
                       (uintptr_t)plane * esz;
  auto go = [&](auto t, auto bytes) {
    return launch_cal<decltype(t), decltype(bytes)::value>(re, im, gain_re, gain_im, plane,
                                                           n_planes, nant, npol, ntimes, per_ch,
                                                           out_re, out_im, stream);
  };
  using B16 = std::integral_constant<int, 16>;
  using B8 = std::integral_constant<int, 8>;
  using B4 = std::integral_constant<int, 4>;
  using B2 = std::integral_constant<int, 2>;
  if (dtype_f16)
    return at % 16 == 0  ? go(__half{}, B16{})
           : at % 8 == 0 ? go(__half{}, B8{})
           : at % 4 == 0 ? go(__half{}, B4{})
                         : go(__half{}, B2{});
  return at % 16 == 0 ? go(float{}, B16{}) : at % 8 == 0 ? go(float{}, B8{}) : go(float{}, B4{});
}

}  // extern "C"
