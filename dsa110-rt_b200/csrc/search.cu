// Search side: fine-DM combine, image masking, boxcar detector, Layer-1
// noise estimate, and the FP64 uv-cell geometry kernel (sm_100a).
#include "dsb_common.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <cstring>
#include <type_traits>

#include <algorithm>

namespace {

int launch_status() { return cudaGetLastError() == cudaSuccess ? DSB_OK : DSB_E_CUDA; }

// ===========================================================================
// uv cells (FP64): ix = rint(-(d / (c / (nu*1e9))) / cell) + N/2
// (grid/sparsity_pattern.py:1090-1170, same operation order as numpy)
// ===========================================================================
__global__ void uv_cells_kernel(const double* __restrict__ du, const double* __restrict__ dv,
                                int n_bl, const double* __restrict__ nu_ghz, int n_ch,
                                double cell_lambda, int half, int* __restrict__ row,
                                int* __restrict__ col) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n_bl * n_ch) return;
  const int b = (int)(idx / n_ch), c = (int)(idx % n_ch);
  const double wl = 299792458.0 / (nu_ghz[c] * 1e9);
  const double u = -(du[b] / wl);
  const double v = -(dv[b] / wl);
  col[idx] = (int)rint(u / cell_lambda) + half;
  row[idx] = (int)rint(v / cell_lambda) + half;
}

// ===========================================================================
// Pipeline combine: Hermitian half-spectrum from stage-2 rings.
//   G_h[f, t, u, w] = 0.5 * sum_e sign_e(D[row_e(f)][t - sf[f, g_e]]) * (-1)^(u+w)
// where each entry e of half-cell (u, w) names a chgroup g, a cell inside
// that chgroup's pattern, and whether it is the conjugate mirror.
// ===========================================================================
struct CombArgs {
  const void* D;         // ring: complex64 (FMT 0), bf16 re/im pairs in 32 bits (1),
                         // or int8 re/im pairs in 16 bits (2) times the row's scale
  const float* scales;   // FMT 2: scales[sc_base[gc] + slot] of each ring row
  const long long* sc_base;
  const long long* seg_base;  // (G * n_coarse) ring segment of (chgroup, coarse DM)
  const int* seg_depth;       // (G * n_coarse) time slots of each segment
  int n_coarse;
  const int* hc_off;     // (n_half_cells + 1) CSR over half cells (u-major)
  const int* e_g;        // chgroup
  const int* e_cell;     // cell within the chgroup (negative = mirror, stored as ~cell)
  const int* d_pitch;    // (G) cells (row pitch) of each chgroup's segments
  const int* sfine;      // (n_fine_total, G) signed shifts
  const int* f2c;        // (n_fine_total) coarse index
  int f0, n_f, G, N;
  long long t0;          // stream time of output t = 0
  int n_t;
  int fftshift;
  float2* out;           // (n_f, n_t, N, N/2+1)
};

// One thread per (half cell, fine DM); time is walked in tiles of CB_T
// samples so every ring row is read sequentially (L1 sector reuse) and each
// output time is written coalesced across the half cells of a warp.
constexpr int CB_T = 8;

template <int FMT>
__global__ void __launch_bounds__(128) combine_rows_kernel(const CombArgs A) {
  const int nh = A.N / 2 + 1;
  const int n_hc = A.N * nh;
  const int hc = blockIdx.x * blockDim.x + threadIdx.x;
  if (hc >= n_hc) return;
  const int fl = blockIdx.y;
  const int f = A.f0 + fl;
  const int c = A.f2c[f];
  const int u = hc / nh, w = hc % nh;
  const bool flip = A.fftshift && ((u + w) & 1);
  float2* out = A.out + (size_t)fl * A.n_t * n_hc + hc;
  const int j0 = A.hc_off[hc], j1 = A.hc_off[hc + 1];
  for (int tt = 0; tt < A.n_t; tt += CB_T) {
    double re[CB_T], im[CB_T];
#pragma unroll
    for (int i = 0; i < CB_T; ++i) re[i] = im[i] = 0.0;
    for (int j = j0; j < j1; ++j) {
      const int g = A.e_g[j];
      int cell = A.e_cell[j];
      const bool mirror = cell < 0;
      if (mirror) cell = ~cell;
      const int gc = g * A.n_coarse + c;
      const long long ts0 = A.t0 + tt - A.sfine[(long long)f * A.G + g];
      const long long e0 = A.seg_base[gc] + cell;
      const long long dep = A.seg_depth[gc];
      const long long pitch = A.d_pitch[g];
      long long slot0 = ts0 % dep;
      if (slot0 < 0) slot0 += dep;
#pragma unroll
      for (int i = 0; i < CB_T; ++i) {
        long long slot = slot0 + i;
        if (slot >= dep) slot -= dep;
        float2 x;
        if constexpr (FMT == 2) {
          const char2 q = static_cast<const char2*>(A.D)[e0 + slot * pitch];
          const float sc = A.scales[A.sc_base[gc] + slot];
          x = make_float2(sc * (float)q.x, sc * (float)q.y);
        } else if constexpr (FMT == 1)
          x = bf16_pair_to_f2(static_cast<const uint32_t*>(A.D)[e0 + slot * pitch]);
        else
          x = static_cast<const float2*>(A.D)[e0 + slot * pitch];
        re[i] += x.x;
        im[i] += mirror ? -(double)x.y : (double)x.y;
      }
    }
#pragma unroll
    for (int i = 0; i < CB_T; ++i) {
      if (tt + i < A.n_t) {
        float o_re = (float)(0.5 * re[i]), o_im = (float)(0.5 * im[i]);
        if (flip) {
          o_re = -o_re;
          o_im = -o_im;
        }
        out[(size_t)(tt + i) * n_hc] = make_float2(o_re, o_im);
      }
    }
  }
}

// ===========================================================================
// Reference-layout dense cint8 combine (image/fused_combine_cuda.py:210-300,
// 560-700): streams [G, T_stream, 2, N, N] int8.  Calibrated forms add
// scale * q + offset per chgroup term, with one scale/offset per chgroup or
// (PER_T) per (chgroup, source time) [G, T_stream] -- the wire's per-tile
// scales (fused_combine_cuda.py:431-505).
// ===========================================================================
template <bool HALF, bool CALIB, bool OUT_F16, bool PER_T>
__global__ void combine_dense_kernel(const int8_t* __restrict__ streams,
                                     const int* __restrict__ shifts,
                                     const float* __restrict__ scales,
                                     const float* __restrict__ off_re,
                                     const float* __restrict__ off_im, void* __restrict__ out,
                                     int G, int t_stream, int t_det, int N, int t_lo,
                                     int fftshift) {
  const int nw = HALF ? N / 2 + 1 : N;
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  const int u = blockIdx.y * blockDim.y + threadIdx.y;
  const int t_out = blockIdx.z * blockDim.z + threadIdx.z;
  const int t = t_out + t_lo;
  if (w >= nw || u >= N || t >= t_det) return;
  const long long nsq = (long long)N * N;
  const int off_cell = u * N + w;
  const int off_m = ((N - u) % N) * N + ((N - w) % N);
  const long long t_stride = 2 * nsq, g_stride = (long long)t_stream * t_stride;
  float o_re, o_im;
  if (!CALIB) {
    int ar = 0, ai = 0, mr = 0, mi = 0;
    for (int g = 0; g < G; ++g) {
      const int ts = t - shifts[g];
      if (ts >= 0 && ts < t_stream) {
        const long long b = g * g_stride + ts * t_stride;
        ar += streams[b + off_cell];
        ai += streams[b + off_cell + nsq];
        if (HALF) {
          mr += streams[b + off_m];
          mi += streams[b + off_m + nsq];
        }
      }
    }
    if (HALF) {
      o_re = 0.5f * (float)(ar + mr);
      o_im = 0.5f * (float)(ai - mi);
    } else {
      o_re = (float)ar;
      o_im = (float)ai;
    }
  } else {
    float ar = 0.f, ai = 0.f, mr = 0.f, mi = 0.f;
    for (int g = 0; g < G; ++g) {
      const int ts = t - shifts[g];
      if (ts >= 0 && ts < t_stream) {
        const long long b = g * g_stride + ts * t_stride;
        const int gt = PER_T ? g * t_stream + ts : g;
        const float sc = scales[gt], orr = off_re[gt], oii = off_im[gt];
        ar = fmaf(sc, (float)streams[b + off_cell], ar) + orr;
        ai = fmaf(sc, (float)streams[b + off_cell + nsq], ai) + oii;
        if (HALF) {
          mr = fmaf(sc, (float)streams[b + off_m], mr) + orr;
          mi = fmaf(sc, (float)streams[b + off_m + nsq], mi) + oii;
        }
      }
    }
    if (HALF) {
      o_re = 0.5f * (ar + mr);
      o_im = 0.5f * (ai - mi);
    } else {
      o_re = ar;
      o_im = ai;
    }
  }
  if (fftshift && ((u + w) & 1)) {
    o_re = -o_re;
    o_im = -o_im;
  }
  const long long o = (long long)t_out * N * nw + (long long)u * nw + w;
  if (OUT_F16)
    reinterpret_cast<__half2*>(out)[o] = __floats2half2_rn(o_re, o_im);
  else
    reinterpret_cast<float2*>(out)[o] = make_float2(o_re, o_im);
}

// The half-spectrum combine on row pairs: CTA (u, t, f) sums full rows u and
// N - u of every chgroup at time t - shift[f][g], four cells per 4-byte load,
// then forms the half cells of both rows from shared memory: every stream
// byte is loaded once (the kernel above loads each one twice, byte by byte,
// for 318 us per fine DM of 64 times at N = 256, 16 chgroups).  Bound by the
// stream reads (n_f x the streams' bytes through L2: fine DMs are the fastest
// grid index, so those that share a time run together): 40 us with 8 fine
// DMs in one launch (dsb_combine_dense_fdm).
// Integers: sums of 4 bytes in two words of 16-bit lanes, the bytes offset to
// unsigned, spilled to 32 bits every 256 chgroups.  Calibrated: each cell's
// float chain over g is the one of the kernel above, bit for bit.
constexpr int CP_MAX_THREADS = 512;
constexpr int CP_G = 256;   // chgroups per staged list (16-bit lanes hold 257)
template <bool CALIB, bool OUT_F16, bool PER_T>
__global__ void __launch_bounds__(CP_MAX_THREADS) combine_pair_kernel(
    const int8_t* __restrict__ streams, const int* __restrict__ shifts,
    const float* __restrict__ scales, const float* __restrict__ off_re,
    const float* __restrict__ off_im, void* __restrict__ out, int G, int t_stream, int N, int n_f,
    int n_t, int t_lo, int fftshift, float prescale) {
  extern __shared__ __align__(16) uint8_t cp_smem[];
  __shared__ size_t s_off[CP_G];
  __shared__ float s_cal[3][CALIB ? CP_G : 1];
  __shared__ int s_n;
  int* acc_s = reinterpret_cast<int*>(cp_smem);   // [row u, row N - u][re, im][N], int or float
  const int f = blockIdx.x % n_f, u = blockIdx.x / n_f;   // u in [0, N/2]
  const int um = (N - u) % N;
  const int t = blockIdx.y, ta = t + t_lo;
  const int nw4 = N / 4, nh = N / 2 + 1;
  const int n_rows = um == u ? 1 : 2;
  const size_t nsq = (size_t)N * N;
  const int* sh = shifts + (size_t)f * G;
  for (int gb = 0; gb < G; gb += CP_G) {
    // the chgroups that have this time, in order, with their planes' offsets
    // (warp 0), so that the loop below has only independent loads
    if (gb) __syncthreads();
    if (threadIdx.x < 32) {
      int n = 0;
      for (int g0 = gb; g0 < min(G, gb + CP_G); g0 += 32) {
        const int g = g0 + (int)threadIdx.x;
        const int ts = g < min(G, gb + CP_G) ? ta - __ldg(sh + g) : -1;
        const bool in = ts >= 0 && ts < t_stream;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) {
          const int i = n + __popc(m & ((1u << threadIdx.x) - 1u));
          s_off[i] = ((size_t)g * t_stream + ts) * 2 * nsq;
          if constexpr (CALIB) {
            const size_t gt = PER_T ? (size_t)g * t_stream + ts : (size_t)g;
            s_cal[0][i] = __ldg(scales + gt);
            s_cal[1][i] = __ldg(off_re + gt);
            s_cal[2][i] = __ldg(off_im + gt);
          }
        }
        n += __popc(m);
      }
      if (threadIdx.x == 0) s_n = n;
    }
    __syncthreads();
    const int n = s_n;
    for (int task = threadIdx.x; task < n_rows * 2 * nw4; task += blockDim.x) {
      const int w4 = task % nw4, part = (task / nw4) & 1, row = task / (2 * nw4);
      const int8_t* src = streams + (size_t)part * nsq + (size_t)(row ? um : u) * N + 4 * w4;
      int* dst = acc_s + (size_t)(row * 2 + part) * N + 4 * w4;
      if constexpr (!CALIB) {
        uint32_t lo = 0u, hi = 0u;
#pragma unroll 8
        for (int i = 0; i < n; ++i) {
          const uint32_t b = __ldg(reinterpret_cast<const uint32_t*>(src + s_off[i])) ^ 0x80808080u;
          lo += b & 0x00ff00ffu;
          hi += (b >> 8) & 0x00ff00ffu;
        }
        int4 q = make_int4((int)(lo & 0xffffu) - 128 * n, (int)(hi & 0xffffu) - 128 * n,
                           (int)(lo >> 16) - 128 * n, (int)(hi >> 16) - 128 * n);
        if (gb) {
          const int4 o = *reinterpret_cast<const int4*>(dst);
          q = make_int4(q.x + o.x, q.y + o.y, q.z + o.z, q.w + o.w);
        }
        *reinterpret_cast<int4*>(dst) = q;
      } else {
        float a[4] = {0.f, 0.f, 0.f, 0.f};
        if (gb) {
          const float4 o = *reinterpret_cast<const float4*>(dst);
          a[0] = o.x; a[1] = o.y; a[2] = o.z; a[3] = o.w;
        }
#pragma unroll 4
        for (int i = 0; i < n; ++i) {
          const uint32_t b = __ldg(reinterpret_cast<const uint32_t*>(src + s_off[i]));
          const float sc = s_cal[0][i], of = s_cal[1 + part][i];
#pragma unroll
          for (int k = 0; k < 4; ++k)
            a[k] = fmaf(sc, (float)(int8_t)(uint8_t)(b >> (8 * k)), a[k]) + of;
        }
        *reinterpret_cast<float4*>(dst) = make_float4(a[0], a[1], a[2], a[3]);
      }
    }
  }
  __syncthreads();
  const size_t o0 = ((size_t)f * n_t + t) * N * nh;
  for (int i = threadIdx.x; i < n_rows * nh; i += blockDim.x) {
    const int row = i / nh, w = i % nh;
    const int ur = row ? um : u, wm = w ? N - w : 0;
    const int* d = acc_s + (size_t)(row * 2) * N;                        // this row
    const int* m = acc_s + (size_t)((n_rows == 1 ? 0 : 1 - row) * 2) * N;  // its mirror
    float o_re, o_im;
    if constexpr (!CALIB) {
      o_re = 0.5f * (float)(d[w] + m[wm]);
      o_im = 0.5f * (float)(d[N + w] - m[N + wm]);
    } else {
      o_re = 0.5f * (__int_as_float(d[w]) + __int_as_float(m[wm]));
      o_im = 0.5f * (__int_as_float(d[N + w]) - __int_as_float(m[N + wm]));
    }
    if (fftshift && ((ur + w) & 1)) {
      o_re = -o_re;
      o_im = -o_im;
    }
    o_re *= prescale;
    o_im *= prescale;
    const size_t o = o0 + (size_t)ur * nh + w;
    if (OUT_F16)
      reinterpret_cast<__half2*>(out)[o] = __floats2half2_rn(o_re, o_im);
    else
      reinterpret_cast<float2*>(out)[o] = make_float2(o_re, o_im);
  }
}

// Whether combine_pair_kernel can take the streams: whole 4-byte words of cells
// in every row (other shapes run one cell per thread above).
bool combine_pair_ok(const void* streams, int N, int n_t) {
  return N % 4 == 0 && N <= 8192 && n_t <= 65535 &&
         (reinterpret_cast<uintptr_t>(streams) & 3) == 0;
}

// Whether it should, for one fine DM.  Its lists, shared sums and barriers cost
// about what four chgroups' loads do, so that few chgroups are faster one cell
// per thread, more of them where that kernel has a float chain to hide its
// byte loads behind: 64 times of 256^2 uncalibrated 23.9 and 25.0 us at one
// chgroup, 28.6 and 25.9 at two; calibrated 22.8 and 26.8 at two, 28.5 and
// 27.1 at three; 16 times of 512^2 calibrated 25.2 and 27.5 at four, 38.3 and
// 33.3 at six; and as many where its CTAs leave SMs idle (2 times of 64^2 at
// three: 2.6 and 2.9).
bool combine_pair_better(bool calib, int G, int N, int n_t) {
  if ((long long)(N / 2 + 1) * n_t < 128) return G >= 5;
  return G >= (!calib ? 2 : N <= 256 ? 3 : 5);
}

int launch_combine_pair(const int8_t* streams, const int* shifts, const float* scales,
                        const float* off_re, const float* off_im, int per_t, void* out,
                        int out_f16, int G, int t_stream, int N, int n_f, int n_t, int t_lo,
                        int fftshift, float prescale, cudaStream_t stream) {
  const long long bx = (long long)(N / 2 + 1) * n_f;
  if (bx > 0x7fffffffLL || n_t > 65535) return DSB_E_ARG;
  const int threads = std::min(CP_MAX_THREADS, (N + 31) / 32 * 32);
  const size_t smem = (size_t)4 * N * 4;
  auto go = [&](auto kern) {
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess)
      return DSB_E_CUDA;
    kern<<<dim3((unsigned)bx, n_t), threads, smem, stream>>>(
        streams, shifts, scales, off_re, off_im, out, G, t_stream, N, n_f, n_t, t_lo, fftshift,
        prescale);
    return cudaGetLastError() == cudaSuccess ? DSB_OK : DSB_E_CUDA;
  };
  if (!scales)
    return out_f16 ? go(combine_pair_kernel<false, true, false>)
                   : go(combine_pair_kernel<false, false, false>);
  if (per_t)
    return out_f16 ? go(combine_pair_kernel<true, true, true>)
                   : go(combine_pair_kernel<true, false, true>);
  return out_f16 ? go(combine_pair_kernel<true, true, false>)
                 : go(combine_pair_kernel<true, false, false>);
}

// ===========================================================================
// image mask / normalise into the detector cube layout
//   cube[t, f, h, w] = img[f, t, h, w] * mask_f[f, h, w]
// ===========================================================================
template <bool OUT_F16>
__global__ void mask_to_cube_kernel(const float* __restrict__ img, const float* __restrict__ mask,
                                    int mask_per_f, int n_f, int n_t, int npix,
                                    void* __restrict__ cube, int cube_f_total, int cube_f0) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)n_f * n_t * npix;
  if (idx >= total) return;
  const int p = (int)(idx % npix);
  const long long r = idx / npix;
  const int t = (int)(r % n_t), f = (int)(r / n_t);
  const float m = mask[(mask_per_f ? (long long)f * npix : 0) + p];
  const float v = img[idx] * m;
  const long long o = ((long long)t * cube_f_total + cube_f0 + f) * npix + p;
  if (OUT_F16)
    reinterpret_cast<__half*>(cube)[o] = __float2half_rn(v);
  else
    reinterpret_cast<float*>(cube)[o] = v;
}

// ===========================================================================
// Compact-layout combine (combine_sparse_v4 + build_sparse_cell_csr,
// image/tiled_combine_cuda.py:966-1060, 1092-1240): streams in the
// time-minor compact layout dense[g][k][t][re, im] int8 (k a pattern cell of
// stream g), a CSR over the active half cells (u, w <= N/2) listing every
// stream g that carries the cell (k) or its mirror (km), -1 where absent.
// out[f][out_row0 + t][u][w] = 0.5 (sum_g q(k) + conj q(km)) at stream time
// t + t_lo - shift[f][g] (zero outside [0, t_rows)), times (-1)^(u+w) when
// fftshift; int32 sums, so exact; fp16 pairs or complex64.  Only active
// cells are written.
//
// Two forms.  A cell at a time (sparse_cell): the cell's entries in shared
// memory, a thread per (fine DM, time) with 2-byte gathers along the time.
//
// Staged (combine_sparse_kernel): a CTA takes 32 or 16 consecutive active
// cells and a tile of CS_T output times for every fine DM.  Each stream row
// (cell k or mirror km of one stream) is staged once in shared memory, the
// tile's times plus the spread of all shifts, zero outside [0, t_rows); a lane
// then owns a cell and sums 8 times at a time, two samples per word (re and im
// bytes offset to unsigned in 16-bit lanes), and a warp's stores go to
// consecutive active cells.  16 fine DMs x 64 times of 28.6k half cells: 380 us
// a cell at a time, 228 us with 32 cells per CTA, 196 us with 16.
// Cells whose rows do not fit together run in groups of 16, 8, ... 1.
//
// The staged form's set-up (shift range, row lists, window) and its few CTAs
// pay only where many outputs share them: 381 cells x 8 fine DMs x 64 times
// take 5.2 us a cell at a time and 6.4 us staged (30 us with 32 cells per
// CTA), 1581 cells 10 and 12 us.  But a CTA per cell costs some 1.5 us per
// thousand cells (16k cells x 4 x 16 times: 26 us, staged 17), so calls of at
// most CS_CELL_MAX cells (times their time tiles) and CS_CELL_OUT outputs go a
// cell at a time.  So does a CTA
// whose windows hold more words than twice the outputs per row (only the
// device knows the shifts), on cells a grid apart, so that those that run
// together write the same sectors: 484 us for 16 fine DMs with shifts spread
// over 3000 times, staged 787 (combine_cell_kernel's fuller SMs take 359).
// ===========================================================================
constexpr int CS_T = 64;
constexpr int CS_MAXE = 64;
constexpr int CS_CELLS = 32;
constexpr int CS_THREADS = 128;
constexpr int CS_WORDS = 10240;                 // staged words (two samples each) of 32 cells
constexpr int CS_ROWS = CS_WORDS / (CS_T / 2);  // most rows of a group
constexpr int CS_CELL_THREADS = 256;
constexpr long long CS_CELL_MAX = 2048, CS_CELL_OUT = 1 << 20;

struct SparseArgs {
  const int16_t* dense;
  const int *cell_uw, *cell_ptr, *ent_g, *ent_k, *ent_km, *shifts;
  void* out;
  int n_act, cpc, words;   // active cells; cells per CTA and staged words of the staged form
  int n_sb, t_rows, t_pad, nfm, N, n_fdm, t_out_len, t_lo, fftshift, out_rows, out_row0;
  int* status;
};
DSB_DEV bool sparse_entry_ok(const SparseArgs& A, int g, int k, int km) {
  return g >= 0 && g < A.n_sb && k < A.nfm && km < A.nfm;
}

template <bool OUT_F16>
DSB_DEV void sparse_put(void* out, long long o, float re, float im, bool flip) {
  if (flip) {
    re = -re;
    im = -im;
  }
  if (OUT_F16)
    reinterpret_cast<__half2*>(out)[o] = __floats2half2_rn(re, im);
  else
    reinterpret_cast<float2*>(out)[o] = make_float2(re, im);
}

// Cell a at output times t0 .. t0 + nt - 1 for every fine DM, by the NT threads
// of the CTA.  s_ent: 3 * CS_MAXE ints.
template <bool OUT_F16, int NT>
DSB_DEV void sparse_cell(const SparseArgs& A, int a, int t0, int nt, int* s_ent) {
  const int e0 = A.cell_ptr[a], ne = A.cell_ptr[a + 1] - e0;
  if (ne > CS_MAXE || ne < 0) {
    if (threadIdx.x == 0) dsb_flag(A.status, DSB_E_CAPACITY);
    return;
  }
  for (int e = threadIdx.x; e < ne; e += NT) {
    const int g = A.ent_g[e0 + e], k = A.ent_k[e0 + e], km = A.ent_km[e0 + e];
    const bool ok = sparse_entry_ok(A, g, k, km);
    s_ent[3 * e] = ok ? g : -1;
    s_ent[3 * e + 1] = k;
    s_ent[3 * e + 2] = km;
    if (!ok) dsb_flag(A.status, DSB_E_ARG);
  }
  __syncthreads();
  const int nh = A.N / 2 + 1, uw = A.cell_uw[a];
  const bool flip = A.fftshift && ((uw / nh + uw % nh) & 1);
  for (int idx = threadIdx.x; idx < A.n_fdm * CS_T; idx += NT) {
    const int f = idx / CS_T, tl = idx % CS_T;
    if (tl >= nt) continue;
    const int t = t0 + tl;
    int re = 0, im = 0;
    for (int e = 0; e < ne; ++e) {
      const int g = s_ent[3 * e], k = s_ent[3 * e + 1], km = s_ent[3 * e + 2];
      if (g < 0) continue;
      const int ts = t + A.t_lo - A.shifts[f * A.n_sb + g];
      if (ts < 0 || ts >= A.t_rows) continue;
      const long long row = (long long)g * A.nfm;
      if (k >= 0) {
        const int16_t v = __ldg(A.dense + (row + k) * A.t_pad + ts);
        re += (int)(int8_t)(v & 0xff);
        im += (int)(int8_t)((v >> 8) & 0xff);
      }
      if (km >= 0) {
        const int16_t v = __ldg(A.dense + (row + km) * A.t_pad + ts);
        re += (int)(int8_t)(v & 0xff);
        im -= (int)(int8_t)((v >> 8) & 0xff);
      }
    }
    sparse_put<OUT_F16>(A.out, ((long long)f * A.out_rows + A.out_row0 + t) * A.N * nh + uw,
                        0.5f * (float)re, 0.5f * (float)im, flip);
  }
}

template <bool OUT_F16>
__global__ void __launch_bounds__(CS_CELL_THREADS) combine_cell_kernel(const SparseArgs A) {
  __shared__ int s_ent[3 * CS_MAXE];
  const int t0 = blockIdx.y * CS_T;
  sparse_cell<OUT_F16, CS_CELL_THREADS>(A, blockIdx.x, t0, min(CS_T, A.t_out_len - t0), s_ent);
}

template <bool OUT_F16>
__global__ void __launch_bounds__(CS_THREADS) combine_sparse_kernel(const SparseArgs A) {
  extern __shared__ uint32_t s_win[];              // [A.words]
  __shared__ long long s_row[CS_ROWS];             // stream row of each staged row
  __shared__ int s_rowg[CS_ROWS];                  // its stream
  __shared__ int s_ptr[CS_CELLS], s_ne[CS_CELLS], s_r0[CS_CELLS + 1], s_rm[CS_CELLS];
  __shared__ int s_min, s_max, s_group;
  const int16_t* dense = A.dense;
  const int *cell_uw = A.cell_uw, *cell_ptr = A.cell_ptr, *ent_g = A.ent_g, *ent_k = A.ent_k,
            *ent_km = A.ent_km, *shifts = A.shifts;
  void* out = A.out;
  const int n_sb = A.n_sb, t_rows = A.t_rows, t_pad = A.t_pad, nfm = A.nfm, N = A.N,
            n_fdm = A.n_fdm, t_lo = A.t_lo, fftshift = A.fftshift, out_rows = A.out_rows,
            out_row0 = A.out_row0;
  int* status = A.status;
  // the streams as aligned words of two samples
  const int dense_off = (int)((reinterpret_cast<uintptr_t>(dense) >> 1) & 1);
  const uint32_t* dense2 = reinterpret_cast<const uint32_t*>(dense - dense_off);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int a0 = blockIdx.x * A.cpc, nc = min(A.cpc, A.n_act - a0);
  const int t0 = blockIdx.y * CS_T, nt = min(CS_T, A.t_out_len - t0);
  const int nh = N / 2 + 1;
  if (tid == 0) {
    s_min = 0x7fffffff;
    s_max = -0x7fffffff - 1;
  }
  __syncthreads();
  int lo = 0x7fffffff, hi = -0x7fffffff - 1;
  for (int i = tid; i < n_fdm * n_sb; i += CS_THREADS) {
    const int v = __ldg(shifts + i);
    lo = min(lo, v);
    hi = max(hi, v);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) {
    atomicMin(&s_min, lo);
    atomicMax(&s_max, hi);
  }
  __syncthreads();
  const int sh_max = s_max;
  const long long spread = (long long)sh_max - s_min;
  // words of a row: the tile's times at every shift, one more for odd starts,
  // odd so that lanes on different rows spread over the banks
  const int pitch = spread > 2 * CS_WORDS ? 0 : (int)((CS_T + spread + 1) / 2 + 1) | 1;
  const int cap = pitch && pitch <= 2LL * n_fdm * nt
                      ? min(CS_ROWS, A.words / pitch) : 0;
  auto entry_ok = [&](int g, int k, int km) { return sparse_entry_ok(A, g, k, km); };
  if (warp == 0) {
    // this lane's cell: its entries and rows (k rows and km rows)
    int ptr = 0, ne = 0, rows = 0;
    if (lane < nc) {
      ptr = cell_ptr[a0 + lane];
      ne = cell_ptr[a0 + lane + 1] - ptr;
      if (ne > CS_MAXE || ne < 0) {
        dsb_flag(status, DSB_E_CAPACITY);
        ne = -1;
      }
      for (int e = 0; e < ne; ++e) {
        const int g = ent_g[ptr + e], k = ent_k[ptr + e], km = ent_km[ptr + e];
        if (entry_ok(g, k, km)) rows += (k >= 0) + (km >= 0);
        else dsb_flag(status, DSB_E_ARG);
      }
    }
    s_ptr[lane] = ptr;
    s_ne[lane] = ne;
    int inc = rows;   // inclusive prefix
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    s_r0[lane + 1] = inc;
    if (lane == 0) s_r0[0] = 0;
    // the largest group of cells whose rows always fit
    int group = 0, sum = rows;
#pragma unroll
    for (int g = 1; g <= 32; g *= 2) {
      if (g <= A.cpc && (int)__reduce_max_sync(0xffffffffu, sum) <= cap) group = g;
      sum += __shfl_xor_sync(0xffffffffu, sum, g);
    }
    if (lane == 0) s_group = group;
  }
  __syncthreads();
  // (the rule of a group is the CTA's own, that of the windows the whole
  // grid's: only then may the cells be dealt out anew)
  const bool wide = cap == 0;
  const int group = s_group;
  if (group == 0) {
    int* s_ent = reinterpret_cast<int*>(s_win);
    for (int i = 0; i < nc || (wide && i < A.cpc); ++i) {
      const int a = wide ? (int)blockIdx.x + i * (int)gridDim.x : a0 + i;
      if (a >= A.n_act) break;
      sparse_cell<OUT_F16, CS_THREADS>(A, a, t0, nt, s_ent);
      __syncthreads();   // the entries' places are the next cell's
    }
    return;
  }
  const int base_t = t0 + t_lo - sh_max;   // stream time of a window's first sample
  const int n_t8 = (nt + 7) / 8, n_task = n_fdm * n_t8;
  for (int cb = 0; cb < nc; cb += group) {
    const int rb = s_r0[cb], n_rows = s_r0[min(cb + group, nc)] - rb;
    // the group's rows, each cell's k rows before its km rows
    for (int c = cb + warp; c < min(cb + group, nc); c += CS_THREADS / 32) {
      const int p = s_ptr[c], ne = s_ne[c];
      int at = s_r0[c] - rb;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        if (m == 1 && lane == 0) s_rm[c] = at;
        for (int e0 = 0; e0 < ne; e0 += 32) {
          const int e = e0 + lane;
          int g = -1, k = -1, km = -1;
          if (e < ne) {
            g = ent_g[p + e];
            k = ent_k[p + e];
            km = ent_km[p + e];
            if (!entry_ok(g, k, km)) k = km = -1;
          }
          const int x = m ? km : k;
          const unsigned has = __ballot_sync(0xffffffffu, x >= 0);
          if (x >= 0) {
            const int r = at + __popc(has & ((1u << lane) - 1u));
            s_row[r] = (long long)g * nfm + x;
            s_rowg[r] = g;
          }
          at += __popc(has);
        }
      }
    }
    __syncthreads();
    for (int r = warp; r < n_rows; r += CS_THREADS / 32) {
      // two samples per aligned word, shifted to the window's start; words
      // that hold no sample of the row are not read
      const long long e0 = s_row[r] * t_pad + base_t + dense_off;   // first sample, from dense2
      const uint32_t* p = dense2 + (e0 >> 1);
      const unsigned sh = (unsigned)(e0 & 1) * 16u;
      const int odd = (int)(e0 & 1);
      for (int j = lane; j < pitch; j += 32) {
        const int ts = base_t + 2 * j;   // the word's samples ts, ts + 1
        auto word = [&](int i) {         // samples ts - odd + 2 i, + 1
          const int a = ts - odd + 2 * i;
          return (a >= 0 && a < t_rows) || (a + 1 >= 0 && a + 1 < t_rows) ? __ldg(p + j + i) : 0u;
        };
        uint32_t w = __funnelshift_r(word(0), odd ? word(1) : 0u, sh);
        if (ts < 0 || ts >= t_rows) w &= 0xffff0000u;
        if (ts + 1 < 0 || ts + 1 >= t_rows) w &= 0x0000ffffu;
        s_win[r * pitch + j] = w ^ 0x80808080u;
      }
    }
    __syncthreads();
    // lane = cell (lane mod group), the rest of the lanes and the warps take
    // the (fine DM, 8 times) tasks
    const int per_warp = 32 / group;
    const int c = cb + lane % group;
    const bool live = c < nc && s_ne[c < nc ? c : 0] >= 0;
    const int uw = live ? cell_uw[a0 + c] : 0;
    const bool flip = fftshift && ((uw / nh + uw % nh) & 1);
    const int r0 = live ? s_r0[c] - rb : 0, rm = live ? s_rm[c] : 0, r1 = live ? s_r0[c + 1] - rb : 0;
    const int nk = rm - r0, nm = r1 - rm;
    for (int task = warp * per_warp + lane / group; task < n_task;
         task += CS_THREADS / 32 * per_warp) {
      if (!live) continue;
      const int f = task / n_t8, o = task % n_t8;
      const int* shf = shifts + f * n_sb;
      uint32_t re[4] = {0u, 0u, 0u, 0u}, im[4] = {0u, 0u, 0u, 0u}, mi[4] = {0u, 0u, 0u, 0u};
      auto row8 = [&](int r, uint32_t (&b)[4]) {
        const int x = 8 * o + sh_max - __ldg(shf + s_rowg[r]);
        const uint32_t* w = s_win + r * pitch + (x >> 1);
        const uint32_t w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3], w4 = w[4];
        const unsigned s = (x & 1) * 16;
        b[0] = __funnelshift_r(w0, w1, s);
        b[1] = __funnelshift_r(w1, w2, s);
        b[2] = __funnelshift_r(w2, w3, s);
        b[3] = __funnelshift_r(w3, w4, s);
      };
      for (int r = r0; r < rm; ++r) {
        uint32_t b[4];
        row8(r, b);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          re[i] += b[i] & 0x00ff00ffu;
          im[i] += (b[i] >> 8) & 0x00ff00ffu;
        }
      }
      for (int r = rm; r < r1; ++r) {
        uint32_t b[4];
        row8(r, b);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          re[i] += b[i] & 0x00ff00ffu;
          mi[i] += (b[i] >> 8) & 0x00ff00ffu;
        }
      }
      const long long o0 = ((long long)f * out_rows + out_row0 + t0 + 8 * o) * N * nh + uw;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (8 * o + j >= nt) break;
        const int h = 16 * (j & 1);
        const int vr = (int)((re[j >> 1] >> h) & 0xffffu) - 128 * (nk + nm);
        const int vi = (int)((im[j >> 1] >> h) & 0xffffu) - 128 * nk -
                       ((int)((mi[j >> 1] >> h) & 0xffffu) - 128 * nm);
        sparse_put<OUT_F16>(out, o0 + (long long)j * N * nh, 0.5f * (float)vr, 0.5f * (float)vi,
                            flip);
      }
    }
    __syncthreads();   // the next group reuses the window
  }
}

// Whether two tables differ: each read once, 16 bytes per access where both
// start on that boundary (n16 words; the rest by bytes).
__global__ void __launch_bounds__(256) tables_differ_kernel(const uint8_t* __restrict__ a,
                                                            const uint8_t* __restrict__ b,
                                                            long long n16, long long n_bytes,
                                                            int* __restrict__ differ) {
  const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long step = (long long)gridDim.x * blockDim.x;
  uint32_t d = 0u;
#pragma unroll 4
  for (long long i = i0; i < n16; i += step) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(a) + i);
    const uint4 y = __ldg(reinterpret_cast<const uint4*>(b) + i);
    d |= (x.x ^ y.x) | (x.y ^ y.y) | (x.z ^ y.z) | (x.w ^ y.w);
  }
  for (long long i = 16 * n16 + i0; i < n_bytes; i += step) d |= (uint32_t)(a[i] ^ b[i]);
  if (d) *differ = 1;
}

// ===========================================================================
// padded cumsum / boxcars (detector/forward.py:250-455,
// detector/triton_boxcar.py:47-360).  Each prefix is accumulated in float64
// and rounded once to float32.
// ===========================================================================
template <typename T>
DSB_DEV float ldf(const T* p, long long i);
template <>
DSB_DEV float ldf<float>(const float* p, long long i) { return p[i]; }
template <>
DSB_DEV float ldf<__half>(const __half* p, long long i) { return __half2float(p[i]); }

template <typename T>
__global__ void padded_cumsum_kernel(const T* __restrict__ x, int n, long long inner, int max_w,
                                     float* __restrict__ cs) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= inner) return;
  const int pl = max_w / 2, pr = max_w - 1 - pl;
  for (int j = 0; j <= pl; ++j) cs[(long long)j * inner + e] = 0.f;
  double run = 0.0;
  float last = 0.f;
  for (int i = 0; i < n; ++i) {
    run += (double)ldf<T>(x, (long long)i * inner + e);
    last = (float)run;
    cs[(long long)(1 + pl + i) * inner + e] = last;
  }
  for (int r = 0; r < pr; ++r) cs[(long long)(1 + pl + n + r) * inner + e] = last;
}

// A CTA walks tt consecutive outputs (BA_T in calls that fill the chip) of
// V x 128 adjacent cells, V cells per thread and access: the prefix rows of one output are the next ones' too, so
// all but the first touch of a row come from L1, and what bounds the kernel
// is the L1 rate of its 2 K loads per output (then memory: every prefix read
// and 6 to 8 bytes written once).  One output per thread, with two 64-bit
// divisions and 2 K 4-byte loads from L2 each, took 309 us for 128 outputs of
// 4 x 256^2 cells at boxcars 1..16; this takes 95 us (tiles of 4, 16, 32 and 64
// times: 100, 108, 123, 120).  Small calls take shorter tiles, down to one
// output, while there are fewer than eight CTAs per SM, and one cell per
// thread below one: 16 outputs of 64^2 cells 2.4 us (6.6 in tiles of 8), 64 of
// 100^2 4.4 (9.3).
//
// CHECK: every prefix row read must lie in [0, cs_rows); an output whose
// widths / offsets would read outside gets S/N NaN and winner -1 instead
// (the rows outside belong to no call's data: the shared scratch array of
// dsb_boxcar_argmax_noalloc).
constexpr int BA_THREADS = 128, BA_T = 8, BA_MAX_K = 32;

template <int V, bool OUT_F16, bool CHECK>
__global__ void __launch_bounds__(BA_THREADS) multi_boxcar_argmax_kernel(
    const float* __restrict__ cs, long long inner, const int* __restrict__ widths,
    const int* __restrict__ offsets, const float* __restrict__ sinv, int K, int n_out, int t_base,
    void* __restrict__ out_max, int16_t* __restrict__ out_win, long long cs_rows, int n_tt, int tt) {
  // each width's first and last row relative to the output's, as offsets into
  // cs, and its scale
  __shared__ longlong2 s_off[BA_MAX_K];
  __shared__ float s_si[BA_MAX_K];
  const bool tab = K <= BA_MAX_K;   // longer lists are read in place
  if (tab && (int)threadIdx.x < K) {
    const long long lo = offsets[threadIdx.x];
    s_off[threadIdx.x] = make_longlong2(lo * inner, (lo + widths[threadIdx.x]) * inner);
    s_si[threadIdx.x] = sinv[threadIdx.x];
  }
  __syncthreads();
  // time tiles fastest: the CTAs that run together share rows in L2
  const long long e = ((long long)(blockIdx.x / n_tt) * BA_THREADS + threadIdx.x) * V;
  const int t0 = (int)(blockIdx.x % n_tt) * tt, t1 = min(n_out, t0 + tt);
  if (e >= inner) return;
  using VT = typename std::conditional<V == 4, float4, float>::type;
  for (int t = t0; t < t1; ++t) {
    const long long ta = (long long)t + t_base;
    const float* row = cs + ta * inner + e;
    float best[V];
    int win[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      best[v] = 0.f;
      win[v] = 0;
    }
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
      if constexpr (CHECK) {
        const long long lo = ta + offsets[k], hi = lo + widths[k];
        if (lo < 0 || hi < 0 || lo >= cs_rows || hi >= cs_rows) {
#pragma unroll
          for (int v = 0; v < V; ++v) {
            best[v] = __int_as_float(0x7fc00000);
            win[v] = -1;
          }
          break;
        }
      }
      const longlong2 o = tab ? s_off[k]
                              : make_longlong2(offsets[k] * inner,
                                               ((long long)offsets[k] + widths[k]) * inner);
      const VT h4 = *reinterpret_cast<const VT*>(row + o.y);
      const VT l4 = *reinterpret_cast<const VT*>(row + o.x);
      const float* h = reinterpret_cast<const float*>(&h4);
      const float* l = reinterpret_cast<const float*>(&l4);
      const float si = tab ? s_si[k] : sinv[k];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const float s = (h[v] - l[v]) * si;
        if (k == 0 || s > best[v]) {
          best[v] = s;
          win[v] = k;
        }
      }
    }
    const long long o = (long long)t * inner + e;
    if constexpr (V == 4) {
      if (OUT_F16) {
        __half2 a = __floats2half2_rn(best[0], best[1]), b = __floats2half2_rn(best[2], best[3]);
        *reinterpret_cast<uint2*>(static_cast<__half*>(out_max) + o) =
            make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
      } else {
        *reinterpret_cast<float4*>(static_cast<float*>(out_max) + o) =
            make_float4(best[0], best[1], best[2], best[3]);
      }
      *reinterpret_cast<short4*>(out_win + o) =
          make_short4((short)win[0], (short)win[1], (short)win[2], (short)win[3]);
    } else {
      if (OUT_F16)
        static_cast<__half*>(out_max)[o] = __float2half_rn(best[0]);
      else
        static_cast<float*>(out_max)[o] = best[0];
      out_win[o] = (int16_t)win[0];
    }
  }
}

// Launch on any shape: four cells per access where the rows of every array
// start on that boundary.
template <bool CHECK>
int launch_argmax(const float* cs, long long inner, const int* widths, const int* offsets,
                  const float* sinv, int K, int n_out, int t_base, void* out_max, int out_f16,
                  int16_t* out_win, long long cs_rows, cudaStream_t stream) {
  const bool aligned = inner % 4 == 0 && (reinterpret_cast<uintptr_t>(cs) % 16) == 0 &&
                    (reinterpret_cast<uintptr_t>(out_max) % (out_f16 ? 8 : 16)) == 0 &&
                    (reinterpret_cast<uintptr_t>(out_win) % 8) == 0;
  // shorter time tiles, then one cell per thread, while the CTAs leave SMs idle
  auto n_blocks = [&](int v, int tt) {
    const long long per = (long long)BA_THREADS * v;
    return (inner + per - 1) / per * ((n_out + tt - 1) / tt);
  };
  int tt = BA_T;
  while (tt > 1 && n_blocks(aligned ? 4 : 1, tt) < 148 * 8) tt /= 2;
  const bool four = aligned && n_blocks(4, tt) >= 148;
  const int n_tt = (n_out + tt - 1) / tt;
  const long long blocks = n_blocks(four ? 4 : 1, tt);
  if (blocks > 0x7fffffffLL) return DSB_E_ARG;
  auto go = [&](auto kern) {
    kern<<<(unsigned)blocks, BA_THREADS, 0, stream>>>(cs, inner, widths, offsets, sinv, K, n_out,
                                                      t_base, out_max, out_win, cs_rows, n_tt, tt);
    return cudaGetLastError() == cudaSuccess ? DSB_OK : DSB_E_CUDA;
  };
  if (four) return out_f16 ? go(multi_boxcar_argmax_kernel<4, true, CHECK>)
                           : go(multi_boxcar_argmax_kernel<4, false, CHECK>);
  return out_f16 ? go(multi_boxcar_argmax_kernel<1, true, CHECK>)
                 : go(multi_boxcar_argmax_kernel<1, false, CHECK>);
}

__global__ void boxcar_from_cs_kernel(const float* __restrict__ cs, long long inner, int width,
                                      int start, int n_out, float* __restrict__ out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n_out * inner) return;
  const int t = (int)(idx / inner);
  const long long e = idx % inner;
  out[idx] = cs[(long long)(start + t + width) * inner + e] - cs[(long long)(start + t) * inner + e];
}

// ===========================================================================
// Fused streaming detector: per pixel, float64 running prefix rounded to
// float32 (identical to the padded cumsum above), a register ring of the
// last MAXW+1 prefixes, boxcar widths 1, 2, 4, ..., MAXW (centred, offsets
// MAXW/2 - w/2), S/N = (hi - lo) * sinv[k], strict '>' over k, and
// compaction of every output cell above threshold.
// ===========================================================================
struct DetCand {
  int t;      // output index (t_abs - t_base)
  int pix;    // (f * H + h) * W + w inside the cube
  float snr;
  int k;
};

// Element e = f * npix + p of time t is read at x[f*f_stride + t*t_stride + p]
// and multiplied by mask[f*npix + p] when a mask is given (the per-fine-DM
// edge mask x 1/sigma), so the detector consumes the FFT output directly.
// Layer-2 score samples (noise_norm/layer2.py, the streaming detector's
// per-kernel subsample, detector/forward.py:1425-1530): entries {eg, t, k,
// slot} sorted by (eg, t), eg = e + pix_off the cell's index over all fine
// DMs, t the output index (ta - t_base); off[gb] the first entry of global
// 256-cell block gb.  Each entry's raw boxcar sum of width 2^k (before the
// 1/sigma_k scale) goes to out[k * m + slot].  out == null: no sampling.
struct L2Samples {
  const int* off;
  const int4* ent;
  float* out;
  int m;
};

DSB_DEV float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// The K boxcar sums (widths 1, 2, ..., 2^(K-1)) of one output, before the
// 1/sigma_k scale.
template <int K>
struct BoxSums {
  float v[K];
};

// Saturation level of the detector's candidate count (capacities are below it).
constexpr int DET_COUNT_MAX = 1 << 30;

// Exact strict-'>' winner over the widths (the lowest k wins ties) and, when
// its S/N passes thr, one appended candidate.  Out of line: called only for
// outputs the screen lets through.
template <int K>
__device__ __noinline__ void det_emit(const BoxSums<K> d, const float* __restrict__ sinv,
                                      float thr, int t_out, int pix,
                                      DetCand* __restrict__ cands, int cap,
                                      int* __restrict__ count) {
  float best = 0.f;
  int win = 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float s = d.v[k] * __ldg(sinv + k);
    if (k == 0 || s > best) {
      best = s;
      win = k;
    }
  }
  if (best > thr) {
    // count[0] stops growing near DET_COUNT_MAX (above any capacity) instead
    // of wrapping to negative slots when nearly every cell passes: once the
    // buffer is full only the count's current value is read, and it is
    // raised while below the saturation level (concurrent raises overshoot
    // it by at most the resident threads)
    int slot = __ldcg(count);
    if (slot < cap)
      slot = atomicAdd(count, 1);
    else if (slot < DET_COUNT_MAX)
      atomicAdd(count, 1);
    if (slot < cap)
      cands[slot] = DetCand{t_out, pix, best, win};
    else  // the largest S/N that did not fit (positive floats order as ints)
      atomicMax(count + 1, __float_as_int(best));
  }
}

// Every Layer-2 entry of (cell eg, output t_out) from entry s_i on: the raw
// boxcar of its width into its slot.  Returns the next entry and its output
// time (0x7fffffff when this cell has no more).
template <int K>
__device__ __noinline__ int2 det_sample(const BoxSums<K> d, const L2Samples l2, int s_i,
                                        int s_end, int eg, int t_out) {
  int s_t = t_out;
  while (s_t == t_out) {
    const int4 en = __ldg(&l2.ent[s_i]);
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (k == en.z) v = d.v[k];
    l2.out[(long long)en.z * l2.m + en.w] = v;
    ++s_i;
    s_t = (s_i < s_end && __ldg(&l2.ent[s_i].x) == eg) ? __ldg(&l2.ent[s_i].y) : 0x7fffffff;
  }
  return make_int2(s_i, s_t);
}

// One thread per cell; it marches the cell's time series once, keeping its
// last MAXW + 1 prefix sums in a register ring.  Time is walked in blocks of
// DB steps (unrolled; det_db): step j of a block writes its prefix to ring slot
// MAXW + j, and the block ends by moving the newest MAXW prefixes down to
// slots 0 .. MAXW-1 (MAXW register moves per DB steps), so the ring indices
// are compile-time constants while the unrolled code stays DB steps long.
// The inputs are prefetched DB steps ahead, one load per step.
// Boxcars to 32 or 64 (MAXW 32, 64): DB = 16 steps per block, inputs
// prefetched DP = 8 steps ahead (a rolling set of DP registers), so that ring
// and prefetch fit 128 registers: two CTAs per SM.  Narrower boxcars keep a
// short ring and run more CTAs per SM (three at 16: 80 registers, 16 steps
// per block; four below: 64 registers, 8 steps per block, 4 ahead), whose
// occupancy hides load latency better (at b16: 116 -> 96 ms per block of the
// 512-DM 256^2 workload against two CTAs per SM).
template <int LOGW>
struct DetCfg {
  // steps per block, prefetch depth, CTAs per SM (64 / 80 / 128 registers)
  static constexpr int DB = LOGW >= 4 ? 16 : 8;
  static constexpr int DP = LOGW >= 4 ? 8 : 4;
  static constexpr int MINB = LOGW >= 5 ? 2 : (LOGW == 4 ? 3 : 4);
};
constexpr int DET_PF = 32;  // L2 prefetch distance (steps)

DSB_DEV void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

template <int LOGW, typename T>
__global__ void __launch_bounds__(256, DetCfg<LOGW>::MINB) detect_kernel(const T* __restrict__ x, int n, int npix,
                                                     long long inner, long long f_stride,
                                                     long long t_stride,
                                                     const float* __restrict__ mask,
                                                     long long mask_f_stride,
                                                     const float* __restrict__ sig_f,
                                                     const float* __restrict__ sinv,
                                                     int t_base, int n_out, float thr,
                                                     DetCand* __restrict__ cands, int cap, int pix_off,
                                                     int* __restrict__ count, const L2Samples l2) {
  constexpr int MAXW = 1 << LOGW;
  constexpr int K = LOGW + 1;
  constexpr int PL = MAXW / 2;
  constexpr int DB = DetCfg<LOGW>::DB, DP = DetCfg<LOGW>::DP;
  constexpr int RS = MAXW + DB;  // ring registers
  static_assert(DB % DP == 0, "the prefetch set cycles within a block");
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= inner) return;
  // this cell's Layer-2 sample entries [s_i, s_end) (a few thousand per
  // kernel over the whole cube), s_t the output index of the next one
  int s_i = 0, s_end = 0, s_t = 0x7fffffff;
  const int eg = (int)e + pix_off;
  if (l2.out) {
    const int gb = pix_off / 256 + (int)blockIdx.x;
    int lo = __ldg(l2.off + gb);
    s_end = __ldg(l2.off + gb + 1);
    while (lo < s_end && __ldg(&l2.ent[lo].x) < eg) ++lo;
    s_i = lo;
    if (s_i < s_end && __ldg(&l2.ent[s_i].x) == eg) s_t = __ldg(&l2.ent[s_i].y);
  }
  const long long fidx = e / npix, p = e % npix;
  const T* cube = x + fidx * f_stride + p;
  // x * 1.0f == x exactly, so an absent mask costs one exact multiply
  float mval = mask ? mask[fidx * mask_f_stride + p] : 1.0f;
  if (sig_f) mval = mval / sig_f[fidx];
  float tau[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    // screen level of width k: a boxcar sum d can give fl(d * si) > thr only
    // if d > thr / si up to two roundings (2^-23 relative), so a level
    // lowered by 2^-20 of its magnitude never misses one
    const float lv = thr / sinv[k];
    tau[k] = lv - fabsf(lv) * 0x1p-20f;
  }
  // ring[i] holds prefix J0 - MAXW + i at the start of the block of steps
  // J0 .. J0 + DB - 1 (prefix index J: 0 for J <= PL, the running sum of
  // inputs 0 .. J-PL-1 up to J = PL + n, then the last sum: the padded
  // cumsum); the output of step J is ta = J - MAXW and reads ring slots
  // j .. j + MAXW
  float ring[RS];
#pragma unroll
  for (int q = 0; q < RS; ++q) ring[q] = 0.f;
  double run = 0.0;
  float last = 0.f;
  const int total = n + MAXW;  // cs length
  // One output: the screen compares each boxcar sum with its lowered level
  // (a superset of what the exact strict-'>' chain of det_emit reports,
  // which decides); the threshold hits and the Layer-2 samples are rare, so
  // both are calls out of the unrolled loop.
  auto output = [&](int j, int ta, auto with_samples) {
    BoxSums<K> d;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int w = 1 << k;
      const int off = PL - w / 2;
      d.v[k] = ring[j + off + w] - ring[j + off];
    }
    bool hit = false;
#pragma unroll
    for (int k = 0; k < K; ++k) hit |= d.v[k] > tau[k];
    if (hit) det_emit<K>(d, sinv, thr, ta - t_base, (int)e + pix_off, cands, cap, count);
    if (decltype(with_samples)::value && ta - t_base == s_t) {
      const int2 r = det_sample<K>(d, l2, s_i, s_end, eg, ta - t_base);
      s_i = r.x;
      s_t = r.y;
    }
  };
  // input of step J: x[J - 1 - PL] (for PL < J <= PL + n); xin[j % DP]
  // holds the input of step J0 + j, loaded DP steps earlier
  auto input = [&](int J) -> float {
    const int i = J - 1 - PL;
    return (i >= 0 && i < n) ? ldf<T>(cube, (long long)i * t_stride) : 0.f;
  };
  float xin[DP];
#pragma unroll
  for (int j = 0; j < DP; ++j) xin[j] = input(j);
  // the first steps produce no output (ta < t_base): prefixes only
  const int warm_end = t_base + MAXW;
  // blocks after the last output step (J = t_base + n_out - 1 + MAXW) feed
  // nothing: the cell is done
  const int out_end = t_base + n_out + MAXW;
  for (int J0 = 0; J0 < total && J0 < out_end; J0 += DB) {
    if (J0 + DB <= warm_end && J0 + DB + DP - 1 - PL <= n) {
#pragma unroll
      for (int j = 0; j < DB; ++j) {
        const int J = J0 + j;
        float v = 0.f;
        if (J > PL) {
          run += (double)(xin[j % DP] * mval);
          v = (float)run;
        }
        ring[MAXW + j] = v;
        xin[j % DP] = input(J + DP);
      }
      last = ring[MAXW + DB - 1];
    } else if (J0 >= PL + 1 && J0 + DB - 1 <= PL + n && J0 - MAXW >= t_base &&
               J0 + DB - 1 - MAXW < t_base + n_out && J0 + DB - 1 + DP - 1 - PL < n) {
      // steady state: every step an input, a prefix and an output, and the
      // prefetched input in range; the Layer-2 test only in the (rare)
      // blocks that hold this cell's next sample
      const T* nxt = cube + (long long)(J0 + DP - 1 - PL) * t_stride;
      // L2 prefetch DET_PF steps ahead, the block's DB lines in one
      // instruction: lane j < DB takes step J0 + j's line of the warp (lane
      // 0's cell), where still inside the cube
      // (lane 0's cell is always active when any lane of its warp is; the
      // branch is warp-uniform, so the warp's live lanes are all here)
      {
        const unsigned lane = threadIdx.x & 31;
        const long long n_live = inner - (e - lane);  // lanes of this warp with a cell
        const unsigned live = n_live >= 32 ? 0xffffffffu : ((1u << n_live) - 1u);
        const T* cube0 = reinterpret_cast<const T*>(
            __shfl_sync(live, reinterpret_cast<unsigned long long>(cube), 0));
        const int ipf = J0 + (int)lane + DET_PF - 1 - PL;
        if (lane < (unsigned)DB && ipf < n) prefetch_l2(cube0 + (long long)ipf * t_stride);
      }
      auto steady = [&](auto with_samples) {
#pragma unroll
        for (int j = 0; j < DB; ++j) {
          run += (double)(xin[j % DP] * mval);
          ring[MAXW + j] = (float)run;
          xin[j % DP] = ldf<T>(nxt, (long long)j * t_stride);
          output(j, J0 + j - MAXW, with_samples);
        }
      };
      if ((unsigned)(s_t - (J0 - MAXW - t_base)) < (unsigned)DB)
        steady(std::true_type{});
      else
        steady(std::false_type{});
      last = ring[MAXW + DB - 1];
    } else {
#pragma unroll
      for (int j = 0; j < DB; ++j) {
        const int J = J0 + j;
        if (J < total) {
          float v;
          if (J <= PL) {
            v = 0.f;
          } else if (J <= PL + n) {
            run += (double)(xin[j % DP] * mval);
            last = (float)run;
            v = last;
          } else {
            v = last;
          }
          ring[MAXW + j] = v;
          const int ta = J - MAXW;
          if (ta >= t_base && ta < t_base + n_out) output(j, ta, std::true_type{});
        }
        xin[j % DP] = input(J + DP);
      }
    }
#pragma unroll
    for (int q = 0; q < MAXW; ++q) ring[q] = ring[q + DB];
  }
}

// The same detector with the cube staged in shared memory by TMA (float
// cubes whose fine DMs are whole warps of cells: npix a multiple of 32).
// Each warp owns 32 consecutive cells of one fine DM and a ring of NST
// shared-memory stages, each one block of DB times x 32 cells (one 3-D tile
// of the cube's tensor map, completing on the stage's mbarrier).  Lane 0
// issues block b + NST - 1 when the warp starts block b, so the copies
// run NST - 1 blocks ahead with no registers held for them and no barrier
// wider than the warp; times outside [0, n) arrive as zeros.  The marching,
// the screen and the rare paths are detect_kernel's, so the outputs are the
// same bits.  A wait that does not complete within DSB_SPIN_LIMIT polls sets
// count[1] to a quiet NaN (DET_TIMEOUT_BITS) and ends the warp after waiting,
// again bounded, for its copies in flight.
constexpr int DET_TIMEOUT_BITS = 0x7fc00000;

// Steps per block and stages of the TMA form: with the inputs out of the
// registers, boxcars to 64 afford 32-step blocks (96 ring registers, half
// the ring moves per step) in three stages of 4 KB per warp; the narrower
// widths keep detect_kernel's blocks in four stages.
template <int LOGW>
struct DetTmaCfg {
  static constexpr int DB = LOGW == 6 ? 32 : DetCfg<LOGW>::DB;
  static constexpr int NST = LOGW == 6 ? 3 : 4;
};

template <int LOGW>
constexpr int det_tma_smem() {
  return 8 * DetTmaCfg<LOGW>::NST * DetTmaCfg<LOGW>::DB * 32 * 4 + 8 * DetTmaCfg<LOGW>::NST * 8;
}

template <int LOGW>
__global__ void __launch_bounds__(256, DetCfg<LOGW>::MINB)
    detect_tma_kernel(const __grid_constant__ CUtensorMap tmap, int n, int npix, long long inner,
                      const float* __restrict__ mask, long long mask_f_stride,
                      const float* __restrict__ sig_f, const float* __restrict__ sinv,
                      int t_base, int n_out, float thr, DetCand* __restrict__ cands, int cap,
                      int pix_off, int* __restrict__ count, const L2Samples l2) {
  constexpr int MAXW = 1 << LOGW;
  constexpr int K = LOGW + 1;
  constexpr int PL = MAXW / 2;
  constexpr int DB = DetTmaCfg<LOGW>::DB;
  constexpr int DET_NST = DetTmaCfg<LOGW>::NST;
  constexpr int RS = MAXW + DB;  // ring registers
  constexpr int SB = DB * 32;    // floats per stage
  extern __shared__ __align__(128) uint8_t det_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* stages = reinterpret_cast<float*>(det_smem) + warp * DET_NST * SB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(det_smem + 8 * DET_NST * SB * 4) + warp * DET_NST;
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  // npix % 32 == 0, so inner is whole warps: a warp is in or out as a whole
  if (e >= inner) return;
  const long long fidx = e / npix, p = e % npix;
  const int p0 = (int)(p - lane);  // the warp's first cell (a multiple of 32)
  const int total = n + MAXW;
  const int warm_end = t_base + MAXW;
  const int out_end = t_base + n_out + MAXW;
  const int n_blk = (min(total, out_end) + DB - 1) / DB;
  // block b holds inputs x[b DB - 1 - PL .. b DB + DB - 2 - PL]; a block with
  // none inside the cube completes its phase with no copy (its inputs are
  // never read)
  // The first blocks' copies leave before the mask, the scales and the
  // Layer-2 entries are loaded (558 -> 547 us for 8 fine DMs x 256 outputs of
  // 512^2 at boxcars to 16: a CTA lives for some 25 us).
  auto issue = [&](int b) {
    uint64_t* bar = bars + b % DET_NST;
    const int y0 = b * DB - 1 - PL;
    if (y0 < n && y0 + DB > 0) {
      mbar_arrive_expect_tx(bar, SB * 4);
      tma_load_3d(stages + (b % DET_NST) * SB, &tmap, p0, y0, (int)fidx, bar);
    } else {
      mbar_arrive(bar);
    }
  };
  if (lane == 0) {
    for (int s = 0; s < DET_NST; ++s) mbar_init(bars + s, 1);
    fence_mbar_init();
    for (int b = 0; b < min(DET_NST - 1, n_blk); ++b) issue(b);
  }
  __syncwarp();
  int s_i = 0, s_end = 0, s_t = 0x7fffffff;
  const int eg = (int)e + pix_off;
  if (l2.out) {
    const int gb = pix_off / 256 + (int)blockIdx.x;
    int lo = __ldg(l2.off + gb);
    s_end = __ldg(l2.off + gb + 1);
    while (lo < s_end && __ldg(&l2.ent[lo].x) < eg) ++lo;
    s_i = lo;
    if (s_i < s_end && __ldg(&l2.ent[s_i].x) == eg) s_t = __ldg(&l2.ent[s_i].y);
  }
  float mval = mask ? mask[fidx * mask_f_stride + p] : 1.0f;
  if (sig_f) mval = mval / sig_f[fidx];
  float tau[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float lv = thr / sinv[k];
    tau[k] = lv - fabsf(lv) * 0x1p-20f;
  }
  // the ring as float32 pairs (slot i in rg[i / 2], .x even, .y odd), so
  // that two consecutive steps' boxcars of one width are one packed
  // float32x2 subtraction where their slots align (widths 4 and up)
  float2 rg[(RS + 1) / 2];
#pragma unroll
  for (int q = 0; q < (RS + 1) / 2; ++q) rg[q] = make_float2(0.f, 0.f);
  auto ring = [&](int i) -> float& { return (i & 1) ? rg[i >> 1].y : rg[i >> 1].x; };
  double run = 0.0;
  float last = 0.f;
  // the screen, the threshold hits and the Layer-2 samples of one output
  // from its boxcar sums
  auto decide = [&](const BoxSums<K>& d, int ta, auto with_samples) {
    bool hit = false;
#pragma unroll
    for (int k = 0; k < K; ++k) hit |= d.v[k] > tau[k];
    if (hit) det_emit<K>(d, sinv, thr, ta - t_base, (int)e + pix_off, cands, cap, count);
    if (decltype(with_samples)::value && ta - t_base == s_t) {
      const int2 r = det_sample<K>(d, l2, s_i, s_end, eg, ta - t_base);
      s_i = r.x;
      s_t = r.y;
    }
  };
  auto output = [&](int j, int ta, auto with_samples) {
    BoxSums<K> d;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int w = 1 << k;
      const int off = PL - w / 2;
      d.v[k] = ring(j + off + w) - ring(j + off);
    }
    decide(d, ta, with_samples);
  };
  // steps j and j + 1 (j even) raise each width's largest boxcar sum m[k]:
  // widths 1 and 2 one by one, the wider ones (both slots even) as packed
  // pairs, with the same roundings.  A three-input maximum takes both steps
  // at once (NaN never raises it), half the instructions of a comparison
  // with tau per step, which is made once per SCR steps: 1133 -> 697 us for
  // 8 fine DMs x 320 times of 512^2 at boxcars to 64 (3.9 TB/s of images).
  auto screen2 = [&](int j, float (&m)[K], bool first) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int w = 1 << k;
      const int off = PL - w / 2;
      float2 dd;
      if (w >= 4 && PL % 2 == 0)
        dd = f2_sub(rg[(j + off + w) >> 1], rg[(j + off) >> 1]);
      else
        dd = make_float2(ring(j + off + w) - ring(j + off),
                         ring(j + 1 + off + w) - ring(j + 1 + off));
      m[k] = first ? fmaxf(dd.x, dd.y) : fmax3(m[k], dd.x, dd.y);
    }
  };
  int b = 0;
  bool ok = true;
  for (; b < n_blk; ++b) {
    const int J0 = b * DB;
    // every lane is done with block b - 1, whose stage takes block
    // b + DET_NST - 1 (generic-proxy reads before the async-proxy write)
    __syncwarp();
    if (lane == 0 && b + DET_NST - 1 < n_blk) {
      fence_proxy_async_smem();
      issue(b + DET_NST - 1);
    }
    if (!__all_sync(0xffffffffu,
                    mbar_wait(bars + b % DET_NST, (uint32_t)((b / DET_NST) & 1)))) {
      ok = false;
      break;
    }
    // input of step J0 + j (x[J0 + j - 1 - PL]) at sx[32 j]
    const float* sx = stages + (b % DET_NST) * SB + lane;
    if (J0 + DB <= warm_end && J0 + DB - 2 - PL < n) {
#pragma unroll
      for (int j = 0; j < DB; ++j) {
        const int J = J0 + j;
        float v = 0.f;
        if (J > PL) {
          run += (double)(sx[32 * j] * mval);
          v = (float)run;
        }
        ring(MAXW + j) = v;
      }
      last = ring(MAXW + DB - 1);
    } else if (J0 >= PL + 1 && J0 + DB - 1 <= PL + n && J0 - MAXW >= t_base &&
               J0 + DB - 1 - MAXW < t_base + n_out) {
      auto steady = [&](auto with_samples) {
        constexpr int SCR = DB < 16 ? DB : 16;
#pragma unroll
        for (int j0 = 0; j0 < DB; j0 += SCR) {
          float m[K];
#pragma unroll
          for (int j = j0; j < j0 + SCR; j += 2) {
            run += (double)(sx[32 * j] * mval);
            ring(MAXW + j) = (float)run;
            run += (double)(sx[32 * (j + 1)] * mval);
            ring(MAXW + j + 1) = (float)run;
            screen2(j, m, j == j0);
          }
          bool hit = false;
#pragma unroll
          for (int k = 0; k < K; ++k) hit |= m[k] > tau[k];
          // rare: a hit or a Layer-2 sample among these steps; the outputs
          // decide from the ring, which still holds all their prefixes.
          // (Against a test per step, same data with lower thresholds: no
          // hits 752 -> 559 us, 0.02 % of the outputs 922 -> 770, 0.3 % 3.79
          // -> 3.75 ms, 2.5 % 32.3 -> 31.4, 15 % 133 -> 140, 48 % 375 -> 380:
          // the appended candidates set the time there.  Screening these
          // steps in pairs first, so that only those with a hit decide, needs
          // their sums formed anew: 559 -> 584 us without hits, 141 ms at 15 %.)
          if (hit || (decltype(with_samples)::value &&
                      (unsigned)(s_t - (J0 + j0 - MAXW - t_base)) < (unsigned)SCR)) {
#pragma unroll
            for (int j = j0; j < j0 + SCR; ++j) output(j, J0 + j - MAXW, with_samples);
          }
        }
      };
      if ((unsigned)(s_t - (J0 - MAXW - t_base)) < (unsigned)DB)
        steady(std::true_type{});
      else
        steady(std::false_type{});
      last = ring(MAXW + DB - 1);
    } else {
#pragma unroll
      for (int j = 0; j < DB; ++j) {
        const int J = J0 + j;
        if (J < total) {
          float v;
          if (J <= PL) {
            v = 0.f;
          } else if (J <= PL + n) {
            run += (double)(sx[32 * j] * mval);
            last = (float)run;
            v = last;
          } else {
            v = last;
          }
          ring(MAXW + j) = v;
          const int ta = J - MAXW;
          if (ta >= t_base && ta < t_base + n_out) output(j, ta, std::true_type{});
        }
      }
    }
    static_assert(DB % 2 == 0, "blocks of whole slot pairs");
#pragma unroll
    for (int q = 0; q < (MAXW + 1) / 2; ++q) rg[q] = rg[q + DB / 2];
  }
  if (!ok && lane == 0) {
    atomicMax(count + 1, DET_TIMEOUT_BITS);
    for (int c = b; c < min(n_blk, b + DET_NST); ++c)
      mbar_wait(bars + c % DET_NST, (uint32_t)((c / DET_NST) & 1));
  }
}

// ===========================================================================
// Layer-1 sigma-clipped std (noise_norm/layer1.py:53-125): one block per
// row, rows of at most L1_MAX samples; bitonic sort, then the clipping
// iterations walk a contiguous range of the sorted row; median is the lower
// median (torch.nanmedian); sums in float64.
// ===========================================================================
constexpr int L1_MAX = 4096;
constexpr int L1_THREADS = 1024;
static_assert(L1_MAX % L1_THREADS == 0, "each thread stages a whole number of samples");

// Where a row's samples come from: a [rows, m] matrix, or (GATHER) the
// images themselves, sample i of row f = img[f*f_stride + times[i / n_pix] *
// t_stride + pix[i % n_pix]] (the Layer-1 subsample of the pipeline).
struct L1Src {
  const float* x;
  long long f_stride, t_stride;
  const int* times;
  const int* pix;
  int n_pix;
  int nonpos_to_one;  // report sigma <= 0 (or NaN) as 1 (the mask divisor)
};

template <bool GATHER>
__global__ void __launch_bounds__(L1_THREADS) clipped_std_kernel(const L1Src src, int m,
                                                                 float n_sigma, int n_iter,
                                                                 float* __restrict__ out) {
  __shared__ __align__(16) float v[L1_MAX];
  __shared__ double red[L1_THREADS / 32];
  __shared__ int s_lo, s_hi;
  if (threadIdx.x == 0) {
    s_lo = 0;
    s_hi = 0;
  }
  __syncthreads();
  const float* row = src.x + (long long)blockIdx.x * (GATHER ? src.f_stride : m);
  // Thread t holds samples 4t .. 4t + 3 in registers (every load issues
  // before the first is used); the padding past m is +inf.  The bitonic
  // network sorts all L1_MAX entries: its stages with partner distance j < 4
  // run inside the thread, 4 <= j <= 64 across the warp by shuffles, and only
  // j >= 128 through shared memory with a barrier (15 of the 78 stages).
  static_assert(L1_MAX == 4 * L1_THREADS, "four samples per thread");
  static_assert(L1_THREADS == 1024, "one sum per lane of a warp");
  float r[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = 4 * threadIdx.x + q;
    r[q] = __int_as_float(0x7f800000);
    if (i < m) {
      if constexpr (GATHER)
        r[q] = row[src.times[i / src.n_pix] * src.t_stride + src.pix[i % src.n_pix]];
      else
        r[q] = row[i];
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (!(r[q] == r[q]) || isinf(r[q])) r[q] = __int_as_float(0x7f800000);  // non-finite -> +inf
  {  // s_hi: the finite samples (the sort's barriers follow)
    const int n_fin = (int)!isinf(r[0]) + (int)!isinf(r[1]) + (int)!isinf(r[2]) + (int)!isinf(r[3]);
    const int w = __reduce_add_sync(0xffffffffu, n_fin);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_hi, w);
  }
  const int i0 = 4 * threadIdx.x;
  float4* v4 = reinterpret_cast<float4*>(v);
  // compare-exchange of positions (i, i ^ j), i the lower: ascending where
  // (i & k) == 0
  auto cx = [](float& lo, float& hi, bool up) {
    if ((lo > hi) == up) {
      const float t = lo;
      lo = hi;
      hi = t;
    }
  };
  for (int k = 2; k <= L1_MAX; k <<= 1) {
    const bool up = (i0 & k) == 0;  // for k >= 4 the same for all four samples
    int j = k >> 1;
    if (j >= 128) {
      v4[threadIdx.x] = make_float4(r[0], r[1], r[2], r[3]);
      __syncthreads();
      for (; j >= 128; j >>= 1) {
        for (int i = threadIdx.x; i < L1_MAX; i += L1_THREADS) {
          const int ixj = i ^ j;
          if (ixj > i) {
            const bool u = (i & k) == 0;
            const float a = v[i], b = v[ixj];
            if ((a > b) == u) {
              v[i] = b;
              v[ixj] = a;
            }
          }
        }
        __syncthreads();
      }
      const float4 w = v4[threadIdx.x];
      r[0] = w.x; r[1] = w.y; r[2] = w.z; r[3] = w.w;
    }
    for (; j >= 4; j >>= 1) {
      const bool lower = (i0 & j) == 0;  // this thread's samples are the lower positions
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float o = __shfl_xor_sync(0xffffffffu, r[q], j >> 2);
        // the lower position keeps the smaller value where ascending
        const bool keep_small = lower == up;
        r[q] = keep_small ? (o < r[q] ? o : r[q]) : (o > r[q] ? o : r[q]);
      }
    }
    if (k >= 4) {  // j = 2: pairs (0, 2), (1, 3)
      cx(r[0], r[2], up);
      cx(r[1], r[3], up);
    }
    {  // j = 1: pairs (0, 1), (2, 3); for k = 2 the direction alternates per pair
      cx(r[0], r[1], k == 2 ? ((i0 & 2) == 0) : up);
      cx(r[2], r[3], k == 2 ? (((i0 + 2) & 2) == 0) : up);
    }
  }
  v4[threadIdx.x] = make_float4(r[0], r[1], r[2], r[3]);
  __syncthreads();
  float sigma = 0.f, med = 0.f;
  for (int it = 0; it <= n_iter; ++it) {
    const int lo = s_lo, hi = s_hi;
    const int cnt = hi - lo;
    if (cnt <= 0) {
      sigma = __int_as_float(0x7fc00000);
      break;
    }
    med = v[lo + (cnt - 1) / 2];
    double acc = 0.0;
    for (int i = lo + threadIdx.x; i < hi; i += L1_THREADS) {
      const float d = v[i] - med;
      acc += (double)(d * d);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    // every warp adds the warps' sums itself (one barrier, no serial chain)
    double tot = red[threadIdx.x & 31];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    sigma = sqrtf((float)tot / (float)cnt);
    if (it == n_iter) break;
    // the clipped range: 32 samples from each end at a time, by warp 0
    if (threadIdx.x < 32) {
      const float lo_v = med - n_sigma * sigma, hi_v = med + n_sigma * sigma;
      int a = lo, b = hi;
      for (;;) {
        const int x = a + (int)threadIdx.x;
        const int n = __ffs(~__ballot_sync(0xffffffffu, x < hi && v[x] < lo_v));
        if (n == 0) {
          a += 32;
          continue;
        }
        a += n - 1;
        break;
      }
      for (;;) {
        const int x = b - 1 - (int)threadIdx.x;
        const int n = __ffs(~__ballot_sync(0xffffffffu, x >= a && v[x] > hi_v));
        if (n == 0) {
          b -= 32;
          continue;
        }
        b -= n - 1;
        break;
      }
      if (threadIdx.x == 0) {
        s_lo = a;
        s_hi = b;
      }
    }
    __syncthreads();   // the new range, and red may be written again
  }
  if (threadIdx.x == 0) {
    float o = (sigma == sigma) ? sigma : 0.f;
    if (src.nonpos_to_one && !(o > 0.f)) o = 1.f;
    out[blockIdx.x] = o;
  }
}

// The driver's tensor-map encoder, looked up once through the runtime.
PFN_cuTensorMapEncodeTiled_v12000 det_tmap_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* q = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &r) ==
            cudaSuccess &&
        r == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(q);
    cudaGetLastError();
  }
  return fn;
}

// The float cube as a 3-D tensor (cell, time, fine DM) with one detector
// block's box (32 cells x db times x 1).  False when the layout does not
// allow it (the caller then runs detect_kernel): npix a multiple of 32, the
// base 16-byte aligned, the strides whole 16-byte units.
bool det_cube_tmap(const float* x, int n, int n_f, int npix, long long f_stride,
                   long long t_stride, int db, CUtensorMap* m) {
  if (npix % 32 || (reinterpret_cast<uintptr_t>(x) & 15) || t_stride % 4 || t_stride < npix ||
      (n_f > 1 && (f_stride % 4 || f_stride < (long long)n * t_stride)))
    return false;
  auto fn = det_tmap_encoder();
  if (!fn) return false;
  const long long fs = n_f > 1 ? f_stride : (long long)n * t_stride;
  const cuuint64_t dims[3] = {(cuuint64_t)npix, (cuuint64_t)n, (cuuint64_t)n_f};
  const cuuint64_t strides[2] = {(cuuint64_t)t_stride * 4, (cuuint64_t)fs * 4};
  const cuuint32_t box[3] = {32u, (cuuint32_t)db, 1u};
  const cuuint32_t es[3] = {1u, 1u, 1u};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(x), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int LOGW>
int det_tma_launch(const float* x, int n, int n_f, int npix, long long f_stride,
                   long long t_stride, const float* mask, long long mask_f_stride,
                   const float* sig_f, const float* sinv, int t_base, int n_out, float thr,
                   DetCand* c, int cap, int pix_off, int* count, const L2Samples& l2,
                   cudaStream_t stream, bool* done) {
  *done = false;
  CUtensorMap tm;
  memset(&tm, 0, sizeof(tm));
  if (!det_cube_tmap(x, n, n_f, npix, f_stride, t_stride, DetTmaCfg<LOGW>::DB, &tm))
    return DSB_OK;
  constexpr int smem = det_tma_smem<LOGW>();
  if (cudaFuncSetAttribute(detect_tma_kernel<LOGW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           smem) != cudaSuccess)
    return DSB_E_CUDA;
  const long long inner = (long long)n_f * npix;
  const unsigned grid = (unsigned)((inner + 255) / 256);
  detect_tma_kernel<LOGW><<<grid, 256, smem, stream>>>(tm, n, npix, inner, mask, mask_f_stride,
                                                       sig_f, sinv, t_base, n_out, thr, c, cap,
                                                       pix_off, count, l2);
  *done = true;
  return launch_status();
}

}  // namespace

extern "C" {

int dsb_uv_cells(const double* du, const double* dv, int n_bl, const double* nu_ghz, int n_ch,
                 double cell_lambda, int n_grid, int* row, int* col, cudaStream_t stream) {
  if (!du || !dv || !nu_ghz || !row || !col || n_bl < 0 || n_ch <= 0 || !(cell_lambda > 0))
    return DSB_E_ARG;
  const long long n = (long long)n_bl * n_ch;
  if (n == 0) return DSB_OK;
  uv_cells_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(du, dv, n_bl, nu_ghz, n_ch,
                                                                   cell_lambda, n_grid / 2, row,
                                                                   col);
  return launch_status();
}

int dsb_combine_rows(const void* D, int d_format, const long long* seg_base, const int* seg_depth,
                     const float* scales, const long long* sc_base, int n_coarse,
                     const int* hc_off, const int* e_g, const int* e_cell, const int* d_pitch,
                     const int* sfine, const int* f2c, int f0, int n_f, int G, int N,
                     long long t0, int n_t, int fftshift, void* out, cudaStream_t stream) {
  if (!D || !seg_base || !seg_depth || n_coarse <= 0 || !hc_off || !e_g || !e_cell ||
      !d_pitch || !sfine || !f2c || !out || d_format < 0 || d_format > 2 ||
      (d_format == 2 && (!scales || !sc_base)))
    return DSB_E_ARG;
  if (N <= 0 || (N & 1) || n_f <= 0 || n_t <= 0 || G <= 0) return DSB_E_ARG;
  CombArgs A{D, scales, sc_base, seg_base, seg_depth, n_coarse, hc_off, e_g, e_cell, d_pitch,
             sfine, f2c, f0, n_f, G, N, t0, n_t, fftshift, (float2*)out};
  const int n_hc = N * (N / 2 + 1);
  dim3 grid((n_hc + 127) / 128, n_f);
  if (d_format == 2)
    combine_rows_kernel<2><<<grid, 128, 0, stream>>>(A);
  else if (d_format == 1)
    combine_rows_kernel<1><<<grid, 128, 0, stream>>>(A);
  else
    combine_rows_kernel<0><<<grid, 128, 0, stream>>>(A);
  return launch_status();
}

int dsb_combine_sparse(const void* dense, const int* cell_uw, const int* cell_ptr,
                       const int* ent_g, const int* ent_k, const int* ent_km, int n_act,
                       const int* shifts, void* out, int out_f16, int n_sb, int t_rows,
                       int t_pad, int n_filled_max, int N, int n_fdm, int t_out_len, int t_lo,
                       int fftshift, int out_rows, int out_row0, int* status,
                       cudaStream_t stream) {
  if (!dense || !cell_uw || !cell_ptr || !shifts || !out || !status || n_act < 0 ||
      n_sb <= 0 || t_rows < 0 || t_pad < t_rows || n_filled_max <= 0 || N <= 0 || (N & 1) ||
      n_fdm <= 0 || t_out_len < 0 || out_row0 < 0 || out_row0 + t_out_len > out_rows)
    return DSB_E_ARG;
  if (n_act > 0 && (!ent_g || !ent_k || !ent_km)) return DSB_E_ARG;
  if ((reinterpret_cast<uintptr_t>(dense) & 1) || (reinterpret_cast<uintptr_t>(out) & 3))
    return DSB_E_ARG;
  if (n_act == 0 || t_out_len == 0) return DSB_OK;
  if ((t_out_len + CS_T - 1) / CS_T > 65535) return DSB_E_ARG;
  SparseArgs A{static_cast<const int16_t*>(dense), cell_uw, cell_ptr, ent_g, ent_k, ent_km, shifts,
               out, n_act, 1, 0, n_sb, t_rows, t_pad, n_filled_max, N, n_fdm, t_out_len, t_lo,
               fftshift, out_rows, out_row0, status};
  const int tiles = (t_out_len + CS_T - 1) / CS_T;
  if ((long long)n_act * tiles <= CS_CELL_MAX &&
      (long long)n_act * n_fdm * t_out_len < CS_CELL_OUT) {
    auto kern = out_f16 ? combine_cell_kernel<true> : combine_cell_kernel<false>;
    kern<<<dim3(n_act, tiles), CS_CELL_THREADS, 0, stream>>>(A);
    return launch_status();
  }
  // 32 cells per CTA (five CTAs per SM) where they fill whole rounds of the
  // chip, else 16 (twice the CTAs), fewer while that leaves SMs idle
  auto ctas = [&](int cpc) { return (long long)((n_act + cpc - 1) / cpc) * tiles; };
  const long long round = 148 * 5, n32 = ctas(CS_CELLS);
  A.cpc = n32 * 10 >= (n32 + round - 1) / round * round * 7 ? CS_CELLS : CS_CELLS / 2;
  A.words = A.cpc == CS_CELLS ? CS_WORDS : CS_WORDS / 2;
  while (A.cpc > 1 && ctas(A.cpc) < 2 * 148) A.cpc /= 2;
  auto kern = out_f16 ? combine_sparse_kernel<true> : combine_sparse_kernel<false>;
  kern<<<dim3((n_act + A.cpc - 1) / A.cpc, tiles), CS_THREADS, (size_t)A.words * 4, stream>>>(A);
  return launch_status();
}

int dsb_tables_differ(const void* a, const void* b, long long n_bytes, int* differ,
                      cudaStream_t stream) {
  if (!a || !b || !differ || n_bytes < 0) return DSB_E_ARG;
  if (n_bytes == 0) return DSB_OK;
  const bool vec = ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
  const long long n16 = vec ? n_bytes / 16 : 0, n = std::max(n16, n_bytes - 16 * n16);
  const unsigned blocks = (unsigned)std::min<long long>((n + 255) / 256, 148 * 8);
  tables_differ_kernel<<<blocks, 256, 0, stream>>>(static_cast<const uint8_t*>(a),
                                                   static_cast<const uint8_t*>(b), n16, n_bytes,
                                                   differ);
  return launch_status();
}

int dsb_combine_dense(const void* streams, const int* shifts, const float* scales,
                      const float* off_re, const float* off_im, int per_t, void* out,
                      int out_f16, int half,
                      int G, int t_stream, int t_det, int N, int t_lo, int fftshift,
                      cudaStream_t stream) {
  if (!streams || !shifts || !out || G <= 0 || N <= 0 || t_det <= t_lo || t_lo < 0) return DSB_E_ARG;
  if (half && (N & 1)) return DSB_E_ARG;
  const bool calib = scales != nullptr;
  if (calib && (!off_re || !off_im)) return DSB_E_ARG;
  if (half && combine_pair_ok(streams, N, t_det - t_lo) &&
      combine_pair_better(calib, G, N, t_det - t_lo))
    return launch_combine_pair(static_cast<const int8_t*>(streams), shifts, scales, off_re, off_im,
                               per_t, out, out_f16, G, t_stream, N, 1, t_det - t_lo, t_lo,
                               fftshift, 1.f, stream);
  const int nw = half ? N / 2 + 1 : N;
  dim3 block(32, 4, 8);
  dim3 grid((nw + 31) / 32, (N + 3) / 4, (t_det - t_lo + 7) / 8);
  const int8_t* s = (const int8_t*)streams;
  auto go = [&](auto h, auto c, auto f, auto pt) {
    combine_dense_kernel<decltype(h)::value, decltype(c)::value, decltype(f)::value,
                         decltype(pt)::value><<<grid, block, 0, stream>>>(
        s, shifts, scales, off_re, off_im, out, G, t_stream, t_det, N, t_lo, fftshift);
  };
  using T = std::true_type;
  using F = std::false_type;
  auto by_f = [&](auto h, auto c, auto pt) { out_f16 ? go(h, c, T{}, pt) : go(h, c, F{}, pt); };
  auto by_c = [&](auto h) {
    if (!calib) by_f(h, F{}, F{});
    else if (per_t) by_f(h, T{}, T{});
    else by_f(h, T{}, F{});
  };
  half ? by_c(T{}) : by_c(F{});
  return launch_status();
}

int dsb_combine_dense_fdm(const void* streams, const int* shifts, int n_f, const float* scales,
                          const float* off_re, const float* off_im, int per_t, void* out, int G,
                          int t_stream, int N, int n_t, int t_lo, int fftshift, float prescale,
                          cudaStream_t stream) {
  if (!streams || !shifts || !out || n_f <= 0 || G <= 0 || N <= 0 || (N & 1) || n_t <= 0 ||
      t_lo < 0 || t_stream <= 0 || (scales && (!off_re || !off_im)))
    return DSB_E_ARG;
  if (!combine_pair_ok(streams, N, n_t)) return DSB_E_UNSUPPORTED;
  return launch_combine_pair(static_cast<const int8_t*>(streams), shifts, scales, off_re, off_im,
                             per_t, out, 0, G, t_stream, N, n_f, n_t, t_lo, fftshift, prescale,
                             stream);
}

int dsb_mask_to_cube(const float* img, const float* mask, int mask_per_f, int n_f, int n_t,
                     int npix, void* cube, int cube_f16, int cube_f_total, int cube_f0,
                     cudaStream_t stream) {
  if (!img || !mask || !cube || n_f <= 0 || n_t <= 0 || npix <= 0) return DSB_E_ARG;
  if (cube_f0 < 0 || cube_f0 + n_f > cube_f_total) return DSB_E_ARG;
  const long long total = (long long)n_f * n_t * npix;
  if (cube_f16)
    mask_to_cube_kernel<true><<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(
        img, mask, mask_per_f, n_f, n_t, npix, cube, cube_f_total, cube_f0);
  else
    mask_to_cube_kernel<false><<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(
        img, mask, mask_per_f, n_f, n_t, npix, cube, cube_f_total, cube_f0);
  return launch_status();
}

int dsb_padded_cumsum(const void* x, int x_f16, int n, long long inner, int max_w, float* cs,
                      cudaStream_t stream) {
  if (!x || !cs || n <= 0 || inner <= 0 || max_w < 1 || max_w > n) return DSB_E_ARG;
  const unsigned grid = (unsigned)((inner + 255) / 256);
  if (x_f16)
    padded_cumsum_kernel<__half><<<grid, 256, 0, stream>>>((const __half*)x, n, inner, max_w, cs);
  else
    padded_cumsum_kernel<float><<<grid, 256, 0, stream>>>((const float*)x, n, inner, max_w, cs);
  return launch_status();
}

int dsb_multi_boxcar_argmax(const float* cs, long long inner, const int* widths,
                            const int* offsets, const float* sigma_inv, int K, int n_out,
                            int t_base, void* out_max, int out_f16, void* out_win,
                            cudaStream_t stream) {
  if (!cs || !widths || !offsets || !sigma_inv || !out_max || !out_win || K < 1 || n_out <= 0)
    return DSB_E_ARG;
  return launch_argmax<false>(cs, inner, widths, offsets, sigma_inv, K, n_out, t_base, out_max,
                              out_f16, static_cast<int16_t*>(out_win), 0, stream);
}

int dsb_boxcar_from_cs(const float* cs, long long inner, int width, int start, int n_out,
                       float* out, cudaStream_t stream) {
  if (!cs || !out || width < 1 || start < 0 || n_out <= 0) return DSB_E_ARG;
  const long long total = (long long)n_out * inner;
  boxcar_from_cs_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(cs, inner, width,
                                                                             start, n_out, out);
  return launch_status();
}

int dsb_detect(const void* cube, int cube_f16, int n, int n_f, int npix, long long f_stride,
               long long t_stride, const float* mask, long long mask_f_stride,
               const float* sig_f, int log_maxw, const float* sigma_inv,
               int t_base, int n_out, float threshold, void* cands, int cap, int pix_off,
               int* count, cudaStream_t stream) {
  return dsb_detect_sampled(cube, cube_f16, n, n_f, npix, f_stride, t_stride, mask,
                            mask_f_stride, sig_f, log_maxw, sigma_inv, t_base, n_out, threshold,
                            cands, cap, pix_off, count, nullptr, nullptr, nullptr, 0, stream);
}

int dsb_detect_sampled(const void* cube, int cube_f16, int n, int n_f, int npix,
                       long long f_stride, long long t_stride, const float* mask,
                       long long mask_f_stride, const float* sig_f, int log_maxw,
                       const float* sigma_inv, int t_base, int n_out, float threshold,
                       void* cands, int cap, int pix_off, int* count, const int* l2_off,
                       const void* l2_ent, float* l2_out, int l2_m, cudaStream_t stream) {
  if (!cube || !sigma_inv || !cands || !count || n <= 0 || n_f <= 0 || npix <= 0 || cap < 0 ||
      cap > DET_COUNT_MAX)
    return DSB_E_ARG;
  if (l2_out && (!l2_off || !l2_ent || l2_m <= 0 || pix_off < 0 || (pix_off % 256) != 0 ||
                 (reinterpret_cast<uintptr_t>(l2_ent) & 15)))
    return DSB_E_ARG;
  if ((long long)n_f * npix + pix_off > 0x7fffffffLL) return DSB_E_ARG;
  const L2Samples l2{l2_off, static_cast<const int4*>(l2_ent), l2_out, l2_m};
  if (log_maxw < 0 || log_maxw > 6 || (1 << log_maxw) > n || t_base < 0 || n_out < 0 ||
      t_base + n_out > n)
    return DSB_E_ARG;
  const long long inner = (long long)n_f * npix;
  const unsigned grid = (unsigned)((inner + 255) / 256);
  DetCand* c = (DetCand*)cands;
  if (!cube_f16) {
    // float cubes of whole-warp fine DMs: the TMA-staged form
    bool done = false;
    int rc = DSB_OK;
#define DSB_DET_TMA(L)                                                                      \
  rc = det_tma_launch<L>((const float*)cube, n, n_f, npix, f_stride, t_stride, mask,         \
                         mask_f_stride, sig_f, sigma_inv, t_base, n_out, threshold, c, cap,  \
                         pix_off, count, l2, stream, &done)
    switch (log_maxw) {
      case 0: DSB_DET_TMA(0); break;
      case 1: DSB_DET_TMA(1); break;
      case 2: DSB_DET_TMA(2); break;
      case 3: DSB_DET_TMA(3); break;
      case 4: DSB_DET_TMA(4); break;
      case 5: DSB_DET_TMA(5); break;
      case 6: DSB_DET_TMA(6); break;
    }
#undef DSB_DET_TMA
    if (done || rc != DSB_OK) return rc;
  }
#define DSB_DET(L)                                                                        \
  do {                                                                                    \
    if (cube_f16)                                                                         \
      detect_kernel<L, __half><<<grid, 256, 0, stream>>>(                                 \
          (const __half*)cube, n, npix, inner, f_stride, t_stride, mask, mask_f_stride,   \
          sig_f, sigma_inv, t_base,                                                       \
          n_out, threshold, c, cap, pix_off, count, l2);                                   \
    else                                                                                  \
      detect_kernel<L, float><<<grid, 256, 0, stream>>>(                                  \
          (const float*)cube, n, npix, inner, f_stride, t_stride, mask, mask_f_stride,    \
          sig_f, sigma_inv, t_base,                                                       \
          n_out, threshold, c, cap, pix_off, count, l2);                                   \
  } while (0)
  switch (log_maxw) {
    case 0: DSB_DET(0); break;
    case 1: DSB_DET(1); break;
    case 2: DSB_DET(2); break;
    case 3: DSB_DET(3); break;
    case 4: DSB_DET(4); break;
    case 5: DSB_DET(5); break;
    case 6: DSB_DET(6); break;
  }
#undef DSB_DET
  return launch_status();
}

int dsb_clipped_std(const float* samples, int rows, int m, float n_sigma, int n_iter, float* out,
                    cudaStream_t stream) {
  if (!samples || !out || rows <= 0 || m <= 0 || n_iter < 0) return DSB_E_ARG;
  if (m > L1_MAX) return DSB_E_CAPACITY;
  L1Src src{samples, 0, 0, nullptr, nullptr, 1, 0};
  clipped_std_kernel<false><<<rows, L1_THREADS, 0, stream>>>(src, m, n_sigma, n_iter, out);
  return launch_status();
}

int dsb_layer1_sigma(const float* img, long long f_stride, long long t_stride, int n_f,
                     const int* times, int n_times, const int* pix, int n_pix, float n_sigma,
                     int n_iter, float* sigma, cudaStream_t stream) {
  if (!img || !times || !pix || !sigma || n_f <= 0 || n_times <= 0 || n_pix <= 0 || n_iter < 0)
    return DSB_E_ARG;
  if ((long long)n_times * n_pix > L1_MAX) return DSB_E_CAPACITY;
  L1Src src{img, f_stride, t_stride, times, pix, n_pix, 1};
  clipped_std_kernel<true><<<n_f, L1_THREADS, 0, stream>>>(src, n_times * n_pix, n_sigma, n_iter,
                                                            sigma);
  return launch_status();
}

}  // extern "C"

// ===========================================================================
// Boxcar S/N argmax without allocation.
//
// dsb_padded_cumsum + dsb_multi_boxcar_argmax need a caller-owned prefix-sum
// buffer of (n + max_w) x inner floats.  Some callers cannot allocate one: a
// host program that hands all of the GPU's memory to its own fixed arena at
// start-up, or a real-time loop where an allocation or free would stall
// every stream on the device (cudaFree synchronises the device).  For them,
// dsb_boxcar_argmax_noalloc keeps the prefix sums in the file-scope array
// below, DSB_NOALLOC_SCRATCH_BYTES (16 MiB) long, which every GPU that
// loads this file's device code holds until the process exits.
// ===========================================================================
#include <cuda.h>

#include <mutex>

static __device__ __align__(256) float g_boxcar_cs_scratch[DSB_NOALLOC_SCRATCH_BYTES / 4];

namespace {

// The scratch array's device address belongs to one CUDA context: after a
// cudaDeviceReset, or under another context on the same device, it is a
// different address.  So the cache is keyed on the current context's unique
// ID (cuCtxGetId, never reused within a process), looked up through the
// runtime's driver entry points so that the library needs no libcuda link.
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

constexpr int kNoallocCache = 64;
struct NoallocEntry {
  unsigned long long ctx_id;
  float* ptr;
};
NoallocEntry g_noalloc_cache[kNoallocCache];
int g_noalloc_n = 0;
std::mutex g_noalloc_mu;
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;

bool load_ctx_fns() {
  if (g_ctx_get_current && g_ctx_get_id) return true;
  void* f1 = nullptr;
  void* f2 = nullptr;
  cudaDriverEntryPointQueryResult q1{}, q2{};
  if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f1, cudaEnableDefault, &q1) != cudaSuccess ||
      cudaGetDriverEntryPoint("cuCtxGetId", &f2, cudaEnableDefault, &q2) != cudaSuccess ||
      q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !f1 || !f2) {
    cudaGetLastError();
    return false;
  }
  g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(f1);
  g_ctx_get_id = reinterpret_cast<CtxGetIdFn>(f2);
  return true;
}

// The unique ID of the context current on this thread; 0 when there is none.
unsigned long long current_ctx_id() {
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (g_ctx_get_current(&ctx) != CUDA_SUCCESS || !ctx) return 0;
  if (g_ctx_get_id(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}

// Device address of the scratch array in the current context (the current
// device's primary context for a runtime caller), looked up on the first
// call in that context and cached.  Null on failure.
float* boxcar_cs_scratch() {
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!load_ctx_fns()) return nullptr;
  unsigned long long id = current_ctx_id();
  if (id) {
    for (int i = 0; i < g_noalloc_n; ++i)
      if (g_noalloc_cache[i].ctx_id == id) return g_noalloc_cache[i].ptr;
  }
  // not seen yet (the runtime makes the device's context current here if
  // no context was)
  void* addr = nullptr;
  if (cudaGetSymbolAddress(&addr, g_boxcar_cs_scratch) != cudaSuccess || !addr) {
    cudaGetLastError();
    return nullptr;
  }
  if (!id) id = current_ctx_id();
  if (id) {
    // the oldest entry goes when the table is full (a process that made
    // more than 64 contexts); its context looks the address up again
    if (g_noalloc_n == kNoallocCache) {
      for (int i = 1; i < kNoallocCache; ++i) g_noalloc_cache[i - 1] = g_noalloc_cache[i];
      --g_noalloc_n;
    }
    g_noalloc_cache[g_noalloc_n++] = NoallocEntry{id, static_cast<float*>(addr)};
  }
  return static_cast<float*>(addr);
}

}  // namespace

extern "C" int dsb_boxcar_argmax_noalloc(const void* x, int x_f16, int n, long long inner,
                                         int max_w, const int* widths, const int* offsets,
                                         const float* sigma_inv, int K, int n_out, int t_base,
                                         void* out_max, int out_f16, void* out_win,
                                         cudaStream_t stream) {
  if (!x || !widths || !offsets || !sigma_inv || !out_max || !out_win) return DSB_E_ARG;
  if (n <= 0 || inner <= 0 || max_w < 1 || max_w > n || K < 1 || n_out <= 0 || t_base < 0 ||
      (long long)t_base + n_out > n)
    return DSB_E_ARG;
  // (n + max_w) rows of inner floats must fit the array; the sum is formed
  // in 64 bits and inner is bounded first, so neither the sum nor the
  // product can overflow
  constexpr long long kCap = (long long)(DSB_NOALLOC_SCRATCH_BYTES / 4);
  const long long rows = (long long)n + max_w;
  if (inner > kCap || rows * inner > kCap) return DSB_E_CAPACITY;
  float* cs = boxcar_cs_scratch();
  if (!cs) return DSB_E_CUDA;
  // padded_cumsum_kernel writes every one of the (n + max_w) x inner prefix
  // values, its zero padding rows included, so nothing left in the array by
  // an earlier call is read; the argmax below checks every row it reads
  // against those (n + max_w) rows.
  const int rc = dsb_padded_cumsum(x, x_f16, n, inner, max_w, cs, stream);
  if (rc != DSB_OK) return rc;
  return launch_argmax<true>(cs, inner, widths, offsets, sigma_inv, K, n_out, t_base, out_max,
                             out_f16, static_cast<int16_t*>(out_win), rows, stream);
}
