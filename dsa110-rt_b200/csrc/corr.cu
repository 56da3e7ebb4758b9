// 4-bit unpack and X-engine correlator kernels (sm_100a).
//
//  * dsb_unpack_int4   : on-wire (npkt, nant, nchan, 2t, 2p) int4 pairs ->
//                        GEMM layout (nchan, 2t, 2p, npkt, nant) int8/fp16/fp32.
//  * dsb_corr_split    : correlator on GEMM-layout voltages (any of the three
//                        dtypes), Stokes-I + channel sum or 2-pol output.
//  * dsb_corr_tc       : fused unpack + correlate from raw on-wire bytes on the
//                        5th-generation tensor cores (tcgen05.mma kind::i8,
//                        int32 accumulators in tensor memory), Stokes-I and
//                        channel sum folded into the contraction dimension.
//                        Epilogue writes strided complex64 visibilities, or
//                        grids them per subband into time-major rows.
#include "dsb_common.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <type_traits>

namespace {

// ===========================================================================
// unpack
// ===========================================================================
template <typename T>
DSB_DEV T from_code(int v, float scale);
template <>
DSB_DEV int8_t from_code<int8_t>(int v, float) { return (int8_t)v; }
template <>
DSB_DEV __half from_code<__half>(int v, float scale) {
  return __float2half_rn((float)v * scale);
}
template <>
DSB_DEV float from_code<float>(int v, float scale) { return (float)v * scale; }

// Tile: 32 (pkt*nant) rows x 32 channels; smem transpose so that the
// 4-byte raw words are read along channels and the outputs are written
// along (pkt, ant).
template <typename T>
__global__ void unpack_kernel(const uint32_t* __restrict__ raw, int rows, int nchan, float scale,
                              T* __restrict__ ore, T* __restrict__ oim) {
  __shared__ uint32_t tile[32][33];
  const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int i = ty; i < 32; i += 8) {
    int r = r0 + i, c = c0 + tx;
    tile[i][tx] = (r < rows && c < nchan) ? raw[(size_t)r * nchan + c] : 0u;
  }
  __syncthreads();
  const size_t plane = (size_t)rows;  // elements per (c, t, pol) plane
  for (int i = ty; i < 32; i += 8) {
    int c = c0 + i, r = r0 + tx;
    if (c >= nchan || r >= rows) continue;
    uint32_t w = tile[tx][i];
#pragma unroll
    for (int tp = 0; tp < 4; ++tp) {  // byte tp = (t, pol)
      int b = (w >> (8 * tp)) & 0xFF;
      int re = (b & 8) ? (b & 0xF) - 16 : (b & 0xF);
      int hi = b >> 4;
      int im = (hi & 8) ? hi - 16 : hi;
      size_t o = ((size_t)c * 4 + tp) * plane + r;
      ore[o] = from_code<T>(re, scale);
      oim[o] = from_code<T>(im, scale);
    }
  }
}

// Four nibbles (code XOR 8, so 0..15) -> four values code * scale, each the
// float32 product rounded once more to T, packed in row order.  2^23 + n is
// exact, so subtracting 2^23 + 8 gives the code without an integer
// conversion (a quarter-rate instruction).
template <typename T>
DSB_DEV void four_codes(const uint32_t (&n)[4], float scale, T* dst);
DSB_DEV float nib_value(uint32_t n, float scale) {
  return (__uint_as_float(0x4B000000u | n) - 8388616.0f) * scale;
}
template <>
DSB_DEV void four_codes<int8_t>(const uint32_t (&n)[4], float, int8_t* dst) {
  const uint32_t w = n[0] | (n[1] << 8) | (n[2] << 16) | (n[3] << 24);
  // code = n - 8 per byte: set a guard bit, subtract, restore the sign bits
  *reinterpret_cast<uint32_t*>(dst) = ((w | 0x80808080u) - 0x08080808u) ^ 0x80808080u;
}
template <>
DSB_DEV void four_codes<__half>(const uint32_t (&n)[4], float scale, __half* dst) {
  const __half2 a = __floats2half2_rn(nib_value(n[0], scale), nib_value(n[1], scale));
  const __half2 b = __floats2half2_rn(nib_value(n[2], scale), nib_value(n[3], scale));
  *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&a),
                                              *reinterpret_cast<const uint32_t*>(&b));
}
template <>
DSB_DEV void four_codes<float>(const uint32_t (&n)[4], float scale, float* dst) {
  *reinterpret_cast<float4*>(dst) = make_float4(nib_value(n[0], scale), nib_value(n[1], scale),
                                                nib_value(n[2], scale), nib_value(n[3], scale));
}

// Tile: 128 rows x 32 channels, four rows per thread and access.  The kernel
// is bound by memory (1 byte read, 2 parts written per sample); the 32 x 32
// tile above writes 64 bytes of a float16 plane at a time, here it is 256.  A
// thread loads four rows of one channel (a warp one 128-byte line per row)
// and stores them as one 16-byte word at column (row / 4) ^ channel, so that
// neither the stores (lanes along channels) nor the loads (lanes along rows)
// of a quarter warp meet in a bank.  A native float16 page (0.3 GB to 1.2 GB):
// 476 -> 265 us (5.7 TB/s).
template <typename T>
__global__ void __launch_bounds__(256) unpack4_kernel(const uint32_t* __restrict__ raw, int rows,
                                                      int nchan, float scale,
                                                      T* __restrict__ ore, T* __restrict__ oim) {
  __shared__ uint4 tile[32][32];
  const int r0 = blockIdx.x * 128, c0 = blockIdx.y * 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t w[4][4];
  const int c = c0 + lane;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = r0 + 4 * (warp + 8 * i) + k;
      w[i][k] = (r < rows && c < nchan) ? __ldg(raw + (size_t)r * nchan + c) : 0u;
    }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    tile[lane][(warp + 8 * i) ^ lane] = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
  __syncthreads();
  const int r = r0 + 4 * lane;
  if (r >= rows) return;   // rows is a multiple of 4
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int cl = warp + 8 * i;
    if (c0 + cl >= nchan) break;
    const uint4 q = tile[cl][lane ^ cl];
    const uint32_t x[4] = {q.x ^ 0x88888888u, q.y ^ 0x88888888u, q.z ^ 0x88888888u,
                           q.w ^ 0x88888888u};
#pragma unroll
    for (int tp = 0; tp < 4; ++tp) {  // byte tp = (t, pol): low nibble re, high im
      uint32_t re[4], im[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        re[k] = (x[k] >> (8 * tp)) & 15u;
        im[k] = (x[k] >> (8 * tp + 4)) & 15u;
      }
      const size_t o = ((size_t)(c0 + cl) * 4 + tp) * rows + r;
      four_codes<T>(re, scale, ore + o);
      four_codes<T>(im, scale, oim + o);
    }
  }
}

// ===========================================================================
// tensor-core correlator (tcgen05, kind::i8)
// ===========================================================================
constexpr int TC_THREADS = 256;
constexpr int TC_TMEM_COLS = 512;   // two accumulators of <= 256 columns
constexpr int TC_SMEM_BUDGET = 224 * 1024;
constexpr int TC_PRE = 4;          // 16-byte raw loads per thread per item (nant <= 128)
// Gridding rows of one (chgroup, subband) whose offsets are kept in shared
// memory, at least: a baseline meets about two cells over a chgroup's
// subbands, so four rows per baseline, between 4096 (wide chgroups: 2404 rows
// at 32 antennas, two chgroups over the band, 512^2) and 12288.  What the
// operand stages leave free holds more (tc_fit_rows).  Groups beyond it read
// their tables in place, which costs a chain of global loads per row: 37 us of
// every unit of some 512^2 patterns of 96 antennas where it was 4096 rows, and
// 261 -> 177 us for those 32 antennas (2 x 512 packets), which 2112 left out.
__host__ __device__ constexpr int tc_min_rows(int nant) {
  const int n = 2 * nant * (nant + 1);
  return n < 4096 ? 4096 : n > 12288 ? 12288 : n;
}
// Every CTA requests more than half an SM's shared memory so that exactly
// one CTA (and one 512-column tensor-memory allocation) lives on each SM.
constexpr int TC_MIN_SMEM = 120 * 1024;

// Adjacent units whose outputs one 32-byte sector holds.
constexpr int TC_QF = 4;

struct TcArgs {
  const uint8_t* raw;
  long long raw_g_stride;  // bytes
  int n_chgroup, npkt, nant, nchan, t_int, csf;
  int ceff, ppfv, n_fv, rows, kc, n_chunks, nkblk, stage_bytes, nstage, n_mma;
  int unit_order;  // 0: fast-vis tile fastest, 1: summed channel fastest
  // mode 0
  float2* out;
  long long o_g, o_f, o_b, o_s;
  // mode 1
  const int* yoff;    // (n_chgroup*ceff) first global row of the group
  const int* ycnt;    // (n_chgroup*ceff) rows in the group
  const int* row_off; // (n_rows + 1) CSR over rows: baselines gridded into each row
  const int* row_bls; // baseline index of each CSR entry
  int cap_rows;       // rows of one group whose offsets fit shared memory
  float2* yout;
  long long y_t_stride;
  long long t_base;
  long long t_mask;
  // (n_chgroup, ceff, nant) complex gains or null: every visibility is
  // multiplied by g_a conj(g_b) of its subband before it is gridded
  const float2* gains;
  // raw staging by TMA (tma != 0): each item's raw bytes, ppk packets x nant
  // antennas x csf channels x 4 bytes, arrive by one 4-D tensor copy into one
  // of nraw shared-memory stages of raw_stage bytes, nraw - 1 items ahead
  int tma, ppk, raw_stage, nraw;
  // TMA form: tensor-memory columns of a CTA (two accumulators), CTAs per SM,
  // unpacking threads, operand stages
  int tmem_cols, ctas, unpackers, ws_nstage;
  // mode 0: outputs of up to TC_QF consecutive units (adjacent elements in
  // memory) staged in shared memory, [unit][baseline] of q_pitch, and written
  // together; 0: each unit's straight from its accumulator
  int q_pitch;
  int* status;
};

DSB_DEV void tc_unit_coords(const TcArgs& A, int u, int& g, int& f, int& s) {
  const int per_g = A.n_fv * A.ceff;
  g = u / per_g;
  const int r = u % per_g;
  if (A.unit_order == 0) {
    f = r % A.n_fv;
    s = r / A.n_fv;
  } else {
    s = r % A.ceff;
    f = r / A.ceff;
  }
}

// The 16-byte raw words of one K chunk of one unit (vectorised path: csf and
// nchan multiples of 4): thread t loads words t, t + 256, ... of the chunk.
DSB_DEV void tc_load(const TcArgs& A, int g, int f, int s, int q, uint4 (&w)[TC_PRE]) {
  const int nv = A.kc / 16;
  const uint8_t* base = A.raw + (size_t)g * A.raw_g_stride;
#pragma unroll
  for (int r = 0; r < TC_PRE; ++r) {
    const int idx = threadIdx.x + r * TC_THREADS;
    if (idx < A.nant * nv) {
      const int a = idx / nv, v = idx % nv;
      const int j = q * (A.kc / 4) + v * 4;
      const int p = j / A.csf, c = j % A.csf;
      w[r] = __ldg(reinterpret_cast<const uint4*>(
          base + ((((size_t)(f * A.ppfv + p) * A.nant + a) * A.nchan + (size_t)s * A.csf + c) * 4)));
    }
  }
}

// Per-thread offsets of the vectorised fill, computed once per kernel (no
// divisions per item): byte offset of word r of chunk 0 inside a unit's raw
// data, and the four shared-memory destinations of its unpacked words.  Valid
// when a chunk covers whole packets (kc/4 a multiple of csf): chunk q is then
// chunk 0 moved by q * (kc/4/csf) packets.
struct TcFillPlan {
  int ld[TC_PRE];
  int lds[TC_PRE];    // the same word in a TMA raw stage [ppk][nant][csf * 4 bytes]
  uint32_t st[TC_PRE][4];
  long long q_step;   // bytes between chunks
  long long f_step;   // bytes between fast-vis tiles
  int s_step;         // bytes between summed channels
};

// thread: of the NT threads that share a chunk
DSB_DEV void tc_fill_plan(const TcArgs& A, TcFillPlan& P, int thread, int NT) {
  const int nv = A.kc / 16;
  const uint32_t region = (uint32_t)A.rows * 128u;
  const long long pkt = (long long)A.nant * A.nchan * 4;
#pragma unroll
  for (int r = 0; r < TC_PRE; ++r) {
    const int idx = thread + r * NT;
    const int a = idx / nv, v = idx % nv;
    const int p = (v * 4) / A.csf, c = (v * 4) % A.csf;
    P.ld[r] = (int)(((long long)p * A.nant + a) * A.nchan * 4 + (long long)c * 4);
    P.lds[r] = ((p * A.nant + a) * A.csf + c) * 4;
    const uint32_t kr = (uint32_t)v * 16u, ki = (uint32_t)A.kc + (uint32_t)v * 16u;
    const uint32_t ra = (uint32_t)a, rb = (uint32_t)(A.nant + a);
    P.st[r][0] = (kr >> 7) * region + sw128_offset(ra, kr & 127u);
    P.st[r][1] = (ki >> 7) * region + sw128_offset(ra, ki & 127u);
    P.st[r][2] = (kr >> 7) * region + sw128_offset(rb, kr & 127u);
    P.st[r][3] = (ki >> 7) * region + sw128_offset(rb, ki & 127u);
  }
  P.q_step = (long long)(A.kc / 4 / A.csf) * pkt;
  P.f_step = (long long)A.ppfv * pkt;
  P.s_step = A.csf * 4;
}

DSB_DEV void tc_load_planned(const TcArgs& A, const TcFillPlan& P, int g, int f, int s, int q,
                             uint4 (&w)[TC_PRE]) {
  const uint8_t* base = A.raw + (size_t)g * A.raw_g_stride + (long long)f * P.f_step +
                        (long long)s * P.s_step + (long long)q * P.q_step;
  const int n = A.nant * (A.kc / 16);
#pragma unroll
  for (int r = 0; r < TC_PRE; ++r)
    if (threadIdx.x + r * TC_THREADS < n)
      w[r] = __ldg(reinterpret_cast<const uint4*>(base + P.ld[r]));
}

DSB_DEV void tc_store_planned(const TcArgs& A, const TcFillPlan& P, uint8_t* st,
                              const uint4 (&w)[TC_PRE], int thread, int NT) {
  const int n = A.nant * (A.kc / 16);
#pragma unroll
  for (int r = 0; r < TC_PRE; ++r) {
    if (thread + r * NT < n) {
      uint4 R, I, N;
      R.x = nib_lo_s8x4(w[r].x); R.y = nib_lo_s8x4(w[r].y);
      R.z = nib_lo_s8x4(w[r].z); R.w = nib_lo_s8x4(w[r].w);
      I.x = nib_hi_s8x4(w[r].x); I.y = nib_hi_s8x4(w[r].y);
      I.z = nib_hi_s8x4(w[r].z); I.w = nib_hi_s8x4(w[r].w);
      N.x = neg_s8x4(R.x); N.y = neg_s8x4(R.y); N.z = neg_s8x4(R.z); N.w = neg_s8x4(R.w);
      *reinterpret_cast<uint4*>(st + P.st[r][0]) = R;
      *reinterpret_cast<uint4*>(st + P.st[r][1]) = I;
      *reinterpret_cast<uint4*>(st + P.st[r][2]) = I;
      *reinterpret_cast<uint4*>(st + P.st[r][3]) = N;
    }
  }
}

// Unpack the words of tc_load into the operand stage (same layout as tc_fill).
DSB_DEV void tc_store(const TcArgs& A, uint8_t* st, const uint4 (&w)[TC_PRE]) {
  const int nv = A.kc / 16;
  const int kc = A.kc;
  const uint32_t region = (uint32_t)A.rows * 128u;
  const int nant = A.nant;
#pragma unroll
  for (int r = 0; r < TC_PRE; ++r) {
    const int idx = threadIdx.x + r * TC_THREADS;
    if (idx < nant * nv) {
      const int a = idx / nv, v = idx % nv;
      uint4 R, I, N;
      R.x = nib_lo_s8x4(w[r].x); R.y = nib_lo_s8x4(w[r].y);
      R.z = nib_lo_s8x4(w[r].z); R.w = nib_lo_s8x4(w[r].w);
      I.x = nib_hi_s8x4(w[r].x); I.y = nib_hi_s8x4(w[r].y);
      I.z = nib_hi_s8x4(w[r].z); I.w = nib_hi_s8x4(w[r].w);
      N.x = neg_s8x4(R.x); N.y = neg_s8x4(R.y); N.z = neg_s8x4(R.z); N.w = neg_s8x4(R.w);
      const uint32_t kr = (uint32_t)v * 16u, ki = (uint32_t)kc + (uint32_t)v * 16u;
      const uint32_t ra = (uint32_t)a, rb = (uint32_t)(nant + a);
      *reinterpret_cast<uint4*>(st + (kr >> 7) * region + sw128_offset(ra, kr & 127u)) = R;
      *reinterpret_cast<uint4*>(st + (ki >> 7) * region + sw128_offset(ra, ki & 127u)) = I;
      *reinterpret_cast<uint4*>(st + (kr >> 7) * region + sw128_offset(rb, kr & 127u)) = I;
      *reinterpret_cast<uint4*>(st + (ki >> 7) * region + sw128_offset(rb, ki & 127u)) = N;
    }
  }
}

// Convert one K chunk of one unit from packed int4 into the operand stage:
// rows [0, nant) = [R | I], rows [nant, 2 nant) = [I | -R] (K-major, SW128).
DSB_DEV void tc_fill(const TcArgs& A, uint8_t* st, int g, int f, int s, int q) {
  const int nw = A.kc / 4;  // 32-bit words (4 complex samples) per antenna per chunk
  const int kc = A.kc;
  const uint32_t region = (uint32_t)A.rows * 128u;
  const uint8_t* base = A.raw + (size_t)g * A.raw_g_stride;
  const int nant = A.nant;
  if ((A.csf & 3) == 0 && (A.nchan & 3) == 0) {
    const int nv = nw / 4;
    for (int idx = threadIdx.x; idx < nant * nv; idx += TC_THREADS) {
      const int a = idx / nv, v = idx % nv;
      const int j = q * nw + v * 4;
      const int p = j / A.csf, c = j % A.csf;
      const uint4 w = __ldg(reinterpret_cast<const uint4*>(
          base + ((((size_t)(f * A.ppfv + p) * nant + a) * A.nchan + (size_t)s * A.csf + c) * 4)));
      uint4 R, I, N;
      R.x = nib_lo_s8x4(w.x); R.y = nib_lo_s8x4(w.y); R.z = nib_lo_s8x4(w.z); R.w = nib_lo_s8x4(w.w);
      I.x = nib_hi_s8x4(w.x); I.y = nib_hi_s8x4(w.y); I.z = nib_hi_s8x4(w.z); I.w = nib_hi_s8x4(w.w);
      N.x = neg_s8x4(R.x); N.y = neg_s8x4(R.y); N.z = neg_s8x4(R.z); N.w = neg_s8x4(R.w);
      const uint32_t kr = (uint32_t)v * 16u, ki = (uint32_t)kc + (uint32_t)v * 16u;
      const uint32_t ra = (uint32_t)a, rb = (uint32_t)(nant + a);
      *reinterpret_cast<uint4*>(st + (kr >> 7) * region + sw128_offset(ra, kr & 127u)) = R;
      *reinterpret_cast<uint4*>(st + (ki >> 7) * region + sw128_offset(ra, ki & 127u)) = I;
      *reinterpret_cast<uint4*>(st + (kr >> 7) * region + sw128_offset(rb, kr & 127u)) = I;
      *reinterpret_cast<uint4*>(st + (ki >> 7) * region + sw128_offset(rb, ki & 127u)) = N;
    }
  } else {
    for (int idx = threadIdx.x; idx < nant * nw; idx += TC_THREADS) {
      const int a = idx / nw, jj = idx % nw;
      const int j = q * nw + jj;
      const int p = j / A.csf, c = j % A.csf;
      const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(
          base + ((((size_t)(f * A.ppfv + p) * nant + a) * A.nchan + (size_t)s * A.csf + c) * 4)));
      const uint32_t R = nib_lo_s8x4(w), I = nib_hi_s8x4(w), N = neg_s8x4(R);
      const uint32_t kr = (uint32_t)jj * 4u, ki = (uint32_t)kc + (uint32_t)jj * 4u;
      const uint32_t ra = (uint32_t)a, rb = (uint32_t)(nant + a);
      *reinterpret_cast<uint32_t*>(st + (kr >> 7) * region + sw128_offset(ra, kr & 127u)) = R;
      *reinterpret_cast<uint32_t*>(st + (ki >> 7) * region + sw128_offset(ra, ki & 127u)) = I;
      *reinterpret_cast<uint32_t*>(st + (kr >> 7) * region + sw128_offset(rb, kr & 127u)) = I;
      *reinterpret_cast<uint32_t*>(st + (ki >> 7) * region + sw128_offset(rb, ki & 127u)) = N;
    }
  }
}

// Read accumulator `buf` (rows b < nant; columns a: Re, nant + a: Im) and
// emit the upper triangle b <= a at bls(a, b) (conj(E_b) E_a).
// Warp w reads TMEM lane quarter (w & 3) (rows 32*(w&3) ...) and every
// other 16-column chunk (w >> 2 picks the parity).
// Shared copies of the gridding CSR of the (chgroup, subband) last used.
struct TcTab {
  int* cached;      // group index whose tables are loaded (-1 none)
  uint16_t* bls;    // (nbase) baseline of each entry
  uint16_t* roff;   // (TcArgs.cap_rows + 1) row offsets relative to the group's first entry
};

// NT threads (warps 0 .. NT / 32 - 1 of the CTA) take part; sync is their
// barrier, done runs once the accumulator has been read.
template <int MODE, int NT, typename Sync, typename Done>
DSB_DEV void tc_epilogue(const TcArgs& A, uint32_t acc, int g, int f, int s, int2* vbuf,
                         const TcTab& tab, Sync sync, Done done, int lu = 0, bool last = true) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int quarter = warp & 3, half = warp >> 2;
  const int nant = A.nant;
  const int b = quarter * 32 + lane;
  if (quarter * 32 < nant) {
    const uint32_t lane_base = acc + ((uint32_t)(quarter * 32) << 16);
    for (int c0 = half * 16; c0 < nant; c0 += NT / 8) {
      if (c0 + 15 < quarter * 32) continue;  // whole chunk below this warp's rows
      __syncwarp();
      uint32_t vr[16], vi[16];
      tmem_ld16(lane_base + (uint32_t)c0, vr);
      tmem_ld16(lane_base + (uint32_t)(nant + c0), vi);
      tmem_ld_wait();
      if (b < nant) {
        auto each = [&](auto emit) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int a = c0 + j;
            if (a < b || a >= nant) continue;
            emit(a, upper_bls(a, b), (int)vr[j], (int)vi[j]);
          }
        };
        if constexpr (MODE == 0) {
          // (a loop of its own per form: the test per output cost the direct
          // one up to a tenth, 34.6 -> 38 us per 2 x 128 packets of 48 antennas)
          if (A.q_pitch) {
            int2* v = vbuf + ((A.unit_order ? s : f) & (TC_QF - 1)) * A.q_pitch;
            each([&](int, int bls, int re, int im) { v[bls] = make_int2(re, im); });
          } else {
            float2* o = A.out + (size_t)g * A.o_g + (size_t)f * A.o_f + (size_t)s * A.o_s;
            each([&](int, int bls, int re, int im) {
              o[(size_t)bls * A.o_b] = make_float2((float)re, (float)im);
            });
          }
        } else if (A.gains) {
          // calibrated: V' = g_a conj(g_b) V (V = conj(E_b) E_a), every
          // product and sum rounded on its own (no contraction)
          const float2* gs = A.gains + ((size_t)g * A.ceff + s) * nant;
          const float2 gb = gs[b];
          each([&](int a, int bls, int re, int im) {
            const float2 ga = gs[a];
            const float pr = __fadd_rn(__fmul_rn(ga.x, gb.x), __fmul_rn(ga.y, gb.y));
            const float pi = __fsub_rn(__fmul_rn(ga.y, gb.x), __fmul_rn(ga.x, gb.y));
            const float fr = (float)re, fi = (float)im;
            reinterpret_cast<float2*>(vbuf)[bls] =
                make_float2(__fsub_rn(__fmul_rn(fr, pr), __fmul_rn(fi, pi)),
                            __fadd_rn(__fmul_rn(fr, pi), __fmul_rn(fi, pr)));
          });
        } else {
          each([&](int, int bls, int re, int im) { vbuf[bls] = make_int2(re, im); });
        }
      }
    }
  }
  tc_fence_before();
  done();
  if constexpr (MODE == 0) {
    // the staged units 8 bytes each, four lanes to a baseline's sector, once
    // the last of them (of their row, or of this CTA's) is in: 8-byte stores
    // of one unit at a time kept L2 busy with quarter sectors (413 us for a
    // native page, 175 us without any stores)
    const int fast = A.unit_order ? s : f, j1 = fast & (TC_QF - 1);
    last = last || fast == (A.unit_order ? A.ceff : A.n_fv) - 1;
    if (A.q_pitch && (j1 == TC_QF - 1 || last)) {
      sync();
      const int j0 = max(0, j1 - lu), nbase = nant * (nant + 1) / 2;
      float2* o = A.out + (size_t)g * A.o_g + (size_t)(A.unit_order ? f : s) *
                                                   (A.unit_order ? A.o_f : A.o_s) + (fast - j1);
      const int j = threadIdx.x & (TC_QF - 1);
      if (j >= j0 && j <= j1)
        for (int bls = threadIdx.x / TC_QF; bls < nbase; bls += NT / TC_QF) {
          const int2 v = vbuf[j * A.q_pitch + bls];
          o[(size_t)bls * A.o_b + j] = make_float2((float)v.x, (float)v.y);
        }
    }
  }
  if constexpr (MODE == 1) {
    // per-cell sum over the baselines gridded into it (exact int32); the
    // group's CSR is copied to shared memory when the group changes (a CTA
    // walks consecutive tiles of one group)
    const int gs = g * A.ceff + s;
    const long long row0 = A.yoff[gs];
    const int cnt = A.ycnt[gs];
    const int e0 = A.row_off[row0];
    const int ne = A.row_off[row0 + cnt] - e0;
    const bool use_tab = cnt <= A.cap_rows && ne <= A.nant * (A.nant + 1) / 2;
    const bool reload = use_tab && *tab.cached != gs;
    if (reload) {
      for (int k = threadIdx.x; k <= cnt; k += NT) tab.roff[k] = (uint16_t)(A.row_off[row0 + k] - e0);
      for (int j = threadIdx.x; j < ne; j += NT) tab.bls[j] = (uint16_t)A.row_bls[e0 + j];
    }
    sync();
    if (reload && threadIdx.x == 0) *tab.cached = gs;
    const long long tp = (A.t_base + f) & A.t_mask;
    float2* yrow = A.yout + tp * A.y_t_stride + row0;
    if (cnt > 0 && !(DSB_INB(row0, A.y_t_stride, A.status) &&
                     DSB_INB(row0 + cnt - 1, A.y_t_stride, A.status)))
      return;
    if (A.gains) {
      // calibrated visibilities: float sums in CSR order
      const float2* fbuf = reinterpret_cast<const float2*>(vbuf);
      for (int k = threadIdx.x; k < cnt; k += NT) {
        const long long r = row0 + k;
        float sr = 0.f, si = 0.f;
        const int j0 = use_tab ? tab.roff[k] + e0 : A.row_off[r];
        const int j1 = use_tab ? tab.roff[k + 1] + e0 : A.row_off[r + 1];
        for (int j = j0; j < j1; ++j) {
          const int bl = use_tab ? (int)tab.bls[j - e0] : A.row_bls[j];
          if (!DSB_INB(bl, A.nant * (A.nant + 1) / 2, A.status)) continue;
          sr = __fadd_rn(sr, fbuf[bl].x);
          si = __fadd_rn(si, fbuf[bl].y);
        }
        yrow[k] = make_float2(sr, si);
      }
    } else if (use_tab) {
      // RW rows at a time, first baselines first (most rows have one): their
      // table and visibility loads overlap (one at a time where a small array
      // has few rows per thread)
      constexpr int RW = NT == 128 ? 1 : 4;
      for (int k0 = threadIdx.x; k0 < cnt; k0 += RW * NT) {
        int j0[RW], j1[RW];
        int2 v[RW];
#pragma unroll
        for (int i = 0; i < RW; ++i) {
          const int k = k0 + i * NT;
          j0[i] = k < cnt ? (int)tab.roff[k] : 0;
          j1[i] = k < cnt ? (int)tab.roff[k + 1] : 0;
        }
#pragma unroll
        for (int i = 0; i < RW; ++i) {
          v[i] = make_int2(0, 0);
          if (j0[i] < j1[i]) {
            const int bl = tab.bls[j0[i]];
            if (DSB_INB(bl, A.nant * (A.nant + 1) / 2, A.status)) v[i] = vbuf[bl];
          }
        }
#pragma unroll
        for (int i = 0; i < RW; ++i) {
          for (int j = j0[i] + 1; j < j1[i]; ++j) {
            if (!DSB_INB(tab.bls[j], A.nant * (A.nant + 1) / 2, A.status)) continue;
            const int2 w = vbuf[tab.bls[j]];
            v[i].x += w.x;
            v[i].y += w.y;
          }
          const int k = k0 + i * NT;
          if (k < cnt) yrow[k] = make_float2((float)v[i].x, (float)v[i].y);
        }
      }
    } else {
      for (int k = threadIdx.x; k < cnt; k += NT) {
        const long long r = row0 + k;
        int sr = 0, si = 0;
        for (int j = A.row_off[r]; j < A.row_off[r + 1]; ++j) {
          if (!DSB_INB(A.row_bls[j], A.nant * (A.nant + 1) / 2, A.status)) continue;
          const int2 v = vbuf[A.row_bls[j]];
          sr += v.x;
          si += v.y;
        }
        yrow[k] = make_float2((float)sr, (float)si);
      }
    }
  }
}

// The raw words loaded by the threads that unpack them (chunks that are not
// whole packets of 16-byte channel runs).
template <int MODE>
__global__ void __launch_bounds__(TC_THREADS, 1) corr_tc_kernel(const TcArgs A) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* stages = smem;
  uint64_t* bar_mma = reinterpret_cast<uint64_t*>(stages + (size_t)A.nstage * A.stage_bytes);
  uint64_t* bar_acc = bar_mma + A.nstage;
  uint64_t* bar_drain = bar_acc + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_drain + 1);
  int2* vbuf = reinterpret_cast<int2*>(tmem_slot + 4);
  TcTab tab{};
  if constexpr (MODE == 1) {
    tab.cached = reinterpret_cast<int*>(vbuf + A.nant * (A.nant + 1) / 2);
    tab.bls = reinterpret_cast<uint16_t*>(tab.cached + 4);
    tab.roff = tab.bls + A.nant * (A.nant + 1) / 2;
  }

  const int tid = threadIdx.x, warp = tid >> 5;
  if (warp == 0) {
    tmem_alloc(tmem_slot, TC_TMEM_COLS);
    tmem_relinquish();
  }
  if (tid == 0) {
    if constexpr (MODE == 1) *tab.cached = -1;
    for (int i = 0; i < A.nstage; ++i) mbar_init(&bar_mma[i], 1);
    mbar_init(&bar_acc[0], 1);
    mbar_init(&bar_acc[1], 1);
    mbar_init(bar_drain, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // each CTA walks a contiguous range of units (consecutive fast-vis tiles
  // of one (chgroup, subband) share the gridding tables)
  const int n_units = A.n_chgroup * A.n_fv * A.ceff;
  const int per_cta = (n_units + (int)gridDim.x - 1) / (int)gridDim.x;
  const int u_begin = (int)blockIdx.x * per_cta;
  const int my_units = max(0, min(per_cta, n_units - u_begin));
  const int n_items = my_units * A.n_chunks;
  const uint32_t idesc = idesc_i8(128u, (uint32_t)(2 * A.nant));
  const bool vec = (A.csf & 3) == 0 && (A.nchan & 3) == 0;
  const bool planned = vec && ((A.kc / 4) % A.csf) == 0;
  TcFillPlan plan{};
  if (planned) tc_fill_plan(A, plan, tid, TC_THREADS);
  bool ok = true;
  // the raw words of the next item are loaded while this one is unpacked
  uint4 pre[TC_PRE];
  if (vec && n_items > 0) {
    int g0, f0, s0;
    tc_unit_coords(A, u_begin, g0, f0, s0);
    if (planned) tc_load_planned(A, plan, g0, f0, s0, 0, pre);
    else tc_load(A, g0, f0, s0, 0, pre);
  }

  for (int it = 0; it < n_items; ++it) {
    const int lu = it / A.n_chunks, q = it % A.n_chunks;
    const int u = u_begin + lu;
    int g, f, s;
    tc_unit_coords(A, u, g, f, s);
    const int slot = it % A.nstage;
    bool w_ok = true;
    if (it >= A.nstage) w_ok = mbar_wait(&bar_mma[slot], (uint32_t)((it / A.nstage - 1) & 1));
    if (!__syncthreads_and(w_ok)) { ok = false; break; }
    uint8_t* st = stages + (size_t)slot * A.stage_bytes;
    if (vec) {
      uint4 cur[TC_PRE];
#pragma unroll
      for (int r = 0; r < TC_PRE; ++r) cur[r] = pre[r];
      if (it + 1 < n_items) {
        const int nlu = (it + 1) / A.n_chunks, nq = (it + 1) % A.n_chunks;
        int ng, nf, ns;
        tc_unit_coords(A, u_begin + nlu, ng, nf, ns);
        if (planned) tc_load_planned(A, plan, ng, nf, ns, nq, pre);
        else tc_load(A, ng, nf, ns, nq, pre);
      }
      if (planned) tc_store_planned(A, plan, st, cur, tid, TC_THREADS);
      else tc_store(A, st, cur);
    } else {
      tc_fill(A, st, g, f, s, q);
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t d = tmem_base + (uint32_t)((lu & 1) * 256);
      const uint32_t sbase = smem_u32(st);
      for (int m = 0; m < A.n_mma; ++m) {
        const uint32_t kb = (uint32_t)m * 32u;
        const uint64_t desc = sdesc_k_sw128(sbase + (kb >> 7) * (uint32_t)A.rows * 128u + (kb & 127u));
        umma_i8_ss(d, desc, desc, idesc, (q > 0 || m > 0) ? 1u : 0u);
      }
      umma_commit(&bar_mma[slot]);
      if (q == A.n_chunks - 1) umma_commit(&bar_acc[lu & 1]);
    }
    if (q == A.n_chunks - 1 && lu >= 1) {
      const int pl = lu - 1;
      const bool a_ok = mbar_wait(&bar_acc[pl & 1], (uint32_t)((pl >> 1) & 1));
      if (!__syncthreads_and(a_ok)) { ok = false; break; }
      tc_fence_after();
      int pg, pf, ps;
      tc_unit_coords(A, u_begin + pl, pg, pf, ps);
      tc_epilogue<MODE, TC_THREADS>(A, tmem_base + (uint32_t)((pl & 1) * 256), pg, pf, ps, vbuf,
                                    tab, [] { __syncthreads(); }, [] {});
    }
  }
  if (ok && my_units > 0) {
    const int pl = my_units - 1;
    const bool a_ok = mbar_wait(&bar_acc[pl & 1], (uint32_t)((pl >> 1) & 1));
    if (__syncthreads_and(a_ok)) {
      tc_fence_after();
      int pg, pf, ps;
      tc_unit_coords(A, u_begin + pl, pg, pf, ps);
      tc_epilogue<MODE, TC_THREADS>(A, tmem_base + (uint32_t)((pl & 1) * 256), pg, pf, ps, vbuf,
                                    tab, [] { __syncthreads(); }, [] {});
    } else {
      ok = false;
    }
  }
  if (!ok) {
    if (tid == 0) dsb_flag(A.status, DSB_E_TIMEOUT);
    // drain every MMA this CTA issued before releasing tensor memory
    if (tid == 0) {
      umma_commit(bar_drain);
      mbar_wait(bar_drain, 0u);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TC_TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// The same correlator with the raw tiles staged by TMA and a role per warp:
// the first warps write out (or grid) the finished unit, the next ones unpack
// raw stages into operand stages, one thread issues the tensor copies and one
// the products; stages pass between them by mbarriers.
//
// What bounds it: shared memory (per 128 samples of 96 antennas 12 KB of raw
// bytes in, 49 KB of operands out, 81 KB read by the products) and the
// products themselves, 0.6 us each per SM.  One role after the other between
// CTA barriers, with the gridding's tables read in place, took 11.0 ms for 16
// native pages gridded into 512^2 patterns and 445 us for one page; this takes
// 3.3 ms and 286 us (175 us a page without the writing).
//
// Where two accumulators need fewer than 512 columns, the CTA takes only
// those (a power of two) and several CTAs share an SM (TcArgs.ctas): a unit
// of a small array is a single chunk whose latency one CTA cannot hide (16
// antennas, 64 samples per unit: 3.7 us per unit with one CTA per SM).
// ---------------------------------------------------------------------------
// NU unpacking threads (TC_PRE words each): 256, or 64 where a chunk is at
// most 256 words; the threads that write out; and the CTAs of that size an
// SM's registers hold.  (Two or four groups of unpacking threads that take the
// chunks in turn were slower: 4.1 -> 4.5 ms gridded, 288 -> 316 us a page.)
template <int NU>
struct WsCfg {
  static constexpr int EPI = NU == 64 ? 128 : 256;
  static constexpr int THREADS = EPI + NU + 64;
  static constexpr int CTAS = NU == 64 ? 4 : 1;
};

template <int MODE, int NU>
__global__ void __launch_bounds__(WsCfg<NU>::THREADS, WsCfg<NU>::CTAS) corr_ws_kernel(
    const TcArgs A, const __grid_constant__ CUtensorMap tmap) {
  constexpr int EPI = WsCfg<NU>::EPI;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* stages = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* raw_st = stages + (size_t)A.nstage * A.stage_bytes;
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(raw_st + (size_t)A.nraw * A.raw_stage);
  uint64_t* bar_free = bar_full + A.nstage;
  uint64_t* bar_raw = bar_free + A.nstage;
  uint64_t* bar_rawfree = bar_raw + A.nraw;
  uint64_t* bar_acc = bar_rawfree + A.nraw;   // [2] accumulator finished
  uint64_t* bar_out = bar_acc + 2;            // [2] accumulator read
  uint64_t* bar_drain = bar_out + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_drain + 1);
  int2* vbuf = reinterpret_cast<int2*>(tmem_slot + 4);
  TcTab tab{};
  if constexpr (MODE == 1) {
    tab.cached = reinterpret_cast<int*>(vbuf + A.nant * (A.nant + 1) / 2);
    tab.bls = reinterpret_cast<uint16_t*>(tab.cached + 4);
    tab.roff = tab.bls + A.nant * (A.nant + 1) / 2;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    tmem_alloc(tmem_slot, (uint32_t)A.tmem_cols);
    tmem_relinquish();
  }
  if (tid == 0) {
    if constexpr (MODE == 1) *tab.cached = -1;
    for (int i = 0; i < A.nstage; ++i) {
      mbar_init(&bar_full[i], NU);
      mbar_init(&bar_free[i], 1);
    }
    for (int i = 0; i < A.nraw; ++i) {
      mbar_init(&bar_raw[i], 1);
      mbar_init(&bar_rawfree[i], NU);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_acc[i], 1);
      mbar_init(&bar_out[i], EPI);
    }
    mbar_init(bar_drain, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t acc_cols = (uint32_t)A.tmem_cols / 2;
  // each CTA walks a contiguous range of units (consecutive fast-vis tiles
  // of one (chgroup, subband) share the gridding tables)
  const int n_units = A.n_chgroup * A.n_fv * A.ceff;
  const int per_cta = (n_units + (int)gridDim.x - 1) / (int)gridDim.x;
  const int u_begin = (int)blockIdx.x * per_cta;
  const int my_units = max(0, min(per_cta, n_units - u_begin));
  const int n_items = my_units * A.n_chunks;
  bool ok = true;

  if (warp < EPI / 32) {
    for (int lu = 0; lu < my_units; ++lu) {
      const int buf = lu & 1;
      ok = mbar_wait(&bar_acc[buf], (uint32_t)((lu >> 1) & 1));
      // (named barrier: the warps agree, and the previous unit's reads
      // of vbuf are done before it is written again)
      int all;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\t"
          "barrier.cta.red.and.pred q, 1, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
          : "=r"(all)
          : "r"((int)ok), "n"(EPI)
          : "memory");
      ok = all != 0;
      if (!ok) break;
      tc_fence_after();
      int g, f, s;
      tc_unit_coords(A, u_begin + lu, g, f, s);
      tc_epilogue<MODE, EPI>(
          A, tmem_base + (uint32_t)buf * acc_cols, g, f, s, vbuf, tab,
          [] { asm volatile("barrier.cta.sync 1, %0;" ::"n"(EPI) : "memory"); },
          [&] { mbar_arrive(&bar_out[buf]); }, lu, lu == my_units - 1);
    }
  } else if (warp < (EPI + NU) / 32) {
    const int ut = tid - EPI;
    TcFillPlan plan;
    tc_fill_plan(A, plan, ut, NU);
    const int n_w = A.nant * (A.kc / 16);
    for (int it = 0; it < n_items; ++it) {
      const int slot = it % A.nstage, r = it % A.nraw;
      if (it >= A.nstage) ok = mbar_wait(&bar_free[slot], (uint32_t)((it / A.nstage - 1) & 1));
      ok = ok && mbar_wait(&bar_raw[r], (uint32_t)((it / A.nraw) & 1));
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        break;
      }
      const uint8_t* rs = raw_st + (size_t)r * A.raw_stage;
      uint4 cur[TC_PRE];
#pragma unroll
      for (int k = 0; k < TC_PRE; ++k)
        if (ut + k * NU < n_w) cur[k] = *reinterpret_cast<const uint4*>(rs + plan.lds[k]);
      tc_store_planned(A, plan, stages + (size_t)slot * A.stage_bytes, cur, ut, NU);
      fence_proxy_async_smem();
      mbar_arrive(&bar_full[slot]);
      mbar_arrive(&bar_rawfree[r]);
    }
  } else if (warp == (EPI + NU) / 32) {
    if (lane == 0) {
      // item's raw bytes: ppk packets x nant x csf channels x 4 bytes of one
      // chgroup page
      int issued = 0;
      for (int it = 0; it < n_items; ++it) {
        const int r = it % A.nraw;
        if (it >= A.nraw) ok = mbar_wait(&bar_rawfree[r], (uint32_t)((it / A.nraw - 1) & 1));
        if (!ok) break;
        const int lu = it / A.n_chunks, q = it % A.n_chunks;
        int g, f, s;
        tc_unit_coords(A, u_begin + lu, g, f, s);
        mbar_arrive_expect_tx(&bar_raw[r], (uint32_t)(A.ppk * A.nant * A.csf * 4));
        tma_load_4d(raw_st + (size_t)r * A.raw_stage, &tmap, s * A.csf * 4, 0,
                    f * A.ppfv + q * A.ppk, g, &bar_raw[r]);
        ++issued;
      }
      // no copy may be in flight into this CTA's shared memory when it ends
      // (each of the last nraw copies' phases; all earlier ones were waited
      // for before their stage was taken again)
      for (int it = max(0, issued - A.nraw); it < issued; ++it)
        mbar_wait(&bar_raw[it % A.nraw], (uint32_t)((it / A.nraw) & 1));
    }
  } else if (lane == 0) {
    const uint32_t idesc = idesc_i8(128u, (uint32_t)(2 * A.nant));
    for (int it = 0; it < n_items; ++it) {
      const int lu = it / A.n_chunks, q = it % A.n_chunks;
      const int slot = it % A.nstage, buf = lu & 1;
      if (q == 0 && lu >= 2) ok = mbar_wait(&bar_out[buf], (uint32_t)(((lu >> 1) - 1) & 1));
      ok = ok && mbar_wait(&bar_full[slot], (uint32_t)((it / A.nstage) & 1));
      if (!ok) break;
      tc_fence_after();
      const uint32_t d = tmem_base + (uint32_t)buf * acc_cols;
      const uint32_t sbase = smem_u32(stages + (size_t)slot * A.stage_bytes);
      for (int m = 0; m < A.n_mma; ++m) {
        const uint32_t kb = (uint32_t)m * 32u;
        const uint64_t desc = sdesc_k_sw128(sbase + (kb >> 7) * (uint32_t)A.rows * 128u + (kb & 127u));
        umma_i8_ss(d, desc, desc, idesc, (q > 0 || m > 0) ? 1u : 0u);
      }
      umma_commit(&bar_free[slot]);
      if (q == A.n_chunks - 1) umma_commit(&bar_acc[buf]);
    }
    // every product issued here ends before tensor memory is given back
    umma_commit(bar_drain);
    mbar_wait(bar_drain, 0u);
  }
  if (!ok) dsb_flag(A.status, DSB_E_TIMEOUT);
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, (uint32_t)A.tmem_cols);
  }
}

// ===========================================================================
// tensor-core correlators on split (GEMM-layout) voltages, float32
// accumulators in TMEM: tcgen05 kind::f16 for int8 codes (exact conversion)
// and float16 voltages (corr_split_mn_kernel), kind::tf32 for float32
// voltages, rounded to tf32 as a float32 tensor-core product does
// (corr_split_tc_kernel).
// ===========================================================================
struct SplitTcArgs {
  const void* re;            // int8, float16: rounded down to 4 bytes, the
  const void* im;            //   first element off_re / off_im elements on
  int off_re, off_im;
  int nchan, npkt, nant, nant_p, ppfv, fuse, csf, ceff;
  int n_fv, n_units, kprime, n_chunks, rows, nstage, stage_bytes;
  int q_pitch;               // staged outputs' pitch (0: none), as in TcArgs
  float2* out;
  int* status;
};

// Output unit u -> the fast-vis tile, its channel range and pols, and the
// output column: Stokes-I unit = (fv, summed channel s), K over (channel of
// the group, pol, t-sub, packet); 2-pol unit = (fv, ch, pol), K over
// (t-sub, packet).
DSB_DEV void split_unit(const SplitTcArgs& A, int u, int& fv, int& ch0, int& pol0, int& npol_u) {
  if (A.fuse) {
    fv = u / A.ceff;
    ch0 = (u % A.ceff) * A.csf;
    pol0 = 0;
    npol_u = 2;
  } else {
    fv = u / (A.nchan * 2);
    ch0 = (u / 2) % A.nchan;
    pol0 = u % 2;
    npol_u = 1;
  }
}

// Element o rounded to tf32 (10 mantissa bits), nearest with ties away from
// zero: add half of the dropped range to the magnitude bits (a carry moves
// into the exponent correctly), clear the dropped bits; infinities and NaNs
// pass unchanged.
DSB_DEV uint32_t split_load_bits(const void* p, size_t o) {
  const uint32_t u = __float_as_uint(static_cast<const float*>(p)[o]);
  if ((u & 0x7F800000u) == 0x7F800000u) return u;
  return (u + 0x1000u) & 0xFFFFE000u;
}

// One K chunk (KC complex samples) of unit u into an operand stage:
// rows [0, nant_p) = [R | I], rows [nant_p, 2 nant_p) = [I | -R] (K-major,
// SW128, one 128-byte row per operand row); samples past the unit's K and
// antennas past nant are zero.
DSB_DEV void split_fill(const SplitTcArgs& A, uint8_t* st, int u, int q) {
  constexpr int KC = 16;           // complex samples per chunk
  constexpr int G = 4;             // samples per 16-byte group
  constexpr int NG = KC / G;       // groups per half row (4)
  int fv, ch0, pol0, npol_u;
  split_unit(A, u, fv, ch0, pol0, npol_u);
  const size_t plane = (size_t)A.npkt * A.nant;
  for (int idx = threadIdx.x; idx < A.nant_p * NG; idx += TC_THREADS) {
    const int a = idx % A.nant_p, j = idx / A.nant_p;
    uint32_t r[G], m[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
      int k = q * KC + j * G + i;
      r[i] = 0u;
      m[i] = 0u;
      if (a < A.nant && k < A.kprime) {
        const int p = k % A.ppfv;
        k /= A.ppfv;
        const int t = k & 1;
        k >>= 1;
        const int pol = pol0 + k % npol_u;
        const int ch = ch0 + k / npol_u;
        const size_t o = (((size_t)ch * 2 + t) * 2 + pol) * plane +
                         (size_t)(fv * A.ppfv + p) * A.nant + a;
        r[i] = split_load_bits(A.re, o);
        m[i] = split_load_bits(A.im, o);
      }
    }
    const uint4 R = make_uint4(r[0], r[1], r[2], r[3]);
    const uint4 I = make_uint4(m[0], m[1], m[2], m[3]);
    const uint4 N = make_uint4(r[0] ^ 0x80000000u, r[1] ^ 0x80000000u, r[2] ^ 0x80000000u,
                               r[3] ^ 0x80000000u);
    const uint32_t kr = (uint32_t)j * 16u, ki = 64u + (uint32_t)j * 16u;
    const uint32_t ra = (uint32_t)a, rb = (uint32_t)(A.nant_p + a);
    *reinterpret_cast<uint4*>(st + sw128_offset(ra, kr)) = R;
    *reinterpret_cast<uint4*>(st + sw128_offset(ra, ki)) = I;
    *reinterpret_cast<uint4*>(st + sw128_offset(rb, kr)) = I;
    *reinterpret_cast<uint4*>(st + sw128_offset(rb, ki)) = N;
  }
}

// Accumulator `buf` of unit u: rows b < nant, columns a (Re) and nant_p + a
// (Im); the upper triangle b <= a goes to bls(a, b) (conj(E_b) E_a).
DSB_DEV void split_epilogue(const SplitTcArgs& A, uint32_t tmem_base, int buf, int u) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int quarter = warp & 3, half = warp >> 2;
  const int nant = A.nant, nbase = nant * (nant + 1) / 2;
  const int b = quarter * 32 + lane;
  int fv, ch0, pol0, npol_u;
  split_unit(A, u, fv, ch0, pol0, npol_u);
  if (quarter * 32 < nant) {
    const uint32_t lane_base =
        tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * 256);
    for (int c0 = half * 16; c0 < nant; c0 += 32) {
      if (c0 + 15 < quarter * 32) continue;  // whole chunk below this warp's rows
      uint32_t vr[16], vi[16];
      tmem_ld16(lane_base + (uint32_t)c0, vr);
      tmem_ld16(lane_base + (uint32_t)(A.nant_p + c0), vi);
      tmem_ld_wait();
      if (b < nant) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int a = c0 + j;
          if (a < b || a >= nant) continue;
          const size_t bls = (size_t)upper_bls(a, b);
          const size_t o = A.fuse ? ((size_t)fv * nbase + bls) * A.ceff + ch0 / A.csf
                                  : (((size_t)fv * nbase + bls) * A.nchan + ch0) * 2 + pol0;
          A.out[o] = make_float2(__uint_as_float(vr[j]), __uint_as_float(vi[j]));
        }
      }
    }
  }
}

__global__ void __launch_bounds__(TC_THREADS, 1) corr_split_tc_kernel(const SplitTcArgs A) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* stages = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bar_mma = reinterpret_cast<uint64_t*>(stages + (size_t)A.nstage * A.stage_bytes);
  uint64_t* bar_acc = bar_mma + A.nstage;
  uint64_t* bar_drain = bar_acc + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_drain + 1);
  const int tid = threadIdx.x, warp = tid >> 5;
  if (warp == 0) {
    tmem_alloc(tmem_slot, TC_TMEM_COLS);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < A.nstage; ++i) mbar_init(&bar_mma[i], 1);
    mbar_init(&bar_acc[0], 1);
    mbar_init(&bar_acc[1], 1);
    mbar_init(bar_drain, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int per_cta = (A.n_units + (int)gridDim.x - 1) / (int)gridDim.x;
  const int u_begin = (int)blockIdx.x * per_cta;
  const int my_units = max(0, min(per_cta, A.n_units - u_begin));
  const int n_items = my_units * A.n_chunks;
  // c_format F32; a/b format TF32 (2); K-major; N = 2 nant_p; M = 128
  constexpr uint32_t fmt = 2u;
  const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) |
                         (((uint32_t)(2 * A.nant_p) >> 3) << 17) | ((128u >> 4) << 24);
  bool ok = true;
  for (int it = 0; it < n_items; ++it) {
    const int lu = it / A.n_chunks, q = it % A.n_chunks;
    const int slot = it % A.nstage;
    bool w_ok = true;
    if (it >= A.nstage) w_ok = mbar_wait(&bar_mma[slot], (uint32_t)((it / A.nstage - 1) & 1));
    if (!__syncthreads_and(w_ok)) { ok = false; break; }
    uint8_t* st = stages + (size_t)slot * A.stage_bytes;
    split_fill(A, st, u_begin + lu, q);
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t d = tmem_base + (uint32_t)((lu & 1) * 256);
      const uint32_t sbase = smem_u32(st);
#pragma unroll
      for (int m = 0; m < 4; ++m) {   // 4 MMAs of 32 bytes of K each
        const uint64_t desc = sdesc_k_sw128(sbase + (uint32_t)m * 32u);
        umma_tf32_ss(d, desc, desc, idesc, (q > 0 || m > 0) ? 1u : 0u);
      }
      umma_commit(&bar_mma[slot]);
      if (q == A.n_chunks - 1) umma_commit(&bar_acc[lu & 1]);
    }
    if (q == A.n_chunks - 1 && lu >= 1) {
      const int pl = lu - 1;
      const bool a_ok = mbar_wait(&bar_acc[pl & 1], (uint32_t)((pl >> 1) & 1));
      if (!__syncthreads_and(a_ok)) { ok = false; break; }
      tc_fence_after();
      split_epilogue(A, tmem_base, pl & 1, u_begin + pl);
      tc_fence_before();
    }
  }
  if (ok && my_units > 0) {
    const int pl = my_units - 1;
    const bool a_ok = mbar_wait(&bar_acc[pl & 1], (uint32_t)((pl >> 1) & 1));
    if (__syncthreads_and(a_ok)) {
      tc_fence_after();
      split_epilogue(A, tmem_base, pl & 1, u_begin + pl);
    } else {
      ok = false;
    }
  }
  if (!ok && tid == 0) {
    dsb_flag(A.status, DSB_E_TIMEOUT);
    // drain every MMA this CTA issued before tensor memory is released
    umma_commit(bar_drain);
    mbar_wait(bar_drain, 0u);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TC_TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// The same correlator for int8 and float16 voltages, operands antenna-major.
//
// What bounds it: the voltages are read once (1.2 GB for a native float16
// page), the products (four real 128 x nant x K ones per unit) need half of
// that time on the tensor cores.  The K-major form above transposes every
// element through 2-byte loads: 7.55 ms for that page (2048 packets, 96
// antennas, 384 channels, 16 channels summed).  Here the operands stay as
// they lie in memory, rows of antennas: tcgen05 reads A and B "MN-major" (128-byte
// swizzle: atoms of 64 antennas x 8 samples, LBO between the two antenna
// atoms, SBO between sample groups of 8), so that staging is a copy of 16-byte
// chunks.  Re and Im get their own accumulators and four products per 16
// samples, R_b R_a + I_b I_a and R_b I_a - I_b R_a, the sign by the
// descriptor's negate-A bit, which drops the second [I | -R] operand copy.
// Roles: warps 0-3 write the finished unit, warps 4-11 stage samples (rows of
// a multiple of 8 float16 antennas by 16-byte asynchronous copies
// MN_LAG stages ahead; other rows through registers, words funnel-shifted
// to the row's offset), one thread of warp 12 issues the products: 0.57 ms for the same
// page, exact sums unchanged.
// ---------------------------------------------------------------------------
constexpr int MN_EPI = 128, MN_LOAD = 256, MN_THREADS = MN_EPI + MN_LOAD + 32;
constexpr int MN_KC = 64;                        // samples per stage
constexpr int MN_PART = 2 * MN_KC * 128;         // bytes of one part (two antenna atoms)
constexpr int MN_STAGE = 2 * MN_PART;            // real and imaginary parts
constexpr int MN_NST = 6;
constexpr int MN_LAG = 4;                        // copy stages in flight per loader thread
constexpr int MN_SMEM = MN_NST * MN_STAGE + 1024 + (2 * MN_NST + 5) * 8 + 16;
static_assert(MN_LAG < MN_NST && MN_SMEM <= 227 * 1024, "stages of one CTA per SM");

// Shared-memory descriptor of an MN-major operand in the 128-byte swizzle:
// atoms of 64 elements x 8 rows of K (1024 bytes), LBO = distance of the next
// 64 elements, SBO = distance of the next 8 rows of K.
DSB_DEV uint64_t sdesc_mn_sw128(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)2u << 61;
  return d;
}

DSB_DEV void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Four int8 codes (one word) as four float16 values: 0x6400 | (x + 128) is
// the half 1024 + x + 128, exactly.
DSB_DEV uint2 s8x4_to_h4(uint32_t w) {
  const uint32_t b = w ^ 0x80808080u;
  const __half2 off = __halves2half2(__ushort_as_half((unsigned short)0x6480),
                                     __ushort_as_half((unsigned short)0x6480));  // 1152
  uint32_t lo = __byte_perm(b, 0x64646464u, 0x4140);
  uint32_t hi = __byte_perm(b, 0x64646464u, 0x4342);
  const __half2 l = __hsub2(*reinterpret_cast<__half2*>(&lo), off);
  const __half2 h = __hsub2(*reinterpret_cast<__half2*>(&hi), off);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&l), *reinterpret_cast<const uint32_t*>(&h));
}

// Eight elements (ESZ bytes each) from element o on, as 16 bytes of float16:
// the aligned words that hold them, shifted to o.  Words past n_words, the
// tensor's last, read as zero.
template <int ESZ>
DSB_DEV void mn_words(const void* p, size_t o, size_t n_words, uint32_t (&w)[2 * ESZ + 1]) {
  const uint32_t* q = static_cast<const uint32_t*>(p);
  const size_t w0 = o * ESZ / 4;
#pragma unroll
  for (int i = 0; i < 2 * ESZ + 1; ++i) w[i] = w0 + i < n_words ? __ldg(q + w0 + i) : 0u;
}
template <int ESZ>
DSB_DEV uint4 mn_shift(size_t o, const uint32_t (&w)[2 * ESZ + 1]) {
  const unsigned sh = (unsigned)(o * ESZ % 4) * 8u;
  uint32_t v[2 * ESZ];
#pragma unroll
  for (int i = 0; i < 2 * ESZ; ++i) v[i] = __funnelshift_r(w[i], w[i + 1], sh);
  if constexpr (ESZ == 2) return make_uint4(v[0], v[1], v[2], v[3]);
  const uint2 a = s8x4_to_h4(v[0]), b = s8x4_to_h4(v[1]);
  return make_uint4(a.x, a.y, b.x, b.y);
}

// The writing warps (the CTA's first NT threads): accumulator lane b, columns
// a (Re), 128 + a (Im); the upper triangle b <= a goes to bls(a, b).  With
// staged outputs (A.q_pitch) those of up to TC_QF adjacent units leave
// together, four lanes to a baseline's 32-byte sector.  False if a wait ran
// out.
template <int NT>
DSB_DEV bool mn_write_units(const SplitTcArgs& A, uint32_t tmem_base, int u_begin, int my_units,
                            uint64_t* bar_acc, uint64_t* bar_out, float2* vbuf) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int quarter = warp & 3, part = warp >> 2;
  const int nant = A.nant, nbase = nant * (nant + 1) / 2;
  const int b = quarter * 32 + lane;
  for (int lu = 0; lu < my_units; ++lu) {
    const int buf = lu & 1;
    const bool ok = mbar_wait(&bar_acc[buf], (uint32_t)((lu >> 1) & 1));
    // (the warps agree, and the previous unit's reads of vbuf are done)
    int all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, 1, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"((int)ok), "n"(NT)
        : "memory");
    if (!all) return false;
    tc_fence_after();
    int fv, ch0, pol0, npol_u;
    split_unit(A, u_begin + lu, fv, ch0, pol0, npol_u);
    const size_t step = A.fuse ? (size_t)A.ceff : (size_t)A.nchan * 2;
    float2* o = A.out + (A.fuse ? (size_t)fv * nbase * A.ceff + ch0 / A.csf
                                : ((size_t)fv * nbase * A.nchan + ch0) * 2 + pol0);
    // place among the adjacent units of its row of outputs
    const int n_fast = A.fuse ? A.ceff : 2 * A.nchan;
    const int fast = (u_begin + lu) % n_fast, j1 = fast & (TC_QF - 1);
    const uint32_t lane_base =
        tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * 256);
    for (int c0 = quarter * 32 + 16 * part; c0 < nant; c0 += NT / 8) {
      __syncwarp();
      uint32_t vr[16], vi[16];
      tmem_ld16(lane_base + (uint32_t)c0, vr);
      tmem_ld16(lane_base + 128u + (uint32_t)c0, vi);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int a = c0 + j;
        if (a < b || a >= nant) continue;
        const float2 z = make_float2(__uint_as_float(vr[j]), __uint_as_float(vi[j]));
        if (A.q_pitch) vbuf[j1 * A.q_pitch + upper_bls(a, b)] = z;
        else o[(size_t)upper_bls(a, b) * step] = z;
      }
    }
    tc_fence_before();
    mbar_arrive(&bar_out[buf]);
    if (A.q_pitch && (j1 == TC_QF - 1 || fast == n_fast - 1 || lu == my_units - 1)) {
      asm volatile("barrier.cta.sync 1, %0;" ::"n"(NT) : "memory");
      const int q = threadIdx.x & (TC_QF - 1);
      if (q >= max(0, j1 - lu) && q <= j1)
        for (int bls = threadIdx.x / TC_QF; bls < nbase; bls += NT / TC_QF)
          o[(size_t)bls * step + q - j1] = vbuf[q * A.q_pitch + bls];
    }
  }
  return true;
}

// The products of one stage of `rows` samples (part_bytes apart, antenna
// atoms rows * 128 bytes apart) into accumulator columns d (Re), d + 128 (Im).
DSB_DEV void mn_products(uint32_t d, uint32_t idesc, uint32_t stage, uint32_t part_bytes,
                         uint32_t rows, int n16, bool first) {
  constexpr uint32_t NEG_A = 1u << 13;
  for (int m = 0; m < n16; ++m) {
    const uint64_t R = sdesc_mn_sw128(stage + (uint32_t)m * 2048u, rows * 128, 1024);
    const uint64_t I = sdesc_mn_sw128(stage + part_bytes + (uint32_t)m * 2048u, rows * 128, 1024);
    const uint32_t acc = (!first || m > 0) ? 1u : 0u;
    umma_f16_ss(d, R, R, idesc, acc);
    umma_f16_ss(d, I, I, idesc, 1u);
    umma_f16_ss(d + 128u, R, I, idesc, acc);
    umma_f16_ss(d + 128u, I, R, idesc | NEG_A, 1u);
  }
}

// ESZ: bytes of a voltage part (1 int8, 2 float16); COPY: float16 rows in
// whole 16-byte chunks, staged by asynchronous copies.
template <int ESZ, bool COPY>
__global__ void __launch_bounds__(MN_THREADS, 1) corr_split_mn_kernel(const SplitTcArgs A) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* stages = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(stages + (size_t)MN_NST * MN_STAGE);
  uint64_t* bar_free = bar_full + MN_NST;
  uint64_t* bar_acc = bar_free + MN_NST;     // [2] accumulator finished
  uint64_t* bar_out = bar_acc + 2;           // [2] accumulator written out
  uint64_t* bar_drain = bar_out + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_drain + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    tmem_alloc(tmem_slot, TC_TMEM_COLS);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < MN_NST; ++i) {
      mbar_init(&bar_full[i], MN_LOAD);
      mbar_init(&bar_free[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_acc[i], 1);
      mbar_init(&bar_out[i], MN_EPI);
    }
    mbar_init(bar_drain, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int per_cta = (A.n_units + (int)gridDim.x - 1) / (int)gridDim.x;
  const int u_begin = (int)blockIdx.x * per_cta;
  const int my_units = max(0, min(per_cta, A.n_units - u_begin));
  const int n_items = my_units * A.n_chunks;
  bool ok = true;

  if (warp < MN_EPI / 32) {
    ok = mn_write_units<MN_EPI>(A, tmem_base, u_begin, my_units, bar_acc, bar_out, nullptr);
  } else if (warp < (MN_EPI + MN_LOAD) / 32) {
    // ---- stage samples: thread (j, r) copies antennas 8j .. 8j + 7 of rows
    //      r, r + 16, ... of the stage ----
    const int lt = tid - MN_EPI;
    const int j = lt & 15, r0 = lt >> 4;
    const bool mine = 8 * j < A.nant;
    const size_t plane = (size_t)A.npkt * A.nant;
    // 4-byte words that hold the tensors (the last one may hold more)
    const size_t n_el = plane * A.nchan * 4;
    const size_t nw_re = ((n_el + A.off_re) * ESZ + 3) / 4, nw_im = ((n_el + A.off_im) * ESZ + 3) / 4;
    const uint32_t jo = (uint32_t)(j >> 3) * (MN_KC * 128);
    const int lag = COPY ? MN_LAG : 0;
    for (int it = 0; it < n_items + lag; ++it) {
      if (it < n_items) {
        const int slot = it % MN_NST;
        if (it >= MN_NST)
          ok = __all_sync(0xffffffffu,
                          mbar_wait(&bar_free[slot], (uint32_t)((it / MN_NST - 1) & 1)));
        if (!ok) break;
        const int q = it % A.n_chunks;
        int fv, ch0, pol0, npol_u;
        split_unit(A, u_begin + it / A.n_chunks, fv, ch0, pol0, npol_u);
        // row k of the unit: plane k / ppfv (Stokes-I: consecutive (ch, t,
        // pol); 2-pol: the unit's pol of t = 0, 1), packet k % ppfv
        const int pl_step = A.fuse ? 1 : 2;
        const size_t base = ((size_t)ch0 * 4 + pol0) * plane + (size_t)fv * A.ppfv * A.nant + 8 * j;
        uint8_t* st = stages + (size_t)slot * MN_STAGE;
        const int rows = (min(MN_KC, A.kprime - q * MN_KC) + 15) & ~15;  // whole products
        if (mine) {
          size_t o[MN_KC / 16];
          bool in[MN_KC / 16];
          uint32_t so[MN_KC / 16];
#pragma unroll
          for (int i = 0; i < MN_KC / 16; ++i) {
            const int r = r0 + 16 * i, k = q * MN_KC + r;
            const int pl = k / A.ppfv, pk = k - pl * A.ppfv;
            in[i] = k < A.kprime;
            o[i] = in[i] ? base + (size_t)(pl * pl_step) * plane + (size_t)pk * A.nant : 0;
            so[i] = jo + (uint32_t)r * 128u + (uint32_t)(((j ^ r) & 7) << 4);
          }
          if constexpr (COPY) {
#pragma unroll
            for (int i = 0; i < MN_KC / 16; ++i) {
              if (r0 + 16 * i >= rows) continue;
              if (in[i]) {
                cp_async16(smem_u32(st + so[i]), static_cast<const __half*>(A.re) + o[i]);
                cp_async16(smem_u32(st + MN_PART + so[i]), static_cast<const __half*>(A.im) + o[i]);
              } else {
                *reinterpret_cast<uint4*>(st + so[i]) = make_uint4(0u, 0u, 0u, 0u);
                *reinterpret_cast<uint4*>(st + MN_PART + so[i]) = make_uint4(0u, 0u, 0u, 0u);
              }
            }
          } else {
            uint32_t wr[MN_KC / 16][2 * ESZ + 1], wi[MN_KC / 16][2 * ESZ + 1];
#pragma unroll
            for (int i = 0; i < MN_KC / 16; ++i)
              if (in[i]) {
                mn_words<ESZ>(A.re, o[i] + A.off_re, nw_re, wr[i]);
                mn_words<ESZ>(A.im, o[i] + A.off_im, nw_im, wi[i]);
              }
#pragma unroll
            for (int i = 0; i < MN_KC / 16; ++i) {
              if (r0 + 16 * i >= rows) continue;
              const uint4 z = make_uint4(0u, 0u, 0u, 0u);
              *reinterpret_cast<uint4*>(st + so[i]) = in[i] ? mn_shift<ESZ>(o[i] + A.off_re, wr[i]) : z;
              *reinterpret_cast<uint4*>(st + MN_PART + so[i]) =
                  in[i] ? mn_shift<ESZ>(o[i] + A.off_im, wi[i]) : z;
            }
          }
        }
      }
      if constexpr (COPY) {
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (it >= lag) asm volatile("cp.async.wait_group %0;" ::"n"(MN_LAG) : "memory");
      }
      if (it >= lag) {
        fence_proxy_async_smem();
        mbar_arrive(&bar_full[(it - lag) % MN_NST]);
      }
    }
    if constexpr (COPY) asm volatile("cp.async.wait_group 0;" ::: "memory");
  } else if (lane == 0) {
    // ---- issue the products ----
    // c_format F32, a/b format F16, both MN-major; N = nant in 16s; M = 128
    const uint32_t n_b = (uint32_t)((A.nant + 15) & ~15);
    const uint32_t idesc = (1u << 4) | (1u << 15) | (1u << 16) | ((n_b >> 3) << 17) |
                           ((128u >> 4) << 24);
    for (int it = 0; ok && it < n_items; ++it) {
      const int lu = it / A.n_chunks, q = it % A.n_chunks;
      const int slot = it % MN_NST, buf = lu & 1;
      if (q == 0 && lu >= 2) ok = mbar_wait(&bar_out[buf], (uint32_t)(((lu >> 1) - 1) & 1));
      ok = ok && mbar_wait(&bar_full[slot], (uint32_t)((it / MN_NST) & 1));
      if (!ok) break;
      tc_fence_after();
      mn_products(tmem_base + (uint32_t)(buf * 256), idesc,
                  smem_u32(stages + (size_t)slot * MN_STAGE), MN_PART, MN_KC,
                  (min(MN_KC, A.kprime - q * MN_KC) + 15) >> 4, q == 0);
      umma_commit(&bar_free[slot]);
      if (q == A.n_chunks - 1) umma_commit(&bar_acc[buf]);
    }
    // a wait that ran out anywhere: every product issued here has to end
    // before tensor memory and the stages are given back
    umma_commit(bar_drain);
    mbar_wait(bar_drain, 0u);
  }
  if (!ok && lane == 0) dsb_flag(A.status, DSB_E_TIMEOUT);
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TC_TMEM_COLS);
  }
}

// The same on float16 voltages whose samples TMA can bring in: rows of a
// multiple of 8 antennas, 16-byte aligned, and stages of whole runs of packets
// (split_tma_plan).  One thread issues up to four copies per stage (real and
// imaginary parts, one or two antenna atoms), so that the load runs at memory
// speed: asynchronous copies by 256 threads took 431 us for a native page by
// themselves.  The stages are short (32 samples) to leave room for the staged
// outputs of four units.  Native float16 page: 0.57 -> 0.36 ms.
constexpr int ST_EPI = 256, ST_THREADS = ST_EPI + 64, ST_MAX_STAGES = 12;
constexpr int ST_EXTRA = 1024 + (2 * ST_MAX_STAGES + 5) * 8 + 32;

__global__ void __launch_bounds__(ST_THREADS, 1) corr_split_tma_kernel(
    const SplitTcArgs A, const __grid_constant__ CUtensorMap map_re,
    const __grid_constant__ CUtensorMap map_im) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* stages = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(stages + (size_t)A.nstage * A.stage_bytes);
  uint64_t* bar_free = bar_full + A.nstage;
  uint64_t* bar_acc = bar_free + A.nstage;   // [2] accumulator finished
  uint64_t* bar_out = bar_acc + 2;           // [2] accumulator written out
  uint64_t* bar_drain = bar_out + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_drain + 1);
  float2* vbuf = reinterpret_cast<float2*>(tmem_slot + 4);   // [TC_QF][q_pitch]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    tmem_alloc(tmem_slot, TC_TMEM_COLS);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < A.nstage; ++i) {
      mbar_init(&bar_full[i], 1);
      mbar_init(&bar_free[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_acc[i], 1);
      mbar_init(&bar_out[i], ST_EPI);
    }
    mbar_init(bar_drain, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int per_cta = (A.n_units + (int)gridDim.x - 1) / (int)gridDim.x;
  const int u_begin = (int)blockIdx.x * per_cta;
  const int my_units = max(0, min(per_cta, A.n_units - u_begin));
  const int n_atoms = A.nant > 64 ? 2 : 1;
  const uint32_t atom = (uint32_t)A.rows * 128u, part = 2 * atom;   // bytes
  bool ok = true;

  if (warp < ST_EPI / 32) {
    ok = mn_write_units<ST_EPI>(A, tmem_base, u_begin, my_units, bar_acc, bar_out, vbuf);
  } else if (warp == ST_EPI / 32) {
    if (lane == 0) {
      int issued = 0, slot = 0;
      uint32_t ph = 1u;   // parity of the stage's previous use (the first passes have none)
      for (int lu = 0; ok && lu < my_units; ++lu) {
        int fv, ch0, pol0, npol_u;
        split_unit(A, u_begin + lu, fv, ch0, pol0, npol_u);
        // sample rows of the unit: packet fastest, then pol, then (ch, t)
        int pk = 0, pl = 0;
        for (int q = 0; q < A.n_chunks; ++q) {
          if (issued >= A.nstage) ok = mbar_wait(&bar_free[slot], ph);
          if (!ok) break;
          const int x1 = fv * A.ppfv + pk;
          const int x2 = npol_u == 2 ? (pl & 1) : pol0, x3 = 2 * ch0 + (npol_u == 2 ? pl >> 1 : pl);
          uint8_t* st = stages + (size_t)slot * A.stage_bytes;
          mbar_arrive_expect_tx(&bar_full[slot], 2u * (uint32_t)n_atoms * atom);
          for (int a = 0; a < n_atoms; ++a) {
            tma_load_4d(st + a * atom, &map_re, 64 * a, x1, x2, x3, &bar_full[slot]);
            tma_load_4d(st + part + a * atom, &map_im, 64 * a, x1, x2, x3, &bar_full[slot]);
          }
          pk += A.rows;   // whole packet runs: a stage ends inside a plane or at its end
          while (pk >= A.ppfv) {
            pk -= A.ppfv;
            ++pl;
          }
          ++issued;
          if (++slot == A.nstage) {
            slot = 0;
            ph ^= 1u;
          }
        }
      }
      // no copy may be in flight into this CTA's shared memory when it ends
      for (int it = max(0, issued - A.nstage); it < issued; ++it)
        mbar_wait(&bar_full[it % A.nstage], (uint32_t)((it / A.nstage) & 1));
    }
  } else if (lane == 0) {
    const uint32_t n_b = (uint32_t)((A.nant + 15) & ~15);
    const uint32_t idesc = (1u << 4) | (1u << 15) | (1u << 16) | ((n_b >> 3) << 17) |
                           ((128u >> 4) << 24);
    int slot = 0;
    uint32_t ph = 0u;
    for (int lu = 0; ok && lu < my_units; ++lu) {
      const int buf = lu & 1;
      if (lu >= 2) ok = mbar_wait(&bar_out[buf], (uint32_t)(((lu >> 1) - 1) & 1));
      for (int q = 0; ok && q < A.n_chunks; ++q) {
        ok = mbar_wait(&bar_full[slot], ph);
        if (!ok) break;
        tc_fence_after();
        mn_products(tmem_base + (uint32_t)(buf * 256), idesc,
                    smem_u32(stages + (size_t)slot * A.stage_bytes), part, (uint32_t)A.rows,
                    A.rows / 16, q == 0);
        umma_commit(&bar_free[slot]);
        if (++slot == A.nstage) {
          slot = 0;
          ph ^= 1u;
        }
      }
      if (ok) umma_commit(&bar_acc[buf]);
    }
    // every product issued here ends before tensor memory is given back
    umma_commit(bar_drain);
    mbar_wait(bar_drain, 0u);
  }
  if (!ok) dsb_flag(A.status, DSB_E_TIMEOUT);
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TC_TMEM_COLS);
  }
}

int g_num_sms = 0;
int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

int launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? DSB_OK : DSB_E_CUDA;
}

// Shared memory beyond the operand stages: mode 0 the staged outputs, mode 1 the upper-triangle
// visibilities of one unit (int2) and the gridding tables of one group.
int tc_extra_bytes(const TcArgs& A, int mode) {
  if (mode != 1) return A.q_pitch * TC_QF * 8;
  const int nbase = A.nant * (A.nant + 1) / 2;
  return nbase * 8 + 16 + nbase * 2 + (A.cap_rows + 1) * 2 + 16;
}

// Offsets of more rows in `room` bytes that the stages leave free (no more
// than the subbands can give: one row per baseline and subband).
void tc_fit_rows(TcArgs& A, int room) {
  const long long most = (long long)A.nant * (A.nant + 1) / 2 * A.ceff;
  A.cap_rows = (int)std::max<long long>(A.cap_rows, std::min<long long>(most, A.cap_rows + room / 2));
}

// Fill the derived geometry; returns DSB_OK or an error code.
int tc_plan(TcArgs& A, int mode) {
  if (A.nant < 16 || A.nant > 128 || (A.nant % 16) != 0) return DSB_E_UNSUPPORTED;
  if (A.t_int <= 0 || (A.t_int % 2) != 0 || A.npkt % (A.t_int / 2) != 0) return DSB_E_ARG;
  if (A.csf <= 0 || A.nchan % A.csf != 0) return DSB_E_ARG;
  A.ppfv = A.t_int / 2;
  A.n_fv = A.npkt / A.ppfv;
  A.ceff = A.nchan / A.csf;
  const int kprime = 2 * A.t_int * A.csf;  // complex samples per antenna per unit
  if (kprime % 16 != 0) return DSB_E_UNSUPPORTED;
  A.kc = std::min(kprime, 128);
  while (kprime % A.kc != 0) A.kc -= 16;
  A.n_chunks = kprime / A.kc;
  A.rows = std::max(128, ((2 * A.nant + 7) / 8) * 8);
  A.nkblk = (2 * A.kc + 127) / 128;
  A.stage_bytes = A.nkblk * A.rows * 128;
  A.n_mma = 2 * A.kc / 32;
  A.tma = 0;
  A.q_pitch = 0;
  A.cap_rows = tc_min_rows(A.nant);
  const int budget = TC_SMEM_BUDGET - tc_extra_bytes(A, mode) - 1024 - 256;
  A.nstage = std::min(4, budget / A.stage_bytes);
  if (A.nstage < 2) return DSB_E_UNSUPPORTED;
  tc_fit_rows(A, budget - A.nstage * A.stage_bytes);
  return DSB_OK;
}

// Plan corr_ws_kernel (A.tma) when a chunk of kc samples is whole packets of
// 16-byte channel runs and four raw stages leave two operand stages: as many
// CTAs per SM as tensor memory, registers and shared memory hold.  q_pitch:
// the staged outputs' pitch (0: none).
bool ws_plan(TcArgs& A, int mode, int kc, int q_pitch) {
  const int kprime = 2 * A.t_int * A.csf;
  if (kc <= 0 || kc > kprime || kprime % kc || kc % 16 || (A.csf % 4) || (A.nchan % 4) ||
      ((kc / 4) % A.csf))
    return false;
  TcArgs P = A;
  P.cap_rows = tc_min_rows(P.nant);
  P.kc = kc;
  P.n_chunks = kprime / kc;
  P.nkblk = (2 * kc + 127) / 128;
  P.stage_bytes = P.nkblk * P.rows * 128;
  P.n_mma = 2 * kc / 32;
  P.q_pitch = q_pitch;
  P.ppk = (kc / 4) / P.csf;
  P.raw_stage = (P.ppk * P.nant * P.csf * 4 + 1023) & ~1023;
  P.nraw = 4;
  P.unpackers = P.nant * (kc / 16) <= 64 * TC_PRE ? 64 : 256;
  P.tmem_cols = 32;
  while (P.tmem_cols < 4 * P.nant) P.tmem_cols *= 2;
  for (P.ctas = std::min(P.unpackers == 64 ? WsCfg<64>::CTAS : WsCfg<256>::CTAS,
                         TC_TMEM_COLS / P.tmem_cols);
       P.ctas >= 1; --P.ctas) {
    const int room = std::min(TC_SMEM_BUDGET, 228 * 1024 / P.ctas - 1024) -
                     tc_extra_bytes(P, mode) - 1024 - 256;
    const int ns = std::min(4, (room - P.nraw * P.raw_stage) / P.stage_bytes);
    if (ns < 2) continue;
    tc_fit_rows(P, room - P.nraw * P.raw_stage - ns * P.stage_bytes);
    P.tma = 1;
    P.ws_nstage = ns;
    A = P;
    return true;
  }
  return false;
}

// The TMA form's plan, if it has one: mode 0 with outputs of adjacent units
// staged where they are adjacent in memory (with 96 antennas that takes
// chunks of 64 samples instead of 128) and the CTAs have TC_QF units or more
// each to write together: 269 -> 116 us for 3072 units of 96 antennas at the
// 262-us cadence, but 10.2 -> 12.7 us for 24 (equal near 600, four per CTA).
void ws_choose(TcArgs& A, int mode, int n_units, int max_ctas) {
  const int nbase = A.nant * (A.nant + 1) / 2;
  // pitch = 4 mod 16 eight-byte words: four units' reads in different banks
  const int pitch = (nbase + 15) / 16 * 16 + 4;
  TcArgs P = A;
  if (mode == 0 && (A.unit_order ? A.o_s : A.o_f) == 1 &&
      (ws_plan(P, mode, P.kc, pitch) || ws_plan(P, mode, 64, pitch)) &&
      n_units > (TC_QF - 1) * (max_ctas > 0 ? max_ctas : P.ctas * num_sms())) {
    A = P;
    return;
  }
  ws_plan(A, mode, A.kc, 0);
}

// The driver's tensor-map encoder, looked up once through the runtime.
PFN_cuTensorMapEncodeTiled_v12000 tmap_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    cudaGetLastError();
  }
  return fn;
}

// The raw pages as a 4-D uint8 tensor (channel bytes, antenna, packet,
// chgroup) with one item's box (csf channels x 4 bytes, every antenna, ppk
// packets, one chgroup).  False if it cannot be encoded (the kernel then
// loads the raw words itself).
bool tc_raw_tmap(const TcArgs& A, CUtensorMap* m) {
  auto fn = tmap_encoder();
  if (!fn) return false;
  const cuuint64_t row = (cuuint64_t)A.nchan * 4;
  const cuuint64_t pkt = row * (cuuint64_t)A.nant;
  const cuuint64_t gs = A.n_chgroup > 1 ? (cuuint64_t)A.raw_g_stride : pkt * (cuuint64_t)A.npkt;
  const cuuint64_t dims[4] = {row, (cuuint64_t)A.nant, (cuuint64_t)A.npkt,
                              (cuuint64_t)A.n_chgroup};
  const cuuint64_t strides[3] = {row, pkt, gs};
  const cuuint32_t box[4] = {(cuuint32_t)(A.csf * 4), (cuuint32_t)A.nant, (cuuint32_t)A.ppk, 1u};
  const cuuint32_t es[4] = {1u, 1u, 1u, 1u};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<uint8_t*>(A.raw), dims, strides, box,
            es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_64B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Launch on the planned geometry: n_units units over at most max_ctas CTAs
// (0: what the device holds).
template <int MODE>
int tc_launch(TcArgs& A, int n_units, int max_ctas, cudaStream_t stream) {
  CUtensorMap tmap;
  memset(&tmap, 0, sizeof(tmap));
  const TcArgs plain = A;
  ws_choose(A, MODE, n_units, max_ctas);
  if (A.tma && !tc_raw_tmap(A, &tmap)) A = plain;
  if (A.tma) {
    A.nstage = A.ws_nstage;
    // at least what keeps more than `ctas` CTAs (and their tensor memory) off an SM
    const int smem = std::max(A.nstage * A.stage_bytes + A.nraw * A.raw_stage + 1024 + 256 +
                                  tc_extra_bytes(A, MODE),
                              228 * 1024 / (A.ctas + 1));
    const int grid = std::min(n_units, max_ctas > 0 ? max_ctas : A.ctas * num_sms());
    auto go = [&](auto kern, int threads) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      kern<<<grid, threads, smem, stream>>>(A, tmap);
      return launch_status();
    };
    return A.unpackers == 64 ? go(corr_ws_kernel<MODE, 64>, WsCfg<64>::THREADS)
                             : go(corr_ws_kernel<MODE, 256>, WsCfg<256>::THREADS);
  }
  const int smem = std::max(A.nstage * A.stage_bytes + 1024 + 256 + tc_extra_bytes(A, MODE),
                            TC_MIN_SMEM);
  cudaFuncSetAttribute(corr_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  corr_tc_kernel<MODE><<<std::min(n_units, max_ctas > 0 ? max_ctas : num_sms()), TC_THREADS, smem,
                         stream>>>(A);
  return launch_status();
}

// Plan corr_split_tma_kernel and its tensor maps, if the unit's samples come
// in stages of `rows` (16 or 32) that are whole packet runs of one box: a
// part as a 4-D float16 tensor (antenna, packet, pol, channel x t).
bool split_tma_plan(SplitTcArgs& A, CUtensorMap* re, CUtensorMap* im) {
  auto fn = tmap_encoder();
  if (!fn || A.nant % 8) return false;
  SplitTcArgs P = A;
  P.rows = P.kprime % 32 == 0 ? 32 : 16;
  if (P.kprime % P.rows) return false;
  const int npol = P.fuse ? 2 : 1;
  int pk, pol, cht;   // box
  if (P.ppfv % P.rows == 0) {
    pk = P.rows; pol = 1; cht = 1;
  } else if (P.rows % P.ppfv == 0) {
    const int planes = P.rows / P.ppfv;
    if (planes % npol) return false;
    pk = P.ppfv; pol = npol; cht = planes / npol;
  } else {
    return false;
  }
  P.n_chunks = P.kprime / P.rows;
  P.stage_bytes = 4 * P.rows * 128;
  const int room = 227 * 1024 - ST_EXTRA, nbase = P.nant * (P.nant + 1) / 2;
  P.q_pitch = (nbase + 15) / 16 * 16 + 4;
  if (room - P.q_pitch * TC_QF * 8 < 4 * P.stage_bytes) P.q_pitch = 0;
  P.nstage = std::min(ST_MAX_STAGES, (room - P.q_pitch * TC_QF * 8) / P.stage_bytes);
  const cuuint64_t row = (cuuint64_t)P.nant * 2, plane = row * (cuuint64_t)P.npkt;
  const cuuint64_t dims[4] = {(cuuint64_t)P.nant, (cuuint64_t)P.npkt, 2u,
                              (cuuint64_t)P.nchan * 2};
  const cuuint64_t strides[3] = {row, plane, 2 * plane};
  const cuuint32_t box[4] = {64u, (cuuint32_t)pk, (cuuint32_t)pol, (cuuint32_t)cht};
  const cuuint32_t es[4] = {1u, 1u, 1u, 1u};
  auto enc = [&](CUtensorMap* m, const void* p) {
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(p), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
  };
  if (!enc(re, P.re) || !enc(im, P.im)) return false;
  A = P;
  return true;
}

}  // namespace

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

int dsb_version(void) { return DSB_VERSION; }

const char* dsb_strerror(int code) {
  switch (code) {
    case DSB_OK: return "ok";
    case DSB_E_ARG: return "invalid argument";
    case DSB_E_CUDA: return "CUDA runtime error";
    case DSB_E_UNSUPPORTED: return "unsupported geometry";
    case DSB_E_TIMEOUT: return "device-side bounded wait ran out";
    case DSB_E_CAPACITY: return "size exceeds a fixed capacity";
    case DSB_E_BOUNDS: return "index out of range (bounds-checked build)";
    default: return "unknown error";
  }
}

int dsb_unpack_int4(const void* raw, int npkt, int nant, int nchan, int out_dtype, float scale,
                    void* out_re, void* out_im, cudaStream_t stream) {
  if (!raw || !out_re || !out_im || npkt <= 0 || nant <= 0 || nchan <= 0) return DSB_E_ARG;
  if (out_dtype != DSB_DT_INT8 && out_dtype != DSB_DT_F16 && out_dtype != DSB_DT_F32)
    return DSB_E_ARG;
  const int rows = npkt * nant;
  const uint32_t* r = static_cast<const uint32_t*>(raw);
  // four rows per store where every plane of rows starts on that boundary, in
  // calls of enough 128 x 32 tiles: with fewer the four times as many small
  // tiles end sooner (32 tiles of float16 3.1 and 3.4 us, 48 3.6 and 3.4;
  // float32, whose stores are 128 bytes either way, 384 tiles 9.0 and 9.5 us,
  // 1152 33.9 and 30.4)
  const size_t esz = out_dtype == DSB_DT_INT8 ? 1 : out_dtype == DSB_DT_F16 ? 2 : 4;
  const long long tiles = (long long)((rows + 127) / 128) * ((nchan + 31) / 32);
  const bool four = rows % 4 == 0 && tiles >= (esz == 4 ? 592 : 40) && (((uintptr_t)out_re | (uintptr_t)out_im) % (4 * esz)) == 0;
  auto go = [&](auto t) {
    using T = decltype(t);
    T *re = static_cast<T*>(out_re), *im = static_cast<T*>(out_im);
    if (four)
      unpack4_kernel<T><<<dim3((rows + 127) / 128, (nchan + 31) / 32), 256, 0, stream>>>(
          r, rows, nchan, scale, re, im);
    else
      unpack_kernel<T><<<dim3((rows + 31) / 32, (nchan + 31) / 32), dim3(32, 8), 0, stream>>>(
          r, rows, nchan, scale, re, im);
    return launch_status();
  };
  if (out_dtype == DSB_DT_INT8) return go(int8_t{});
  if (out_dtype == DSB_DT_F16) return go(__half{});
  return go(float{});
}

int dsb_corr_split(const void* re, const void* im, int in_dtype, int nchan, int npkt, int nant,
                   int t_int, int fuse_stokes_i, int csf, void* out, int* status,
                   cudaStream_t stream) {
  if (!re || !im || !out || nchan <= 0 || npkt <= 0 || nant <= 0) return DSB_E_ARG;
  if (t_int <= 0 || t_int % 2 || npkt % (t_int / 2)) return DSB_E_ARG;
  if (nant > 128) return DSB_E_UNSUPPORTED;
  if (in_dtype != DSB_DT_INT8 && in_dtype != DSB_DT_F16 && in_dtype != DSB_DT_F32)
    return DSB_E_ARG;
  SplitTcArgs A{};
  A.re = re; A.im = im;
  A.nchan = nchan; A.npkt = npkt; A.nant = nant;
  A.nant_p = (nant + 7) & ~7;
  A.ppfv = t_int / 2;
  A.n_fv = npkt / A.ppfv;
  A.fuse = fuse_stokes_i ? 1 : 0;
  if (A.fuse) {
    if (csf <= 0 || nchan % csf) return DSB_E_ARG;
    A.csf = csf;
    A.ceff = nchan / csf;
    A.n_units = A.n_fv * A.ceff;
    A.kprime = 2 * csf * t_int;     // (channel, pol, t-sub, packet)
  } else {
    A.csf = 1;
    A.ceff = nchan;
    A.n_units = A.n_fv * nchan * 2;
    A.kprime = t_int;               // (t-sub, packet)
  }
  const int kc = in_dtype == DSB_DT_F32 ? 16 : MN_KC;
  A.n_chunks = (A.kprime + kc - 1) / kc;
  A.out = static_cast<float2*>(out);
  A.status = status;
  const int grid = std::min(A.n_units, num_sms());
  if (in_dtype == DSB_DT_F32) {
    A.rows = std::max(128, 2 * A.nant_p);
    A.stage_bytes = A.rows * 128;
    A.nstage = 4;
    const int smem = A.nstage * A.stage_bytes + 1024 + (A.nstage + 3) * 8 + 16;
    cudaFuncSetAttribute(corr_split_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    corr_split_tc_kernel<<<grid, TC_THREADS, smem, stream>>>(A);
    return launch_status();
  }
  const uintptr_t at_re = reinterpret_cast<uintptr_t>(re), at_im = reinterpret_cast<uintptr_t>(im);
  const bool copy = in_dtype == DSB_DT_F16 && nant % 8 == 0 && (at_re | at_im) % 16 == 0;
  const int esz = in_dtype == DSB_DT_INT8 ? 1 : 2;
  if ((at_re | at_im) % esz) return DSB_E_ARG;
  A.off_re = (int)(at_re % 4) / esz;
  A.off_im = (int)(at_im % 4) / esz;
  A.re = reinterpret_cast<const void*>(at_re & ~(uintptr_t)3);
  A.im = reinterpret_cast<const void*>(at_im & ~(uintptr_t)3);
  auto go = [&](auto kern) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MN_SMEM);
    kern<<<grid, MN_THREADS, MN_SMEM, stream>>>(A);
    return launch_status();
  };
  if (in_dtype == DSB_DT_INT8) return go(corr_split_mn_kernel<1, false>);
  if (copy) {
    CUtensorMap map_re, map_im;
    if (split_tma_plan(A, &map_re, &map_im)) {
      // more than half an SM's shared memory: one CTA (and its 512 tensor
      // memory columns) per SM
      const int smem = std::max(A.nstage * A.stage_bytes + A.q_pitch * TC_QF * 8 + ST_EXTRA,
                                TC_MIN_SMEM);
      cudaFuncSetAttribute(corr_split_tma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           smem);
      corr_split_tma_kernel<<<grid, ST_THREADS, smem, stream>>>(A, map_re, map_im);
      return launch_status();
    }
    return go(corr_split_mn_kernel<2, true>);
  }
  return go(corr_split_mn_kernel<2, false>);
}

int dsb_corr_tc(const void* raw, long long raw_g_stride, int n_chgroup, int npkt, int nant,
                int nchan, int t_int, int csf, int unit_order, void* out, long long o_g,
                long long o_f, long long o_b, long long o_s, int max_ctas, int* status,
                cudaStream_t stream) {
  if (!raw || !out || n_chgroup <= 0 || npkt <= 0) return DSB_E_ARG;
  if (((uintptr_t)raw & 15) || (raw_g_stride & 15)) return DSB_E_ARG;
  TcArgs A{};
  A.raw = static_cast<const uint8_t*>(raw);
  A.raw_g_stride = raw_g_stride;
  A.n_chgroup = n_chgroup; A.npkt = npkt; A.nant = nant; A.nchan = nchan;
  A.t_int = t_int; A.csf = csf; A.unit_order = unit_order;
  A.out = static_cast<float2*>(out);
  A.o_g = o_g; A.o_f = o_f; A.o_b = o_b; A.o_s = o_s;
  A.status = status;
  int rc = tc_plan(A, 0);
  if (rc) return rc;
  const int n_units = n_chgroup * A.n_fv * A.ceff;
  return tc_launch<0>(A, n_units, max_ctas, stream);
}

int dsb_corr_tc_grid(const void* raw, long long raw_g_stride, int n_chgroup, int npkt, int nant,
                     int nchan, int t_int, int csf, const int* yoff, const int* ycnt,
                     const int* row_off, const int* row_bls, void* yout, long long y_t_stride,
                     long long t_base, long long t_mask, int max_ctas, const void* gains,
                     int* status, cudaStream_t stream) {
  if (!raw || !yout || !yoff || !ycnt || !row_off || !row_bls) return DSB_E_ARG;
  if (((uintptr_t)raw & 15) || (raw_g_stride & 15)) return DSB_E_ARG;
  TcArgs A{};
  A.raw = static_cast<const uint8_t*>(raw);
  A.raw_g_stride = raw_g_stride;
  A.n_chgroup = n_chgroup; A.npkt = npkt; A.nant = nant; A.nchan = nchan;
  A.t_int = t_int; A.csf = csf; A.unit_order = 0;
  A.yoff = yoff; A.ycnt = ycnt; A.row_off = row_off; A.row_bls = row_bls;
  A.yout = static_cast<float2*>(yout);
  A.y_t_stride = y_t_stride; A.t_base = t_base; A.t_mask = t_mask;
  A.gains = static_cast<const float2*>(gains);
  A.status = status;
  int rc = tc_plan(A, 1);
  if (rc) return rc;
  const int n_units = n_chgroup * A.n_fv * A.ceff;
  return tc_launch<1>(A, n_units, max_ctas, stream);
}

}  // extern "C"
