// Gridding, stage-1 coarse-DM shift + grid, static-sky subtraction and the
// stage-2 per-coarse-DM delay (sm_100a).
//
// Drop-in forms (reference layouts):
//   dsb_grid_vis          FastVisGridder.compute       (n_fv, nbase, C) -> (n_fv, n_filled)
//   dsb_dedisp_vis        Stage1MultiDMCoarseDM window (T, nbase, C)    -> (n_dm, T_d, n_filled)
//   dsb_static_sky        StaticSkyMean.apply          (n_fv, n_filled) -> same
//   dsb_stage2_roll       Stage2InterChgroupShiftFifo  ring of cubes    -> aligned cube
// Pipeline form (time-major rows, ring buffers indexed by absolute time):
//   dsb_stage1_rows       per-subband gridded rows Y -> per-(chgroup, DM,
//                         cell) rows written at t + shift2 into the stage-2
//                         ring, static-sky subtraction fused.
#include "dsb_common.cuh"

#include <algorithm>
#include <type_traits>

namespace {

__global__ void grid_vis_kernel(const float2* __restrict__ vis, int n_fv, long long nsrc,
                                const int* __restrict__ off, const int* __restrict__ src,
                                int n_filled, float2* __restrict__ out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n_fv * n_filled) return;
  const int f = (int)(idx / n_filled), cell = (int)(idx % n_filled);
  const float2* v = vis + (size_t)f * nsrc;
  float re = 0.f, im = 0.f;
  for (int j = off[cell]; j < off[cell + 1]; ++j) {
    const float2 x = v[src[j]];
    re += x.x;
    im += x.y;
  }
  out[idx] = make_float2(re, im);
}

// Stage 1 on visibilities: out[d, t, cell] = sum_{src in cell}
// vis_joined[t + shift[s(src), d], src], vis_joined = concat(prev[0:n_prev],
// cur) along time.
//
// What bounds it: every visibility is needed once per coarse DM, at a
// different time for each, so the adds read n_dm x the input.  Read straight
// from global memory (one thread per output) those were 8-byte gathers a row
// of sources apart, a sector each: 23.9 ms for 32 DMs of a native page (512
// tiles, 4656 baselines x 24 subbands, 0.46 GB).  So a CTA takes 4 adjacent
// cells, 64 output times and up to 32 DMs, and stages each source's time
// window (the 64 times plus the spread of its subband's shifts over the DMs)
// in shared memory by 8-byte asynchronous copies, one batch of sources ahead:
// lanes run over the sources of a row, which are consecutive in memory where
// a baseline's subbands share a cell.  A warp then owns DPW DMs and its lanes
// the times, so that the adds read consecutive 8-byte words (no bank
// conflicts).  A batch is as many of the CTA's sources as fit, each in a
// window of its own length, across cell ends: half as many batches as with
// windows of the longest length and a batch end at each cell's (1.32 -> 0.98
// ms for the same page).  What is left is the adds' shared-memory reads (0.73
// ms without the copies) beside the copies (0.63 ms without the adds).  Each
// cell's sources are added in CSR order, as before.
constexpr int DV_TT = 64;        // output times per CTA
constexpr int DV_CELLS = 4;      // cells per CTA (32 bytes of an output row)
constexpr int DV_THREADS = 256;
constexpr int DV_SLOTS = 6144;   // float2 slots of one window buffer (offsets fit 16 bits)
constexpr int DV_MAXB = 96;      // most sources of a batch
constexpr int DV_MAX_C = 512;    // subbands whose shift tables fit

// dynamic shared memory: two window buffers, two offset tables [warp][source][its DMs],
// the subbands' shifts relative to their smallest [subband][DM] and their
// smallest and largest shift
__host__ __device__ inline size_t dv_smem_bytes(int ceff, int dg) {
  return (size_t)2 * DV_SLOTS * 8 + (size_t)2 * DV_MAXB * dg * 2 + (size_t)ceff * dg * 2 +
         (size_t)ceff * 8 + 16;
}

DSB_DEV void cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
DSB_DEV void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}
DSB_DEV void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
DSB_DEV void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int DPW>
__global__ void __launch_bounds__(DV_THREADS, 2)
    dedisp_vis_kernel(const float2* __restrict__ prev, const float2* __restrict__ cur, int n_prev,
                      long long nsrc, int ceff, const int* __restrict__ off,
                      const int* __restrict__ src, const int* __restrict__ shifts, int n_dm,
                      int n_filled, int t_dedisp, int n_tiles, float2* __restrict__ out) {
  constexpr int DG = DPW * (DV_THREADS / 32);  // DMs per CTA
  constexpr int TPL = DV_TT / 32;              // times per lane
  extern __shared__ __align__(16) uint8_t dv_smem[];
  __shared__ int s_w, s_off[DV_CELLS + 1];     // the widest spread; the cells' sources
  float2* win = reinterpret_cast<float2*>(dv_smem);                    // [2][DV_SLOTS]
  uint16_t* boff = reinterpret_cast<uint16_t*>(win + 2 * DV_SLOTS);    // [2][8][DV_MAXB][DPW]
  uint16_t* rel = boff + 2 * DV_MAXB * DG;                             // [ceff][DG]
  int* s_lo = reinterpret_cast<int*>(rel + (size_t)ceff * DG);         // [ceff]
  int* s_hi = s_lo + ceff;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t0 = (int)(blockIdx.x % n_tiles) * DV_TT;
  const int nt = min(DV_TT, t_dedisp - t0);
  const int d0 = blockIdx.y * DG;
  const int nd = min(DG, n_dm - d0);
  const int cell0 = (int)(blockIdx.x / n_tiles) * DV_CELLS;
  const int nc = min(DV_CELLS, n_filled - cell0);

  // each subband's shift range over this CTA's DMs, and the widest of them:
  // whether every source's window fits a buffer
  if (tid == 0) s_w = 0;
  __syncthreads();
  int w_max = 0;
  for (int sb = tid; sb < ceff; sb += DV_THREADS) {
    const int* sh = shifts + (long long)sb * n_dm + d0;
    int lo = sh[0], hi = sh[0];
    for (int d = 1; d < nd; ++d) {
      lo = min(lo, sh[d]);
      hi = max(hi, sh[d]);
    }
    s_lo[sb] = lo;
    s_hi[sb] = hi;
    // a spread too wide for the buffers (or for 16 bits) sends the CTA to
    // the direct path; clamped so that the sum stays an int
    w_max = max(w_max, (int)min((long long)hi - lo, (long long)DV_SLOTS));
  }
  atomicMax(&s_w, w_max);
  __syncthreads();
  const bool windowed = s_w + DV_TT <= DV_SLOTS;
  const int c_end = cell0 + nc;
  float2 acc[DPW][TPL], res[DV_CELLS][DPW][TPL];
#pragma unroll
  for (int k = 0; k < DPW; ++k)
#pragma unroll
    for (int h = 0; h < TPL; ++h) acc[k][h] = make_float2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < DV_CELLS; ++c)
#pragma unroll
    for (int k = 0; k < DPW; ++k)
#pragma unroll
      for (int h = 0; h < TPL; ++h) res[c][k][h] = make_float2(0.f, 0.f);
  auto finish = [&](int c) {
#pragma unroll
    for (int x = 0; x < DV_CELLS; ++x)
      if (x == c)
#pragma unroll
        for (int k = 0; k < DPW; ++k)
#pragma unroll
          for (int h = 0; h < TPL; ++h) res[x][k][h] = acc[k][h];
#pragma unroll
    for (int k = 0; k < DPW; ++k)
#pragma unroll
      for (int h = 0; h < TPL; ++h) acc[k][h] = make_float2(0.f, 0.f);
  };
  auto row_of = [&](long long r) {
    return r < n_prev ? prev + r * nsrc : cur + (r - n_prev) * nsrc;
  };

  if (windowed) {
    for (int i = tid; i < ceff * DG; i += DV_THREADS) {
      const int sb = i / DG, d = i % DG;
      rel[i] = (uint16_t)(d < nd ? shifts[(long long)sb * n_dm + d0 + d] - s_lo[sb] : 0);
    }
    if (tid <= DV_CELLS) s_off[tid] = off[min(cell0 + tid, c_end)];
    __syncthreads();
    const int j_end = s_off[DV_CELLS];
    auto src_at = [&](int j) { return j + lane < j_end ? __ldg(src + j + lane) : 0; };
    int pre = src_at(s_off[0]);   // this lane's source of the next batch
    // The batch that starts at source j: as many of the CTA's sources as fit
    // the buffer, returned.  Every warp works out the same layout, a lane per
    // source, copies its share of the rows and notes its own DMs' offsets.
    auto load = [&](int buf, int j) {
      float2* wb = win + buf * DV_SLOTS;
      uint16_t* bo = boff + (buf * (DV_THREADS / 32) + warp) * DV_MAXB * DPW;
      int nb = 0, base0 = 0;
      for (int ch = 0; ch < DV_MAXB; ch += 32) {
        const int sj = ch ? src_at(j + ch) : pre, sb = sj % ceff;
        const int l = s_lo[sb], spread = s_hi[sb] - l;
        int n = spread + nt;   // rows t0 + l .. t0 + l + n - 1
        // padded so that a row's copies by consecutive lanes meet in no bank
        const int w = n + ((__shfl_down_sync(0xffffffffu, l, 1) - l + 1 - n) & 15);
        int end = w;
#pragma unroll
        for (int o = 1; o < 32; o *= 2) {
          const int v = __shfl_up_sync(0xffffffffu, end, o);
          if (lane >= o) end += v;
        }
        const int base = base0 + end - w;
        const bool fits = j + ch + lane < j_end && base + spread + DV_TT <= DV_SLOTS;
        const int cnt = __popc(__ballot_sync(0xffffffffu, fits));
        if (cnt == 0) break;
        if (fits) {
          if constexpr (DPW == 4) {   // no carry between the halves: offsets fit 16 bits
            const uint2 d = *reinterpret_cast<const uint2*>(rel + sb * DG + warp * DPW);
            const uint32_t b2 = (uint32_t)base * 0x10001u;
            *reinterpret_cast<uint2*>(bo + (ch + lane) * DPW) = make_uint2(d.x + b2, d.y + b2);
          } else {
#pragma unroll
            for (int k = 0; k < DPW; ++k)
              bo[(ch + lane) * DPW + k] = (uint16_t)(base + rel[sb * DG + warp * DPW + k]);
          }
        }
        if (!fits) n = 0;
        const int lo = __reduce_min_sync(0xffffffffu, fits ? l : 0x7fffffff);
        const int hi = __reduce_max_sync(0xffffffffu, fits ? l + n : -0x7fffffff);
        const uint32_t dst = smem_u32(wb) + 8 * (base - l);
        auto copy = [&](const float2* rows, int first, int last) {   // rows: that of shift 0
          const float2* p = rows + (long long)first * nsrc + sj;
          for (int r = first; r < last; r += DV_THREADS / 32, p += (DV_THREADS / 32) * nsrc)
            if ((unsigned)(r - l) < (unsigned)n) cp_async8(dst + 8 * r, p);
        };
        const int in_prev = max(lo, min(hi, n_prev - t0));
        copy(prev + (long long)t0 * nsrc, lo + warp, in_prev);
        // the first of this warp's rows in cur
        const int first = lo + warp + max(0, (in_prev - lo - warp + 7) / 8) * 8;
        copy(cur + ((long long)t0 - n_prev) * nsrc, first, hi);
        nb += cnt;
        base0 += __shfl_sync(0xffffffffu, end, 31);
        if (cnt < 32) break;
      }
      cp_async_commit();
      pre = src_at(j + nb);
      return nb;
    };
    int j = s_off[0], buf = 0, cl = 0;
    int nb = j < j_end ? load(0, j) : 0;
    while (j < j_end) {
      const int jn = j + nb;
      int nbn = 0;
      if (jn < j_end) {
        nbn = load(buf ^ 1, jn);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      if (warp * DPW < nd) {
        const float2* wb = win + buf * DV_SLOTS + lane;
        const uint16_t* bo = boff + (buf * (DV_THREADS / 32) + warp) * DV_MAXB * DPW;
        for (int i = 0;;) {
          const int e = s_off[cl + 1] - j, stop = min(nb, e);
#pragma unroll 2
          for (; i < stop; ++i) {
            uint16_t o[DPW];
            if constexpr (DPW == 4) {
              const uint2 w = *reinterpret_cast<const uint2*>(bo + i * DPW);
              o[0] = (uint16_t)w.x; o[1] = (uint16_t)(w.x >> 16);
              o[2] = (uint16_t)w.y; o[3] = (uint16_t)(w.y >> 16);
            } else {
#pragma unroll
              for (int k = 0; k < DPW; ++k) o[k] = bo[i * DPW + k];
            }
#pragma unroll
            for (int k = 0; k < DPW; ++k)
#pragma unroll
              for (int h = 0; h < TPL; ++h) acc[k][h] = f2_add(acc[k][h], wb[o[k] + 32 * h]);
          }
          if (i < e) break;   // the cell goes on in the next batch
          finish(cl);
          if (++cl == nc) break;
        }
      }
      j = jn;
      nb = nbn;
      buf ^= 1;
      __syncthreads();   // the buffer just read is the next batch's target
    }
  } else {
    for (int c = cell0; c < c_end; ++c) {
      for (int j = off[c]; j < off[c + 1]; ++j) {
        const int sj = src[j];
        const int* sh = shifts + (long long)(sj % ceff) * n_dm + d0;
#pragma unroll
        for (int k = 0; k < DPW; ++k)
#pragma unroll
          for (int h = 0; h < TPL; ++h)
            if (warp * DPW + k < nd && lane + 32 * h < nt)
              acc[k][h] = f2_add(acc[k][h], row_of((long long)t0 + lane + 32 * h +
                                                   sh[warp * DPW + k])[sj]);
      }
      finish(c - cell0);
    }
  }
  // four lanes exchange (cell, time) so that they write the 4 cells of one
  // time together (one sector instead of four)
  const int q = lane & 3;
#pragma unroll
  for (int k = 0; k < DPW; ++k)
#pragma unroll
    for (int h = 0; h < TPL; ++h) {
      float2 a[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) a[c] = res[c][k][h];
      // lane q's a[c] (cell c, time 4 (lane / 4) + q) -> lane c's a[q]
#pragma unroll
      for (int m = 1; m <= 2; m *= 2)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (!(c & m)) {
            const bool up = q & m;
            const float2 give = up ? a[c] : a[c | m];
            float2 got;
            got.x = __shfl_xor_sync(0xffffffffu, give.x, m);
            got.y = __shfl_xor_sync(0xffffffffu, give.y, m);
            if (up) a[c] = got;
            else a[c | m] = got;
          }
      const int d = warp * DPW + k;
      if (d < nd && q < nc) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int t = 32 * h + (lane & ~3) + c;
          if (t < nt)
            out[((long long)(d0 + d) * t_dedisp + t0 + t) * n_filled + cell0 + q] = a[c];
        }
      }
    }
}

// More subbands than the shift tables hold: one thread per output.
__global__ void dedisp_vis_wide_kernel(const float2* __restrict__ prev,
                                       const float2* __restrict__ cur, int n_prev,
                                       long long nsrc, int ceff, const int* __restrict__ off,
                                       const int* __restrict__ src,
                                       const int* __restrict__ shifts, int n_dm, int n_filled,
                                       int t_dedisp, float2* __restrict__ out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long per_d = (long long)t_dedisp * n_filled;
  if (idx >= per_d * n_dm) return;
  const int d = (int)(idx / per_d);
  const long long r = idx % per_d;
  const int t = (int)(r / n_filled), cell = (int)(r % n_filled);
  float re = 0.f, im = 0.f;
  for (int j = off[cell]; j < off[cell + 1]; ++j) {
    const int sj = src[j];
    const int tt = t + shifts[(sj % ceff) * n_dm + d];
    const float2 x = tt < n_prev ? prev[(size_t)tt * nsrc + sj] : cur[(size_t)(tt - n_prev) * nsrc + sj];
    re += x.x;
    im += x.y;
  }
  out[idx] = make_float2(re, im);
}

template <int DPW>
int launch_dedisp_vis(const float2* prev, const float2* cur, int n_prev, long long nsrc, int ceff,
                      const int* off, const int* src, const int* shifts, int n_dm, int n_filled,
                      int t_dedisp, float2* out, cudaStream_t stream) {
  constexpr int DG = DPW * (DV_THREADS / 32);
  const size_t smem = dv_smem_bytes(ceff, DG);
  if (cudaFuncSetAttribute(dedisp_vis_kernel<DPW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess)
    return DSB_E_CUDA;
  const int n_tiles = (t_dedisp + DV_TT - 1) / DV_TT;
  const long long blocks = (long long)n_tiles * ((n_filled + DV_CELLS - 1) / DV_CELLS);
  // times fastest: CTAs that run together share a cell group's input rows and
  // complete the output rows' sectors in L2
  const dim3 grid((unsigned)blocks, (n_dm + DG - 1) / DG);
  dedisp_vis_kernel<DPW><<<grid, DV_THREADS, smem, stream>>>(
      prev, cur, n_prev, nsrc, ceff, off, src, shifts, n_dm, n_filled, t_dedisp, n_tiles, out);
  return cudaGetLastError() == cudaSuccess ? DSB_OK : DSB_E_CUDA;
}

// Static-sky mean (per cell): mean of the past `count` block means held in
// ring[cell*window + w] (float64), subtracted once `subtract` is set; this
// block's float64 time-mean is written to ring[cell*window + head].
__global__ void static_sky_kernel(const float2* __restrict__ in, float2* __restrict__ out,
                                  int n_t, int n_cells, double2* __restrict__ ring, int window,
                                  int head, int count, int subtract) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= n_cells) return;
  double2 m = make_double2(0.0, 0.0);
  if (subtract && count > 0) {
    for (int w = 0; w < count; ++w) {
      const double2 r = ring[(size_t)cell * window + w];
      m.x += r.x;
      m.y += r.y;
    }
    m.x /= count;
    m.y /= count;
  }
  double sr = 0.0, si = 0.0;
  for (int t = 0; t < n_t; ++t) {
    const float2 x = in[(size_t)t * n_cells + cell];
    sr += x.x;
    si += x.y;
    if (subtract && count > 0)
      out[(size_t)t * n_cells + cell] =
          make_float2((float)((double)x.x - m.x), (float)((double)x.y - m.y));
    else
      out[(size_t)t * n_cells + cell] = x;
  }
  ring[(size_t)cell * window + head] = make_double2(sr / n_t, si / n_t);
}

// Stage-2 aligned cube: out[c, t, :] = stream_c[t - shift[c]] where the
// stream is the concatenation of past cubes; hist[c][j] points at the cube
// pushed j ticks ago (j = 0 newest).  warm[c] == 0 -> zeros.
__global__ void stage2_roll_kernel(const float2* const* __restrict__ hist, int depth,
                                   const int* __restrict__ kblk, const int* __restrict__ rsmp,
                                   const int* __restrict__ warm, int n_dm, int t_len,
                                   long long inner, float2* __restrict__ out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long per_c = (long long)t_len * inner;
  if (idx >= per_c * n_dm) return;
  const int c = (int)(idx / per_c);
  const long long r = idx % per_c;
  const int t = (int)(r / inner);
  const long long e = r % inner;
  float2 v = make_float2(0.f, 0.f);
  if (warm[c]) {
    const int k = kblk[c], rr = rsmp[c];
    int j, ts;
    if (t < rr) {
      j = k + 1;
      ts = t_len - rr + t;
    } else {
      j = k;
      ts = t - rr;
    }
    if (j < depth) {
      const float2* cube = hist[j];
      v = cube[((size_t)c * t_len + ts) * inner + e];
    }
  }
  out[idx] = v;
}

// Pipeline stage 1 over per-subband gridded rows, time-major rings:
//   Y[(t & y_mask) * y_rows + y_base[g] + s * pitch[g] + cell],
//   D[seg_base[g*n_dm + d] + (t mod seg_depth[g*n_dm + d]) * pitch[g] + cell]
// (each (chgroup, coarse DM) a ring segment as deep as its own stage-2 delay
// needs); the sky ring is indexed by d_base[g] + d * pitch[g] + cell.
//
// A CTA owns 4 adjacent cells of one chgroup and a group of DG coarse
// DMs, and walks the output times in tiles of S1_TT.  For each tile it
// stages every subband's Y samples that any of its DMs needs (the tile plus
// the spread of that subband's shifts over the DM group) in shared memory,
// two planes of two cells, and then every (DM, time) output of the tile sums
// its ceff subbands from there: each Y sample is read from L2 once per DM
// group instead of once per DM.  Thread (dl, ln) = (tid / L, tid % L), with
// L = 256 / DG lanes per DM, owns DM dl of the group and times ln, ln + L,
// ...; DG is 32, 16 or 8: the largest whose windows fit in shared memory
// (a wide DM spread per group, as with few coarse DMs over a wide range,
// needs a smaller group); its D writes are whole
// 32-byte sectors (4 cells).
struct S1Args {
  const float2* Y;
  long long y_rows, y_mask;
  const int* blk_g;       // chgroup of each block
  const int* blk_c0;      // first cell of each block (a multiple of 4)
  const int* y_base;      // (G) first Y row of the chgroup (a multiple of 4)
  const int* pitch;       // (G) row pitch between subbands / coarse DMs (a multiple of 4)
  const int* shift1;      // (G, ceff, n_dm)
  const int* shift2;      // (G, n_dm)
  const int* d_base;      // (G) first sky-ring row of the chgroup
  const int* n_filled;    // (G)
  void* D;                // complex64 elements, or (BF16) bf16 re/im pairs in 32 bits
  const long long* seg_base;  // (G * n_dm) first element of each ring segment (a multiple of 4)
  const int* seg_depth;       // (G * n_dm) time slots of each segment
  float* amax;            // (G * n_dm) or null: raised to the largest |part| written
  long long t0;           // absolute time of the first output
  int n_t, n_dm, ceff;
  int win_len;            // S1_TT + largest shift spread over a DM group
  int sbc;                // subbands per staged chunk (0: all at once)
  double2* sky_ring;      // (D rows, window) or null
  int sky_window, sky_head, sky_count, sky_subtract;
  int* status;
};

constexpr int S1_THREADS = 256;
constexpr int S1_MAX_C = 64;
constexpr int S1_TT = 64;   // output times per tile
constexpr int S1_DG = 32;   // largest DM group (coarse DMs per CTA)
// CTAs per SM of the chunked form with 8 DMs (80 registers, 56 bytes of them
// spilled): the 312 CTAs of the small configuration then run in one wave (two
// per SM, without spills: 245 us, not 190)
constexpr int S1_CHUNK_CTAS8 = 3;

__host__ __device__ inline size_t s1_smem_bytes(int ceff, int dg, int win_len) {
  return (size_t)ceff * dg * 4 + (size_t)S1_MAX_C * 8 + (size_t)ceff * win_len * 32 + 16;
}

// CHUNK: where every subband's window together leaves one CTA per SM (few
// coarse DMs over a wide range: the small plain configuration's 8 DMs of 600
// pc cm^-3 / 32 need 219 KB), the subbands are staged A.sbc at a time in two
// buffers, the next ones copied under the current ones' sums, which stay in
// registers: several CTAs per SM and no exposed load.  300 -> 190 us per block of
// that configuration (512 times, 32 DMs, 314 cells).
template <bool BF16, int DG, bool CHUNK>
__global__ void __launch_bounds__(S1_THREADS, CHUNK && DG == 8 ? S1_CHUNK_CTAS8 : 2)
    stage1_rows_kernel(const S1Args A) {
  constexpr int L = S1_THREADS / DG;  // time lanes per DM
  static_assert(L >= 8 && L <= 32 && S1_TT % L == 0, "unsupported DM group");
  extern __shared__ __align__(16) uint8_t s1_smem[];
  const int ceff = A.ceff;
  int* s_sh = reinterpret_cast<int*>(s1_smem);              // [s][dl] shift - lo[s]
  int* s_lo = s_sh + ceff * DG;                             // [s] smallest shift
  int* s_len = s_lo + S1_MAX_C;                             // [s] window length
  float4* win0 = reinterpret_cast<float4*>(s1_smem + ((size_t)ceff * DG * 4 +
                                                      (size_t)S1_MAX_C * 8 + 15) / 16 * 16);
  const int n_win = CHUNK ? 2 * A.sbc : ceff;                // windows staged
  float4* win1 = win0 + (size_t)n_win * A.win_len;           // cells 2-3

  const int g = A.blk_g[blockIdx.x];
  const int c0 = A.blk_c0[blockIdx.x];
  const int dg0 = blockIdx.y * DG;
  const int nd = min(DG, A.n_dm - dg0);
  const int pitch = A.pitch[g];
  const int tid = threadIdx.x;
  for (int sb = tid; sb < ceff; sb += S1_THREADS) {
    const int* sh = A.shift1 + ((long long)g * ceff + sb) * A.n_dm + dg0;
    int lo = sh[0], hi = sh[0];
    for (int dl = 1; dl < nd; ++dl) {
      lo = min(lo, sh[dl]);
      hi = max(hi, sh[dl]);
    }
    s_lo[sb] = lo;
    s_len[sb] = S1_TT + hi - lo;
  }
  __syncthreads();
  // a window longer than the caller sized the shared memory for: flag, stop
  bool fits = true;
  for (int sb = 0; sb < ceff; ++sb) fits = fits && s_len[sb] <= A.win_len;
  if (!fits) {
    if (tid == 0) dsb_flag(A.status, DSB_E_CAPACITY);
    return;
  }
  for (int i = tid; i < ceff * DG; i += S1_THREADS) {
    const int sb = i / DG, dl = i % DG;
    s_sh[i] = dl < nd ? A.shift1[((long long)g * ceff + sb) * A.n_dm + dg0 + dl] - s_lo[sb] : 0;
  }

  const int dl = tid / L, ln = tid % L;
  const bool active = dl < nd;
  const int d = dg0 + (active ? dl : 0);
  const int gd = g * A.n_dm + d;
  const long long seg = A.seg_base[gd] + c0;
  const long long dep = A.seg_depth[gd];
  const int sh2 = A.shift2[gd];
  const long long drow = (long long)A.d_base[g] + (long long)d * pitch + c0;
  double mr[4] = {0, 0, 0, 0}, mi[4] = {0, 0, 0, 0};
  const bool sub = A.sky_ring && A.sky_subtract && A.sky_count > 0;
  if (sub && active) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      for (int w = 0; w < A.sky_count; ++w) {
        const double2 r = A.sky_ring[(drow + c) * A.sky_window + w];
        mr[c] += r.x;
        mi[c] += r.y;
      }
      mr[c] /= A.sky_count;
      mi[c] /= A.sky_count;
    }
  }
  double sr[4] = {0, 0, 0, 0}, si[4] = {0, 0, 0, 0};
  float amax = 0.f;  // largest |part| this thread writes
  const float4* Y4 = reinterpret_cast<const float4*>(A.Y);
  const long long ycol = (long long)A.y_base[g] + c0;   // a multiple of 4

  // the sums (a0, a1) of the four cells at tile time tl, into ring slot `slot`
  auto emit = [&](float4 a0, float4 a1, long long slot) {
    sr[0] += a0.x; si[0] += a0.y; sr[1] += a0.z; si[1] += a0.w;
    sr[2] += a1.x; si[2] += a1.y; sr[3] += a1.z; si[3] += a1.w;
    float4 o0 = a0, o1 = a1;
    if (sub) {
      o0 = make_float4((float)((double)a0.x - mr[0]), (float)((double)a0.y - mi[0]),
                       (float)((double)a0.z - mr[1]), (float)((double)a0.w - mi[1]));
      o1 = make_float4((float)((double)a1.x - mr[2]), (float)((double)a1.y - mi[2]),
                       (float)((double)a1.z - mr[3]), (float)((double)a1.w - mi[3]));
    }
    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(o0.x), fabsf(o0.y)), fmaxf(fabsf(o0.z), fabsf(o0.w))));
    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(o1.x), fabsf(o1.y)), fmaxf(fabsf(o1.z), fabsf(o1.w))));
    const long long o = seg + slot * pitch;  // element of cell c0, a multiple of 4
    if (!(DSB_INB(slot, dep, A.status) && DSB_INB(c0 + 3, pitch, A.status))) return;
    if constexpr (BF16) {
      reinterpret_cast<uint4*>(A.D)[o / 4] =
          make_uint4(bf16_pair(o0.x, o0.y), bf16_pair(o0.z, o0.w), bf16_pair(o1.x, o1.y),
                     bf16_pair(o1.z, o1.w));
    } else {
      float4* D4 = reinterpret_cast<float4*>(A.D);
      D4[o / 2] = o0;
      D4[o / 2 + 1] = o1;
    }
  };

  if constexpr (CHUNK) {
    constexpr int KT = S1_TT / L;
    static_assert(KT <= 4, "a thread's sums stay in registers");
    const int n_ch = (ceff + A.sbc - 1) / A.sbc;
    const int n_items = (A.n_t + S1_TT - 1) / S1_TT * n_ch;   // (tile, subbands)
    // four warps per subband's copies: with windows so long that a chunk is one
    // subband, one warp issuing them all took 343 us where the whole windows
    // take 278, four 271 (64 DMs in 16s, 6 subbands, shifts spread over 1000)
    auto load = [&](int item) {
      const int tt = item / n_ch * S1_TT, s0 = item % n_ch * A.sbc;
      const int w0 = (item & 1) * A.sbc;
      for (int q = tid / 128; q < min(A.sbc, ceff - s0); q += S1_THREADS / 128) {
        const int sb = s0 + q;
        for (int tau = tid % 128; tau < s_len[sb]; tau += 128) {
          const long long r2 = ((((A.t0 + tt + s_lo[sb] + tau) & A.y_mask) * A.y_rows) + ycol +
                                (long long)sb * pitch) / 2;
          if (!DSB_INB(r2 + 1, (A.y_mask + 1) * A.y_rows / 2, A.status)) continue;
          const int e = (w0 + q) * A.win_len + tau;
          cp_async16(win0 + e, Y4 + r2);
          cp_async16(win1 + e, Y4 + r2 + 1);
        }
      }
      cp_async_commit();
    };
    float4 acc[KT][2];
    __syncthreads();   // the shift tables
    load(0);
    for (int item = 0; item < n_items; ++item) {
      const int tt = item / n_ch * S1_TT, ch = item % n_ch, s0 = ch * A.sbc;
      if (item + 1 < n_items) {
        load(item + 1);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      if (active) {
        if (ch == 0) {
#pragma unroll
          for (int k = 0; k < KT; ++k) acc[k][0] = acc[k][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const int w0 = (item & 1) * A.sbc;
        for (int q = 0; q < min(A.sbc, ceff - s0); ++q) {
          const int idx = (w0 + q) * A.win_len + ln + s_sh[(s0 + q) * DG + dl];
#pragma unroll
          for (int k = 0; k < KT; ++k) {
            acc[k][0] = f4_add(acc[k][0], win0[idx + L * k]);
            acc[k][1] = f4_add(acc[k][1], win1[idx + L * k]);
          }
        }
        if (ch == n_ch - 1) {
          long long slot = (A.t0 + tt + ln + sh2) % dep;
          if (slot < 0) slot += dep;
#pragma unroll
          for (int k = 0; k < KT; ++k, slot += L) {
            if (slot >= dep) slot -= dep;
            if (tt + ln + L * k < A.n_t) emit(acc[k][0], acc[k][1], slot);
          }
        }
      }
      __syncthreads();   // the windows just read are the next item's target
    }
  } else {
    for (int tt = 0; tt < A.n_t; tt += S1_TT) {
      __syncthreads();  // the previous tile's windows are no longer read
      // stage the windows: entry (sb, tau) = Y at time t0 + tt + lo[sb] + tau,
      // flattened over (sb, tau) so that each thread's loads are independent
      {
        constexpr int U = 4;
        const int n_e = ceff * A.win_len;
        for (int e0 = 0; e0 < n_e; e0 += U * S1_THREADS) {
          float4 v0[U], v1[U];
          int ei[U];
#pragma unroll
          for (int q = 0; q < U; ++q) {
            const int e = e0 + q * S1_THREADS + tid;
            ei[q] = -1;
            if (e < n_e) {
              const int sb = e / A.win_len, tau = e - sb * A.win_len;
              if (tau < s_len[sb]) {
                const long long r2 = ((((A.t0 + tt + s_lo[sb] + tau) & A.y_mask) * A.y_rows) +
                                      ycol + (long long)sb * pitch) / 2;
                if (DSB_INB(r2 + 1, (A.y_mask + 1) * A.y_rows / 2, A.status)) {
                  v0[q] = Y4[r2];
                  v1[q] = Y4[r2 + 1];
                  ei[q] = e;
                }
              }
            }
          }
#pragma unroll
          for (int q = 0; q < U; ++q) {
            if (ei[q] >= 0) {
              win0[ei[q]] = v0[q];
              win1[ei[q]] = v1[q];
            }
          }
        }
      }
      __syncthreads();
      if (!active) continue;
      long long slot = (A.t0 + tt + ln + sh2) % dep;
      if (slot < 0) slot += dep;
      for (int k = 0; k < S1_TT / L; ++k, slot += L) {
        if (slot >= dep) slot -= dep;
        const int tl = ln + L * k;
        if (tt + tl >= A.n_t) break;
        float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
        for (int sb = 0; sb < ceff; ++sb) {
          const int idx = sb * A.win_len + tl + s_sh[sb * DG + dl];
          const float4 v0 = win0[idx], v1 = win1[idx];
          a0 = f4_add(a0, v0);  // packed pairs: 4 adds instead of 8
          a1 = f4_add(a1, v1);
        }
        emit(a0, a1, slot);
      }
    }
  }
  // the bound of the (chgroup, DM) rows: max over the L lanes that share
  // the DM, one atomic per DM and block (non-negative floats order as ints)
  if (A.amax) {
#pragma unroll
    for (int o = 1; o < L; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (active && ln == 0) atomicMax(reinterpret_cast<int*>(A.amax) + gd, __float_as_int(amax));
  }
  // sky: block mean of every (DM, cell) over the chunk, summed over the L
  // lanes that share the DM (L-aligned inside the warp)
  if (A.sky_ring) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
      for (int o = 1; o < L; o <<= 1) {
        sr[c] += __shfl_xor_sync(0xffffffffu, sr[c], o);
        si[c] += __shfl_xor_sync(0xffffffffu, si[c], o);
      }
    }
    if (active && ln == 0) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        A.sky_ring[(drow + c) * A.sky_window + A.sky_head] =
            make_double2(sr[c] / A.n_t, si[c] / A.n_t);
    }
  }
}

int launch_status() { return cudaGetLastError() == cudaSuccess ? DSB_OK : DSB_E_CUDA; }

}  // namespace

extern "C" {

int dsb_grid_vis(const void* vis, int n_fv, long long nsrc, const int* cell_off,
                 const int* cell_src, int n_filled, void* out, cudaStream_t stream) {
  if (!vis || !out || !cell_off || !cell_src || n_fv <= 0 || n_filled < 0) return DSB_E_ARG;
  const long long n = (long long)n_fv * n_filled;
  if (n == 0) return DSB_OK;
  grid_vis_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(
      (const float2*)vis, n_fv, nsrc, cell_off, cell_src, n_filled, (float2*)out);
  return launch_status();
}

int dsb_dedisp_vis(const void* prev, const void* cur, int n_prev, long long nsrc, int ceff,
                   const int* cell_off, const int* cell_src, const int* shifts, int n_dm,
                   int n_filled, int t_dedisp, void* out, cudaStream_t stream) {
  if (!cur || !out || !cell_off || !cell_src || !shifts || ceff <= 0 || n_dm <= 0) return DSB_E_ARG;
  if (n_prev > 0 && !prev) return DSB_E_ARG;
  const long long n = (long long)n_dm * t_dedisp * n_filled;
  if (n <= 0) return DSB_OK;
  const auto* p = (const float2*)prev;
  const auto* v = (const float2*)cur;
  auto* o = (float2*)out;
  // the windowed kernel while the subbands' shift tables fit beside the
  // window buffers; DMs per warp as few as cover the DMs of the call, so that
  // no warp of a short list idles
  if (ceff <= DV_MAX_C && (n_dm + 31) / 32 <= 65535) {
    if (n_dm <= 8)
      return launch_dedisp_vis<1>(p, v, n_prev, nsrc, ceff, cell_off, cell_src, shifts, n_dm,
                                  n_filled, t_dedisp, o, stream);
    if (n_dm <= 16)
      return launch_dedisp_vis<2>(p, v, n_prev, nsrc, ceff, cell_off, cell_src, shifts, n_dm,
                                  n_filled, t_dedisp, o, stream);
    return launch_dedisp_vis<4>(p, v, n_prev, nsrc, ceff, cell_off, cell_src, shifts, n_dm,
                                n_filled, t_dedisp, o, stream);
  }
  dedisp_vis_wide_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(
      p, v, n_prev, nsrc, ceff, cell_off, cell_src, shifts, n_dm, n_filled, t_dedisp, o);
  return launch_status();
}

int dsb_static_sky(const void* in, void* out, int n_t, int n_cells, void* ring, int window,
                   int head, int count, int subtract, cudaStream_t stream) {
  if (!in || !out || !ring || n_t <= 0 || n_cells < 0 || window <= 0) return DSB_E_ARG;
  if (head < 0 || head >= window || count < 0 || count > window) return DSB_E_ARG;
  if (n_cells == 0) return DSB_OK;
  static_sky_kernel<<<(n_cells + 127) / 128, 128, 0, stream>>>(
      (const float2*)in, (float2*)out, n_t, n_cells, (double2*)ring, window, head, count,
      subtract);
  return launch_status();
}

int dsb_stage2_roll(const void* const* hist, int depth, const int* kblk, const int* rsmp,
                    const int* warm, int n_dm, int t_len, long long inner, void* out,
                    cudaStream_t stream) {
  if (!hist || !kblk || !rsmp || !warm || !out || depth <= 0 || n_dm <= 0 || t_len <= 0)
    return DSB_E_ARG;
  const long long n = (long long)n_dm * t_len * inner;
  if (n == 0) return DSB_OK;
  stage2_roll_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(
      (const float2* const*)hist, depth, kblk, rsmp, warm, n_dm, t_len, inner, (float2*)out);
  return launch_status();
}

int dsb_stage1_rows(const void* Y, long long y_rows, long long y_mask, int n_blocks,
                    const int* blk_g, const int* blk_c0, const int* y_base, const int* pitch,
                    const int* shift1, const int* shift2, const int* d_base, const int* n_filled,
                    void* D, int d_bf16, const long long* seg_base, const int* seg_depth,
                    float* amax, long long t0, int n_t, int n_dm, int ceff, int dm_group, int max_spread,
                    void* sky_ring, int sky_window,
                    int sky_head, int sky_count, int sky_subtract, int* status,
                    cudaStream_t stream) {
  if (!Y || !D || !blk_g || !blk_c0 || !y_base || !pitch || !shift1 || !shift2 ||
      !d_base || !n_filled || !seg_base || !seg_depth || n_t <= 0 || n_dm <= 0 || ceff <= 0 ||
      max_spread < 0 || (dm_group != 32 && dm_group != 16 && dm_group != 8))
    return DSB_E_ARG;
  // four cells per 32-byte access: rings 16-byte aligned, row counts multiples of 4
  if ((reinterpret_cast<uintptr_t>(Y) & 15) || (reinterpret_cast<uintptr_t>(D) & 15) ||
      (y_rows & 3))
    return DSB_E_ARG;
  if (ceff > S1_MAX_C) return DSB_E_CAPACITY;
  const int win_len = S1_TT + max_spread;
  const size_t smem = s1_smem_bytes(ceff, dm_group, win_len);
  if (smem > 227 * 1024) return DSB_E_CAPACITY;
  if (sky_ring && (sky_window <= 0 || sky_head < 0 || sky_head >= sky_window ||
                   sky_count < 0 || sky_count > sky_window))
    return DSB_E_ARG;
  if (n_blocks <= 0) return DSB_OK;
  S1Args A{};
  A.Y = (const float2*)Y; A.y_rows = y_rows; A.y_mask = y_mask;
  A.blk_g = blk_g; A.blk_c0 = blk_c0; A.y_base = y_base; A.pitch = pitch;
  A.shift1 = shift1; A.shift2 = shift2; A.d_base = d_base; A.n_filled = n_filled;
  A.D = D; A.seg_base = seg_base; A.seg_depth = seg_depth; A.amax = amax;
  A.t0 = t0; A.n_t = n_t; A.n_dm = n_dm; A.ceff = ceff; A.win_len = win_len;
  A.sky_ring = (double2*)sky_ring; A.sky_window = sky_window; A.sky_head = sky_head;
  A.sky_count = sky_count; A.sky_subtract = sky_subtract; A.status = status;
  // chunks where the whole windows leave room for one CTA per SM only (and
  // a DM group narrow enough to keep its sums in registers): as many subbands
  // as two buffers in half an SM hold, at most eight.  A grid that gives the
  // SMs one CTA each keeps the whole windows: 111 us for 100 CTAs of 8 DMs
  // (121 in chunks), 86 for 80 (91); 100 CTAs of 16 DMs 129 and 120.
  size_t bytes = smem;
  const size_t tables = s1_smem_bytes(ceff, dm_group, 0), per_sb = (size_t)2 * win_len * 32;
  const size_t room = 227 * 1024 / (dm_group == 8 ? S1_CHUNK_CTAS8 : 2) - 1024;
  const long long ctas = (long long)n_blocks * ((n_dm + dm_group - 1) / dm_group);
  if (dm_group <= 16 && smem > 113 * 1024 && tables + per_sb <= room &&
      ctas > (dm_group == 8 ? 148 : 74)) {
    A.sbc = (int)std::min<size_t>(S1_THREADS / 32, (room - tables) / per_sb);
    A.sbc = std::min(A.sbc, ceff);
    bytes = tables + (size_t)A.sbc * per_sb;
  }
  auto pick = [&](auto bf) {
    constexpr bool B = decltype(bf)::value;
    if (A.sbc)
      return dm_group == 16 ? stage1_rows_kernel<B, 16, true> : stage1_rows_kernel<B, 8, true>;
    return dm_group == 32   ? stage1_rows_kernel<B, 32, false>
           : dm_group == 16 ? stage1_rows_kernel<B, 16, false>
                            : stage1_rows_kernel<B, 8, false>;
  };
  auto kern = d_bf16 ? pick(std::true_type{}) : pick(std::false_type{});
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) !=
      cudaSuccess)
    return DSB_E_CUDA;
  dim3 grid(n_blocks, (n_dm + dm_group - 1) / dm_group);
  kern<<<grid, S1_THREADS, bytes, stream>>>(A);
  return launch_status();
}

int dsb_stage1_block_size(void) { return 4; }
int dsb_stage1_dm_group(void) { return S1_DG; }

long long dsb_stage1_smem_bytes(int ceff, int dm_group, int max_spread) {
  if (ceff <= 0 || ceff > S1_MAX_C || max_spread < 0 ||
      (dm_group != 32 && dm_group != 16 && dm_group != 8))
    return -1;
  return (long long)s1_smem_bytes(ceff, dm_group, S1_TT + max_spread);
}

}  // extern "C"
