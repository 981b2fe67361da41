// Transmission builder: per-slice projected potential in Fourier space, inverse 2-D FFT, and
// T = exp(i * sigma/1000 * V).
//
// Reference: cal_p / initKernel_P (cuda_source_lobato.cu:585-956, cuda_source_peng_and_corr.cu
// :785-1156) and the correction potential p_corr (cuda_source_peng_and_corr.cu:587-779); the CPU
// statement of the same sums is GetPotential4AllSlice_multicore_lotabo_peng(_corr).m.
//
// Differences by design:
//  * one thread owns each pixel's accumulator for all atoms of a slice (the reference launches
//    one thread per (atom, pixel) and adds into the same pixel without atomics,
//    cuda_source_lobato.cu:82-83);
//  * the phase exp(-2 pi i (kx x + ky y)) is reduced modulo one in FP64 before the FP32
//    sincospi (the reference forms the angle in FP32 with pi = 3.14159265, :80-81); on the
//    reference's separable grids the two factors are tabulated per atom and tile;
//  * the ifftshift before the inverse FFT is folded into a (-1)^(r+c) factor after it, and
//    APERTURE is applied while the sum is written.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "fft.cuh"
#include "tx_grid.cuh"

namespace totem {

namespace {

constexpr int TX_TC = 32;      // tile columns (one per lane)
constexpr int TX_PR = 4;       // rows per thread
constexpr int TX_TR = 32;      // tile rows (8 warps x 4)
constexpr int TX_CH = 32;      // atoms staged per chunk
constexpr int TX_MAXC = 24;    // widest coefficient block (ionic Lobato row without x, y)

struct TxSmem {
  double pos[TX_CH][2];
  float coef[TX_CH][TX_MAXC];
  float absorp[TX_CH][10];
  float2 ex[TX_CH][TX_TC];
  float2 ey[TX_CH][TX_TR];
};

// kind: 0 neutral, 1 ionic, 2 correction (neutral), 3 correction (ionic)
template <bool SEP>
__device__ void accumulate_rows(const TxGrid& g, const AtomRowsDev& rows, int kind, int slice, TxSmem& sm,
                                int tx, int ty, int c, int r0, int c_tile, int r_tile, const float* s2v,
                                const double* kxv, const double* kyv, const int* pix, float2* acc) {
  if (rows.beg == nullptr) return;
  const int a_begin = rows.beg[slice], a_end = rows.beg[slice + 1];
  const long plane = (long)g.p_h * g.p_w;
  for (int a0 = a_begin; a0 < a_end; a0 += TX_CH) {
    const int na = min(TX_CH, a_end - a0);
    __syncthreads();
    for (int e = threadIdx.x; e < na * 2; e += blockDim.x) sm.pos[e >> 1][e & 1] = rows.pos[(long)(a0 + (e >> 1)) * 2 + (e & 1)];
    for (int e = threadIdx.x; e < na * rows.ncoef; e += blockDim.x) {
      const int a = e / rows.ncoef, k = e - a * rows.ncoef;
      sm.coef[a][k] = rows.coef[(long)(a0 + a) * rows.ncoef + k];
    }
    if (rows.absorp != nullptr)
      for (int e = threadIdx.x; e < na * 10; e += blockDim.x) sm.absorp[e / 10][e % 10] = rows.absorp[(long)a0 * 10 + e];
    __syncthreads();
    if (SEP) {
      for (int e = threadIdx.x; e < na * (TX_TC + TX_TR); e += blockDim.x) {
        const int a = e / (TX_TC + TX_TR), k = e - a * (TX_TC + TX_TR);
        if (k < TX_TC) {
          const int cc = min(c_tile + k, g.p_w - 1);
          sm.ex[a][k] = phase_of(g.kx_axis[cc] * sm.pos[a][0]);
        } else {
          const int rr = min(r_tile + k - TX_TC, g.p_h - 1);
          sm.ey[a][k - TX_TC] = phase_of(g.ky_axis[rr] * sm.pos[a][1]);
        }
      }
      __syncthreads();
    }
    for (int a = 0; a < na; ++a) {
      const float* cf = sm.coef[a];
      float2 ex = make_float2(1.f, 0.f);
      if (SEP) ex = sm.ex[a][tx];
#pragma unroll
      for (int i = 0; i < TX_PR; ++i) {
        const float s2 = s2v[i];
        float2 ph;
        if (SEP) ph = cmul(ex, sm.ey[a][ty * TX_PR + i]);
        else ph = phase_of(kxv[i] * sm.pos[a][0] + kyv[i] * sm.pos[a][1]);
        float fr, fi = 0.f;
        if (kind <= 1) {
          row_form(kind, g.lobato, cf, rows.absorp != nullptr ? sm.absorp[a] : nullptr, s2, fr, fi);
        } else if (kind == 2) {
          const int idx = (int)cf[2] - 1;
          const float m = (idx >= 0 && idx < g.cim_len && pix[i] >= 0) ? g.cim[idx * plane + pix[i]] : 0.f;
          fr = cf[1] * m * __expf(-cf[0] * s2);
        } else {
          const int i1 = (int)cf[3] - 1, i2 = (int)cf[5] - 1;
          float m = 0.f;
          if (pix[i] >= 0) {
            if (i1 >= 0 && i1 < g.cim_len) m = fmaf(cf[2], g.cim[i1 * plane + pix[i]], m);
            if (i2 >= 0 && i2 < g.cim_len) m = fmaf(cf[4], g.cim[i2 * plane + pix[i]], m);
          }
          fr = cf[1] * m * __expf(-cf[0] * s2);
        }
        acc[i].x = fmaf(fr, ph.x, fmaf(-fi, ph.y, acc[i].x));
        acc[i].y = fmaf(fr, ph.y, fmaf(fi, ph.x, acc[i].y));
      }
    }
  }
}

template <bool SEP>
__global__ void __launch_bounds__(256) k_tx_structure(TxGrid g, AtomRowsDev nr, AtomRowsDev ir, AtomRowsDev cn,
                                                      AtomRowsDev ci, float2* __restrict__ out, int accumulate) {
  __shared__ TxSmem sm;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int slice = blockIdx.z;
  const int c_tile = blockIdx.x * TX_TC, r_tile = blockIdx.y * TX_TR;
  const int c = c_tile + tx, r0 = r_tile + ty * TX_PR;
  float s2v[TX_PR];
  double kxv[TX_PR], kyv[TX_PR];
  int pix[TX_PR];
  float2 acc[TX_PR];
#pragma unroll
  for (int i = 0; i < TX_PR; ++i) {
    const int r = r0 + i;
    const bool in = (r < g.p_h) && (c < g.p_w);
    pix[i] = in ? r * g.p_w + c : -1;
    s2v[i] = in ? g.s2[pix[i]] : 0.f;
    kxv[i] = (!SEP && in) ? g.kx[pix[i]] : 0.0;
    kyv[i] = (!SEP && in) ? g.ky[pix[i]] : 0.0;
    acc[i] = make_float2(0.f, 0.f);
  }
  accumulate_rows<SEP>(g, nr, 0, slice, sm, tx, ty, c, r0, c_tile, r_tile, s2v, kxv, kyv, pix, acc);
  accumulate_rows<SEP>(g, ir, 1, slice, sm, tx, ty, c, r0, c_tile, r_tile, s2v, kxv, kyv, pix, acc);
  accumulate_rows<SEP>(g, cn, 2, slice, sm, tx, ty, c, r0, c_tile, r_tile, s2v, kxv, kyv, pix, acc);
  accumulate_rows<SEP>(g, ci, 3, slice, sm, tx, ty, c, r0, c_tile, r_tile, s2v, kxv, kyv, pix, acc);
  float2* dst = out + (long)slice * g.p_h * g.p_w;
#pragma unroll
  for (int i = 0; i < TX_PR; ++i) {
    if (pix[i] < 0) continue;
    const float ap = (g.aper_true != nullptr) ? g.aper_true[pix[i]] : 1.f;
    float2 v = cscale(acc[i], g.parameter * ap);
    if (accumulate) v = cadd(dst[pix[i]], v);
    dst[pix[i]] = v;
  }
}

// ---------------------------------------------------------------------------------------------
// By species.  A 256-thread block owns a 64 x 64 pixel tile of one slice; thread (tx, ty) owns the
// 16 pixels (r_tile + ty + 16 i, c_tile + tx + 16 j).  Per species the block accumulates
//   S(r, c) = sum_atoms ey_a(r) * ex_a(c),  ex_a(c) = exp(-2 pi i kx(c) x_a), ey_a(r) likewise,
// a complex rank-K update from per-atom tables staged in shared memory (16 atoms at a time),
// then adds f_species(s^2) * S.  Table entries are stored so that one complex multiply-add is two
// packed FMAs: ex as (re, im, -im, re), ey as (re, re, im, im).
// ---------------------------------------------------------------------------------------------
constexpr int SP_T = 64;
constexpr int SP_CH = 16;

struct SpSmem {
  double pos[SP_CH][2];
  float4 ex[SP_CH][SP_T];
  float4 ey[SP_CH][SP_T];
};

__global__ void __launch_bounds__(256, 2) k_tx_species(TxGrid g, SpeciesSet spset, float2* __restrict__ out) {
  __shared__ SpSmem sm;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int slice = blockIdx.z;
  const int c_tile = blockIdx.x * SP_T, r_tile = blockIdx.y * SP_T;
  float2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  for (int kind = 0; kind < 4; ++kind) {
    const SpeciesDev& d = spset.k[kind];
    if (d.seg_beg == nullptr) continue;
    const int s_end = d.seg_beg[slice + 1];
    for (int sidx = d.seg_beg[slice]; sidx < s_end; ++sidx) {
      const int sp = d.seg[3 * sidx], a_begin = d.seg[3 * sidx + 1], a_end = d.seg[3 * sidx + 2];
      float2 S[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) S[i][j] = make_float2(0.f, 0.f);
      for (int a0 = a_begin; a0 < a_end; a0 += SP_CH) {
        const int na = min(SP_CH, a_end - a0);
        __syncthreads();  // previous chunk's tables fully read
        if (threadIdx.x < 2 * na) sm.pos[threadIdx.x >> 1][threadIdx.x & 1] = d.pos[(long)a0 * 2 + threadIdx.x];
        __syncthreads();
        for (int e = threadIdx.x; e < na * 2 * SP_T; e += blockDim.x) {
          const int a = e / (2 * SP_T), k = e - a * (2 * SP_T);
          if (k < SP_T) {
            const int cc = min(c_tile + k, g.p_w - 1);
            const float2 p = phase_of(g.kx_axis[cc] * sm.pos[a][0]);
            sm.ex[a][k] = make_float4(p.x, p.y, -p.y, p.x);
          } else {
            const int rr = min(r_tile + k - SP_T, g.p_h - 1);
            const float2 p = phase_of(g.ky_axis[rr] * sm.pos[a][1]);
            sm.ey[a][k - SP_T] = make_float4(p.x, p.x, p.y, p.y);
          }
        }
        __syncthreads();
#pragma unroll 2
        for (int a = 0; a < na; ++a) {
          float4 exv[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) exv[j] = sm.ex[a][tx + 16 * j];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 ey = sm.ey[a][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              S[i][j] = __ffma2_rn(make_float2(ey.x, ey.y), make_float2(exv[j].x, exv[j].y), S[i][j]);
              S[i][j] = __ffma2_rn(make_float2(ey.z, ey.w), make_float2(exv[j].z, exv[j].w), S[i][j]);
            }
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int r = min(r_tile + ty + 16 * i, g.p_h - 1), c = min(c_tile + tx + 16 * j, g.p_w - 1);
          const long pix = (long)r * g.p_w + c;
          float fr, fi;
          species_form(kind, g, d, sp, __ldg(g.s2 + pix), pix, fr, fi);
          acc[i][j].x = fmaf(fr, S[i][j].x, fmaf(-fi, S[i][j].y, acc[i][j].x));
          acc[i][j].y = fmaf(fr, S[i][j].y, fmaf(fi, S[i][j].x, acc[i][j].y));
        }
    }
  }
  float2* dst = out + (long)slice * g.p_h * g.p_w;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = r_tile + ty + 16 * i, c = c_tile + tx + 16 * j;
      if (r >= g.p_h || c >= g.p_w) continue;
      const long pix = (long)r * g.p_w + c;
      const float ap = (g.aper_true != nullptr) ? g.aper_true[pix] : 1.f;
      dst[pix] = cscale(acc[i][j], g.parameter * ap);
    }
}

// ---------------------------------------------------------------------------------------------
// Gridding (tx_grid.cuh): the kernels that do not depend on the transform length.
// ---------------------------------------------------------------------------------------------
constexpr int GR_T = 256;

// Kaiser-Bessel shape parameter for GR_W points at oversampling 2, and I0 by its power series
// (arguments up to 18.7; the terms left out are below 1e-17 of the sum).
constexpr double GR_BETA = 18.638814;  // pi sqrt((GR_W / 2)^2 (3 / 2)^2 - 0.8)
__host__ __device__ inline double bessel_i0(double z) {
  const double q = 0.25 * z * z;
  double t = 1.0, s = 1.0;
#pragma unroll
  for (int k = 1; k <= 48; ++k) {
    t *= q * (1.0 / ((double)k * k));
    s += t;
  }
  return s;
}

// Exclusive prefix sum of cnt[0 .. n) in shared memory, in place; returns the total.
__device__ int block_exclusive_scan(int* cnt, int n, int* warp_sum) {
  const int per = (n + GR_T - 1) / GR_T, lo = min(n, (int)threadIdx.x * per), hi = min(n, lo + per);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  int s = 0;
  for (int i = lo; i < hi; ++i) s += cnt[i];
  int x = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sum[wid] = x;
  __syncthreads();
  int before = x - s, total = 0;
  for (int i = 0; i < GR_T / 32; ++i) {
    if (i < wid) before += warp_sum[i];
    total += warp_sum[i];
  }
  for (int i = lo; i < hi; ++i) {
    const int c = cnt[i];
    cnt[i] = before;
    before += c;
  }
  __syncthreads();
  return total;
}

// Fine-grid place of an atom: v in [0, nf], first row b = ceil(v - GR_W / 2) mod nf (nf = 2 n rows).
__device__ __forceinline__ double fine_row(double y, double dky, int nf) {
  const double t = dky * y;
  return (t - floor(t)) * nf;
}
__device__ __forceinline__ int first_row(double v, int nf) {
  const int b = (int)ceil(v - GR_W / 2);
  return min(max(b < 0 ? b + nf : b, 0), nf - 1);
}

// One CTA per job: counting sort of its atoms by first fine row (stable: one warp places 32 atoms
// at a time in order, so the result does not depend on timing), groups of adjacent atoms with the
// same y, the first group of every fine row, and the blocks of fine rows a group reaches.
__global__ void __launch_bounds__(GR_T) k_grid_sort(GridPlanDev gp, SpeciesSet spset, GridWork w) {
  extern __shared__ int cnt[];  // [2 n + 1]
  __shared__ int warp_sum[GR_T / 32];
  const int nf = 2 * gp.n, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int4 jb = gp.jobs[blockIdx.x];
  const int K = jb.w - jb.z;
  const double* pos = spset.k[jb.x & 3].pos + 2L * jb.z;
  const int at0 = gp.atom_beg[blockIdx.x];
  int* bin = w.bin + at0;
  int* base = w.base + at0;
  int* order = w.order + at0;
  int* first = w.first + at0 + blockIdx.x;
  int* ptr = w.ptr + (long)blockIdx.x * (nf + 1);
  unsigned char* used = w.used + (long)blockIdx.x * (nf / GR_ROWS);
  for (int i = tid; i < nf; i += GR_T) cnt[i] = 0;
  __syncthreads();
  for (int a = tid; a < K; a += GR_T) {
    const int b = first_row(fine_row(pos[2 * a + 1], gp.dky, nf), nf);
    bin[a] = b;
    atomicAdd(&cnt[b], 1);
  }
  block_exclusive_scan(cnt, nf, warp_sum);  // its barriers make bin visible to the CTA
  if (wid == 0) {
    constexpr int AHEAD = 4;  // chunks whose bins are loaded ahead of their placing
    int nb[AHEAD];
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) nb[k] = 32 * k + lane < K ? bin[32 * k + lane] : -1;
    for (int a0 = 0; a0 < K; a0 += 32 * AHEAD) {
#pragma unroll
      for (int k = 0; k < AHEAD; ++k) {
        const int a = a0 + 32 * k + lane, b = nb[k];
        nb[k] = a + 32 * AHEAD < K ? bin[a + 32 * AHEAD] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, b);  // lanes past the end: b = -1
        const int at = b >= 0 ? cnt[b] : 0;
        __syncwarp();
        if (b >= 0) {
          if (lane == __ffs(peers) - 1) cnt[b] = at + __popc(peers);
          order[at + __popc(peers & ((1u << lane) - 1u))] = a;
        }
        __syncwarp();
      }
    }
  }
  __syncthreads();  // the whole CTA sees the sorted order
  for (int i = tid; i < nf; i += GR_T) cnt[i] = 0;
  int groups = 0;  // groups before the chunk
  for (int i0 = 0; i0 < K; i0 += GR_T) {
    const int i = i0 + tid;
    bool head = false;
    int row = 0;
    if (i < K) {
      const int a = order[i];
      row = bin[a];
      head = i == 0 || !(pos[2 * order[i - 1] + 1] == pos[2 * a + 1]);
    }
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    __syncthreads();  // warp_sum of the previous chunk is read
    if (lane == 0) warp_sum[wid] = __popc(heads);
    __syncthreads();
    int gi = groups + __popc(heads & ((1u << lane) - 1u));
    for (int k = 0; k < GR_T / 32; ++k) {
      if (k < wid) gi += warp_sum[k];
      groups += warp_sum[k];
    }
    if (head) {
      first[gi] = i;
      base[gi] = row;
      atomicAdd(&cnt[row], 1);
    }
  }
  block_exclusive_scan(cnt, nf, warp_sum);
  if (tid == 0) {
    cnt[nf] = groups;
    first[groups] = K;
    w.groups[blockIdx.x] = groups;
  }
  __syncthreads();
  for (int i = tid; i <= nf; i += GR_T) ptr[i] = cnt[i];
  for (int b = tid; b < nf / GR_ROWS; b += GR_T) {
    const int f0 = b * GR_ROWS;
    bool u = cnt[max(f0 - GR_W + 1, 0)] != cnt[f0 + GR_ROWS];
    if (b == 0) u = u || cnt[nf - GR_W + 1] != cnt[nf];  // groups that wrap around
    used[b] = u;
  }
}

// exp(-2 pi i t) for t given in FP64, reduced to [-1/2, 1/2]: half the rounding of phase_of's [0, 1).
__device__ __forceinline__ float2 near_phase_of(double t) {
  float s, c;
  sincospif(2.f * (float)(t - rint(t)), &s, &c);
  return make_float2(c, -s);
}

// E[group][column]: the direct x phases, summed over the group's atoms in FP64, and the groups' spreading
// weights, for the groups [g0, g0 + ex_rows).  A CTA takes 128 columns of every gridDim.y-th chunk of 16
// groups of one job.
__global__ void __launch_bounds__(128) k_grid_phases(GridPlanDev gp, SpeciesSet spset, TxGrid g, int job0,
                                                     int col0, int g0, GridWork w) {
  const int h = col0 + blockIdx.x * 128 + threadIdx.x, job = job0 + blockIdx.z;
  const int4 jb = gp.jobs[job];
  const double* pos = spset.k[jb.x & 3].pos + 2L * jb.z;
  const int* order = w.order + gp.atom_beg[job];
  const int* first = w.first + gp.atom_beg[job] + job;
  double* wgt = w.wgt + (long)GR_W * gp.atom_beg[job];
  float2* ex = w.ex + (long)blockIdx.z * w.ex_rows * w.ex_cols + (h - col0);
  const int groups = min(w.groups[job], g0 + w.ex_rows);
  // half: column h holds kx = h dkx, the last of them +p_w / 2 (the grid's own -p_w / 2 is its
  // conjugate); columns beyond ``cols`` pad the pitch
  const double kx = h >= w.cols ? 0.0
                    : !w.half   ? g.kx_axis[h]
                    : 2 * h < g.p_w ? g.kx_axis[g.p_w / 2 + h]
                                    : -g.kx_axis[0];
  for (int q0 = g0 + blockIdx.y * 16; q0 < groups; q0 += gridDim.y * 16) {
    if (h < 128) {  // thread (q, k): weight k of group q
      const int q = q0 + threadIdx.x / GR_W, k = threadIdx.x % GR_W;
      if (q < groups) {
        const double v = fine_row(pos[2L * order[first[q]] + 1], gp.dky, 2 * gp.n);
        const double d = (ceil(v - GR_W / 2) + k - v) / (GR_W / 2);
        wgt[GR_W * q + k] = bessel_i0(GR_BETA * sqrt(fmax(1.0 - d * d, 0.0))) * (1.0 / bessel_i0(GR_BETA));
      }
    }
    if (h >= w.pitch) continue;
    for (int q = q0; q < min(q0 + 16, groups); ++q) {
      double2 s = make_double2(0.0, 0.0);
      for (int i = first[q]; i < first[q + 1]; ++i) {
        const double* p = pos + 2L * order[i];
        const float2 e = near_phase_of(kx * p[0] + (w.half ? 0.0 : gp.sy * p[1]));
        s = make_double2(s.x + e.x, s.y + e.y);
      }
      ex[(long)(q - g0) * w.ex_cols] = make_float2((float)s.x, (float)s.y);
    }
  }
}

// Adds weight times x of a group whose first fine row lies D rows from the block's.
template <int D>
__device__ __forceinline__ void spread_at(double2 (&acc)[GR_ROWS], const double* wt, double2 x) {
#pragma unroll
  for (int k = 0; k < GR_W; ++k)
    if (D + k >= 0 && D + k < GR_ROWS)
      acc[D + k] = make_double2(fma(wt[k], x.x, acc[D + k].x), fma(wt[k], x.y, acc[D + k].y));
}

// One block of GR_ROWS fine rows of one job and 128 columns, a column per thread: the groups that
// reach the block in sorted order.  All lanes take the same group, so its offset picks one of the 23
// unrolled bodies without divergence; the weights and rows of the next 16 groups are staged in shared
// memory while the present ones are added, and E is loaded four groups ahead of its use.
// The sums are FP64 and rounded once, whatever the atoms per row (25 000 terms on a row of 64^2: the
// transmission 1.3e-7 from 64 bits, with FP32 sums 2.0e-5; on grids filled with SrTiO3 it was 0.1-0.9 %
// further off with FP32 sums and phases reduced to [0, 1)).  64 instead of 32 registers of sums and half
// the FMA rate cost 27 us on 66 at 2048^2 with 10 jobs of 1024 atoms, 4.6 % of a build.  Slower still:
// weights read from global memory by every thread (+20 us), a thread per real component, half the
// registers and twice the threads (+42 us), E loaded eight groups ahead (126 registers, +12 us).
// PIECES: of the groups only [g0, g0 + ex_rows) are held.  The sums go on from one piece to the next in
// fine64, in the same order (the groups that wrap around sort last), so the pieces change no bit.
template <bool PIECES>
__global__ void __launch_bounds__(128) k_grid_spread(GridPlanDev gp, int job0, int col0, int g0, GridWork w) {
  const int nf = 2 * gp.n, f0 = blockIdx.y * GR_ROWS, job = job0 + blockIdx.z;
  const int h = col0 + blockIdx.x * 128 + threadIdx.x;
  if (!w.used[(long)job * (nf / GR_ROWS) + blockIdx.y]) return;
  constexpr int GR_Q = 128 / GR_W;  // groups whose weights and rows are staged at a time
  __shared__ double s_w[GR_Q][GR_W];
  __shared__ int s_row[GR_Q];
  const int hc = min(h, w.pitch - 1);
  const int* __restrict__ ptr = w.ptr + (long)job * (nf + 1);
  const int* __restrict__ base = w.base + gp.atom_beg[job];
  const double* __restrict__ wgt = w.wgt + (long)GR_W * gp.atom_beg[job];
  const float2* __restrict__ ex = w.ex + ((long)blockIdx.z * w.ex_rows - (PIECES ? g0 : 0)) * w.ex_cols + (hc - col0);
  const long at = ((long)blockIdx.z * nf + f0) * w.pitch + hc;
  // the groups of the block, and those that wrap around into the first one
  int lo = ptr[max(f0 - GR_W + 1, 0)], hi = ptr[f0 + GR_ROWS];
  int wlo = f0 == 0 ? ptr[nf - GR_W + 1] : 0, whi = f0 == 0 ? ptr[nf] : 0;
  const bool last = !PIECES || g0 + w.ex_rows >= w.kmax;
  if (PIECES) {
    lo = max(lo, g0), hi = min(hi, g0 + w.ex_rows);
    wlo = max(wlo, g0), whi = min(whi, g0 + w.ex_rows);
    if (g0 > 0 && !last && lo >= hi && wlo >= whi) return;
  }
  double2 acc[GR_ROWS];
#pragma unroll
  for (int t = 0; t < GR_ROWS; ++t)
    acc[t] = PIECES && g0 > 0 ? w.fine64[at + (long)t * w.pitch] : make_double2(0.0, 0.0);
  const int tq = threadIdx.x / GR_W, tk = threadIdx.x % GR_W;
  for (int wrap = 0; wrap < 2; ++wrap, lo = wlo, hi = whi) {
    const int shift = (wrap ? nf : 0) + f0;
    double next_w = 0.0;
    int next_row = 0;
    if (lo + tq < hi) {
      next_w = __ldg(wgt + (long)GR_W * (lo + tq) + tk);
      next_row = __ldg(base + lo + tq);
    }
    for (int q0 = lo; q0 < hi; q0 += GR_Q) {
      __syncthreads();  // the previous groups' weights are read
      s_w[tq][tk] = next_w;
      if (tk == 0) s_row[tq] = next_row - shift;
      __syncthreads();
      if (q0 + GR_Q + tq < hi) {
        next_w = __ldg(wgt + (long)GR_W * (q0 + GR_Q + tq) + tk);
        next_row = __ldg(base + q0 + GR_Q + tq);
      }
      const int m = min(GR_Q, hi - q0);
      for (int i0 = 0; i0 < m; i0 += 4) {
        float2 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          x[i] = i0 + i < m ? __ldg(ex + (long)(q0 + i0 + i) * w.ex_cols) : make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i0 + i >= m) break;
          const double2 xi = make_double2(x[i].x, x[i].y);
          const double* wt = s_w[i0 + i];
          switch (s_row[i0 + i]) {
#define TOTEM_SPREAD(D) \
  case D: spread_at<D>(acc, wt, xi); break;
            TOTEM_SPREAD(-7) TOTEM_SPREAD(-6) TOTEM_SPREAD(-5) TOTEM_SPREAD(-4) TOTEM_SPREAD(-3) TOTEM_SPREAD(-2)
            TOTEM_SPREAD(-1) TOTEM_SPREAD(0) TOTEM_SPREAD(1) TOTEM_SPREAD(2) TOTEM_SPREAD(3) TOTEM_SPREAD(4)
            TOTEM_SPREAD(5) TOTEM_SPREAD(6) TOTEM_SPREAD(7) TOTEM_SPREAD(8) TOTEM_SPREAD(9) TOTEM_SPREAD(10)
            TOTEM_SPREAD(11) TOTEM_SPREAD(12) TOTEM_SPREAD(13) TOTEM_SPREAD(14) TOTEM_SPREAD(15)
#undef TOTEM_SPREAD
          }
        }
      }
    }
  }
  if (h >= w.pitch) return;
#pragma unroll
  for (int t = 0; t < GR_ROWS; ++t) {
    if (last) w.fine[at + (long)t * w.pitch] = make_float2((float)acc[t].x, (float)acc[t].y);
    else w.fine64[at + (long)t * w.pitch] = acc[t];
  }
}

// V(r, c) of slices s_lo.. from the jobs [j_lo, j_hi): f_species(s^2) S summed over the jobs,
// PARAMETER * APERTURE as in k_tx_species.  A slice whose first jobs ran in an earlier batch adds
// to what that batch wrote.
__global__ void __launch_bounds__(256) k_grid_combine(TxGrid g, SpeciesSet spset, GridPlanDev gp, GridWork w, int s_lo,
                                                      int j_lo, int j_hi, float2* __restrict__ out) {
  const long plane = (long)g.p_h * g.p_w;
  const int s = s_lo + blockIdx.y;
  const int jb0 = max(gp.job_beg[s], j_lo), jb1 = min(gp.job_beg[s + 1], j_hi);
  const bool add = gp.job_beg[s] < j_lo;
  float2* dst = out + (long)s * plane;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < plane; i += (long)gridDim.x * blockDim.x) {
    const int r = (int)(i / g.p_w), c = (int)(i - (long)r * g.p_w);
    const float s2 = g.s2[i];
    float2 acc = make_float2(0.f, 0.f);
    for (int jj = jb0; jj < jb1; ++jj) {
      const int4 jb = gp.jobs[jj];
      const ColumnOfS col(w, w.s + (long)(jj - j_lo) * (g.p_h + 1) * w.pitch, g.p_h, g.p_w, c);
      float2 S = col.at(r);
      S.y *= col.sign;
      float fr, fi;
      species_form(jb.x & 3, g, spset.k[jb.x & 3], jb.y, s2, i, fr, fi);
      acc.x = fmaf(fr, S.x, fmaf(-fi, S.y, acc.x));
      acc.y = fmaf(fr, S.y, fmaf(fi, S.x, acc.y));
    }
    const float ap = (g.aper_true != nullptr) ? g.aper_true[i] : 1.f;
    float2 v = cscale(acc, g.parameter * ap);
    if (add) v = cadd(dst[i], v);
    dst[i] = v;
  }
}

// Columns of E held at a time: all, or as many whole 128s as keep a row for each of kmax atoms within 4 p_h
// rows (at least 128).
int grid_ex_cols(int p_h, int pitch, int kmax) {
  const long long cols = 4LL * p_h * pitch / kmax / 128 * 128;
  return (int)std::min<long long>(pitch, std::max(cols, 128LL));
}

// Where the parts of the work memory lie (base may be null: sizes only); returns its bytes.
// ``batch`` jobs in a batch.
size_t grid_work(int p_h, int p_w, int half, int kmax, int ex_rows, int jobs, long long atoms, int batch, char* base,
                 GridWork* w) {
  const size_t n = grid_transform(p_h);
  w->kmax = kmax;
  w->half = half;
  w->cols = half ? p_w / 2 + 1 : p_w;
  w->pitch = (int)grid_pitch(p_w, half);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* p = base + off;
    off += (bytes + 255) & ~size_t(255);
    return p;
  };
  const size_t nj = jobs, na = (size_t)atoms, nb = batch, row = w->pitch * sizeof(float2);
  w->wgt = reinterpret_cast<double*>(take(na * GR_W * sizeof(double)));
  w->bin = reinterpret_cast<int*>(take(na * sizeof(int)));
  w->base = reinterpret_cast<int*>(take(na * sizeof(int)));
  w->order = reinterpret_cast<int*>(take(na * sizeof(int)));
  w->first = reinterpret_cast<int*>(take((na + nj) * sizeof(int)));
  w->ptr = reinterpret_cast<int*>(take(nj * (2 * n + 1) * sizeof(int)));
  w->groups = reinterpret_cast<int*>(take(nj * sizeof(int)));
  w->used = reinterpret_cast<unsigned char*>(take(nj * (2 * n / GR_ROWS)));
  // E: ``ex_rows`` groups, in pieces of columns where the largest job's atoms would be more than 4 p_h rows
  w->ex_cols = grid_ex_cols(p_h, w->pitch, kmax);
  w->ex_rows = ex_rows;
  w->ex = reinterpret_cast<float2*>(take(nb * w->ex_rows * w->ex_cols * sizeof(float2)));
  w->fine = reinterpret_cast<float2*>(take(nb * 2 * n * row));
  w->s = reinterpret_cast<float2*>(take(nb * (p_h + 1) * row));
  w->fine64 = reinterpret_cast<double2*>(take(ex_rows < kmax ? nb * 2 * n * w->pitch * sizeof(double2) : 0));
  return off;
}

// Batches of whole slices of at most jobs_per_batch jobs; empty if a slice has more.
std::vector<GridBatch> whole_slice_batches(const std::vector<int>& job_beg, int jobs_per_batch) {
  std::vector<GridBatch> out;
  const int slices = (int)job_beg.size() - 1;
  for (int s = 0; s < slices;) {
    int e = s + 1;
    if (job_beg[e] - job_beg[s] > jobs_per_batch) return {};
    while (e < slices && job_beg[e + 1] - job_beg[s] <= jobs_per_batch) ++e;
    out.push_back(GridBatch{s, e, job_beg[s], job_beg[e]});
    s = e;
  }
  return out;
}

__global__ void k_sign_exp(float2* __restrict__ data, long total, int p_h, int p_w, float sig) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long plane = (long)p_h * p_w;
    const long k = i % plane;
    const int r = (int)(k / p_w), c = (int)(k % p_w);
    // ifftshift of the input == multiplication of the output by (-1)^(r+c) (even sizes only;
    // the uploader rejects odd grids, as the reference's quadrant-swap ifftShift assumes).
    data[i] = exp_i_sigma(data[i], r + c, sig);
  }
}

}  // namespace

bool fused_fft_size_ok(int n) {
  return (n >= 64 && n <= 4096 && (n & (n - 1)) == 0) || radix_window_ops(n) != nullptr;
}

namespace {
template <int N>
constexpr int2 tx_tiles() { return make_int2(RowCfg<N>::G, GridColCfg<N>::G); }
// (rows per row tile, columns per column tile) of the transmission FFT at edge n; (0, 0) if none
int2 tx_tiles_of(int n) {
  switch (n) {
#define TOTEM_TX_TILES(NN) \
  case NN: return tx_tiles<NN>();
    TOTEM_TX_TILES(64) TOTEM_TX_TILES(128) TOTEM_TX_TILES(256) TOTEM_TX_TILES(512) TOTEM_TX_TILES(1024)
    TOTEM_TX_TILES(2048) TOTEM_TX_TILES(4096)
#undef TOTEM_TX_TILES
  }
  if (const WindowOps* o = radix_window_ops(n)) return make_int2(o->row_tile_rows, o->col_tile_cols);
  return make_int2(0, 0);
}
}  // namespace

bool tx_fft_shape_ok(int p_h, int p_w, int slices) {
  const int2 rw = tx_tiles_of(p_w), ch = tx_tiles_of(p_h);
  return rw.x > 0 && ch.y > 0 && ((long)slices * p_h) % rw.x == 0 && p_w % ch.y == 0;
}

Status launch_tx_structure(const TxGrid& g, const AtomRowsDev& neutral, const AtomRowsDev& ion,
                           const AtomRowsDev& corr_n, const AtomRowsDev& corr_i, float2* out, cudaStream_t st,
                           bool accumulate) {
  dim3 grid((g.p_w + TX_TC - 1) / TX_TC, (g.p_h + TX_TR - 1) / TX_TR, g.slices);
  if (g.slices == 0) return Status::Ok();
  if (g.separable) k_tx_structure<true><<<grid, 256, 0, st>>>(g, neutral, ion, corr_n, corr_i, out, accumulate);
  else k_tx_structure<false><<<grid, 256, 0, st>>>(g, neutral, ion, corr_n, corr_i, out, accumulate);
  return cuda_status(cudaGetLastError(), "k_tx_structure");
}

Status launch_tx_species(const TxGrid& g, const SpeciesSet& sp, float2* out, cudaStream_t st) {
  if (g.slices == 0) return Status::Ok();
  if (!g.separable) return Status::Err(TOTEM_ERR_UNSUPPORTED, "species builder needs separable reciprocal grids");
  dim3 grid((g.p_w + SP_T - 1) / SP_T, (g.p_h + SP_T - 1) / SP_T, g.slices);
  k_tx_species<<<grid, 256, 0, st>>>(g, sp, out);
  return cuda_status(cudaGetLastError(), "k_tx_species");
}

int grid_transform(int p_h) {
  if (p_h < 1 || p_h > 4096) return 0;
  int n = 64;  // the powers of two, then a mixed-radix edge below the one found
  while (n < p_h) n *= 2;
  for (int m = p_h; m < n; ++m)
    if (radix_window_ops(m)) return m;
  return n;
}

std::vector<float2> grid_deconvolution(int p_h, int n) {
  // transform of the spreading kernel at xi = k / (2 n): W sinh(z) / (z I0(beta))
  const double pi = 3.14159265358979323846, i0 = bessel_i0(GR_BETA);
  std::vector<float2> t(2 * ((size_t)p_h + 1));
  for (int r = 0; r <= p_h; ++r) {
    const double k = r - p_h / 2, a = pi * GR_W * k / (2.0 * n);
    const double z = std::sqrt(GR_BETA * GR_BETA - a * a);
    const double d = z * i0 / (GR_W * std::sinh(z));
    t[2 * r] = make_float2((float)d, 0.f);
    t[2 * r + 1] = make_float2((float)(d * std::cos(pi * k / n)), (float)(-d * std::sin(pi * k / n)));
  }
  return t;
}

GridBytes grid_bytes(int p_h, int p_w, int half, int kmax, int ex_rows, int jobs, long long atoms) {
  GridWork w;
  const size_t tables = grid_work(p_h, p_w, half, kmax, ex_rows, jobs, atoms, 0, nullptr, &w);
  // (each part of a batch is rounded up to 256 bytes as a whole, so the batch never needs more)
  return GridBytes{tables, grid_work(p_h, p_w, half, kmax, ex_rows, jobs, atoms, 1, nullptr, &w) - tables};
}

int grid_piece_rows(int p_h, int p_w, int half, int kmax, size_t job_bytes) {
  const size_t rest = grid_bytes(p_h, p_w, half, kmax, 0, 1, 0).per_job;
  const int pitch = (int)grid_pitch(p_w, half), cols = grid_ex_cols(p_h, pitch, kmax);
  const long long least = std::max(4LL * p_h * pitch, 1LL << 20) / cols;
  const long long room = job_bytes > rest ? (long long)((job_bytes - rest) / (cols * sizeof(float2))) : 0;
  return (int)std::min<long long>(kmax, std::max(least, room));
}

std::vector<GridBatch> grid_batches(const std::vector<int>& job_beg, int jobs_per_batch) {
  std::vector<GridBatch> out;
  const int slices = (int)job_beg.size() - 1;
  if (slices <= 0 || jobs_per_batch < 1) return out;
  const int total = job_beg[slices];
  int s_lo = 0, j_lo = 0;
  while (s_lo < slices) {
    const int j_hi = std::min(j_lo + jobs_per_batch, total);
    int s_hi = s_lo;
    if (j_hi == total) s_hi = slices;
    else
      while (s_hi < slices && job_beg[s_hi] < j_hi) ++s_hi;
    out.push_back(GridBatch{s_lo, s_hi, j_lo, j_hi});
    const bool partial = job_beg[s_hi] > j_hi;  // slice s_hi - 1 continues in the next batch
    s_lo = partial ? s_hi - 1 : s_hi;
    j_lo = j_hi;
  }
  return out;
}

namespace {
// One instantiation per transform length: F(n) returns the Status of the launch.
#define TOTEM_GRID_DISPATCH(NN, FN, OP, ...)                                             \
  [&]() -> Status {                                                                      \
    switch (NN) {                                                                        \
      case 64: return FN<64>(__VA_ARGS__);                                               \
      case 128: return FN<128>(__VA_ARGS__);                                             \
      case 256: return FN<256>(__VA_ARGS__);                                             \
      case 512: return FN<512>(__VA_ARGS__);                                             \
      case 1024: return FN<1024>(__VA_ARGS__);                                           \
      case 2048: return FN<2048>(__VA_ARGS__);                                           \
      case 4096: return FN<4096>(__VA_ARGS__);                                           \
    }                                                                                    \
    if (const WindowOps* o = radix_window_ops(NN)) return o->OP(__VA_ARGS__);            \
    return Status::Err(TOTEM_ERR_UNSUPPORTED, "gridding builder: unsupported grid edge"); \
  }()
}  // namespace

Status launch_tx_gridding(const TxGrid& g, const SpeciesSet& sp, const GridPlanDev& gp,
                          const std::vector<int>& job_beg, int kmax, int ex_rows, long long atoms, const float2* tw_w,
                          const float2* tw_h, void* scratch, size_t scratch_bytes, bool finish, float sig, float2* out,
                          cudaStream_t st, int* launches, bool* finished) {
  *finished = false;
  if (g.slices == 0) return Status::Ok();
  if ((int)job_beg.size() != g.slices + 1) return Status::Err(TOTEM_ERR_STATE, "gridding job table size");
  const long plane = (long)g.p_h * g.p_w;
  const int jobs = job_beg.back();
  const GridBytes need = grid_bytes(g.p_h, g.p_w, gp.half, kmax, ex_rows, jobs, atoms);
  if (scratch_bytes < need.tables + need.per_job) return Status::Err(TOTEM_ERR_STATE, "gridding scratch below one job");
  // at most 65535: the job is a grid dimension
  const int per_batch = (int)std::min<size_t>((scratch_bytes - need.tables) / need.per_job, 65535);
  GridWork w;
  grid_work(g.p_h, g.p_w, gp.half, kmax, ex_rows, jobs, atoms, per_batch, static_cast<char*>(scratch), &w);
  // whole slices in every batch: their sums do not depend on the batch size.  Where a batch does not hold
  // a slice, its later jobs add to what the earlier ones wrote.
  std::vector<GridBatch> batches = whole_slice_batches(job_beg, per_batch);
  if (batches.empty()) {
    finish = false;
    batches = grid_batches(job_beg, per_batch);
  }
  // The inverse row transform runs with each batch; where a batch's rows are no whole row tiles (2048 rows
  // of 160 columns in batches of 111 slices: tiles of 20 rows) once after the last, over the whole stack,
  // whose rows are (tx_fft_shape_ok).
  bool rows_by_batch = true;
  for (const GridBatch& b : batches)
    if (finish && (long)(b.s_hi - b.s_lo) * g.p_h % tx_tiles_of(g.p_w).x) rows_by_batch = false;
  if (jobs > 0) {
    const size_t smem = sizeof(int) * (2 * (size_t)gp.n + 1);
    TOTEM_TRY(ensure_smem((const void*)k_grid_sort, smem));
    k_grid_sort<<<jobs, GR_T, smem, st>>>(gp, sp, w);
    TOTEM_TRY(cuda_status(cudaGetLastError(), "k_grid_sort"));
    ++*launches;
  }
  for (const GridBatch& b : batches) {
    const int nj = b.j_hi - b.j_lo;
    if (nj > 0) {
      for (int col0 = 0; col0 < w.pitch; col0 += w.ex_cols) {
        const unsigned cx = (std::min(w.ex_cols, w.pitch - col0) + 127) / 128;
        for (int g0 = 0; g0 < kmax; g0 += w.ex_rows) {
          const int ng = std::min(w.ex_rows, kmax - g0);
          k_grid_phases<<<dim3(cx, (unsigned)std::min((ng + 15) / 16, 1024), nj), 128, 0, st>>>(gp, sp, g, b.j_lo, col0,
                                                                                               g0, w);
          TOTEM_TRY(cuda_status(cudaGetLastError(), "k_grid_phases"));
          (w.ex_rows < kmax ? k_grid_spread<true> : k_grid_spread<false>)<<<dim3(cx, 2 * gp.n / GR_ROWS, nj), 128, 0, st>>>(
              gp, b.j_lo, col0, g0, w);
          TOTEM_TRY(cuda_status(cudaGetLastError(), "k_grid_spread"));
          *launches += 2;
        }
      }
      TOTEM_TRY(TOTEM_GRID_DISPATCH(gp.n, grid_cols, grid_cols, w, b.j_lo, nj, g.p_h, gp.ay, gp.tw, st));
      ++*launches;
    }
    if (finish) {
      float2* first = out + (long)b.s_lo * plane;
      TOTEM_TRY(TOTEM_GRID_DISPATCH(g.p_h, grid_cols_inv, grid_cols_inv, g, sp, gp, w, b.s_lo, b.s_hi, b.j_lo, out,
                                    tw_h, st));
      ++*launches;
      if (rows_by_batch) {
        TOTEM_TRY(TOTEM_GRID_DISPATCH(g.p_w, rows_exp, tx_rows_exp, first, (long)(b.s_hi - b.s_lo) * g.p_h, tw_w, sig,
                                      st));
        ++*launches;
      }
      continue;
    }
    const unsigned cx = (unsigned)std::min<long>((plane + 255) / 256, 2048);
    for (int s0 = b.s_lo; s0 < b.s_hi; s0 += 65535) {
      const int ns = std::min(b.s_hi - s0, 65535);
      k_grid_combine<<<dim3(cx, ns), 256, 0, st>>>(g, sp, gp, w, s0, b.j_lo, b.j_hi, out);
      TOTEM_TRY(cuda_status(cudaGetLastError(), "k_grid_combine"));
      ++*launches;
    }
  }
  if (finish && !rows_by_batch) {
    TOTEM_TRY(TOTEM_GRID_DISPATCH(g.p_w, rows_exp, tx_rows_exp, out, (long)g.slices * g.p_h, tw_w, sig, st));
    ++*launches;
  }
  *finished = finish;
  return Status::Ok();
}

Status launch_tx_fft_exp(float2* data, int slices, int p_h, int p_w, float sig, const float2* tw_w,
                         const float2* tw_h, cudaStream_t st) {
  if (!tx_fft_shape_ok(p_h, p_w, slices))
    return Status::Err(TOTEM_ERR_UNSUPPORTED, "fused transmission FFT: unsupported grid shape");
  const long nrows = (long)slices * p_h;
  switch (p_w) {
#define TOTEM_TX_ROWS_CASE(NN) \
  case NN: TOTEM_TRY(rows_inv<NN>(data, nrows, tw_w, st)); break;
    TOTEM_TX_ROWS_CASE(64) TOTEM_TX_ROWS_CASE(128) TOTEM_TX_ROWS_CASE(256) TOTEM_TX_ROWS_CASE(512)
    TOTEM_TX_ROWS_CASE(1024) TOTEM_TX_ROWS_CASE(2048) TOTEM_TX_ROWS_CASE(4096)
#undef TOTEM_TX_ROWS_CASE
    default: TOTEM_TRY(radix_window_ops(p_w)->tx_rows_inv(data, nrows, tw_w, st));
  }
  switch (p_h) {
#define TOTEM_TX_COLS_CASE(NN) \
  case NN: return cols_exp<NN>(data, slices, p_w, tw_h, sig, st);
    TOTEM_TX_COLS_CASE(64) TOTEM_TX_COLS_CASE(128) TOTEM_TX_COLS_CASE(256) TOTEM_TX_COLS_CASE(512)
    TOTEM_TX_COLS_CASE(1024) TOTEM_TX_COLS_CASE(2048) TOTEM_TX_COLS_CASE(4096)
#undef TOTEM_TX_COLS_CASE
  }
  return radix_window_ops(p_h)->tx_cols_exp(data, slices, p_w, tw_h, sig, st);
}

Status launch_sign_exp(float2* data, long total, int p_h, int p_w, float sig, cudaStream_t st) {
  if (total == 0) return Status::Ok();
  int blocks = (int)std::min<long>((total + 255) / 256, 148L * 16);
  k_sign_exp<<<blocks, 256, 0, st>>>(data, total, p_h, p_w, sig);
  return cuda_status(cudaGetLastError(), "k_sign_exp");
}

}  // namespace totem
