// The gridding transmission builder (TOTEM_TX_GRIDDING) and the form factors it shares with the
// direct sums, instantiated per grid height by transmission.cu (powers of two) and windows_mr_*.cu
// (mixed-radix heights).
//
// Per job (one species of one slice) the builder needs, on a separable grid with a uniform ky axis
// (ky(r) = ky(P/2) + (r - P/2) dky, P = p_h),
//   S(r, c) = sum_a exp(-2 pi i kx(c) x_a) exp(-2 pi i ky(r) y_a).
// The x factor is evaluated directly; the y factor is a type-1 non-uniform FFT per column, with N the
// smallest edge of the fused transforms that is at least P (GridPlanDev::n; N = P where the height is
// such an edge, and the inverse transform is fused too):
//   k_grid_sort    sorts the job's atoms by their place on a fine y grid of 2N rows and joins atoms
//                  of equal y into one group;
//   k_grid_phases  E[group][c] = sum over the group's atoms of exp(-2 pi i kx(c) x_a), and the
//                  group's GR_W spreading weights;
//   k_grid_spread  the fine rows: sum over groups of weight times E, sixteen rows of a column in
//                  one thread's registers, the lanes of a warp along c;
//   k_grid_cols    per column tile: the fine column's transform (two N-point FFTs, fine rows of
//                  even and odd index), its P central frequencies divided by the spreading kernel's
//                  transform: S;
//   k_grid_cols_inv  form factors, the sum over the slice's jobs, and the inverse column FFT;
//   k_rows_exp       the inverse row FFT and T = exp(i sigma V).
// (k_grid_combine in transmission.cu writes the sum itself instead, where per-atom correction rows
// are still to be added, a batch splits a slice, or cuFFT runs the transform.)
//
// Spreading: Kaiser-Bessel, phi(t) = I0(beta sqrt(1 - (2t/W)^2)) / I0(beta) on W = 8 fine rows with
// oversampling 2 and beta = pi sqrt((W/2)^2 (3/2)^2 - 0.8) (Beatty, Nishimura & Pauly, IEEE Trans.
// Med. Imaging 24 (2005) 799-808), whose transform W sinh(z)/(z I0(beta)), z = sqrt(beta^2 -
// (pi W xi)^2), is divided out.  The aliasing error is ~2e-8 of S at the largest |ky| and less
// below, under the FP32 rounding of the transforms; the weights and the fine rows' sums are FP64.
//
// Why this split: a 2-D fine grid (2P x 2P points per job) was 64 bytes per pixel and job of clearing,
// spreading, row and column passes: 29-44 ps per pixel and job.  With the x factor direct, nothing
// needs clearing and no atomics are used, so results are reproducible bit by bit.  On a grid
// centred on zero (kx(P_W/2) = ky(P/2) = 0, the axis antisymmetric: the reference's always is)
// S(-k) = conj S(k), so only the columns kx >= 0 are formed (GridWork::half).  Fine rows are handled
// in blocks of GR_ROWS; a block no group touches is neither written nor read.  (Spreading inside
// k_grid_cols, in shared memory, ran 6 times longer: its lanes hold four columns of eight row
// blocks, and atoms of a crystal crowd into a few blocks, so most lanes waited.)
#pragma once
#include "common.cuh"
#include "fft.cuh"
#include "tx_fft.cuh"

namespace totem {

namespace {

__device__ __forceinline__ float peng5(const float* c, float s2) {
  float f = 0.f;
#pragma unroll
  for (int i = 0; i < 5; ++i) f = fmaf(c[2 * i], __expf(-c[2 * i + 1] * s2), f);
  return f;
}

__device__ __forceinline__ float lobato5(const float* c, float g2) {
  float f = 0.f;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const float b = c[2 * i + 1];
    const float d = fmaf(b, g2, 1.f);
    f = fmaf(c[2 * i], __fdividef(fmaf(b, g2, 2.f), d * d), f);
  }
  return f;
}

// Form factor of one neutral (kind 0) or ionic (kind 1) coefficient row at s^2: real part fr
// (Peng: occ * sum a_i exp(-b_i s^2); Lobato: occ * sum a_i (2 + b_i g^2) / (1 + b_i g^2)^2 *
// exp(-B s^2), g^2 = 4 s^2; ionic rows mix the ion and atom sums by their fractions) and the
// absorptive imaginary part fi (occ * Peng sum of the absorptive row, or 0).
__device__ __forceinline__ void row_form(int kind, int lobato, const float* cf, const float* absorp, float s2,
                                         float& fr, float& fi) {
  if (kind == 0) {
    if (lobato) fr = cf[0] * lobato5(cf + 1, 4.f * s2) * __expf(-cf[11] * s2);
    else fr = cf[0] * peng5(cf + 1, s2);
  } else {
    if (lobato)
      fr = cf[0] * (cf[1] * lobato5(cf + 2, 4.f * s2) + cf[12] * lobato5(cf + 13, 4.f * s2)) * __expf(-cf[23] * s2);
    else fr = cf[0] * (cf[1] * peng5(cf + 2, s2) + cf[12] * peng5(cf + 13, s2));
  }
  fi = absorp != nullptr ? cf[0] * peng5(absorp, s2) : 0.f;
}

// Form factor of species ``sp`` of kind ``kind`` (SpeciesSet) at pixel ``pix`` (s^2 = s2):
// kinds 0 / 1 as row_form; the Peng-extended correction kinds 2 / 3
// (cuda_source_peng_and_corr.cu:587-779, GetPotential4AllSlice_multicore_lotabo_peng_corr.m:13-60)
// amplitude * exp(-B s^2) * the correction plane(s) at the pixel (planes numbered from 1).
__device__ __forceinline__ void species_form(int kind, const TxGrid& g, const SpeciesDev& d, int sp, float s2,
                                             long pix, float& fr, float& fi) {
  const float* cf = d.coef + (long)sp * d.ncoef;
  if (kind <= 1) {
    row_form(kind, g.lobato, cf, d.absorp != nullptr ? d.absorp + (long)sp * 10 : nullptr, s2, fr, fi);
    return;
  }
  const long plane = (long)g.p_h * g.p_w;
  float m = 0.f;
  if (kind == 2) {
    const int idx = (int)cf[2] - 1;
    if (idx >= 0 && idx < g.cim_len) m = g.cim[idx * plane + pix];
  } else {
    const int i1 = (int)cf[3] - 1, i2 = (int)cf[5] - 1;
    if (i1 >= 0 && i1 < g.cim_len) m = fmaf(cf[2], g.cim[i1 * plane + pix], m);
    if (i2 >= 0 && i2 < g.cim_len) m = fmaf(cf[4], g.cim[i2 * plane + pix], m);
  }
  fr = cf[1] * m * __expf(-cf[0] * s2);
  fi = 0.f;
}

// exp(-2 pi i t) for t given in FP64, reduced to [0, 1) before the FP32 evaluation.
__device__ __forceinline__ float2 phase_of(double t) {
  const double fr = t - floor(t);
  float s, c;
  sincospif(2.f * (float)fr, &s, &c);
  return make_float2(c, -s);
}

constexpr int GR_W = 8;      // fine rows an atom spreads over
constexpr int GR_ROWS = 16;  // fine rows of one block

// Column tile of k_grid_cols: the column pass's width, four columns from P = 2048 on (two 256-thread
// CTAs per SM; a 32-byte segment of a row is whole sectors).
template <int N>
using GridTile = ColCfg<N, 4, (N >= 2048) ? 4 : 0>;

// S of the jobs of a batch from their fine rows.  The even and odd spectra are added through S itself
// (the same thread writes and reads back its elements).
// WHOLE: the grid has N rows (known at compile time, so that no row is tested).
template <int N, bool WHOLE>
__global__ void __launch_bounds__(GridTile<N>::G * GridTile<N>::T, GridTile<N>::MINB)
    k_grid_cols(GridWork w, int job0, int rows, const float4* __restrict__ ay, int tiles, const float2* __restrict__ tw) {
  constexpr int P = GridTile<N>::P, T = GridTile<N>::T, G = GridTile<N>::G;
  const int p_h = WHOLE ? N : rows;
  extern __shared__ float2 sh[];
  float2* s_tw = sh;
  float2* s_x = sh + Fft<N>::tw_size;
  const int job = blockIdx.x / tiles, col0 = (blockIdx.x - job * tiles) * G;
  const int j = threadIdx.x / G, g = threadIdx.x - j * G;
  const float2* __restrict__ fine = w.fine + (long)job * 2 * N * w.pitch + col0 + g;
  const unsigned char* __restrict__ used = w.used + (long)(job0 + job) * (2 * N / GR_ROWS);
  float2* S = w.s + (long)job * (p_h + 1) * w.pitch + col0 + g;
  load_twiddles<N>(s_tw, tw);
  static_for<0, 2>([&](auto parity) {
    constexpr int e = decltype(parity)::value;
    float2 v[P];
#pragma unroll
    for (int m = 0; m < P; ++m) {
      const int f = 2 * (j + m * T) + e;
      v[m] = __ldg(used + f / GR_ROWS) ? __ldg(fine + f * w.pitch) : make_float2(0.f, 0.f);
    }
    __syncthreads();  // twiddles staged; the previous parity's exchanges are done
    fft_regs<N, false>(v, j, g, s_tw, s_x, ColLayout<N, G>(), SyncBlock());
#pragma unroll
    for (int m = 0; m < P; ++m) {
      if (m % 8 == 0) asm volatile("" ::: "memory");  // eight loads of S in flight: all of them would spill
      // frequency ky = k or k - N is row r = ky + p_h / 2; one row more, ky = +p_h / 2, is what the
      // conjugate half of row 0 (ky = -p_h / 2) needs.  With p_h = N that is row 0's own frequency
      // with the odd half's phase turned by pi.
      const int k = j + m * T, r = (m < P / 2 ? k : k - N) + p_h / 2;
      if (WHOLE || (r >= 0 && r <= p_h)) {
        const float4 a = __ldg(ay + r);
        float2* dst = S + r * w.pitch;
        if (e == 0) {
          *dst = cscale(v[m], a.x);
        } else {
          const float2 odd = cmul(v[m], make_float2(a.z, a.w)), even = *dst;
          *dst = cadd(even, odd);
          if (WHOLE && m == P / 2 && j == 0) S[N * w.pitch] = csub(even, odd);
        }
      }
    }
  });
}

// S of one job along column c of the grid, from the columns held: row r of the grid is row
// ``at(r)`` of the held column and its conjugate on the kx < 0 side of a half plane,
// S(ky, kx) = conj S(-ky, -kx).  ``sign`` is that of its imaginary part.
struct ColumnOfS {
  const float2* p;
  int step;
  float sign;
  __device__ __forceinline__ ColumnOfS(const GridWork& w, const float2* sj, int p_h, int p_w, int c) {
    const int kx = c - p_w / 2;
    const bool conj = w.half && kx < 0;
    p = conj ? sj + (long)p_h * w.pitch - kx : sj + (w.half ? kx : c);
    step = conj ? -w.pitch : w.pitch;
    sign = conj ? -1.f : 1.f;
  }
  __device__ __forceinline__ float2 at(int r) const { return __ldg(p + r * step); }
};

// exp(x) of a coefficient sum with the factor log2(e) already in x.
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Adds one job's f S at the thread's rows to its slots acc[k * G] (k = r + N / 2 mod N the transform's
// index of grid row r = j, j + T, .. < N).  The form factor's kind is a template parameter (FORM: 0
// neutral Peng without absorption, 1 neutral Lobato likewise, 2 any), so the row loop holds one
// short body, and the loads of B rows are issued together.
template <int N, int G, int T, int FORM>
__device__ __forceinline__ void add_job(float2* acc, int j, int c, const TxGrid& g, const SpeciesDev& d, int4 jb,
                                        const ColumnOfS& col) {
  constexpr int P = N / T, B = P % 8 == 0 ? 8 : 4;
  constexpr float L2E = 1.4426950408889634f;
  static_assert(P % B == 0, "whole batches of rows");
  float cf[12];
  if (FORM < 2) {
#pragma unroll
    for (int i = 0; i < (FORM ? 12 : 11); ++i) cf[i] = __ldg(d.coef + (long)jb.y * d.ncoef + i);
    if (FORM == 0)
#pragma unroll
      for (int i = 0; i < 5; ++i) cf[2 * i + 2] *= -L2E;
    else cf[11] *= -L2E;
  }
  const float* __restrict__ s2p = g.s2 + c;
#pragma unroll 1
  for (int r0 = j; r0 < N; r0 += B * T) {
    float2 S[B];
    float s2[B];
#pragma unroll
    for (int i = 0; i < B; ++i) {
      S[i] = col.at(r0 + i * T);
      s2[i] = __ldg(s2p + (r0 + i * T) * g.p_w);
    }
#pragma unroll
    for (int i = 0; i < B; ++i) {
      const int r = r0 + i * T;
      float fr = 0.f, fi = 0.f;
      if (FORM == 0) {
#pragma unroll
        for (int q = 0; q < 5; ++q) fr = fmaf(cf[2 * q + 1], exp2_fast(cf[2 * q + 2] * s2[i]), fr);
        fr *= cf[0];
      } else if (FORM == 1) {
        fr = cf[0] * lobato5(cf + 1, 4.f * s2[i]) * exp2_fast(cf[11] * s2[i]);
      } else {
        species_form(jb.x & 3, g, d, jb.y, s2[i], (long)r * g.p_w + c, fr, fi);
      }
      float2& a = acc[(r < N / 2 ? r + N / 2 : r - N / 2) * G];
      const float sy = S[i].y * col.sign;
      float2 v = a;
      v.x = fmaf(fr, S[i].x, v.x);
      v.y = fmaf(fr, sy, v.y);
      if (FORM == 2) {
        v.x = fmaf(-fi, sy, v.x);
        v.y = fmaf(fi, S[i].x, v.y);
      }
      a = v;
    }
  }
}

// V of whole slices and its inverse column FFT: thread (j, g) sums f S over the slice's jobs at its
// own rows k (natural FFT order, so the ifftshift along y needs no sign), scales by PARAMETER *
// APERTURE and transforms.  The sums stand in the thread's own slots of the exchange region until
// the transform takes them, so the loop over rows need not be unrolled (unrolled 32 times, with the
// form factors inside, it ran from instruction-cache misses: 158 us a slice at 2048^2).
template <int N>
__global__ void __launch_bounds__(GridTile<N>::G * GridTile<N>::T, GridTile<N>::MINB)
    k_grid_cols_inv(TxGrid g, SpeciesSet spset, GridPlanDev gp, GridWork w, int s_lo, int j_lo,
                    float2* __restrict__ out, const float2* __restrict__ tw) {
  constexpr int P = GridTile<N>::P, T = GridTile<N>::T, G = GridTile<N>::G;
  extern __shared__ float2 sh[];
  float2* s_tw = sh;
  float2* s_x = sh + Fft<N>::tw_size;
  const int nblk = g.p_w / G;
  const int slice = blockIdx.x / nblk, cb = blockIdx.x - slice * nblk;
  const int j = threadIdx.x / G, cg = threadIdx.x - j * G;
  const int c = cb * G + cg;
  load_twiddles<N>(s_tw, tw);
  float2* acc = s_x + cg;
  for (int k = j; k < N; k += T) acc[k * G] = make_float2(0.f, 0.f);
  const int jb0 = gp.job_beg[s_lo + slice], jb1 = gp.job_beg[s_lo + slice + 1];
  for (int jj = jb0; jj < jb1; ++jj) {
    const int4 jb = gp.jobs[jj];
    const SpeciesDev& d = spset.k[jb.x & 3];
    const ColumnOfS col(w, w.s + (long)(jj - j_lo) * (N + 1) * w.pitch, N, g.p_w, c);
    if ((jb.x & 3) == 0 && d.absorp == nullptr) {
      if (g.lobato) add_job<N, G, T, 1>(acc, j, c, g, d, jb, col);
      else add_job<N, G, T, 0>(acc, j, c, g, d, jb, col);
    } else {
      add_job<N, G, T, 2>(acc, j, c, g, d, jb, col);
    }
  }
  float2 v[P];
#pragma unroll
  for (int m = 0; m < P; ++m) {
    const int k = j + m * T, r = m < P / 2 ? k + N / 2 : k - N / 2;
    const float ap = (g.aper_true != nullptr) ? g.aper_true[(long)r * g.p_w + c] : 1.f;
    v[m] = cscale(acc[k * G], g.parameter * ap);
  }
  __syncthreads();  // every slot is read, and the twiddles staged, before the exchange region is used
  fft_regs<N, true>(v, j, cg, s_tw, s_x, ColLayout<N, G>(), SyncBlock());
  float2* p = out + (long)(s_lo + slice) * N * g.p_w + c;
#pragma unroll
  for (int m = 0; m < P; ++m) p[(j + m * T) * g.p_w] = v[m];
}

// In-place inverse FFT of rows of length N, (-1)^c (the ifftshift along x), exp(i sig V).
template <int N>
__global__ void __launch_bounds__(RowCfg<N>::G * RowCfg<N>::T, RowCfg<N>::MINB)
    k_rows_exp(float2* __restrict__ data, const float2* __restrict__ tw, float sig) {
  constexpr int P = RowCfg<N>::P, T = RowCfg<N>::T, G = RowCfg<N>::G;
  extern __shared__ float2 sh[];
  float2* s_tw = sh;
  float2* s_x = sh + Fft<N>::tw_size;
  const int g = threadIdx.x / T, j = threadIdx.x - g * T;
  float2* p = data + ((long)blockIdx.x * G + g) * N;
  load_twiddles<N>(s_tw, tw);
  float2 v[P];
#pragma unroll
  for (int m = 0; m < P; ++m) v[m] = p[j + m * T];
  __syncthreads();
  fft_regs<N, true>(v, j, g, s_tw, s_x, RowLayout<N>(), group_sync<N>(g));
#pragma unroll
  for (int m = 0; m < P; ++m) p[j + m * T] = exp_i_sigma(v[m], j + m * T, sig);
}

template <int N>
Status grid_cols(const GridWork& w, int job0, int jobs, int p_h, const float2* ay, const float2* tw, cudaStream_t st) {
  constexpr int T = GridTile<N>::T, G = GridTile<N>::G;
  static_assert(2 * N % GR_ROWS == 0, "whole blocks of fine rows");
  const size_t smem = sizeof(float2) * (Fft<N>::tw_size + ColLayout<N, G>::size(G));
  const auto kernel = p_h == N ? k_grid_cols<N, true> : k_grid_cols<N, false>;
  TOTEM_TRY(ensure_smem((const void*)kernel, smem));
  if (w.pitch % G) return Status::Err(TOTEM_ERR_STATE, "gridding pitch not a multiple of the column tile");
  const int tiles = (w.cols + G - 1) / G;
  kernel<<<(unsigned)((long)jobs * tiles), G * T, smem, st>>>(w, job0, p_h, reinterpret_cast<const float4*>(ay), tiles, tw);
  return cuda_status(cudaGetLastError(), "k_grid_cols");
}

template <int N>
Status grid_cols_inv(const TxGrid& g, const SpeciesSet& sp, const GridPlanDev& gp, const GridWork& w, int s_lo,
                     int s_hi, int j_lo, float2* out, const float2* tw, cudaStream_t st) {
  constexpr int T = GridTile<N>::T, G = GridTile<N>::G;
  const size_t smem = sizeof(float2) * (Fft<N>::tw_size + ColLayout<N, G>::size(G));
  TOTEM_TRY(ensure_smem((const void*)k_grid_cols_inv<N>, smem));
  if (g.p_w % G) return Status::Err(TOTEM_ERR_UNSUPPORTED, "potential width not a multiple of the column tile");
  k_grid_cols_inv<N><<<(unsigned)((long)(s_hi - s_lo) * (g.p_w / G)), G * T, smem, st>>>(g, sp, gp, w, s_lo, j_lo, out,
                                                                                         tw);
  return cuda_status(cudaGetLastError(), "k_grid_cols_inv");
}

template <int N>
Status rows_exp(float2* data, long nrows, const float2* tw, float sig, cudaStream_t st) {
  constexpr int T = RowCfg<N>::T, G = RowCfg<N>::G;
  const size_t smem = sizeof(float2) * (Fft<N>::tw_size + RowLayout<N>::size(G));
  TOTEM_TRY(ensure_smem((const void*)k_rows_exp<N>, smem));
  if (nrows % G) return Status::Err(TOTEM_ERR_UNSUPPORTED, "row count not a multiple of the row tile");
  k_rows_exp<N><<<(unsigned)(nrows / G), G * T, smem, st>>>(data, tw, sig);
  return cuda_status(cudaGetLastError(), "k_rows_exp");
}

}  // namespace

}  // namespace totem
