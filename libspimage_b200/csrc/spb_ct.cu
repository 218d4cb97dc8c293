// Passes of 192, 384 and 1000-point lines with the radix plan, the strides and
// the divisions of the stages known at compile time: one butterfly a thread and
// stage, the projection's and the update's operands fetched with the line.
// The mixed-radix kernels (spb_mixed.cuh) run every length and do better on
// most grids; these are kept for the grids where they are the faster ones,
// by the rules beside the launchers.  Figures there are us per HIO slot with an
// area update every 20 slots on one B200, both sides in turn on one box.
#include <math.h>

#include "spb_internal.h"
#include "spb_passes.cuh"
#include "spb_pointwise.cuh"

namespace spb {
namespace ct {

// The canonical radix plan: 16s first, then one 8/4/2 (a trailing 2 after a 16
// turns that 16 into 8*4), then 3s and 5s.
__host__ __device__ constexpr int plan(int n, int *r) {
  int k = 0, m = n, n16 = 0;
  while (m % 16 == 0) { r[k++] = 16; m /= 16; n16++; }
  if (m % 8 == 0) { r[k++] = 8; m /= 8; }
  else if (m % 4 == 0) { r[k++] = 4; m /= 4; }
  else if (m % 2 == 0) {
    if (n16 > 0) { r[k - 1] = 8; r[k++] = 4; }
    else r[k++] = 2;
    m /= 2;
  }
  while (m % 3 == 0) { r[k++] = 3; m /= 3; }
  while (m % 5 == 0) { r[k++] = 5; m /= 5; }
  return k;
}
__host__ __device__ constexpr int plan_len(int n) {
  int r[32] = {};
  return plan(n, r);
}
__host__ __device__ constexpr int plan_radix(int n, int s) {
  int r[32] = {};
  plan(n, r);
  return r[s];
}
// the largest number of butterflies of any stage: threads per line that give
// every thread at most one butterfly per stage
__host__ __device__ constexpr int max_butterflies(int n) {
  int r[32] = {};
  const int k = plan(n, r);
  int m = 0;
  for (int s = 0; s < k; s++) m = (n / r[s] > m) ? n / r[s] : m;
  return m;
}

// The stages from S on, between the buffers x and y (points es apart); twiddles
// from the per-stage table ([stage][m-1][k]).  All threads of the block call
// it; returns the buffer of the result.
template <int N, int S, int NS, bool INV>
struct Stages {
  static __device__ float2 *run(float2 *x, float2 *y, const float2 *__restrict__ stw, int es, int t0, int tn) {
    constexpr int R = plan_radix(N, S);
    constexpr int NB = N / R;
    for (int b = t0; b < NB; b += tn) {
      const int k = b % NS;
      float2 a[R];
#pragma unroll
      for (int m = 0; m < R; m++) a[m] = x[(b + m * NB) * es];
      if (NS > 1 && k) {
#pragma unroll
        for (int m = 1; m < R; m++) {
          float2 w = stw[(m - 1) * NS + k];
          if (INV) w.y = -w.y;
          a[m] = cmulw(a[m], w.x, w.y);
        }
      }
      bfly<R, INV>(a);
      const int base = (b / NS) * NS * R + k;
#pragma unroll
      for (int m = 0; m < R; m++) y[(base + m * NS) * es] = a[m];
    }
    __syncthreads();
    if constexpr (S + 1 < plan_len(N)) return Stages<N, S + 1, NS * R, INV>::run(y, x, stw + (R - 1) * NS, es, t0, tn);
    else return y;
  }
};
template <int N, bool INV>
__device__ __forceinline__ float2 *line_fft(float2 *x, float2 *y, const float2 *stw, int es, int t0, int tn) {
  return Stages<N, 0, 1, INV>::run(x, y, stw, es, t0, tn);
}

// ---------------------------------------------------------------- row pass
// rpb rows a block, tpr threads each.  Shared memory: two buffers a row (four
// in the difference map's iteration), then (iterations) g0 and the flags of
// the rows.  Stage twiddles are read from device memory.
template <int MODE, int N>
__device__ __forceinline__ void row_pass(const float2 *stw, const PassArgs &a, int tpr, int rpb, long long nrows) {
  extern __shared__ float2 smem[];
  const int lr = threadIdx.x / tpr, t = threadIdx.x % tpr;
  const long long row = (long long)blockIdx.x * rpb + lr;
  const bool valid = row < nrows;
  const long long base = row * N;
  const size_t slab = (size_t)rpb * N;
  float2 *A = smem + (size_t)lr * N;
  float2 *B = A + slab;
  float2 *Cb = A + 2 * slab;
  float2 *D = A + 3 * slab;
  constexpr bool UPD = MODE == ROW_ITER || MODE == ROW_DM_ITER;
  constexpr int NBUF = MODE == ROW_DM_ITER ? 4 : 2;
  float2 *G0S = smem + (size_t)NBUF * slab + (size_t)lr * N;
  uint8_t *FLS = reinterpret_cast<uint8_t *>(smem + (size_t)(NBUF + 1) * slab) + (size_t)lr * N;

  for (int i = t; i < N; i += tpr) {
    float2 v = make_float2(0.0f, 0.0f), w = make_float2(0.0f, 0.0f);
    if (valid) {
      if constexpr (MODE == ROW_FWD_DEPHASE) {
        v = make_float2(cabs_ref(a.src[base + i]), 0.0f);
      } else {
        v = a.src[base + i];
        if constexpr (MODE == ROW_DM_ITER) w = a.src2[base + i];
      }
    }
    A[i] = v;
    if constexpr (MODE == ROW_DM_ITER) Cb[i] = w;
    if constexpr (UPD) {
      if (valid) {
        G0S[i] = a.g0[base + i];
        FLS[i] = a.flags[base + i];
      }
    }
  }
  __syncthreads();

  if constexpr (MODE == ROW_FWD_DEPHASE) {
    float2 *r = line_fft<N, false>(A, B, stw, 1, t, tpr);
    if (valid)
      for (int i = t; i < N; i += tpr) a.dst[base + i] = r[i];
  } else if constexpr (MODE == ROW_ITER) {
    const float beta = iter_beta(a);
    const float one_m2b = fsub(1.0f, fmul(2.0f, beta));  // 1 - 2*beta in float, as the reference
    float2 *r = line_fft<N, true>(A, B, stw, 1, t, tpr);
    for (int i = t; i < N; i += tpr) {
      float2 g = make_float2(0.0f, 0.0f);
      if (valid) {
        const long long idx = base + i;
        const float2 gp = scale_cmul_dev(r[i], a.inv_n);
        if (a.gp) a.gp[idx] = gp;
        const uint8_t f = FLS[i];
        if (f & FLAG_INSIDE) {
          g = gp;
        } else if (a.alg == ALG_HIO) {
          const float2 g0 = G0S[i];
          g = make_float2(fsub(g0.x, fmul(gp.x, beta)), fsub(g0.y, fmul(gp.y, beta)));
        } else if (a.alg == ALG_RAAR) {
          const float2 g0 = G0S[i];
          g = make_float2(fadd(fmul(gp.x, one_m2b), fmul(g0.x, beta)),
                          fadd(fmul(gp.y, one_m2b), fmul(g0.y, beta)));
        }
        g = apply_constraints(g, f, a.constraints);
        a.g1[idx] = g;
      }
      r[i] = g;
    }
    __syncthreads();
    float2 *x = line_fft<N, false>(r, r == A ? B : A, stw, 1, t, tpr);
    if (valid)
      for (int i = t; i < N; i += tpr) a.dst[base + i] = x[i];
  } else {
    static_assert(MODE == ROW_DM_ITER, "a mode without a pass");
    const float beta = iter_beta(a);
    float2 *rho = line_fft<N, true>(A, B, stw, 1, t, tpr);
    float2 *fr = line_fft<N, true>(Cb, D, stw, 1, t, tpr);
    for (int i = t; i < N; i += tpr) {
      float2 g = make_float2(0.0f, 0.0f), f1 = g;
      if (valid) {
        const long long idx = base + i;
        if (a.gp) a.gp[idx] = rho[i];
        const uint8_t f = FLS[i];
        g = dm_point(rho[i], fr[i], G0S[i], f, beta, a);
        a.g1[idx] = g;
        f1 = (f & FLAG_INSIDE) ? g : make_float2(fmul(-a.gamma1, g.x), fmul(-a.gamma1, g.y));
      }
      rho[i] = g;
      fr[i] = f1;
    }
    __syncthreads();
    float2 *x = line_fft<N, false>(rho, rho == A ? B : A, stw, 1, t, tpr);
    float2 *xf = line_fft<N, false>(fr, fr == Cb ? D : Cb, stw, 1, t, tpr);
    if (valid)
      for (int i = t; i < N; i += tpr) {
        a.dst[base + i] = x[i];
        a.dst2[base + i] = xf[i];
      }
  }
}
template <int MODE, int N>
__global__ void __launch_bounds__(256) row_kernel(const float2 *stw, PassArgs a, int tpr, int rpb, long long nrows) {
  row_pass<MODE, N>(stw, a, tpr, rpb, nrows);
}

// ------------------------------------------------------------- column pass
// byte offset of the stage table behind a column block's buffers (16-byte aligned)
__host__ __device__ constexpr size_t tw_offset(int n, int nl) { return ((size_t)n * nl * (2 * 8 + 5) + 15) / 16 * 16; }

// The projection of nl columns a block, tpc threads each.  Shared memory: two
// buffers, the columns' amplitudes and flags, the stage table.
template <int MODE, int N>
__device__ __forceinline__ void col_pass(const float2 *stw, const PassArgs &a, int nl, int tpc) {
  extern __shared__ float2 smem[];
  const int cc = threadIdx.x % nl, t = threadIdx.x / nl;
  const long long o = a.outer0 + blockIdx.y;
  const int c = blockIdx.x * nl + cc;
  const bool valid = c < a.ncols;
  float2 *A = smem + cc;
  float2 *B = smem + (size_t)N * nl + cc;
  const long long lbase = o * a.ostride + c;
  float *AMc = reinterpret_cast<float *>(smem + (size_t)2 * N * nl) + cc;
  uint8_t *FLc = reinterpret_cast<uint8_t *>(reinterpret_cast<float *>(smem + (size_t)2 * N * nl) + (size_t)N * nl) + cc;
  const long long ai0 = lbase % a.n_start;  // amplitude index of element 0
  float2 *TW = reinterpret_cast<float2 *>(reinterpret_cast<unsigned char *>(smem) + tw_offset(N, nl));
  for (int i = threadIdx.x; i < N - 1; i += blockDim.x) TW[i] = stw[i];

  for (int i = t; i < N; i += tpc) {
    float2 v = make_float2(0.0f, 0.0f);
    if (valid) {
      v = a.src[lbase + i * a.estride];
      AMc[(size_t)i * nl] = a.amp[ai0 + i * a.estride];
      FLc[(size_t)i * nl] = a.flags[lbase + i * a.estride];
    }
    A[(size_t)i * nl] = v;
  }
  __syncthreads();

  float2 *f = line_fft<N, false>(A, B, TW, nl, t, tpc);
  if (valid) {
    for (int i = t; i < N; i += tpc) {
      float2 &G = f[(size_t)i * nl];
      G = project_vals(G, FLc[(size_t)i * nl], AMc[(size_t)i * nl], ai0 + i * a.estride, a, MODE == COL_PROJECT);
    }
  }
  __syncthreads();
  float2 *r = line_fft<N, true>(f, f == A ? B : A, TW, nl, t, tpc);
  if (valid)
    for (int i = t; i < N; i += tpc) a.dst[lbase + i * a.estride] = r[(size_t)i * nl];
}
template <int MODE, int N>
__global__ void __launch_bounds__(1024) col_kernel(const float2 *stw, PassArgs a, int nl, int tpc) {
  col_pass<MODE, N>(stw, a, nl, tpc);
}
// 1000-point columns, four of 200 threads a block: with at most 32 registers
// two blocks share an SM (43.2 -> 39.9 us a slot with rows of the same cap)
template <int MODE>
__global__ void __maxnreg__(32) col_kernel_1000(const float2 *stw, PassArgs a, int nl, int tpc) {
  col_pass<MODE, 1000>(stw, a, nl, tpc);
}

// ---------------------------------------------------------------- launches
template <int MODE, int N>
static cudaError_t launch_row(const LinePlan &px, const PassArgs &a, cudaStream_t st) {
  constexpr bool UPD = MODE == ROW_ITER || MODE == ROW_DM_ITER;
  constexpr int NBUF = MODE == ROW_DM_ITER ? 4 : 2;
  constexpr int tpr = max_butterflies(N) > 64 ? max_butterflies(N) : 64;  // at least two warps a row
  const long long nrows = a.n / N;
  long long rpb = nrows / 296;  // no fewer blocks than two per SM when the rows allow it
  if (rpb > 256 / tpr) rpb = 256 / tpr;
  if (rpb < 1) rpb = 1;
  const size_t smem = (size_t)(NBUF + (UPD ? 1 : 0)) * rpb * N * sizeof(float2) + (UPD ? (size_t)rpb * N : 0);
  const cudaError_t e = ensure_smem<row_kernel<MODE, N>>(smem);
  if (e != cudaSuccess) return e;
  row_kernel<MODE, N><<<(unsigned)((nrows + rpb - 1) / rpb), (int)rpb * tpr, smem, st>>>(px.stw, a, tpr, (int)rpb, nrows);
  return cudaGetLastError();
}

template <int MODE, int N>
static cudaError_t launch_col(const LinePlan &pl, const PassArgs &a, cudaStream_t st) {
  constexpr int tpc = max_butterflies(N);
  // four columns: a full 32-byte sector of every row, and more blocks than
  // wider ones give a single pattern (192^2 at 16/8/4/2/1 columns
  // 13.6/12.2/11.6/11.9/12.6, 384^2 -/16.4/14.9/15.9/17.8)
  const int nl = a.col_width > 0 ? a.col_width : 4;
  const size_t smem = tw_offset(N, nl) + (size_t)(N - 1) * sizeof(float2);
  const dim3 grid((a.ncols + nl - 1) / nl, a.nouter);
  if constexpr (N == 1000) {
    const cudaError_t e = ensure_smem<col_kernel_1000<MODE>>(smem);
    if (e != cudaSuccess) return e;
    col_kernel_1000<MODE><<<grid, nl * tpc, smem, st>>>(pl.stw, a, nl, tpc);
  } else {
    const cudaError_t e = ensure_smem<col_kernel<MODE, N>>(smem);
    if (e != cudaSuccess) return e;
    col_kernel<MODE, N><<<grid, nl * tpc, smem, st>>>(pl.stw, a, nl, tpc);
  }
  return cudaGetLastError();
}

}  // namespace ct

// Which grids run here (the measured pairs are mixed-radix / these kernels for
// the pass, the other pass as it is built in).
// Rows of 192 points: one wave of 1024 threads an SM, up to 2368 rows on 148 SMs:
// 192^2 x 1 12.5 / 11.2, x 8 16.3 / 15.2, x 12 17.9 / 17.5, x 14 20.5 / 21.0, x 16 21.1 /
// 23.6.  Rows of 384 points: half a wave, up to 592: 384^2 x 1 14.4 / 13.8, x 2 17.0
// / 17.1, 1000 rows 21.8 / 22.1.  Rows of 1000 points: only the difference map's,
// where its projections run here.
static bool row_here(int mode, int n, long long nrows, int sms) {
  if (mode == ROW_DM_ITER) return n == 1000 && 2 * nrows > 16LL * sms;
  if (mode != ROW_ITER && mode != ROW_FWD_DEPHASE) return false;
  return (n == 192 && nrows * 64 <= 1024LL * sms) || (n == 384 && nrows * 128 <= 512LL * sms);
}
// Projections of 192 and 384-point columns: one wave of 1024 threads an SM, up to
// 2368 and 1184 columns: 192^2 x 1 13.5 / 12.5, x 12 20.6 / 17.9, x 14 20.4 / 20.5, x 16
// 21.1 / 21.5; 384^2 x 1 15.7 / 14.4, x 3 19.1 / 18.2, x 6 26.5 / 28.1.
// Of 1000-point columns (four of 200 threads a block, two blocks an SM): not where
// the mixed-radix pass has a block for every SM and runs in two waves at most:
// 1000^2 x 1 37.1 / 39.2, x 2 68.6 / 70.4, x 3 107.1 / 104.2, x 4 142.5 / 131.4, x 8 261 /
// 248; 384 columns 22.7 / 21.8, 1000 x 64 x 64 132 / 121.  The difference map projects
// two images an iteration (rows here too): DM 1000^2 x 1 65.8 / 68.4, x 2 135.6 /
// 130.8, x 8 487 / 451.
static bool col_here(int mode, int n, long long lines, int alg, int sms) {
  if (mode != COL_PROJECT && mode != COL_PROJECT_NOFC) return false;
  if (n == 192 || n == 384) return lines * ct::max_butterflies(n) <= 1024LL * sms;
  return n == 1000 && (lines <= 4LL * sms || (alg == ALG_DM ? 2 * lines : lines) > 16LL * sms);
}

bool ct_columns(int mode, int n, long long lines, const PassArgs &a) {
  int sms = 0;
  return device_sms(&sms) == cudaSuccess && col_here(mode, n, lines, a.alg, sms);
}

cudaError_t launch_row_ct(int mode, const LinePlan &px, const PassArgs &a, cudaStream_t st) {
  if (px.n != 192 && px.n != 384 && px.n != 1000) return cudaErrorNotSupported;
  int sms = 0;
  const cudaError_t e = device_sms(&sms);
  if (e != cudaSuccess) return e;
  // rows a block were asked for: the mixed-radix kernels take any number
  if (a.row_lpb > 0 || !row_here(mode, px.n, a.n / px.n, sms)) return cudaErrorNotSupported;
  switch (mode) {
    case ROW_DM_ITER: return ct::launch_row<ROW_DM_ITER, 1000>(px, a, st);
    case ROW_ITER: return px.n == 192 ? ct::launch_row<ROW_ITER, 192>(px, a, st) : ct::launch_row<ROW_ITER, 384>(px, a, st);
    case ROW_FWD_DEPHASE:
      return px.n == 192 ? ct::launch_row<ROW_FWD_DEPHASE, 192>(px, a, st) : ct::launch_row<ROW_FWD_DEPHASE, 384>(px, a, st);
  }
  return cudaErrorNotSupported;
}

template <int N>
static cudaError_t launch_col_n(int mode, const LinePlan &pl, const PassArgs &a, cudaStream_t st) {
  return mode == COL_PROJECT ? ct::launch_col<COL_PROJECT, N>(pl, a, st) : ct::launch_col<COL_PROJECT_NOFC, N>(pl, a, st);
}
cudaError_t launch_col_ct(int mode, const LinePlan &pl, const PassArgs &a, cudaStream_t st) {
  if (!ct_columns(mode, pl.n, (long long)a.ncols * a.nouter, a)) return cudaErrorNotSupported;
  return pl.n == 192 ? launch_col_n<192>(mode, pl, a, st)
                     : pl.n == 384 ? launch_col_n<384>(mode, pl, a, st) : launch_col_n<1000>(mode, pl, a, st);
}

}  // namespace spb
