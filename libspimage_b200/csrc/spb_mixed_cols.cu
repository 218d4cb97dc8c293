// Column passes of the mixed-radix lines (spb_mixed.cuh).
#include "spb_mixed.cuh"

namespace spb {
namespace mix {

// nl neighbouring columns per block (a power of two, lg its logarithm).
// Shared memory: two buffers of nl lines of `pitch` points, point i of column p
// at (i nl + p), then the stage tables.
template <int MODE, bool PRIME>
__global__ void __launch_bounds__(512, 2)
    col_kernel(const __grid_constant__ MixPlan mp, const __grid_constant__ PassArgs a, int nl, int lg) {
  constexpr bool PROJ = MODE == COL_PROJECT || MODE == COL_PROJECT_NOFC || MODE == COL_PROJECT_PAIR;
  constexpr bool MID = PROJ || MODE == COL_BLUR;  // forward, pointwise, inverse; else one transform
  constexpr bool FWD = MID || MODE == COL_FWD;
  const int n = mp.n;
  const int by = 8 * nl * mp.pitch, tw = 2 * by;
  const long long o = a.outer0 + blockIdx.y;
  const int p = threadIdx.x & (nl - 1);  // blockDim.x is a multiple of nl
  const int c0 = blockIdx.x * nl, c = c0 + p;
  const Lay L{8 * p, 8 * nl, (int)threadIdx.x >> lg, (int)blockDim.x >> lg};
  const long long base = o * a.ostride + c0;  // the block's first point
  const int es = (int)a.estride;              // a start has fewer than 2^31 points
  const bool valid = c < a.ncols;
  const bool second = MODE == COL_PROJECT_PAIR && blockIdx.z;  // the second image
  const float2 *src = (second ? a.src2 : a.src) + base;
  const float *f32 = a.f32src + base;
  float2 *dst = (second ? a.dst2 : a.dst) + base;
  stage_tables(mp, tw);
  pdl_wait();
  const float2 zero = make_float2(0.0f, 0.0f);
  auto load = [&](int i) -> float2 {
    const int k = i * es + p;
    if (!valid) return zero;
    if constexpr (MODE == COL_INV_SQUARE_F32) return make_float2(fmul(f32[k], f32[k]), 0.0f);
    else return src[k];
  };
  auto store = [&](int i, float2 v) {
    if (valid) dst[i * es + p] = v;
  };
  cp_async_wait_all();
  __syncthreads();  // the tables
  int r = 0;
#pragma unroll 1
  for (int ph = FWD ? 0 : 1; ph < 2; ph++) {  // ph 0: forward, 1: inverse
    const bool end = !MID || ph == 1;
    r = line_fft<PRIME ? 2 : MID>(r, r ? 0 : by, mp, L, tw, ph ? -1.0f : 1.0f, !MID || ph == 0, end, load, store);
    if (end) break;
    if constexpr (PROJ) {
      const long long ai0 = base % a.n_start;  // the amplitude side holds one start
      const uint8_t *fl = a.flags + base;
      const float *am = a.amp + ai0;
      const bool amp_ok = a.objective == 0 && !(a.constraints & C_MARGIN) && a.amp_bad && !*a.amp_bad;
      if (valid)
        for (int i0 = L.t; i0 < n; i0 += 4 * L.tpl) {
          uint8_t f[4];
          float amp[4];
          long long ai[4];
          float2 G[4];
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int i = i0 + u * L.tpl, k = i * es + p;
            f[u] = i < n ? fl[k] : (uint8_t)0;
            amp[u] = i < n && a.amp ? am[k] : 0.0f;
            ai[u] = ai0 + k;
          }
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int i = i0 + u * L.tpl;
            G[u] = i < n ? at(r + L.base + i * L.es) : zero;
            if (MODE == COL_PROJECT_PAIR && !second && (a.constraints & C_CENTROSYM)) G[u].y = 0.0f;
          }
          project_many<4, MODE == COL_PROJECT>(G, f, amp, ai, amp_ok, a);
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int i = i0 + u * L.tpl;
            if (i < n) at(r + L.base + i * L.es) = G[u];
          }
        }
    } else if constexpr (MODE == COL_BLUR) {
      const bool zl = a.line_axis == 2;  // lines along z: column c is pixel (c % nx, c / nx)
      const int x = zl ? c % a.nx : c, y = zl ? c / a.nx : 0, z = (int)(o % a.nz);
      if (valid)
#pragma unroll 4
        for (int i = L.t; i < n; i += L.tpl) {
          float2 &v = at(r + L.base + i * L.es);
          v = zl ? blur_point(v, x, y, i, a) : blur_point(v, x, i, z, a);
        }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- launches
template <int MODE>
static cudaError_t launch_col(const LinePlan &pl, const PassArgs &a, cudaStream_t st) {
  // four columns a block (a 32-byte sector of every row); eight when that
  // still gives two blocks per SM
  constexpr int IMAGES = MODE == COL_PROJECT_PAIR ? 2 : 1;
  const long long lines = (long long)a.ncols * a.nouter * IMAGES;
  const MixPlan &mp = choose_plan(pl, lines);
  int nl = lines / 8 >= 2 * num_sms() ? 8 : 4;
  if ((MODE == COL_PROJECT || MODE == COL_PROJECT_NOFC || MODE == COL_PROJECT_PAIR) && a.col_width > 0) nl = a.col_width;
  while (nl > 1 && smem_bytes(mp, nl) > kMixSmem) nl >>= 1;
  const size_t smem = smem_bytes(mp, nl);
  if (smem > kMixSmem) return cudaErrorNotSupported;
  int lg = 0;
  while ((1 << lg) < nl) lg++;
  const cudaError_t e = mp.primes ? ensure_smem<col_kernel<MODE, true>>(smem) : ensure_smem<col_kernel<MODE, false>>(smem);
  if (e != cudaSuccess) return e;
  int threads = (nl * threads_per_line(mp, lines, 512 / nl) + 31) / 32 * 32;
  if (threads > 512) threads = 512;
  const dim3 grid((a.ncols + nl - 1) / nl, a.nouter, IMAGES);
  return launch_maybe_pdl(mp.primes ? col_kernel<MODE, true> : col_kernel<MODE, false>, grid, dim3(threads), smem, st,
                          a.pdl != 0, mp, a, nl, lg);
}

}  // namespace mix

cudaError_t launch_col_mixed(int mode, const LinePlan &pl, const PassArgs &a, cudaStream_t st) {
  if (!pl.mix) return cudaErrorNotSupported;
  switch (mode) {
    case COL_FWD: return mix::launch_col<COL_FWD>(pl, a, st);
    case COL_INV: return mix::launch_col<COL_INV>(pl, a, st);
    case COL_PROJECT: return mix::launch_col<COL_PROJECT>(pl, a, st);
    case COL_PROJECT_NOFC: return mix::launch_col<COL_PROJECT_NOFC>(pl, a, st);
    case COL_PROJECT_PAIR: return mix::launch_col<COL_PROJECT_PAIR>(pl, a, st);
    case COL_BLUR: return mix::launch_col<COL_BLUR>(pl, a, st);
    case COL_INV_SQUARE_F32: return mix::launch_col<COL_INV_SQUARE_F32>(pl, a, st);
  }
  return cudaErrorNotSupported;
}

}  // namespace spb
