// Row passes of the mixed-radix lines (spb_mixed.cuh), and the plan of a line.
#include <string.h>

#include "spb_mixed.cuh"

namespace spb {
namespace mix {

// The update of spb_pointwise.cuh's UpdateRule, every rule without a branch: flipping
// positivity and ER are selects too, and the -0 of the products is the plan's.  The
// branch for those two (spb_split.cu, the persistent kernels) is slower here: HIO
// 1000^2 x 4 134.5 instead of 132.1 us per slot, 384^3 1887 instead of 1858.
struct RowRule {
  float a, b;
  float lim_x, lim_y;  // a part below its limit becomes 0, or its absolute value (flip)
  bool er, flip, real;
  float2 z;
};
__device__ __forceinline__ RowRule row_rule(const PassArgs &p, float beta, float neg0) {
  RowRule r;
  r.er = p.alg == ALG_ER;
  r.a = p.alg == ALG_HIO ? -beta : fsub(1.0f, fmul(2.0f, beta));  // 1 - 2*beta in float, as the reference
  r.b = p.alg == ALG_HIO ? 1.0f : beta;
  const int c = p.constraints;
  const float none = -INFINITY;
  r.real = (c & (C_REAL | C_POS_REAL)) != 0;
  r.lim_x = !(c & C_REAL) && (c & (C_POS_REAL | C_POS_COMPLEX)) ? 0.0f : none;
  r.lim_y = !r.real && (c & C_POS_COMPLEX) ? 0.0f : none;
  r.flip = (c & C_FLIP) != 0;
  r.z = make_float2(neg0, neg0);
  return r;
}
__device__ __forceinline__ float2 row_point(float2 gp, float2 g0, bool inside, const RowRule &r) {
  const float2 x = __ffma2_rn(gp, make_float2(r.a, r.a), r.z), y = __ffma2_rn(g0, make_float2(r.b, r.b), r.z);
  float2 o = __fadd2_rn(x, y);
  if (r.er) o = make_float2(0.0f, 0.0f);
  float2 i = gp;
  if (i.x < r.lim_x) i.x = r.flip ? -i.x : 0.0f;
  if (i.y < r.lim_y) i.y = r.flip ? -i.y : 0.0f;
  if (r.real) i.y = 0.0f;
  return inside ? i : o;
}
// scale_cmul_dev
__device__ __forceinline__ float2 scale_point(float2 v, float s, float2 z) {
  const float2 p = __ffma2_rn(v, make_float2(s, s), z);
  const float2 q = __ffma2_rn(make_float2(v.y, v.x), make_float2(0.0f, 0.0f), z);
  return __ffma2_rn(q, make_float2(-1.0f, 1.0f), p);
}

// nl lines per block, tpl threads each: one row a line, or in the difference
// map's iteration lines 2j and 2j + 1 the rows of Y and Yf.  Shared memory: two
// buffers of nl lines of `pitch` points, then the stage tables.
template <int MODE, bool PRIME>
__global__ void __launch_bounds__(512, 2)
    row_kernel(const __grid_constant__ MixPlan mp, const __grid_constant__ PassArgs a, int nl, int tpl, int nrows) {
  constexpr bool DM = MODE == ROW_DM_ITER;
  constexpr bool UPD = MODE == ROW_ITER || DM;  // inverse, update, forward; else one transform
  constexpr bool INV = UPD || MODE == ROW_INV || MODE == ROW_INV_SCALE || MODE == ROW_INV_ABS;
  const int n = mp.n;
  const int by = 8 * nl * mp.pitch, tw = 2 * by;
  const int p = threadIdx.x / tpl;  // threads past the last line (p >= nl) only synchronise
  const Lay L{8 * p * mp.pitch, 8, p < nl ? (int)threadIdx.x - p * tpl : 1 << 30, tpl};
  const int rl = DM ? p >> 1 : p, row0 = blockIdx.x * (DM ? nl >> 1 : nl);
  const bool valid = row0 + rl < nrows;
  const long long base = (long long)row0 * n;  // the block's first point; the line's from there:
  const int pl = rl * n;
  const bool second = DM && (p & 1);
  const float2 *src = (second ? a.src2 : a.src) + base;
  float2 *dst = (second ? a.dst2 : a.dst) + base;
  const uint8_t *flags = a.flags + base;
  const float *f32 = a.f32src + base;
  float *absout = a.absout + base;
  stage_tables(mp, tw);
  pdl_wait();
  const float2 zero = make_float2(0.0f, 0.0f);
  auto load = [&](int i) -> float2 {
    i += pl;
    if (!valid) return zero;
    if constexpr (MODE == ROW_FWD_F32) return make_float2(f32[i], 0.0f);
    else if constexpr (MODE == ROW_FWD_SQUARE_F32) return make_float2(fmul(f32[i], f32[i]), 0.0f);
    else if constexpr (MODE == ROW_FWD_DEPHASE) return make_float2(cabs_ref(src[i]), 0.0f);
    else if constexpr (MODE == ROW_DM_F1_FWD) {
      const float2 v = src[i];
      return (flags[i] & FLAG_INSIDE) ? v : make_float2(fmul(-a.gamma1, v.x), fmul(-a.gamma1, v.y));
    } else return src[i];
  };
  auto store = [&](int i, float2 v) {
    i += pl;
    if (!valid) return;
    if constexpr (MODE == ROW_INV_ABS) absout[i] = cabs_ref(v);
    else dst[i] = MODE == ROW_INV_SCALE ? scale_cmul_dev(v, a.inv_n) : v;
  };
  cp_async_wait_all();
  __syncthreads();  // the tables
  int r = 0;
#pragma unroll 1
  for (int ph = INV ? 0 : 1; ph < 2; ph++) {  // ph 0: inverse, 1: forward
    const bool end = !UPD || ph == 1;
    r = line_fft<PRIME ? 2 : 0>(r, r ? 0 : by, mp, L, tw, ph ? 1.0f : -1.0f, !UPD || ph == 0, end, load, store);
    if (end) break;
    if constexpr (UPD) {
      const float beta = iter_beta(a);
      const float2 *g0 = a.g0 + base + pl;
      float2 *g1 = a.g1 + base + pl, *gp = a.gp ? a.gp + base + pl : nullptr;
      const uint8_t *fl = flags + pl;
      if constexpr (DM) {
        // the two lines' threads share their row's pixels
        const int ra = r + L.base - (second ? 8 * mp.pitch : 0), rb = ra + 8 * mp.pitch;
        for (int i = L.t + (second ? tpl : 0); i < n; i += 2 * tpl) {
          float2 x = zero, y = zero;
          if (valid) {
            const uint8_t f = fl[i];
            const float2 rho = at(ra + 8 * i);
            if (gp) gp[i] = rho;
            x = dm_point(rho, at(rb + 8 * i), g0[i], f, beta, a);
            g1[i] = x;
            y = (f & FLAG_INSIDE) ? x : make_float2(fmul(-a.gamma1, x.x), fmul(-a.gamma1, x.y));
          }
          at(ra + 8 * i) = x;
          at(rb + 8 * i) = y;
        }
      } else if (valid) {
        const RowRule rule = row_rule(a, beta, mp.neg0);
        for (int i0 = L.t; i0 < n; i0 += 4 * tpl) {
          uint8_t f[4];
          float2 g[4];
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int i = i0 + u * tpl;
            f[u] = 0;
            g[u] = zero;
            if (i < n) {
              f[u] = fl[i];
              if (!rule.er) g[u] = g0[i];
            }
          }
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int i = i0 + u * tpl, m = r + L.base + 8 * i;
            if (i < n) {
              const float2 w = scale_point(at(m), a.inv_n, rule.z);
              if (gp) gp[i] = w;
              const float2 x = row_point(w, g[u], f[u] & FLAG_INSIDE, rule);
              g1[i] = x;
              at(m) = x;
            }
          }
        }
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------- launches
template <int MODE>
static cudaError_t launch_row(const LinePlan &px, const PassArgs &a, cudaStream_t st) {
  constexpr int PER = MODE == ROW_DM_ITER ? 2 : 1;  // lines of a row
  const long long nrows = a.n / px.n;
  const MixPlan &mp = choose_plan(px, nrows * PER);
  if (nrows > 0x7fffffff / PER) return cudaErrorNotSupported;
  const int tpl = threads_per_line(mp, nrows * PER, 512 / PER);
  // about 128 threads a block, and two blocks per SM while the rows last
  long long rows = 128 / (tpl * PER);
  if (rows > nrows / (2 * num_sms())) rows = nrows / (2 * num_sms());
  if (a.row_lpb > 0) rows = a.row_lpb;
  if (rows > 512 / (tpl * PER)) rows = 512 / (tpl * PER);
  if (rows < 1) rows = 1;
  while (rows > 1 && smem_bytes(mp, (int)rows * PER) > kMixSmem) rows--;
  const int nl = (int)rows * PER;
  const size_t smem = smem_bytes(mp, nl);
  if (smem > kMixSmem) return cudaErrorNotSupported;
  const dim3 grid((unsigned)((nrows + rows - 1) / rows)), block((nl * tpl + 31) / 32 * 32);
  const cudaError_t e = mp.primes ? ensure_smem<row_kernel<MODE, true>>(smem) : ensure_smem<row_kernel<MODE, false>>(smem);
  if (e != cudaSuccess) return e;
  return launch_maybe_pdl(mp.primes ? row_kernel<MODE, true> : row_kernel<MODE, false>, grid, block, smem, st, a.pdl != 0, mp,
                          a, nl, tpl, (int)nrows);
}

}  // namespace mix

cudaError_t launch_row_mixed(int mode, const LinePlan &px, const PassArgs &a, cudaStream_t st) {
  if (!px.mix) return cudaErrorNotSupported;
  switch (mode) {
    case ROW_FWD: return mix::launch_row<ROW_FWD>(px, a, st);
    case ROW_FWD_DEPHASE: return mix::launch_row<ROW_FWD_DEPHASE>(px, a, st);
    case ROW_INV: return mix::launch_row<ROW_INV>(px, a, st);
    case ROW_INV_SCALE: return mix::launch_row<ROW_INV_SCALE>(px, a, st);
    case ROW_INV_ABS: return mix::launch_row<ROW_INV_ABS>(px, a, st);
    case ROW_ITER: return mix::launch_row<ROW_ITER>(px, a, st);
    case ROW_DM_F1_FWD: return mix::launch_row<ROW_DM_F1_FWD>(px, a, st);
    case ROW_DM_ITER: return mix::launch_row<ROW_DM_ITER>(px, a, st);
    case ROW_FWD_F32: return mix::launch_row<ROW_FWD_F32>(px, a, st);
    case ROW_FWD_SQUARE_F32: return mix::launch_row<ROW_FWD_SQUARE_F32>(px, a, st);
  }
  return cudaErrorNotSupported;
}

// The steps of a line of n points with the canonical radices r[0..ns): the
// fewest steps, consecutive stages run as one where a kernel for the pair
// exists (mix_pair_ok).  False when a prime factor's table lacks the
// symmetry the prime stages use (tw: the n forward twiddles).  The free
// elements after the first step are left out where a line would not fit.
static bool make_mix_plan_as(MixPlan &mp, int n, const int *r, int ns, const float2 *tw, bool pairs, bool pads) {
  mp = MixPlan{};
  mp.n = n;
  mp.neg0 = -0.0f;
  int best[SPB_MAX_STAGES + 1], two[SPB_MAX_STAGES + 1];
  best[ns] = 0;
  for (int s = ns - 1; s >= 0; s--) {
    best[s] = best[s + 1] + 1;
    two[s] = 0;
    if (pairs && s + 1 < ns && mix_pair_ok(r[s], r[s + 1]) && best[s + 2] + 1 < best[s]) {
      best[s] = best[s + 2] + 1;
      two[s] = 1;
    }
  }
  if (best[0] > kMixMaxSteps || best[0] < 1) return false;
  int tws = 0, pws = 0, stride = 1, pad = 0, s = 0;  // stride: ns of the stage
  mp.pitch = n;
  while (s < ns) {
    MixStep &st = mp.step[mp.nsteps];
    const int r1 = r[s], r2 = two[s] ? r[s + 1] : 1;
    st.kind = mix_single_ok(r1) ? mix_kind(r1, r2) : 0;
    st.r = r1 * r2;
    st.ns = stride;
    st.nb = n / st.r;
    st.ns_magic = stride > 1 ? (unsigned)((0x100000000ull + stride - 1) / stride) : 0u;
    st.nb_magic = st.nb > 1 ? (unsigned)((0x100000000ull + st.nb - 1) / st.nb) : 0u;
    st.tw1 = 8 * tws;
    tws += (r1 - 1) * stride;
    st.tw2 = 8 * tws;
    if (r2 > 1) tws += (r2 - 1) * stride * r1;
    // the first step's outputs: an element free after every even r
    const int dout = (pads && mp.nsteps == 0 && s + (r2 > 1 ? 2 : 1) < ns && st.r % 2 == 0) ? 1 : 0;
    st.din = pad;
    st.qout = stride * st.r + dout;
    st.sin = st.nb / stride * (stride + st.din);
    if (dout) mp.pitch = n + n / st.r;
    pad = dout;
    if (!st.kind) {
      mp.primes = true;
      st.pw = pws;
      pws += r1;
      const int step = n / r1;
      for (int e = 1; e < r1; e++) {
        const float2 w = tw[(size_t)e * step], v = tw[(size_t)(r1 - e) * step];
        if (memcmp(&w.x, &v.x, 4)) return false;
        const float m = -w.y;
        if (memcmp(&m, &v.y, 4)) return false;
      }
    }
    stride *= st.r;
    s += r2 > 1 ? 2 : 1;
    mp.nsteps++;
  }
  return mix::smem_bytes(mp, 1) <= kMixSmem;
}

bool make_mix_plan(MixPlan &mp, int n, const int *r, int ns, const float2 *tw, bool pairs) {
  return make_mix_plan_as(mp, n, r, ns, tw, pairs, true) || make_mix_plan_as(mp, n, r, ns, tw, pairs, false);
}

}  // namespace spb
