// Transforms of the pass kernels for every line length without a register kernel of its own
// (spb_fast.cuh, spb_split.cu): 2^a 3^b 5^c lengths that are not powers of
// two, and lengths with larger prime factors.
//
// Same transform as spb_fft.cuh, operation for operation: the canonical radix
// plan, its butterflies and twiddle floats, explicitly rounded arithmetic.
// The organisation is for sm_100a:
//  * (re, im) pairs are computed in packed f32x2 instructions, whose operands
//    may be swapped, repeated or negated for free: a complex add is one
//    instruction, a twiddle product three, x + i y one.  A packed product is
//    formed as fma(a, b, -0): the sum of an exact product with -0 rounds once,
//    to the product's own bits (signed zeros included), and unlike a packed
//    multiply it is not contracted with the add that follows (the -0 is a
//    kernel argument, which the compiler cannot fold).
//  * Short consecutive stages are run as one (3 x 3, 3 x 5, 4 x 3, ...): the
//    butterflies of the second stage whose inputs a thread has just computed
//    stay in its registers, with the second stage's own twiddles, so the
//    roundings do not change and one exchange through shared memory is saved.
//  * A prime factor R >= 7 costs R^2 products per butterfly in the recipe.
//    Its inputs are multiplied by their twiddles once (not once per output),
//    and outputs m and R - m of a butterfly are computed together by one
//    thread: W^(q(R-m)) is the conjugate of W^(qm) to the bit (checked when the
//    plan is made), so the four products of a term serve both.
//  * One body serves both directions: the direction enters as a sign
//    multiplied in by fma(v, +-1, t), which rounds like the add or subtract it
//    replaces, so the code the SM fetches is half of two bodies'.
// The first step reads its inputs from device memory and the last one writes
// there; in between, lines go through two shared-memory buffers.  After the
// first step, whose outputs are R apart, an element is left free after every
// even R so that the stores do not meet in one bank.
//
// Bounds and figures (one B200).  Grids of one wave are bound by the latency of
// the steps (load, butterfly, store, barrier), larger ones by instruction
// issue (55-59 % issue active at 192^3 before the pointwise loops were made
// branch-free).  Per iteration slot, the run-time stage loops these kernels
// replaced / these kernels: HIO 600^2 38 / 22 us, 768^2 51 / 28.5, 1200^2 95 / 54.5,
// 100^3 83 / 48.5, 192^3 384 / 187, 384^3 3270 / 1858, 1000^2 39.0 / 37.3 (a
// compile-time plan before), RAAR 650x670 (2.5.5.13 x 2.5.67) 1816 / 57,
// 257x263 49000 / 80.  Two lines a thread (shared index arithmetic and
// twiddle loads, 128 registers) was slower everywhere: 1000^2 39.6 against
// 36.0, 8 x 384^2 57.5 against 44.9.
#pragma once
#include <math.h>

#include "spb_internal.h"
#include "spb_passes.cuh"
#include "spb_pointwise.cuh"

namespace spb {
namespace mix {

// What a butterfly multiplies by: d = +1 forward, -1 backward; w = (d, -d),
// so that x + W4 y = fma(swapped y, w, x); z = (-0, -0)
struct Dir {
  float2 w, z;
};
__device__ __forceinline__ Dir make_dir(float d, float z) { return Dir{make_float2(d, -d), make_float2(z, z)}; }

__device__ __forceinline__ float2 swp(float2 a) { return make_float2(a.y, a.x); }
__device__ __forceinline__ float2 neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 mul(float2 a, float b, const Dir &g) { return __ffma2_rn(a, make_float2(b, b), g.z); }
// cmulw by w, or by its conjugate backward: d (im * w.im) rounds to d times the rounded product
__device__ __forceinline__ float2 mulw(float2 a, float wr, float wi, const Dir &g) {
  return __ffma2_rn(mul(swp(a), wi, g), neg(g.w), mul(a, wr, g));
}
// t + W4 v and t - W4 v (W4 = -i forward, +i backward)
__device__ __forceinline__ float2 add_w4(float2 t, float2 v, const Dir &g) { return __ffma2_rn(swp(v), g.w, t); }
__device__ __forceinline__ float2 sub_w4(float2 t, float2 v, const Dir &g) { return __ffma2_rn(swp(v), neg(g.w), t); }
__device__ __forceinline__ float2 mul_w4(float2 a, const Dir &g) { return __ffma2_rn(swp(a), g.w, g.z); }
__device__ __forceinline__ float2 mul_w8_1(float2 a, const Dir &g) { return mul(add_w4(a, a, g), SPB_C8, g); }
__device__ __forceinline__ float2 mul_w8_3(float2 a, const Dir &g) {
  const float2 v = add_w4(a, a, g);
  return __ffma2_rn(swp(v), make_float2(SPB_C8 * g.w.x, SPB_C8 * g.w.y), g.z);
}

__device__ __forceinline__ void bf4(float2 &a0, float2 &a1, float2 &a2, float2 &a3, const Dir &g) {
  const float2 t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), d = csub(a1, a3);
  a0 = cadd(t0, t2);
  a1 = add_w4(t1, d, g);
  a2 = csub(t0, t2);
  a3 = sub_w4(t1, d, g);
}

// DFT of R points held at a[0], a[ST], a[2 ST], ... (in place)
template <int R, int ST>
__device__ __forceinline__ void bfly(float2 *a, const Dir &g) {
  if constexpr (R == 2) {
    const float2 t = a[0];
    a[0] = cadd(t, a[ST]);
    a[ST] = csub(t, a[ST]);
  } else if constexpr (R == 3) {
    const float2 t1 = cadd(a[ST], a[2 * ST]), d = csub(a[ST], a[2 * ST]);
    const float2 m = csub(a[0], mul(t1, 0.5f, g)), e = mul(d, SPB_S3, g);
    a[0] = cadd(a[0], t1);
    a[ST] = add_w4(m, e, g);
    a[2 * ST] = sub_w4(m, e, g);
  } else if constexpr (R == 4) {
    bf4(a[0], a[ST], a[2 * ST], a[3 * ST], g);
  } else if constexpr (R == 5) {
    const float2 b1 = cadd(a[ST], a[4 * ST]), b2 = cadd(a[2 * ST], a[3 * ST]);
    const float2 d1 = csub(a[ST], a[4 * ST]), d2 = csub(a[2 * ST], a[3 * ST]);
    const float2 x = a[0];
    const float2 m1 = cadd(cadd(x, mul(b1, SPB_C51, g)), mul(b2, SPB_C52, g));
    const float2 m2 = cadd(cadd(x, mul(b1, SPB_C52, g)), mul(b2, SPB_C51, g));
    const float2 n1 = cadd(mul(d1, SPB_S51, g), mul(d2, SPB_S52, g));
    const float2 n2 = csub(mul(d1, SPB_S52, g), mul(d2, SPB_S51, g));
    a[0] = cadd(cadd(x, b1), b2);
    a[ST] = add_w4(m1, n1, g);
    a[4 * ST] = sub_w4(m1, n1, g);
    a[2 * ST] = add_w4(m2, n2, g);
    a[3 * ST] = sub_w4(m2, n2, g);
  } else if constexpr (R == 8) {
    bf4(a[0], a[2 * ST], a[4 * ST], a[6 * ST], g);
    bf4(a[ST], a[3 * ST], a[5 * ST], a[7 * ST], g);
    const float2 o1 = mul_w8_1(a[3 * ST], g), o3 = mul_w8_3(a[7 * ST], g);
    const float2 e0 = a[0], e1 = a[2 * ST], e2 = a[4 * ST], e3 = a[6 * ST], o0 = a[ST], d2 = a[5 * ST];
    a[0] = cadd(e0, o0);
    a[4 * ST] = csub(e0, o0);
    a[ST] = cadd(e1, o1);
    a[5 * ST] = csub(e1, o1);
    a[2 * ST] = add_w4(e2, d2, g);
    a[6 * ST] = sub_w4(e2, d2, g);
    a[3 * ST] = cadd(e3, o3);
    a[7 * ST] = csub(e3, o3);
  } else if constexpr (R == 16) {
    static_assert(ST == 1, "radix 16 runs alone");
#pragma unroll
    for (int q = 0; q < 4; q++) bf4(a[q], a[q + 4], a[q + 8], a[q + 12], g);
    a[5] = mulw(a[5], SPB_C16, -SPB_S16, g);
    a[9] = mul_w8_1(a[9], g);
    a[13] = mulw(a[13], SPB_S16, -SPB_C16, g);
    a[6] = mul_w8_1(a[6], g);
    a[10] = mul_w4(a[10], g);
    a[14] = mul_w8_3(a[14], g);
    a[7] = mulw(a[7], SPB_S16, -SPB_C16, g);
    a[11] = mul_w8_3(a[11], g);
    a[15] = mulw(a[15], -SPB_C16, SPB_S16, g);
    // output k1 + 4 k2 of the second layer's row k1 lands at 4 k1 + k2: transpose
#pragma unroll
    for (int k = 0; k < 4; k++) bf4(a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3], g);
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++)
#pragma unroll
      for (int k2 = k1 + 1; k2 < 4; k2++) {
        const float2 t = a[4 * k1 + k2];
        a[4 * k1 + k2] = a[4 * k2 + k1];
        a[4 * k2 + k1] = t;
      }
  }
}

extern __shared__ float4 mix_smem[];
// the point (or table entry) at byte offset i of shared memory
__device__ __forceinline__ float2 &at(int i) {
  return *reinterpret_cast<float2 *>(reinterpret_cast<unsigned char *>(mix_smem) + i);
}

// How a block's lines lie in a buffer and are shared out.  Rows: line p at p *
// pitch points, points side by side; it has threads [p * tpl, (p + 1) * tpl).
// Columns: lines side by side (nl a power of two), points 8 nl bytes apart;
// the threads are dealt to the lines in turn.
struct Lay {
  int base, es;  // byte offset of the thread's line, bytes between its points
  int t, tpl;    // the thread's first task of its line, the distance to its next
};

// One stage R1, or two consecutive stages R1, R2 in one step (R2 > 1), of the
// thread's line, from the buffer at x to the buffer at y (byte offsets).  b
// runs over the nb = n / (R1 R2) composite butterflies; q = b / ns, k = b %
// ns.  Input j = m R2 + m2 of a butterfly is point b + j nb; the first stage's
// butterflies run over m for each m2, the second's over m2 for each output m0
// of the first, at k + m0 ns of its twiddles.
// load(i), when set (first), gives point i of the line from device memory;
// store(i, v), when set (last), takes the transform's point i.
template <int R1, int R2, class Load, class Store>
__device__ __forceinline__ void stage(int x, int y, const Lay &L, int tw, const MixStep &s, const Dir &g, bool first,
                                      bool last, Load load, Store store) {
  constexpr int R = R1 * R2;
  const int ns = s.ns, nb = s.nb, sin = s.sin * L.es, sout = ns * L.es, tws = 8 * ns;
  x += L.base;
  y += L.base;
  for (int b = L.t; b < nb; b += L.tpl) {
    const int q = ns == 1 ? b : (int)__umulhi((unsigned)b, s.ns_magic);
    const int k = b - q * ns;
    float2 a[R];
    if (first) {
#pragma unroll
      for (int j = 0; j < R; j++) a[j] = load(b + j * nb);
    } else {
      const int in = x + (b + q * s.din) * L.es;
#pragma unroll
      for (int j = 0; j < R; j++) a[j] = at(in + j * sin);
    }
    if (k) {
      const int t1 = tw + s.tw1 + 8 * k;
#pragma unroll
      for (int m = 1; m < R1; m++) {
        const float2 w = at(t1 + (m - 1) * tws);
#pragma unroll
        for (int m2 = 0; m2 < R2; m2++) a[m * R2 + m2] = mulw(a[m * R2 + m2], w.x, w.y, g);
      }
    }
#pragma unroll
    for (int m2 = 0; m2 < R2; m2++) bfly<R1, R2>(a + m2, g);
    if constexpr (R2 > 1) {
      const int t2 = tw + s.tw2 + 8 * k;
#pragma unroll
      for (int m0 = 0; m0 < R1; m0++) {
        if (m0 > 0 || k) {
#pragma unroll
          for (int m2 = 1; m2 < R2; m2++) {
            const float2 w = at(t2 + ((m2 - 1) * R1 + m0) * tws);
            a[m0 * R2 + m2] = mulw(a[m0 * R2 + m2], w.x, w.y, g);
          }
        }
        bfly<R2, 1>(a + m0 * R2, g);
      }
    }
    if (last) {  // one group of outputs: q = 0, ns = nb, output o is point b + o nb
#pragma unroll
      for (int m0 = 0; m0 < R1; m0++)
#pragma unroll
        for (int m2 = 0; m2 < R2; m2++) store(b + (m0 + R1 * m2) * nb, a[m0 * R2 + m2]);
    } else {
      const int out = y + (q * s.qout + k) * L.es;
#pragma unroll
      for (int m0 = 0; m0 < R1; m0++)
#pragma unroll
        for (int m2 = 0; m2 < R2; m2++) at(out + (m0 + R1 * m2) * sout) = a[m0 * R2 + m2];
    }
  }
}

// The outputs of a prime stage from its twiddled inputs: y_m = a_0 + sum_q a_q
// W_R^(mq mod R), added left to right.  A task is output m and output R - m
// (m = 0: the plain sum) of JB butterflies, b and b + (nb + 1) / 2: the index
// mq mod R, the table's entry and the loop are shared by them (670-point rows:
// 1826 -> 1378 instructions a point, 48.8 -> 39.9 us a pass at 650 rows).
// Neighbouring threads take neighbouring butterflies, so a warp reads the
// table at few places.
template <int JB, class Store>
__device__ __forceinline__ void prime_outputs(int x, int y, const Lay &L, const float2 *__restrict__ wr,
                                              const MixStep &s, const Dir &g, bool last, Store store) {
  const int R = s.r, ns = s.ns, nb = s.nb, sin = s.sin * L.es;
  const int groups = (nb + JB - 1) / JB, half = (R + 1) / 2;
  const unsigned group_magic = 0xffffffffu / groups + 1;  // quotients by groups > 1 as a high product
  for (int t = L.t; t < groups * half; t += L.tpl) {
    const int m = groups == 1 ? t : (int)__umulhi((unsigned)t, group_magic);
    const int b0 = t - m * groups;
    int in[JB], out[JB];
    float2 u[JB], v[JB];
    bool ok[JB];
#pragma unroll
    for (int j = 0; j < JB; j++) {
      ok[j] = b0 + j * groups < nb;
      const int b = ok[j] ? b0 + j * groups : b0;
      const int q0 = ns == 1 ? b : (int)__umulhi((unsigned)b, s.ns_magic);
      in[j] = x + (b + q0 * s.din) * L.es;
      out[j] = b + q0 * ns * (R - 1);  // point of output 0
      u[j] = v[j] = at(in[j]);
    }
    if (m == 0) {
#pragma unroll 4
      for (int q = 1; q < R; q++)
#pragma unroll
        for (int j = 0; j < JB; j++) u[j] = cadd(u[j], at(in[j] += sin));
    } else {
      const unsigned step = 8 * m, wrap = 8 * R;
      unsigned e = 0;  // byte offset of W_R^(mq mod R)
#pragma unroll 4
      for (int q = 1; q < R; q++) {
        e += step;
        e = min(e, e - wrap);  // unsigned: e - wrap is huge while e < wrap
        const float2 w = __ldg(reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(wr) + e));
#pragma unroll
        for (int j = 0; j < JB; j++) {
          const float2 aq = at(in[j] += sin);
          // the products of a term serve both outputs: a w = p + (-i, i) h, a conj(w) = p - (-i, i) h
          const float2 p = mul(aq, w.x, g), h = mul(swp(aq), w.y, g);
          u[j] = cadd(u[j], __ffma2_rn(h, neg(g.w), p));
          v[j] = cadd(v[j], __ffma2_rn(h, g.w, p));
        }
      }
    }
#pragma unroll
    for (int j = 0; j < JB; j++) {
      if (!ok[j]) continue;
      const int ou = out[j] + m * ns, ov = out[j] + (R - m) * ns;
      if (last) {
        store(ou, u[j]);
        if (m) store(ov, v[j]);
      } else {
        at(y + ou * L.es) = u[j];
        if (m) at(y + ov * L.es) = v[j];
      }
    }
  }
}

// A prime stage R >= 7: its inputs take their twiddles in place, once, then
// its outputs are formed.
template <int PRIMES, class Load, class Store>
__device__ __forceinline__ void stage_prime(int x, int y, const Lay &L, int tw, const float2 *__restrict__ wr,
                                            const MixStep &s, const Dir &g, bool first, bool last, Load load,
                                            Store store) {
  const int R = s.r, ns = s.ns, nb = s.nb, sin = s.sin * L.es;
  x += L.base;
  y += L.base;
  if (first) {  // every input is read by many threads: into shared memory first
#pragma unroll 4
    for (int i = L.t; i < nb * R; i += L.tpl) at(x + i * L.es) = load(i);
    __syncthreads();
  }
  if (ns > 1) {
    for (int t = L.t; t < nb * (R - 1); t += L.tpl) {  // input m + 1 of butterfly b
      const int m = nb == 1 ? t : (int)__umulhi((unsigned)t, s.nb_magic);
      const int b = t - m * nb;
      const int q = (int)__umulhi((unsigned)b, s.ns_magic);
      const int k = b - q * ns;
      const int in = x + (b + q * s.din) * L.es + (m + 1) * sin;
      if (k) {
        const float2 w = at(tw + s.tw1 + (m * ns + k) * 8);
        at(in) = mulw(at(in), w.x, w.y, g);
      }
    }
    __syncthreads();
  }
  if constexpr (PRIMES == 2) {
    if (nb > 1) prime_outputs<2>(x, y, L, wr, s, g, last, store);
    else prime_outputs<1>(x, y, L, wr, s, g, last, store);
  } else {  // one butterfly a task, a plainer loop (line_fft)
    const int half = (R + 1) / 2;
    for (int t = L.t; t < nb * half; t += L.tpl) {
      const int m = nb == 1 ? t : (int)__umulhi((unsigned)t, s.nb_magic);
      const int b = t - m * nb;
      const int q0 = ns == 1 ? b : (int)__umulhi((unsigned)b, s.ns_magic);
      int in = x + (b + q0 * s.din) * L.es;
      const int out = b + q0 * ns * (R - 1);  // point of output 0
      const float2 a0 = at(in);
      float2 u = a0, v = a0;
      if (m == 0) {
#pragma unroll 4
        for (int q = 1; q < R; q++) u = cadd(u, at(in += sin));
      } else {
        int e = 0;
#pragma unroll 4
        for (int q = 1; q < R; q++) {
          e += m;
          e = e >= R ? e - R : e;
          const float2 w = __ldg(wr + e), aq = at(in += sin);
          const float2 p = mul(aq, w.x, g), h = mul(swp(aq), w.y, g);
          u = cadd(u, __ffma2_rn(h, neg(g.w), p));
          v = cadd(v, __ffma2_rn(h, g.w, p));
        }
      }
      const int ou = out + m * ns, ov = out + (R - m) * ns;
      if (last) {
        store(ou, u);
        if (m) store(ov, v);
      } else {
        at(y + ou * L.es) = u;
        if (m) at(y + ov * L.es) = v;
      }
    }
  }
}

// Every stage of the block's lines, from the buffer at x (or, with from_mem,
// from load()) to a buffer, or with to_mem to store(); returns the buffer (x
// or y) of the result.  All threads call it; it synchronises after every step
// that ends in shared memory.  tw: where the stage tables start.  PRIMES: 2
// for plans with prime steps; the kernels of plans without any leave them out
// (0), except for the columns' forward and inverse passes (1): no plan of theirs
// reaches the plain loop either, but without it the compiler allocates their 64
// registers worse (24 + 48 bytes of spill stores and loads in the projection,
// 12 + 16 with it).  Projection and blur without / with, us a pass at 192^3: 76.0 /
// 71.5 and 57.6 / 53.6; in the passes of one transform it costs (192^3, one
// direction 39.5 / 40.2, |blur| rows 31.1 / 32.5).
template <int PRIMES, class Load, class Store>
__device__ __forceinline__ int line_fft(int x, int y, const MixPlan &mp, const Lay &L, int tw, float d, bool from_mem,
                                         bool to_mem, Load load, Store store) {
  const Dir g = make_dir(d, mp.neg0);
#pragma unroll 1
  for (int i = 0; i < mp.nsteps; i++) {
    const MixStep &s = mp.step[i];
    const bool first = from_mem && i == 0, last = to_mem && i == mp.nsteps - 1;
    if (last) pdl_release();
#define SPB_MIX_STEP(r1, r2) \
  case mix_kind(r1, r2): stage<r1, r2>(x, y, L, tw, s, g, first, last, load, store); break;
    switch (s.kind) {
      SPB_MIX_KINDS(SPB_MIX_STEP)
      default:
        if constexpr (PRIMES != 0) stage_prime<PRIMES>(x, y, L, tw, mp.pw + s.pw, s, g, first, last, load, store);
        break;
    }
#undef SPB_MIX_STEP
    if (!last) __syncthreads();
    const int t = x;
    x = y;
    y = t;
  }
  return x;
}

__device__ __forceinline__ void stage_tables(const MixPlan &mp, int tw) {
  for (int i = threadIdx.x; i < mp.n - 1; i += blockDim.x)
    cp_async8(reinterpret_cast<unsigned char *>(mix_smem) + tw + 8 * i, mp.stw + i);
}

// ---------------------------------------------------------------- launches
inline int num_sms() {
  static int nsm = 0;
  if (!nsm && cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, 0) != cudaSuccess) nsm = 148;
  return nsm;
}

// shared memory of nl lines
inline size_t smem_bytes(const MixPlan &mp, int nl) {
  return (size_t)2 * nl * mp.pitch * sizeof(float2) + (size_t)mp.n * sizeof(float2);
}

// tasks of a line in a step, and in its widest step
inline int tasks_of(const MixStep &st) {
  return st.kind ? st.nb : (st.nb > 1 ? (st.nb + 1) / 2 : 1) * ((st.r + 1) / 2);
}
inline int most_tasks(const MixPlan &mp) {
  int t = 1;
  for (int i = 0; i < mp.nsteps; i++) t = tasks_of(mp.step[i]) > t ? tasks_of(mp.step[i]) : t;
  return t;
}

// Threads per line (at most `most`): a task of the widest step each, or one
// of every `rounds` tasks, whichever lets `lines` lines finish first by this
// model: a step takes 8 + rounds * (6 + R) units, an SM holds 1024 threads (64
// registers each) and kMixSmem bytes of lines, and lines beyond what the SMs
// hold at once wait.  Few lines are fastest with a thread per task, many with
// more lines in flight.  Measured at 1 / 2 / 4 rounds (us per HIO slot):
// 1000^2 37.4 / 40.4 / 45.6, 16 x 1000^2 565 / 530 / 589, 1200^2 58.3 / 54.6 /
// 67.4, 8 x 384^2 41.2 / 38.0 / 35.3, 192^3 188 / 236 / 322, 100^3 49.4 / 48.0 /
// 54.8; the model picks 1, 2, 2, 2, 1, 2.
inline int threads_per_line(const MixPlan &mp, long long lines, int most) {
  const int tasks = most_tasks(mp);
  int best = 0;
  double best_cost = 0.0;
  for (int rounds = 1; rounds <= 8; rounds++) {
    int t = (tasks + rounds - 1) / rounds;
    if (t > most) t = most;
    double time = 0.0;
    for (int i = 0; i < mp.nsteps; i++) {
      const MixStep &st = mp.step[i];
      time += 8.0 + (tasks_of(st) + t - 1) / t * (6.0 + st.r);
    }
    const double by_threads = 1024.0 / t, by_smem = (double)kMixSmem / (16.0 * mp.pitch);
    const double waves = (double)lines / (num_sms() * (by_threads < by_smem ? by_threads : by_smem));
    const double cost = time * (waves > 1.0 ? waves : 1.0);
    if (!best || cost < best_cost) {
      best = t;
      best_cost = cost;
    }
    if (t == 1) break;
  }
  return best;
}

// Stages run as one save an exchange but leave fewer, longer tasks: not where
// their tasks do not give the SMs two warps each (120^2 13.8 -> 12.0 us per slot,
// 240^2 17.5 -> 13.9).
inline const MixPlan &choose_plan(const LinePlan &pl, long long lines) {
  return pl.mix[lines * most_tasks(pl.mix[0]) < 64LL * num_sms() ? 1 : 0];
}

}  // namespace mix
}  // namespace spb
