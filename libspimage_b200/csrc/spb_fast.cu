// Persistent and plane forms of the power-of-two lines, the self-check of the
// branch-free roundings, and the choice between the column passes' sources
// (spb_fast.cuh holds the transforms and the pass kernels).
#include "spb_fast.cuh"

namespace spb {

// ------------------------------------------------ persistent small patterns
// One block per start of an N x N pattern (N = 32, 64, 128) runs every
// iteration of a call with the start's spectrum resident in shared memory:
// X (the row transform of the model) stays in the block between iterations,
// and each iteration is the column pass (forward y, projection, inverse y)
// and the row pass (inverse x, update, forward x) of the two-pass kernels,
// separated by block barriers instead of kernel boundaries.  The previous
// iterate, the flags and the amplitude lines are read from global memory
// (L2); the new iterate is written there.  Same transforms and pointwise
// steps, so the bits are those of the two-pass kernels.
//
// Shared memory: [twiddles N][N rows of pitch P = N + N/16].  Element (row i,
// column x) of X sits at i*P + x; a row's exchanges use the padded positions
// of its own P slots, a column's exchanges use its own elements (stride P).
namespace reg {
// The twiddles of a stage on a thread's points in packed products; k = 0 takes
// none.  They run under a branch (a select costs two instructions a point in
// packed form), where T is a multiple of NS one for the J butterflies of a
// thread, which then share k and the table's loads, elsewhere only for a
// butterfly whose T j is a multiple of NS.
template <int N, int R, int NS, bool INV>
__device__ __forceinline__ void twiddle_points(float2 (&v)[16], int t, const float2 *stw) {
  constexpr int T = N / 16, J = 16 / R;
  if constexpr (NS > 1 && T % NS == 0) {
    const int k = t & (NS - 1);
    if (k) {
#pragma unroll
      for (int m = 1; m < R; m++) {
        const float2 w = stw[(m - 1) * NS + k];  // shared-memory stage table
#pragma unroll
        for (int j = 0; j < J; j++) v[j + m * J] = packed::cmulw(v[j + m * J], w.x, INV ? -w.y : w.y);
      }
    }
  } else if constexpr (NS > 1) {
#pragma unroll
    for (int j = 0; j < J; j++) {
      const int k = (t + T * j) & (NS - 1);
      if ((T * j) % NS != 0 || k) {
#pragma unroll
        for (int m = 1; m < R; m++) {
          const float2 w = stw[(m - 1) * NS + k];
          v[j + m * J] = packed::cmulw(v[j + m * J], w.x, INV ? -w.y : w.y);
        }
      }
    }
  }
}

template <int N, int S, int NS, bool INV, int STRIDE>
struct PStages {
  // storage address of line index i: padded within a row (STRIDE 0) or down a column
  static __device__ __forceinline__ int at(int i) { return STRIDE == 0 ? pad(i) : i * STRIDE; }
  static __device__ __forceinline__ void run(float2 (&v)[16], float2 *line, int t, const float2 *stw) {
    constexpr int R = plan_radix(N, S);
    constexpr int T = N / 16;
    constexpr int J = 16 / R;
    constexpr bool LAST = (S == plan_len(N) - 1);
    twiddle_points<N, R, NS, INV>(v, t, stw);
#pragma unroll
    for (int j = 0; j < J; j++) {
      float2 a[R];
#pragma unroll
      for (int m = 0; m < R; m++) a[m] = v[j + m * J];
      const int b = t + T * j;
      const int k = b & (NS - 1);
      if constexpr (R == 16) packed::bf16<INV>(a);
      else if constexpr (R == 8) packed::bf8<INV>(a);
      else if constexpr (R == 4) packed::bf4<INV>(a[0], a[1], a[2], a[3]);
      else bfly<R, INV>(a);
      if constexpr (LAST) {
#pragma unroll
        for (int m = 0; m < R; m++) v[j + m * J] = a[m];
      } else {
        const int base = (b / NS) * NS * R + k;
#pragma unroll
        for (int m = 0; m < R; m++) line[at(base + m * NS)] = a[m];
      }
    }
    if constexpr (!LAST) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 16; q++) v[q] = line[at(t + T * q)];
      __syncthreads();
      PStages<N, S + 1, NS * R, INV, STRIDE>::run(v, line, t, stw + (R - 1) * NS);
    }
  }
};
}  // namespace reg

// blocks per SM the register budget is sized for (64 registers a thread)
template <int N>
__host__ __device__ constexpr int persist_min_blocks() {
  return N >= 128 ? 1 : (N == 64 ? 4 : 16);
}

template <int N>
__global__ void __launch_bounds__(N * N / 16, persist_min_blocks<N>())
    persist_kernel(PassArgs a, const float2 *__restrict__ stw, float2 *gbuf0, float2 *gbuf1, int cur0, int iters,
                   int keep_gp) {
  constexpr int T = N / 16;
  constexpr int P = N + N / 16;
  constexpr int W = proj_words(N);
  extern __shared__ __align__(16) float2 sm[];
  float2 *tw_s = sm;
  float2 *Xs = sm + N;
  const size_t off = (size_t)blockIdx.x * N * N;
  const uint8_t *flags = a.flags + off;
  float2 *Xg = a.dst + off;
  stage_twiddles<N>(tw_s, stw);
  for (int i = threadIdx.x; i < N * N; i += blockDim.x) Xs[(i / N) * P + (i % N)] = Xg[i];
  cp_async_wait_all();
  __syncthreads();
  int cur = cur0;
  for (int it = 0; it < iters; it++) {
    cur ^= 1;
    const float2 *g0 = (cur ? gbuf0 : gbuf1) + off;  // the previous model
    float2 *g1 = (cur ? gbuf1 : gbuf0) + off;        // the new one
    const float beta = a.alg == ALG_ER ? 0.0f : (a.beta_tab ? a.beta_tab[*a.beta_base + it] : a.beta);
    const UpdateRule rule = update_rule(a, beta);
    {  // column pass: column c, thread t of its T
      const int c = threadIdx.x % N, t = threadIdx.x / N;
      float2 v[16];
#pragma unroll
      for (int q = 0; q < 16; q++) v[q] = Xs[(t + T * q) * P + c];
      __syncthreads();  // every column read before its elements serve as exchange space
      reg::PStages<N, 0, 1, false, P>::run(v, Xs + c, t, tw_s);
      project16<T, true>(v, a.amp_line + (size_t)c * N, a.meas_bits + (size_t)c * W, t, (size_t)t * N + c,
                         (size_t)T * N, a);
      reg::PStages<N, 0, 1, true, P>::run(v, Xs + c, t, tw_s);
#pragma unroll
      for (int q = 0; q < 16; q++) Xs[(t + T * q) * P + c] = v[q];
      __syncthreads();
    }
    {  // row pass: row r, thread t of its T
      const int r = threadIdx.x / T, t = threadIdx.x % T;
      float2 v[16];
#pragma unroll
      for (int q = 0; q < 16; q++) v[q] = Xs[r * P + t + T * q];
      __syncthreads();  // every row read before its slots serve as exchange space
      reg::PStages<N, 0, 1, true, 0>::run(v, Xs + r * P, t, tw_s);
      const bool last = keep_gp && it == iters - 1;
      const int idx = r * N + t;
      update_points(v, g0 + idx, flags + idx, last ? a.gp + off + idx : nullptr, g1 + idx, rule, a,
                    [](int q) { return T * q; });
      reg::PStages<N, 0, 1, false, 0>::run(v, Xs + r * P, t, tw_s);
#pragma unroll
      for (int q = 0; q < 16; q++) Xs[r * P + t + T * q] = v[q];
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < N * N; i += blockDim.x) Xg[i] = Xs[(i / N) * P + (i % N)];
}

template <int N>
static cudaError_t persist_launch(const LinePlan &px, const PassArgs &a, float2 *g0, float2 *g1, int cur0, int iters,
                                  int keep_gp, int nb, cudaStream_t st) {
  const size_t smem = (size_t)(N + N * (N + N / 16)) * sizeof(float2);
  cudaError_t e = ensure_smem<persist_kernel<N>>(smem);
  if (e != cudaSuccess) return e;
  persist_kernel<N><<<nb, N * N / 16, smem, st>>>(a, px.stw, g0, g1, cur0, iters, keep_gp);
  return cudaGetLastError();
}

cudaError_t launch_persist(const LinePlan &px, const PassArgs &a, float2 *g0, float2 *g1, int cur0, int iters,
                           int keep_gp, int nb, cudaStream_t st) {
  if (!px.stw || a.meas_words != proj_words(px.n)) return cudaErrorNotSupported;
  switch (px.n) {
    case 32: return persist_launch<32>(px, a, g0, g1, cur0, iters, keep_gp, nb, st);
    case 64: return persist_launch<64>(px, a, g0, g1, cur0, iters, keep_gp, nb, st);
    case 128: return persist_launch<128>(px, a, g0, g1, cur0, iters, keep_gp, nb, st);
  }
  return cudaErrorNotSupported;
}

// ------------------------------------------------- 3-D plane pass (ny = nz)
// The y and z passes of a 3-D iteration in one launch: one block per x-plane
// of a start holds the plane's N x N points (rows along y, one per z) in
// shared memory and runs the forward y transforms (rows), then per column
// (one per y) the forward z transform, the projection and the inverse z
// transform, then the inverse y transforms (rows).  That is the work of the
// forward y, z projection and inverse y column passes, with one read and one
// write of the volume instead of three of each.  Same transforms, projection
// and order, so the bits are those of the three passes.
//
// Shared memory: [twiddles N][N rows of pitch P = N + N/16] as in the
// persistent form: point (z, y) of the plane at z*P + y; a row's exchanges
// use the padded positions of its own P slots, a column's use its own
// elements (stride P).  Plane loads and stores are 8-byte accesses at stride
// nx points; the neighbouring planes' blocks run at the same time and share
// the sectors in L2.
template <int N, int MODE>
__global__ void __launch_bounds__(N * N / 16, 1) plane_kernel(PassArgs a, const float2 *__restrict__ stw) {
  constexpr int T = N / 16;
  constexpr int P = N + N / 16;
  constexpr int W = proj_words(N);
  extern __shared__ __align__(16) float2 sm[];
  float2 *tw_s = sm;
  float2 *Ps = sm + N;
  const int x = blockIdx.x;
  const long long b = a.outer0 + blockIdx.y;
  const long long nxy = (long long)a.nx * N;  // points per z-slice (ny = N)
  const long long off = b * a.n_start + x;     // point (z, y) of the plane at off + z*nxy + y*nx
  stage_twiddles<N>(tw_s, stw);
  pdl_wait();
  {  // forward y: row r (z = r), thread t of its T, straight from global memory
    const int r = threadIdx.x / T, t = threadIdx.x % T;
    const float2 *src = a.src + off + (long long)r * nxy + (long long)t * a.nx;
    float2 v[16];
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = src[(long long)(T * q) * a.nx];
    cp_async_wait_all();
    __syncthreads();  // twiddles in
    reg::PStages<N, 0, 1, false, 0>::run(v, Ps + r * P, t, tw_s);
#pragma unroll
    for (int q = 0; q < 16; q++) Ps[r * P + t + T * q] = v[q];
    __syncthreads();
  }
  {  // column c (y = c), thread t of its T: forward z, projection, inverse z
    const int c = threadIdx.x % N, t = threadIdx.x / N;
    float2 v[16];
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = Ps[(t + T * q) * P + c];
    __syncthreads();  // every column read before its elements serve as exchange space
    reg::PStages<N, 0, 1, false, P>::run(v, Ps + c, t, tw_s);
    const long long line = (long long)c * a.nx + x;  // z-line index y*nx + x
    project16<T, MODE == COL_PROJECT>(v, a.amp_line + line * N, a.meas_bits + line * W, t,
                                      (size_t)(off + (long long)c * a.nx + (long long)t * nxy), (size_t)T * nxy, a);
    reg::PStages<N, 0, 1, true, P>::run(v, Ps + c, t, tw_s);
#pragma unroll
    for (int q = 0; q < 16; q++) Ps[(t + T * q) * P + c] = v[q];
    __syncthreads();
  }
  {  // inverse y: row r, thread t
    const int r = threadIdx.x / T, t = threadIdx.x % T;
    float2 v[16];
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = Ps[r * P + t + T * q];
    __syncthreads();  // every row read before its slots serve as exchange space
    reg::PStages<N, 0, 1, true, 0>::run(v, Ps + r * P, t, tw_s);
    pdl_release();
    float2 *dst = a.dst + off + (long long)r * nxy + (long long)t * a.nx;
#pragma unroll
    for (int q = 0; q < 16; q++) dst[(long long)(T * q) * a.nx] = v[q];
  }
}

template <int N, int MODE>
static cudaError_t plane_launch_n(const LinePlan &pl, const PassArgs &a, cudaStream_t st) {
  const size_t smem = (size_t)(N + N * (N + N / 16)) * sizeof(float2);
  cudaError_t e = ensure_smem<plane_kernel<N, MODE>>(smem);
  if (e != cudaSuccess) return e;
  return launch_maybe_pdl(plane_kernel<N, MODE>, dim3(a.nx, a.nouter), dim3(N * N / 16), smem, st, a.pdl != 0, a,
                          pl.stw);
}

// Whether the plane pass serves this projection: a 3-D volume with ny = nz =
// 64 or 128, a projection mode, the line-major amplitudes and measured bits.
bool plane_fits(int mode, const LinePlan &pl, const PassArgs &a) {
  if (mode != COL_PROJECT && mode != COL_PROJECT_NOFC) return false;
  if (a.nz == 1 || pl.n != a.ny || a.ny != a.nz || (pl.n != 64 && pl.n != 128)) return false;
  return pl.stw && a.amp_line && a.meas_bits && a.meas_words == proj_words(pl.n);
}

// The plane pass (cudaErrorNotSupported where plane_fits says no); a.nouter
// starts from a.outer0 (at most 65535 per launch).
cudaError_t launch_plane(int mode, const LinePlan &pl, const PassArgs &a, cudaStream_t st) {
  if (!plane_fits(mode, pl, a)) return cudaErrorNotSupported;
  switch (pl.n) {
    case 64:
      return mode == COL_PROJECT ? plane_launch_n<64, COL_PROJECT>(pl, a, st) : plane_launch_n<64, COL_PROJECT_NOFC>(pl, a, st);
    case 128:
      return mode == COL_PROJECT ? plane_launch_n<128, COL_PROJECT>(pl, a, st)
                                 : plane_launch_n<128, COL_PROJECT_NOFC>(pl, a, st);
  }
  return cudaErrorNotSupported;
}

// ------------------------------------------- self-check of the roundings
// Bit-for-bit comparisons of the branch-free forms with the IEEE intrinsics,
// counting differences: every float x with bit pattern in [lo, hi) inside the
// square-root domain (square root) and inside [2^-63, 2^63] (reciprocal);
// n pseudo-random quotients a/b with a and b drawn over their domains; and the
// quotients of significand pairs a in [1, 2) (every a_stride-th significand)
// and b in [1, 2) (every significand; for divisor significand mb the
// dividend's run over (mb * 2654435761 + seed) mod a_stride + k * a_stride, so
// the calls with seed = 0 .. a_stride-1 cover every pair once).
__global__ void check_sqrt_rcp_kernel(unsigned lo, unsigned hi, unsigned long long *bad) {
  unsigned long long nsq = 0, nrc = 0;
  for (unsigned long long u = lo + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; u < hi;
       u += (unsigned long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float((unsigned)u);
    if (sqrt_rn_nb_domain(x)) nsq += __float_as_uint(sqrt_rn_nb(x)) != __float_as_uint(__fsqrt_rn(x));
    if (x >= 0x1p-63f && x <= 0x1p63f) nrc += __float_as_uint(rcp_rn_nb(x)) != __float_as_uint(__frcp_rn(x));
  }
  if (nsq) atomicAdd(bad, nsq);
  if (nrc) atomicAdd(bad + 1, nrc);
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;  // splitmix64 finaliser
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void check_div_kernel(unsigned long long n, unsigned long long seed, unsigned long long *bad) {
  unsigned long long nbad = 0;
  for (unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long r = mix64(seed ^ mix64(k));
    // a: random sign and significand, exponent in [-60, 60) (one in 64 draws: zero)
    const unsigned ea = 67u + (unsigned)((r >> 24) % 120u);
    const float a = ((r >> 58) == 0) ? 0.0f : __uint_as_float(((unsigned)r & 0x807FFFFFu) | (ea << 23));
    // b: exponent in [-63, 63), random significand
    const unsigned eb = 64u + (unsigned)((r >> 32) % 126u);
    const float b = __uint_as_float((eb << 23) | ((unsigned)(r >> 40) & 0x7FFFFFu));
    nbad += __float_as_uint(div_rn_nb(a, b)) != __float_as_uint(__fdiv_rn(a, b));
  }
  if (nbad) atomicAdd(bad, nbad);
}

__global__ void check_div_significands_kernel(unsigned a_stride, unsigned phase, unsigned long long *bad) {
  unsigned long long nbad = 0;
  for (unsigned mb = blockIdx.x * blockDim.x + threadIdx.x; mb < (1u << 23); mb += gridDim.x * blockDim.x) {
    const float b = __uint_as_float(0x3F800000u | mb);
    for (unsigned ma = (mb * 2654435761u + phase) % a_stride; ma < (1u << 23); ma += a_stride) {
      const float a = __uint_as_float(0x3F800000u | ma);
      nbad += __float_as_uint(div_rn_nb(a, b)) != __float_as_uint(__fdiv_rn(a, b));
    }
  }
  if (nbad) atomicAdd(bad, nbad);
}

cudaError_t check_roundings(unsigned lo, unsigned hi, unsigned long long ndiv, unsigned long long seed,
                            unsigned a_stride, unsigned long long *d_bad) {
  if (hi > lo) check_sqrt_rcp_kernel<<<148 * 8, 256>>>(lo, hi, d_bad);
  if (ndiv) check_div_kernel<<<148 * 8, 256>>>(ndiv, seed, d_bad + 2);
  if (a_stride) check_div_significands_kernel<<<148 * 8, 256>>>(a_stride, (unsigned)(seed % a_stride), d_bad + 3);
  return cudaGetLastError();
}

// Columns per block the projection pass offers besides the built-in width:
// lines of 256, 512 and 1024 points, C a power of two with C*N/16 <= 256
// threads and C <= 16 (the shared-memory skew is 16/C words); and the
// lengths 192, 384 and 1000 (general_col_width_ok).
bool col_width_ok(int n, int w) {
  if (w < 1 || w > 16 || (w & (w - 1))) return false;
  if (n != 256 && n != 512 && n != 1024) return general_col_width_ok(n, w);
  return w * (n / 16) <= 256;
}

cudaError_t launch_col_fast_short(int mode, const LinePlan &pl, const PassArgs &a, cudaStream_t st);
cudaError_t launch_col_fast_long(int mode, const LinePlan &pl, const PassArgs &a, cudaStream_t st);

cudaError_t launch_col_fast(int mode, const LinePlan &pl, const PassArgs &a, cudaStream_t st) {
  if (!pl.stw) return cudaErrorNotSupported;
  return pl.n <= 256 ? launch_col_fast_short(mode, pl, a, st) : launch_col_fast_long(mode, pl, a, st);
}

}  // namespace spb
