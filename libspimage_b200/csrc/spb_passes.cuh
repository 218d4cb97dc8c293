// Helpers shared by the register-resident pass kernels (spb_fast.cuh: 16
// points per thread; spb_split.cu: 8 points per thread): asynchronous copies,
// programmatic dependent launch, stage twiddles in shared memory, the
// Fourier projection with its operands at hand, the layout of the
// line-major projection operands in shared memory, and the launch helpers.
#pragma once
#include <math.h>

#include <atomic>
#include <mutex>

#include "spb_internal.h"
#include "spb_pointwise.cuh"

namespace spb {

// ------------------------------------------------------ async copy helpers
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Programmatic dependent launch.  What a pass kernel does before this point
// reads only data written two or more kernels earlier in the stream (twiddles,
// the previous iterate, flags, line-major operands) and writes only shared
// memory; the predecessor's output is read after the wait.  The successor may
// start its own prologue once this kernel's predecessor has completed, which
// keeps that two-kernel distance for every prologue; the release comes just
// before the final stores, so that the successor's blocks do not take SM
// residency from this kernel's.  Without the launch attribute both
// instructions return at once.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
// called before the final stores: the successor launches during this kernel's tail
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

template <typename K, typename... Args>
inline cudaError_t launch_maybe_pdl(K k, dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool pdl,
                                    Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

// stage-twiddle table of an N-point line into shared memory (N-1 entries)
template <int N>
__device__ __forceinline__ void stage_twiddles(float2 *tw_s, const float2 *__restrict__ stw) {
  for (int i = threadIdx.x; i < N - 1; i += blockDim.x) cp_async8(tw_s + i, stw + i);
}

// Fourier projection with the amplitude and measured bit already at hand
__device__ __forceinline__ float2 project_with(float2 G, float amp, bool measured, long long idx, const PassArgs &a,
                                               bool fourier_constraints) {
  if (fourier_constraints && (a.constraints & C_CENTROSYM)) G.y = 0.0f;
  if (!measured) return G;
  if (a.objective != 0) return a.phased_amp[idx % a.n_start];
  float m = 1.0f;
  if (!(a.constraints & C_MARGIN)) {
    m = __fdiv_rn(amp, cabs_ref(G));
  } else {
    const float av = cabs_ref(G);
    const float lo = a.amp_min[idx % a.n_start], hi = a.amp_max[idx % a.n_start];
    if (av < lo) m = __fdiv_rn(lo, av);
    else if (av > hi) m = __fdiv_rn(hi, av);
  }
  if (isfinite(m)) return make_float2(fmul(G.x, m), fmul(G.y, m));
  return make_float2(amp, 0.0f);
}

// The update of a thread's U points after the inverse transform: v becomes the
// new model, gp (when set) and g1 take the model before projection and the
// new model.  Point q lies off(q) behind g0, fl, gp and g1.
template <int U, class Off>
__device__ __forceinline__ void update_points(float2 (&v)[U], const float2 *g0, const uint8_t *fl, float2 *gp, float2 *g1,
                                              const UpdateRule &r, const PassArgs &a, Off off) {
#pragma unroll
  for (int q = 0; q < U; q++) v[q] = packed::cmulw(v[q], a.inv_n, 0.0f);  // scale_cmul_dev
  if (gp)
#pragma unroll
    for (int q = 0; q < U; q++) gp[off(q)] = v[q];
  if (r.rare) {
#pragma unroll
    for (int q = 0; q < U; q++) v[q] = update_point_any(v[q], g0[off(q)], fl[off(q)], r, a);
  } else {
#pragma unroll
    for (int q = 0; q < U; q++) v[q] = update_point(v[q], g0[off(q)], fl[off(q)], r);
  }
#pragma unroll
  for (int q = 0; q < U; q++) g1[off(q)] = v[q];
}

// words per line of the measured-bit bitmap (a multiple of 4 words)
__host__ __device__ constexpr int proj_words(int n) { return ((n + 127) / 128) * 4; }
template <int N, int C>
__host__ __device__ constexpr int amp_stride() {
  return N + (C == 1 ? 0 : (C <= 8 ? 32 / C : 4));
}
template <int N, int C>
__host__ __device__ constexpr int bits_stride() {
  return C == 1 ? proj_words(N) : proj_words(N) + ((((C <= 8 ? 32 / C : 4) - proj_words(N) % 32) + 32) % 32);
}

// multiprocessors of the device
inline cudaError_t device_sms(int *n) {
  static int nsm = 0;
  cudaError_t e = cudaSuccess;
  if (!nsm) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, 0);
  *n = nsm;
  return e;
}

// Dynamic shared memory limit of kernel K raised to at least smem.  One kernel
// serves many line lengths, so host threads with contexts of different sizes
// ask for different limits: the comparison, the call and the record are one
// step under a lock, and the limit only grows (a launch that fits the recorded
// limit takes no lock).
template <auto K>
static cudaError_t ensure_smem(size_t smem) {
  static std::atomic<size_t> have{0};
  static std::mutex lock;
  if (smem <= have.load(std::memory_order_acquire)) return cudaSuccess;
  std::lock_guard<std::mutex> hold(lock);
  if (smem <= have.load(std::memory_order_relaxed)) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) have.store(smem, std::memory_order_release);
  return e;
}

}  // namespace spb
