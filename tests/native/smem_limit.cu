// Two host threads raise one kernel's dynamic shared memory limit to different
// sizes at the same time.  The runtime's attribute call is replaced by one that
// keeps the limit it was given and makes the calls overlap: the smaller
// request takes effect after the larger one, and the larger one returns last.
// Needs no GPU.
#include <cuda_runtime.h>
#include <stdio.h>

#include <atomic>
#include <chrono>
#include <thread>

static std::atomic<int> limit{0};
static const int kSmall = 60 << 10, kLarge = 100 << 10;

static void nap(int ms) { std::this_thread::sleep_for(std::chrono::milliseconds(ms)); }

template <class F>
static cudaError_t set_attribute(F *, cudaFuncAttribute, int v) {
  if (v == kSmall) nap(150);
  limit = v;
  if (v == kLarge) nap(300);
  return cudaSuccess;
}
#define cudaFuncSetAttribute set_attribute
#include "spb_passes.cuh"

__global__ void kernel() {}

int main() {
  std::thread a([] { spb::ensure_smem<kernel>(kSmall); }), b([] { spb::ensure_smem<kernel>(kLarge); });
  a.join();
  b.join();
  if (spb::ensure_smem<kernel>(kLarge) != cudaSuccess) return 2;
  printf("limit %d, launch asks for %d\n", (int)limit, kLarge);
  return limit >= kLarge ? 0 : 1;
}
