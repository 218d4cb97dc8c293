// The transform tables of a new context are on the device when it is handed
// out, ordered before the first pass of its (non-blocking) stream.  The CUDA
// calls are replaced by ones that keep account: a copy from pageable memory,
// on whatever stream, is in flight until that stream is waited for; waiting for
// a non-blocking stream says nothing about the legacy one.  Needs no GPU.
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>

#include <map>

static std::map<cudaStream_t, int> in_flight;  // copies by stream (null: the legacy stream)
static int copies;

template <class T>
static cudaError_t fake_malloc(T **p, size_t bytes) {
  *p = (T *)malloc(bytes);
  return cudaSuccess;
}
static cudaError_t fake_free(void *p) {
  free(p);
  return cudaSuccess;
}
static cudaError_t fake_copy_async(void *, const void *, size_t, cudaMemcpyKind k, cudaStream_t st) {
  if (k == cudaMemcpyHostToDevice) in_flight[st]++, copies++;
  return cudaSuccess;
}
static cudaError_t fake_copy(void *d, const void *s, size_t n, cudaMemcpyKind k) { return fake_copy_async(d, s, n, k, nullptr); }
static cudaError_t fake_memset_async(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
static cudaError_t fake_stream_create(cudaStream_t *st, unsigned) {
  *st = (cudaStream_t)malloc(1);
  return cudaSuccess;
}
static cudaError_t fake_stream_destroy(cudaStream_t st) {
  free((void *)st);
  return cudaSuccess;
}
static cudaError_t fake_stream_sync(cudaStream_t st) {
  in_flight[st] = 0;
  return cudaSuccess;
}
#define cudaMalloc fake_malloc
#define cudaFree fake_free
#define cudaMemcpy fake_copy
#define cudaMemcpyAsync fake_copy_async
#define cudaMemsetAsync fake_memset_async
#define cudaStreamCreateWithFlags fake_stream_create
#define cudaStreamDestroy fake_stream_destroy
#define cudaStreamSynchronize fake_stream_sync
#include "spb_capi.cu"

int main() {
  const int shapes[][3] = {{30, 1, 1}, {16, 21, 1}, {12, 10, 14}, {64, 64, 257}};
  int bad = 0;
  for (auto &s : shapes) {
    spb_ctx *c = nullptr;
    copies = 0;
    if (transform_ctx(&c, s[0], s[1], s[2], 0)) return 2;
    int left = 0;
    for (auto &f : in_flight) left += f.second;
    printf("%d x %d x %d: %d copies, %d in flight\n", s[0], s[1], s[2], copies, left);
    bad += left || copies < 3;
    in_flight.clear();
    spb_ctx_destroy(c);
  }
  return bad ? 1 : 0;
}
