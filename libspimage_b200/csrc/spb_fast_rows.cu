// Row passes of the power-of-two lines (spb_fast.cuh).
#include "spb_fast.cuh"

namespace spb {

// Returns cudaErrorNotSupported when no register kernel exists for the line
// length or mode; the caller then uses the general kernels.
cudaError_t launch_row_fast(int mode, const LinePlan &px, const PassArgs &a, cudaStream_t st) {
  if (!px.stw) return cudaErrorNotSupported;
  switch (px.n) {
    case 16: return row_fast_mode<16>(mode, px, a, st);
    case 32: return row_fast_mode<32>(mode, px, a, st);
    case 64: return row_fast_mode<64>(mode, px, a, st);
    case 128: return row_fast_mode<128>(mode, px, a, st);
    case 256: return row_fast_mode<256>(mode, px, a, st);
    case 512: return row_fast_mode<512>(mode, px, a, st);
    case 1024: return row_fast_mode<1024>(mode, px, a, st);
    case 2048: return row_fast_mode<2048>(mode, px, a, st);
    case 4096: return row_fast_mode<4096>(mode, px, a, st);
  }
  return cudaErrorNotSupported;
}

}  // namespace spb
