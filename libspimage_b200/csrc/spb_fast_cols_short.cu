// Column passes of the power-of-two lines of 16 to 256 points (spb_fast.cuh).
#include "spb_fast.cuh"

namespace spb {

cudaError_t launch_col_fast_short(int mode, const LinePlan &pl, const PassArgs &a, cudaStream_t st) {
  switch (pl.n) {
    case 16: return col_fast_mode<16>(mode, pl, a, st);
    case 32: return col_fast_mode<32>(mode, pl, a, st);
    case 64: return col_fast_mode<64>(mode, pl, a, st);
    case 128: return col_fast_mode<128>(mode, pl, a, st);
    case 256: return col_fast_mode<256>(mode, pl, a, st);
  }
  return cudaErrorNotSupported;
}

}  // namespace spb
