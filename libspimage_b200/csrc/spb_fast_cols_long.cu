// Column passes of the power-of-two lines of 512 to 4096 points (spb_fast.cuh).
#include "spb_fast.cuh"

namespace spb {

cudaError_t launch_col_fast_long(int mode, const LinePlan &pl, const PassArgs &a, cudaStream_t st) {
  switch (pl.n) {
    case 512: return col_fast_mode<512>(mode, pl, a, st);
    case 1024: return col_fast_mode<1024>(mode, pl, a, st);
    case 2048: return col_fast_mode<2048>(mode, pl, a, st);
    case 4096: return col_fast_mode<4096>(mode, pl, a, st);
  }
  return cudaErrorNotSupported;
}

}  // namespace spb
