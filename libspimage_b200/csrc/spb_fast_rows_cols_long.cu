// Row passes of the power-of-two lines, and column passes of those of 512 to
// 4096 points (spb_fast.cuh).  One file on purpose: compiled in a file without a
// blur pass (COL_BLUR) the row kernels come out with other registers
// (row_fast_kernel<128, ROW_ITER, false> 70 instead of 60, <64, ...> 66 instead
// of 59) and slower: per slot with area updates every 20, HIO 32 x 512^2 105.6
// instead of 105.0 us, ER 100.5 instead of 99.8, HIO 128^2 10.46 instead of 10.32.
// Only the passes of spb_fast_rows_late.cu are faster so.
#include "spb_fast.cuh"

namespace spb {

// Returns cudaErrorNotSupported when no register kernel exists for the line
// length or mode; the caller then uses the mixed-radix kernels.
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
