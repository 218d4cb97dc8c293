// ROW_ITER passes of 128 and 256-point lines with g0 fetched between the
// transforms (grids of several waves).  A file of their own: compiled beside a
// blur pass they take 57 and 55 registers instead of 58 and 56 and are slower
// (HIO 128^3 39.2 instead of 38.8 us per slot, 32 x 256^2 27.9 instead of 27.7).
#include "spb_fast.cuh"

namespace spb {

template <int N>
cudaError_t row_iter_late(const LinePlan &px, const PassArgs &a, int LPB, size_t smem, cudaStream_t st) {
  return row_late_launch<N, ROW_ITER>(px, a, LPB, smem, st);
}
template cudaError_t row_iter_late<128>(const LinePlan &, const PassArgs &, int, size_t, cudaStream_t);
template cudaError_t row_iter_late<256>(const LinePlan &, const PassArgs &, int, size_t, cudaStream_t);

}  // namespace spb
