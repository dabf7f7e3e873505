// fss_align_shape.cu -- instantiations of the fused alignment kernel for the shape mode (FP32-lane variants and tensor-core sums).
#include "fss_align_spread.cuh"

namespace fss {

int launch_align_shape(int lpp, int acc, int var, const AlignParams& prm, int fewest, int cps, size_t smem,
         cudaStream_t st) {
  if (acc == 1) return launch_align<32, FSS_MODE_SHAPE, 1, 0>(prm, fewest, cps, smem, st);
  if (acc == 2) return launch_align<32, FSS_MODE_SHAPE, 2, 0>(prm, fewest, cps, smem, st);
  switch (var) {
    case 0: return dispatch_lanes<FSS_MODE_SHAPE, 0>(lpp, prm, fewest, cps, smem, st);
    case 1: return dispatch_lanes<FSS_MODE_SHAPE, 1>(lpp, prm, fewest, cps, smem, st);
    case 2: return dispatch_lanes<FSS_MODE_SHAPE, 2>(lpp, prm, fewest, cps, smem, st);
    case 3: return dispatch_lanes<FSS_MODE_SHAPE, 3>(lpp, prm, fewest, cps, smem, st);
    case 4: return dispatch_lanes<FSS_MODE_SHAPE, 4>(lpp, prm, fewest, cps, smem, st);
    default: return set_error(FSS_ERR_INVALID, "fss_align: kernel_variant must be 0..5");
  }
}

}  // namespace fss
