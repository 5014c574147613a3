// toed_qad.cu -- the MATLAB "quick and dirty" orientation mode
// (third_order_edge_detector.m:91-141 with QaD_flag set): the edgel kernel
// with the subpixel orientation.
//
// In this mode the emitted orientation is the third-order direction
// atan2(Fx, -Fy) (:127-141) built from the nine derivatives interpolated
// with MATLAB's interp2 'cubic' -- cubic convolution, Keys a = -1/2, the
// kernel the reference also restates as cubic_kernel
// (subpix_to_correction.cpp:57-67) -- at the edgel's subpixel point, instead
// of the direction at its 2x-grid point (cpu_toed.cpp:227-232).  The
// derivatives are the C++ detector's own (2x grid, zero padding,
// cpu_toed.cpp:204-344); positions and strengths are unchanged.
#include "toed_edgels.cuh"

namespace toed {

cudaError_t prepare_qad(int radius) { return prepare_edgels_as<true>(radius); }
cudaError_t launch_qad(const BatchParams& p, cudaStream_t stream) { return launch_edgels_as<true>(p, stream); }

}  // namespace toed
