// The derivation kernels of the frame-code build for simple tables
// (PGA_SIMPLE_PARAMS: scalars, block values and the custom attribute): engines
// with such a table, no Rotate and a single phase launch these (pga::simple).
// Their adjoint is that of derive.cu or derive_blk.cu, whose tape is the same.
#define PGA_SIMPLE_PARAMS 1
#define PGA_INLINE_BLOCKS 1
#include "derive_kernels.cuh"

namespace pga {
FrameKernels simple_frame_kernels() { return frame_kernels(); }
}  // namespace pga
