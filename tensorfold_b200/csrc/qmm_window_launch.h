// Host-side launch interface of qmm_window_kernel; one translation unit per bit width (qmm_window_inst.cu with
// -DTF_BITS=b).  8-bit codes, whose two nibble planes need a second operand 16 x, stay with the tiled kernel.
#pragma once

#include <cuda_runtime.h>

#include "qmm_window.cuh"

namespace tf {

// Rows a tile's registers and buffers hold: 32, 48 or 64.
inline int window_rows(int tile_rows) { return tile_rows <= 32 ? 32 : tile_rows <= 48 ? 48 : 64; }

#define TF_DECLARE_BITS(B)                                                                                              \
  cudaError_t qmm_window_launch_b##B(const CUtensorMap& tmx, const WindowParams& p, int gs, int rows, int grid, cudaStream_t stream, bool pdl); \
  cudaError_t qmm_window_configure_b##B();
TF_DECLARE_BITS(2)
TF_DECLARE_BITS(3)
TF_DECLARE_BITS(4)
TF_DECLARE_BITS(5)
TF_DECLARE_BITS(6)
#undef TF_DECLARE_BITS

}  // namespace tf
