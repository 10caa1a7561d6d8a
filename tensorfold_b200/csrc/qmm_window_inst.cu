// Instantiates qmm_window_kernel for one bit width (TF_BITS) over every group size and row tile.
#include "qmm_window_launch.h"

#ifndef TF_BITS
#error "compile with -DTF_BITS=<2|3|4|5|6>"
#endif

namespace tf {

namespace {

template <int GS, int ROWS>
cudaError_t launch(const CUtensorMap& tmx, const WindowParams& p, int grid, cudaStream_t stream, bool pdl) {
  using Geo = WindowGeo<TF_BITS, GS, ROWS>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(Geo::THREADS);
  cfg.dynamicSmemBytes = Geo::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, qmm_window_kernel<TF_BITS, GS, ROWS>, tmx, p);
}

template <int GS, int ROWS>
cudaError_t configure() {
  using Geo = WindowGeo<TF_BITS, GS, ROWS>;
  // The roles' shares (setmaxnreg) add up to 96 registers a thread.  A kernel compiled to fewer would wait for ever for its
  // epilogue warps' share, so it must not be launched.
  cudaFuncAttributes compiled;
  cudaError_t e = cudaFuncGetAttributes(&compiled, qmm_window_kernel<TF_BITS, GS, ROWS>);
  if (e == cudaSuccess && compiled.numRegs < 96) e = cudaErrorLaunchOutOfResources;
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(qmm_window_kernel<TF_BITS, GS, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Geo::SMEM);
}

}  // namespace

#define TF_CAT2(a, b) a##b
#define TF_CAT(a, b) TF_CAT2(a, b)
#define TF_WINDOW_SHAPES(X) X(32, 32) X(32, 48) X(32, 64) X(64, 32) X(64, 48) X(64, 64) X(128, 32) X(128, 48) X(128, 64)

cudaError_t TF_CAT(qmm_window_launch_b, TF_BITS)(const CUtensorMap& tmx, const WindowParams& p, int gs, int rows, int grid,
                                                 cudaStream_t stream, bool pdl) {
#define TF_CASE(GS, ROWS) \
  if (gs == GS && rows == ROWS) return launch<GS, ROWS>(tmx, p, grid, stream, pdl);
  TF_WINDOW_SHAPES(TF_CASE)
#undef TF_CASE
  return cudaErrorInvalidValue;
}

cudaError_t TF_CAT(qmm_window_configure_b, TF_BITS)() {
  cudaError_t e = cudaSuccess;
#define TF_CASE(GS, ROWS) \
  if (e == cudaSuccess) e = configure<GS, ROWS>();
  TF_WINDOW_SHAPES(TF_CASE)
#undef TF_CASE
  return e;
}

}  // namespace tf
