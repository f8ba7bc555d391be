// The FP64 column slice pass (kernels_col.cuh) and what both precisions share on
// the host: the dispatch, tile widths, twiddle tables and tensor maps.
#include "kernels_col.cuh"

#include <cudaTypedefs.h>

namespace msf {

cudaError_t launch_col32(bool last, const PassArgs& a, const CUtensorMap& map, int* err,
                         cudaStream_t s);  // kernels_col32.cu

cudaError_t launch_col_slice(bool fp64, bool last, const PassArgs& a, const void* tensor_map,
                             int* err, cudaStream_t s) {
  const CUtensorMap& map = *static_cast<const CUtensorMap*>(tensor_map);
  if (!fp64) return launch_col32(last, a, map, err, s);
  if (a.slots) return cudaErrorInvalidValue;  // slot lanes run FP32
  switch (a.nx) {
#define MSF_CASE(N)                                                     \
  case N:                                                               \
    return last ? col_launch<double2, N, true, false>(a, map, err, s)   \
                : col_launch<double2, N, false, false>(a, map, err, s);
    MSF_COL_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
  return cudaErrorInvalidValue;
}

int col_tile(int nx, bool fp64) {
  switch (nx) {
#define MSF_CASE(N) case N: return fp64 ? tile_cols<double2, N>() : tile_cols<Pair, N>();
    MSF_COL_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
  return 0;
}

void fill_col_twiddles(int n, std::vector<float>& out) {
  out.clear();
  switch (n) {
#define MSF_CASE(N) case N: line_twiddles<ColShape<N>>(out); break;
    MSF_COL_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
}
void fill_col_twiddles(int n, std::vector<double>& out) {
  out.clear();
  switch (n) {
#define MSF_CASE(N) case N: line_twiddles<ColShape<N>>(out); break;
    MSF_COL_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
}

// Tensor map over a batch of planes [nb*nx rows][ny columns] of 8-byte words
// (one a complex value in FP32, two in FP64): box {tile columns, min(256, nx)}
// rows, no multicast.  Up to
// 512 points swizzled over the 128-byte tile row, so that eight consecutive
// rows of an element column lie in eight different 16-byte bank groups; the wide
// tiles are read a whole row at a time and need no swizzle.
cudaError_t encode_col_map(bool fp64, void* psi, int nb, int nx, int ny, void* map_out) {
  // looked up once per process (a thread-safe static: lanes of the request
  // loop encode maps from their worker thread)
  static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
    cudaDriverEntryPointQueryResult q;
    void* fn = nullptr;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    return (e == cudaSuccess && q == cudaDriverEntryPointSuccess)
               ? reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn)
               : nullptr;
  }();
  if (!encode) return cudaErrorNotSupported;
  const int cols = col_tile(nx, fp64), words = fp64 ? 2 : 1;
  if (!cols) return cudaErrorInvalidValue;
  cuuint64_t dims[2] = {(cuuint64_t)ny * words, (cuuint64_t)nx * (cuuint64_t)nb};
  cuuint64_t strides[1] = {(cuuint64_t)ny * 8 * words};
  cuuint32_t box[2] = {(cuuint32_t)(cols * words), (cuuint32_t)(nx < 256 ? nx : 256)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode(static_cast<CUtensorMap*>(map_out), CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, psi,
                      dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      nx < 1024 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace msf
