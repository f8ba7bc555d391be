// The FP32 column slice pass (kernels_col.cuh).
#include "kernels_col.cuh"

namespace msf {

cudaError_t launch_col32(bool last, const PassArgs& a, const CUtensorMap& map, int* err,
                         cudaStream_t s) {
  switch (a.nx) {
#define MSF_CASE(N)                                                              \
  case N:                                                                        \
    return a.slots ? col_launch<Pair, N, false, true>(a, map, err, s)            \
           : last  ? col_launch<Pair, N, true, false>(a, map, err, s)            \
                   : col_launch<Pair, N, false, false>(a, map, err, s);
    MSF_COL_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
  return cudaErrorInvalidValue;
}

}  // namespace msf
