// Instantiations of the potential-block apply for double blocks.
#include "bsl_vapply.cuh"

namespace bsl {

int launch_vapply_f64(const double* vb, cudaStream_t s, int nn, const double* v, const double* uk,
                     const double* rot, double* out, long long N, int mode, double* partials, unsigned int* counter,
                     double* scalars, double* hist, int j, long long dpk) {
  const unsigned g = (unsigned)((N + kVapplyThreads - 1) / kVapplyThreads);
  // Up to 26,000 points there are fewer than 1.35 warps of points per FP64 pipe
  // (4 per SM), so rows are split over warps: 14 against 32 us at 15^3 and 33
  // against 39 us at 27^3, 51 against 48 us at 33^3 (odd l <= 5).
  if (N <= 26000) {
    const unsigned gr = (unsigned)((N + 31) / 32);
#define BSL_ROWS(K, G)                                                                                          \
  if (nn == K) {                                                                                                \
    k_vapply_rows<K, G><<<gr, 32 * G, 0, s>>>(vb, v, uk, rot, out, N, mode, partials, counter, scalars, hist, j, \
                                              dpk);                                                             \
    BSL_CUDA(cudaGetLastError());                                                                               \
    return BSL_OK;                                                                                              \
  }
    BSL_ROWS(9, 3)
    BSL_ROWS(10, 5)
    BSL_ROWS(15, 5)
    BSL_ROWS(16, 4)
    BSL_ROWS(21, 7)
    BSL_ROWS(25, 5)
    BSL_ROWS(28, 7)
    BSL_ROWS(36, 6)
#undef BSL_ROWS
  }
#define BSL_CASE(K)                                                                                            \
  case K:                                                                                                      \
    k_vapply<K, double><<<g, kVapplyThreads, 0, s>>>(vb, v, uk, rot, out, N, mode, partials, counter, scalars, \
                                                     hist, j, dpk);                                            \
    break;
  switch (nn) {
    BSL_CASE(1)
    BSL_CASE(3)
    BSL_CASE(4)
    BSL_CASE(6)
    BSL_CASE(9)
    BSL_CASE(10)
    BSL_CASE(15)
    BSL_CASE(16)
    BSL_CASE(21)
    BSL_CASE(25)
    BSL_CASE(28)
    BSL_CASE(36)
    default:
      k_vapply_generic<<<(unsigned)grid_for(N), kThreads, 0, s>>>(vb, v, uk, rot, out, N, nn, mode, partials, counter, scalars, hist, j,
                                              dpk);
  }
#undef BSL_CASE
  BSL_CUDA(cudaGetLastError());
  return BSL_OK;
}

}  // namespace bsl
