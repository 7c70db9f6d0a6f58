// Potential-block apply kernels (templated on the block size), shared by the
// FP32 and FP64 instantiation units.
#pragma once

#include "bsl_device.cuh"

namespace bsl {
namespace {

// ---------------------------------------------------------------------------
// potential apply + rotor + (optionally) the first Lanczos step
//   mode 0: u = T v + rot v + V v          (u = out)
//   mode 1: r += T v + rot v + V v; partial alpha = v . r   (r = out, in place)
// ---------------------------------------------------------------------------
// The FP64 apply is bound by the FP64 pipe (nn^2 + 4 nn operations a point at
// 2 lanes a clock and SM: 131 us at 54^3 and 21 functions).  Blocks of 128 points
// at 4 per SM, so that an SM holds warps in different phases and no last wave of
// large blocks idles: 187 us there against 229 us with blocks of 256 points (4.05
// waves of one block per SM), 86 against 98 us at 41^3.
constexpr int kVapplyThreads = 128;
template <int NN, typename VT>
__global__ void __launch_bounds__(kVapplyThreads, NN <= 21 ? 4 : 1) k_vapply(const VT* __restrict__ vb, const double* __restrict__ vec,
                                                     const double* __restrict__ ukin, const double* __restrict__ rot,
                                                     double* __restrict__ out, long long npts, int mode,
                                                     double* partials, unsigned int* counter, double* scalars,
                                                     double* hist, int j, long long dpk) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  // logical Lanczos vectors are v = sv vec and r = sr out; r + H v is kept as
  // sr (out + (sv/sr) H vec): out' = out + c H vec, alpha = sv sr (vec . out')
  const double c = mode ? scalars[6] : 1.0;
  double dot = 0.0;
  if (p < npts) {
    double v[NN], acc[NN];
    VT vv[NN], va[NN];
#pragma unroll
    for (int s = 0; s < NN; ++s) {
      v[s] = vec[s * npts + p];
      vv[s] = (VT)v[s];
      va[s] = (VT)0;
      acc[s] = ukin[s * npts + p] + __ldg(rot + s) * v[s];
    }
    int t = 0;
#pragma unroll
    for (int s = 0; s < NN; ++s) {
#pragma unroll
      for (int q = s; q < NN; ++q, ++t) {
        const VT x = vb[(long long)t * npts + p];
        va[s] += x * vv[q];
        if (q != s) va[q] += x * vv[s];
      }
    }
#pragma unroll
    for (int s = 0; s < NN; ++s) {
      const double hv = acc[s] + (double)va[s];
      if (mode == 0) {
        out[s * npts + p] = hv;
      } else {
        const double r = fma(c, hv, out[s * npts + p]);
        out[s * npts + p] = r;
        dot += v[s] * r;
      }
    }
  }
  if (mode == 1) {
    if (p == 0) dot += vec[dpk] * out[dpk];  // the coordinate outside the symmetry block (H acts on it as 0)
    double total;
    if (reduce_grid(dot, partials, counter, &total) && threadIdx.x == 0) {
      scalars[0] = scalars[7] * total;
      hist[j - 1] = scalars[7] * total;
    }
  }
}

// The same for grids whose points are too few warps to fill the FP64 pipes:
// a CTA takes 32 points, and each of its kG warps NN / kG rows of their blocks.
// A row's sum runs over the columns in the order in which k_vapply adds them,
// so H v is the same bits.
template <int NN, int kG>
__global__ void __launch_bounds__(32 * kG) k_vapply_rows(const double* __restrict__ vb,
                                                         const double* __restrict__ vec,
                                                         const double* __restrict__ ukin,
                                                         const double* __restrict__ rot, double* __restrict__ out,
                                                         long long npts, int mode, double* partials,
                                                         unsigned int* counter, double* scalars, double* hist, int j,
                                                         long long dpk) {
  constexpr int R = NN / kG;
  static_assert(R * kG == NN, "the rows are split evenly");
  const int s0 = (threadIdx.x >> 5) * R;
  const long long p = (long long)blockIdx.x * 32 + (threadIdx.x & 31);
  const double c = mode ? scalars[6] : 1.0;
  double dot = 0.0;
  if (p < npts) {
    double v[NN], va[R], acc[R], vr[R];
#pragma unroll
    for (int q = 0; q < NN; ++q) v[q] = vec[q * npts + p];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int s = s0 + r;
      va[r] = 0.0;
      vr[r] = vec[s * npts + p];
      acc[r] = ukin[s * npts + p] + __ldg(rot + s) * vr[r];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int s = s0 + r;
#pragma unroll
      for (int q = 0; q < NN; ++q) {
        const int a = q < s ? q : s, b = q < s ? s : q;  // element (a, b), a <= b, of the triangle
        va[r] += vb[(long long)(a * NN - a * (a - 1) / 2 + b - a) * npts + p] * v[q];
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long i = (s0 + r) * npts + p;
      const double hv = acc[r] + va[r];
      if (mode == 0) {
        out[i] = hv;
      } else {
        const double x = fma(c, hv, out[i]);
        out[i] = x;
        dot += vr[r] * x;
      }
    }
  }
  if (mode == 1) {
    if (blockIdx.x == 0 && threadIdx.x == 0) dot += vec[dpk] * out[dpk];
    double total;
    if (reduce_grid(dot, partials, counter, &total) && threadIdx.x == 0) {
      scalars[0] = scalars[7] * total;
      hist[j - 1] = scalars[7] * total;
    }
  }
}

// generic fallback (local-memory arrays) for block sizes without an instantiation
__global__ void __launch_bounds__(kThreads) k_vapply_generic(const double* __restrict__ vb,
                                                             const double* __restrict__ vec,
                                                             const double* __restrict__ ukin,
                                                             const double* __restrict__ rot, double* __restrict__ out,
                                                             long long npts, int nn, int mode, double* partials,
                                                             unsigned int* counter, double* scalars, double* hist,
                                                             int j, long long dpk) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  // logical Lanczos vectors are v = sv vec and r = sr out; r + H v is kept as
  // sr (out + (sv/sr) H vec): out' = out + c H vec, alpha = sv sr (vec . out')
  const double c = mode ? scalars[6] : 1.0;
  double dot = 0.0;
  if (p < npts) {
    double v[kMaxNN], acc[kMaxNN];
    for (int s = 0; s < nn; ++s) {
      v[s] = vec[s * npts + p];
      acc[s] = ukin[s * npts + p] + __ldg(rot + s) * v[s];
    }
    int t = 0;
    for (int s = 0; s < nn; ++s)
      for (int q = s; q < nn; ++q, ++t) {
        const double x = vb[(long long)t * npts + p];
        acc[s] += x * v[q];
        if (q != s) acc[q] += x * v[s];
      }
    for (int s = 0; s < nn; ++s) {
      if (mode == 0) {
        out[s * npts + p] = acc[s];
      } else {
        const double r = fma(c, acc[s], out[s * npts + p]);
        out[s * npts + p] = r;
        dot += v[s] * r;
      }
    }
  }
  if (mode == 1) {
    if (p == 0) dot += vec[dpk] * out[dpk];
    double total;
    if (reduce_grid(dot, partials, counter, &total) && threadIdx.x == 0) {
      scalars[0] = scalars[7] * total;
      hist[j - 1] = scalars[7] * total;
    }
  }
}

}  // namespace
}  // namespace bsl
