// The kinetic contractions of a mixed-precision H v in one launch, for small
// grids (sm_103a).
//
// Reference: Tv_5D_oneCompositeIndex / Mv_5D_oneCompositeIndex,
// Hv-calculators/linRotor/cartSphBasis/HvCalc/linRotCartSphHvRoutines.cpp:1807-1969.
//
// One CTA per (function s, z plane k), one thread per point of the plane.  A
// thread loads its whole z column of v, so the CTA holds everything the three
// contractions of its plane need: the z term straight from the column's
// registers, the x and y terms from the plane's slices in shared memory.  The
// slices are those of the tensor-core kernels (bsl_slices.cuh: per-plane
// scales, four 9-bit integers) and the class sums are exact integers in FP32,
// so u_kin is the same bits.
//
// What bounds a small grid is the latency of a launch: below 20^3 a tensor-core
// kernel takes 6-8 us whatever its work, most of it set-up (tensor memory, the T
// image, 128 KiB of zeroed stages).  The column loads and their slicing grow as n
// per point, which ends the range (kin_small_supported).
#include <algorithm>

#include "bsl_device.cuh"
#include "bsl_slices.cuh"

namespace bsl {
namespace {

struct SmallArgs {
  const float2* v;    // the Lanczos v as double-float pairs
  float2* out;        // u_kin
  const float *tx, *tz;  // slices of T as FP32 integers, [slice][n][n]
  int n, nz, e_txy, e_tz;
  long long npts;
  // the first CTA finishes the previous update's deferred beta (null: none)
  double *partials, *scalars, *hist;
  int* jdev;
  int* status;
  int fin_count, hist_stride;
};

// class sums of one pair of sliced operands
__device__ __forceinline__ void add_products(float (&c)[4], const float (&a)[kVS], const float (&b)[kTS]) {
#pragma unroll
  for (int k = 0; k < kVS; ++k)
#pragma unroll
    for (int l = 0; l < kTS - k; ++l) c[k + l] = __fmaf_rn(a[k], b[l], c[k + l]);
}

constexpr int kMaxN = 16;
__global__ void __launch_bounds__(kMaxN * kMaxN + 32) k_kin_small(const SmallArgs a) {
  extern __shared__ float sh[];
  const int n = a.n, nz = a.nz, np = n * n, tid = threadIdx.x, lane = tid & 31;
  float* tx = sh;                   // [4][n][n]
  float* sv = tx + kTS * np;        // [4][n][n]: slices of the plane
  float* tz = sv + kVS * np;        // [nz][4]: row k of Tz
  int* row_max = reinterpret_cast<int*>(tz + kTS * nz);  // [n]: max |v| over (z, x) per y
  __shared__ int plane_max;
  const int k0 = blockIdx.x, s = blockIdx.y;
  for (int e = tid; e < kTS * np; e += blockDim.x) tx[e] = __ldg(a.tx + e);
  for (int e = tid; e < kTS * nz; e += blockDim.x) tz[e] = __ldg(a.tz + ((e & 3) * nz + k0) * nz + (e >> 2));
  if (tid < n) row_max[tid] = 0;
  if (tid == 0) plane_max = 0;
  __syncthreads();
  pdl_launch_dependents();
  pdl_wait();
  const int beta_warp = (int)blockDim.x / 32 - 1;  // beside the points' warps
  const bool point = tid < np;
  const int y = tid / n, x = tid - y * n;
  const long long i0 = (long long)s * a.npts + (long long)k0 * np + tid;
  float2 col[kMaxN], vx = make_float2(0.f, 0.f);
  if (tid / 32 == beta_warp) {
    if (a.partials && blockIdx.x == 0 && blockIdx.y == 0) {
      int* si = reinterpret_cast<int*>(a.scalars);
      if (*(volatile int*)(si + kPendingSlot)) {
        // the sum of finish_deferred_beta by 256 threads, one of their warps after the other
        double total = 0.0;
        for (int w = 0; w < 256 && w < a.fin_count; w += 32) {
          double acc = 0.0;
          for (int b = w + lane; b < a.fin_count; b += 256) acc += __ldcg(a.partials + kBetaPartials + b);
          total += warp_sum(acc);
        }
        if (lane == 0) {
          const int j = *a.jdev;
          finish_update_pair(total, si[20], a.scalars, a.hist, a.hist_stride, j, a.status);
          *a.jdev = j + 1;
          si[kPendingSlot] = 0;
        }
      }
    }
  } else if (point) {
    const float2* src = a.v + (long long)s * a.npts + tid;
#pragma unroll
    for (int z = 0; z < kMaxN; ++z) col[z] = z < nz ? __ldg(src + (long long)z * np) : make_float2(0.f, 0.f);
    vx = __ldg(a.v + i0);
    float m = 0.f;
#pragma unroll
    for (int z = 0; z < kMaxN; ++z) m = fmaxf(m, fabsf(col[z].x));
    atomicMax(&row_max[y], __float_as_int(m));
    atomicMax(&plane_max, __float_as_int(fabsf(vx.x)));
  }
  __syncthreads();
  const int e_xy = plane_exponent(__int_as_float(plane_max));
  if (point) {
    const float sc = pow2f(8 - e_xy);
    float sl[kVS];
    slice4(__fmul_rn(vx.x, sc), __fmul_rn(vx.y, sc), sl);
#pragma unroll
    for (int k = 0; k < kVS; ++k) sv[k * np + tid] = sl[k];
  }
  __syncthreads();
  if (point) {
    float c[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};
    const int e_z = plane_exponent(__int_as_float(row_max[y]));
    const float sc = pow2f(8 - e_z);
#pragma unroll
    for (int z = 0; z < kMaxN; ++z) {
      if (z < nz) {
        float sl[kVS];
        slice4(__fmul_rn(col[z].x, sc), __fmul_rn(col[z].y, sc), sl);
        const float4 t = reinterpret_cast<const float4*>(tz)[z];
        const float b[kTS] = {t.x, t.y, t.z, t.w};
        add_products(d, sl, b);
      }
    }
    for (int q = 0; q < n; ++q) {
      float av[kVS], b[kTS];
#pragma unroll
      for (int k = 0; k < 4; ++k) {  // y: sum_q v(q, x) Ty[y][q], T symmetric, Tx = Ty
        av[k] = sv[k * np + q * n + x];
        b[k] = tx[k * np + q * n + y];
      }
      add_products(c, av, b);
#pragma unroll
      for (int k = 0; k < 4; ++k) {  // x: sum_q v(y, q) Tx[x][q]
        av[k] = sv[k * np + y * n + q];
        b[k] = tx[k * np + q * n + x];
      }
      add_products(c, av, b);
    }
    a.out[i0] = df_add_fast(combine_classes(c[0], c[1], c[2], c[3], pow2f(e_xy + a.e_txy - 16)),
                            combine_classes(d[0], d[1], d[2], d[3], pow2f(e_z + a.e_tz - 16)));
  }
}

}  // namespace

// Up to 16 points per axis (the z column in registers).  Against the tensor cores'
// one launch, us: H v at 16^3 with 9, 15, 21 and 36 functions 16.5 against 20.7, 22.7
// against 24.7, 27.1 against 37.2, 41.2 against 55.5; an iteration at 15^3 with 15
// and 21 functions 20.1 against 21.4, 23.4 against 35.1, at 10^3 with 10 14.8
// against 18.5.  At 16^3 the iterations with 9, 10 and 15 functions are the other
// way round (24.1 against 22.3, 19.1 against 18.9, 21.7 against 20.6); they keep the
// kernel of their H v.  The same kernel with columns of up to 24 points gains 1.1x
// at 17^3 against two launches and loses from 20^3 on.
bool kin_small_supported(const bsl_handle* h) {
  const Tables& t = h->t;
  return h->d.tx_slices32 && h->kin_slices == 4 && t.nx <= kMaxN && t.nz <= kMaxN;
}

// u_kin of v; fin_count > 0: the block totals of a deferred beta to finish
int launch_kin_small(bsl_handle* h, const float2* v, int fin_count, cudaStream_t s) {
  const Tables& t = h->t;
  DeviceState& d = h->d;
  SmallArgs a{};
  a.v = v;
  a.out = reinterpret_cast<float2*>(d.ukin);
  a.tx = d.tx_slices32;
  a.tz = d.tz_slices32;
  a.n = t.nx;
  a.nz = t.nz;
  a.e_txy = d.e_txy;
  a.e_tz = d.e_tz;
  a.npts = t.npts;
  a.status = d.status;
  if (fin_count > 0) {
    a.partials = d.partials;
    a.scalars = d.scalars;
    a.hist = d.hist;
    a.jdev = d.jdev;
    a.fin_count = fin_count;
    a.hist_stride = d.hist_cap;
  }
  const int threads = (a.n * a.n + 31) / 32 * 32 + 32;  // the points and the warp of the deferred beta
  const size_t smem = sizeof(float) * ((size_t)(kTS + kVS) * a.n * a.n + kTS * a.nz + a.n);
  const cudaError_t e = launch_pdl(k_kin_small, dim3(a.nz, t.nn), dim3(threads), smem, s, a);
  return e == cudaSuccess ? BSL_OK : cuda_fail(e, "small-grid kinetic launch");
}

}  // namespace bsl
