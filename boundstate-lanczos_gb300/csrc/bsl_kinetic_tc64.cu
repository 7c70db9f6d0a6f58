// FP64 sinc-DVR kinetic contractions on the tensor cores (tcgen05.mma kind::f16,
// FP32 accumulation in tensor memory), sm_103a.
//
// Reference: Tv_5D_oneCompositeIndex / Mv_5D_oneCompositeIndex,
// Hv-calculators/linRotor/cartSphBasis/HvCalc/linRotCartSphHvRoutines.cpp:1807-1969.
//
// The contractions of bsl_kinetic_tc.cu (the same plane pairs, tiles, swizzle
// and accumulator layout) for FP64 vectors: v and T are cut into seven 9-bit
// integer slices instead of four (after Ozaki, Ogita, Oishi and Rump, Numer.
// Algorithms 59, 2012), 62 bits below the plane's and the matrix's largest
// element, and the 28 products of the classes k + l <= 6 are kept.  What is left
// out is 2^-62 of max|v| max|T| per term, below the rounding of an FP64 dot
// product (2^-53 of its partial sums): see test_kinetic_f64_slicing.py.
// The class sums 0-3 are integers below 2^24 and exact; the sums of classes 4-6
// could pass 2^24 only for a v that follows the signs of T's low slices, and
// one unit there is 2^-52 and less of the FP64 unit.  The classes are put
// together in 64-bit integers and rounded once to FP64.
//
// Why: the FP64 pipe executes 2 lanes a clock and SM, so 3 x 54 multiply-adds
// per coefficient take 0.85 ms at 54^3 and 21 functions; the 28 slice products
// are 18 us of tensor-core time.  Measured at 54^3, 21
// functions, x/y and z: 70 and 57 us against 656 and 337 us, and 28 and 24 us
// against 49 and 29 us at 27^3; bound by the shared-memory reads of the MMA
// operands (x/y) and the FP64 conversions and read-modify-write of the epilogue
// (z).
//
// Pipeline: as there, 8 epilogue warps, 8 producer warps and one MMA thread, but
// with one shared-memory stage (112 KiB) and one accumulator (448 columns): the
// producers slice the next pair while the epilogue reads the finished one.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "bsl_device.cuh"
#include "bsl_internal.h"
#include "bsl_tc.cuh"

namespace bsl {
namespace {

constexpr int kS = 7;                           // slices of v and of T
constexpr uint32_t kTile = 64 * 128;            // 64 rows x 64 FP16, one 128-byte swizzled row each
constexpr uint32_t kPlane = kS * kTile;         // the slices of one plane
constexpr uint32_t kAccCols = kS * 64;          // classes 0..6
constexpr int kEpiWarps = 8, kProdWarps = 8, kMmaWarp = kEpiWarps + kProdWarps;
constexpr int kThreads64 = (kMmaWarp + 1) * 32;
constexpr int kProdThreads = kProdWarps * 32, kEpiThreads = kEpiWarps * 32;
constexpr int kMaxItems = 64 * 16 / kProdThreads;  // (row, 4-column group) items per producer thread
constexpr int kNonFinite = 1 << 20;                // plane exponent of a plane with an infinity or a NaN

struct Kin64 {
  const uint4* timage;  // the T tiles as laid out in shared memory
  int timage16;
  int e_t;
  const double* v;
  double* out;
  int nx, ny, nz, nplanes;
  int* status;
};

// 512^0 + ... + 512^6, times 256: added to the 62-bit fixed-point value, every
// 9-bit digit d stands for d - 256
constexpr unsigned long long kBias = 256ull * ((1ull << 54) + (1ull << 45) + (1ull << 36) + (1ull << 27) +
                                               (1ull << 18) + (1ull << 9) + 1ull);

__device__ __forceinline__ uint32_t quad_offset64(int r, int k) {
  return (uint32_t)(r * 128 + (((k >> 3) ^ (r & 7)) << 4) + ((k & 7) << 1));
}

// v 2^(62 - e) + kBias for |v| < 2^e (truncated below 2^-62 of 2^e)
__device__ __forceinline__ unsigned long long fixed_point(double v, int e) {
  const long long b = __double_as_longlong(v);
  const int ev = (int)(((unsigned long long)b >> 52) & 0x7ff);
  unsigned long long m = ((unsigned long long)b & 0xfffffffffffffull) | (1ull << 52);
  const int sh = ev - 1013 - e;  // at most 9
  m = sh >= 0 ? m << min(sh, 9) : m >> min(-sh, 63);
  if (ev == 0) m = 0;
  return kBias + (b < 0 ? 0ull - m : m);
}

// digits k of two values as FP16 integers in [-256, 256]
template <int kDigit>
__device__ __forceinline__ uint32_t slice2(unsigned long long a, unsigned long long b) {
  const uint32_t mask = kDigit == kS - 1 ? 0x3ffu : 0x1ffu;  // the top digit reaches 512
  const uint32_t x = (uint32_t)(a >> (9 * kDigit)) & mask, y = (uint32_t)(b >> (9 * kDigit)) & mask;
  // 0x6400 + d is 1024 + d in FP16 for d < 1024
  uint32_t r = (x | (y << 16)) + 0x64006400u;
  const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&r), __floats2half2_rn(1280.f, 1280.f));
  return *reinterpret_cast<const uint32_t*>(&h);
}

template <bool kXY>
struct Planes64 {
  int nx, ny, nz;
  __device__ __forceinline__ long long base(int plane) const {
    if (kXY) return (long long)plane * nx * ny;
    return (long long)(plane / ny) * nz * nx * ny + (long long)(plane % ny) * nx;
  }
  __device__ __forceinline__ long long row_stride() const { return kXY ? (long long)nx : (long long)nx * ny; }
  __device__ __forceinline__ int rows() const { return kXY ? ny : nz; }
};

// x 2^s rounded to FP64, |x| < 2^62, on the integer pipe (a conversion and a
// product on the FP64 pipe would take 16 clocks of the SM each)
__device__ __forceinline__ double scaled(long long x, int s) {
  if (x == 0) return 0.0;
  const unsigned long long m = (unsigned long long)(x < 0 ? -x : x);
  const int lz = __clzll((long long)m);  // at least 2
  // the leading 53 bits, rounded to nearest (ties up), the leading one at bit 52
  const unsigned long long r = ((m << (lz - 1)) + 0x200ull) >> 10;
  const int e = s + 1085 - lz;  // biased exponent less 1: r's leading one adds 1 to it
  const unsigned long long sign = (unsigned long long)x & 0x8000000000000000ull;
  if ((unsigned int)e < 2045u) return __longlong_as_double((long long)(sign | (((unsigned long long)e << 52) + r)));
  // out of the normal range
  return ldexp(__longlong_as_double((long long)(sign | ((1074ull << 52) + r))), e - 1074);
}

// 4 consecutive columns of the seven classes as FP64 values times 2^s
__device__ __forceinline__ void combine4(uint32_t taddr, int s, double (&out)[4]) {
  float c[kS][4];
#pragma unroll
  for (int k = 0; k < kS; ++k) tc::tmem_ld4_nowait(taddr + 64u * k, c[k]);
  tc::tmem_wait_ld();
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    // units of 2^-41 of class 0's: below 2^62, and 2^-57 of 2^(e + e_t)
    const float low = __fmaf_rn(c[6][u], 0x1p-18f, __fmaf_rn(c[5][u], 0x1p-9f, c[4][u]));
    const int h01 = __float2int_rn(c[0][u]) * 512 + __float2int_rn(c[1][u]);
    const long long h23 = (long long)__float2int_rn(c[2][u]) * 512 + __float2int_rn(c[3][u]);
    const long long x = (((long long)h01 << 18) + h23) * 16384 + __float2int_rn(__fmul_rn(low, 32.f));
    out[u] = scaled(x, s);
  }
}

template <bool kXY>
__device__ __forceinline__ void kin64_body(const Kin64& a) {
  extern __shared__ uint8_t smraw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~(uintptr_t)1023);
  // T tiles: x/y as Z T0 .. T6 Z (Z = zero tile), z as T0 .. T6; then the v stage
  constexpr int kTTiles = kXY ? kS + 2 : kS;
  uint8_t* V = sm + kTTiles * kTile;
  __shared__ uint64_t v_full, v_empty, acc_full, acc_empty, e_full, stage_zeroed, t_ready;
  __shared__ uint32_t tmem_slot;
  __shared__ int e_stage[2], e_acc[2];
  __shared__ unsigned int red[2][kProdWarps];
  __shared__ int prod_go, failed, skip;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Planes64<kXY> pg{a.nx, a.ny, a.nz};
  const int npairs = (a.nplanes + 1) / 2, p_first = blockIdx.x, p_stride = gridDim.x;

  // a time-out recorded before this launch: leave before any allocation or wait
  if (tid == 0) skip = *(volatile int*)(a.status + 3);
  __syncthreads();
  if (skip) return;
  if (tid == 0) {
    tc::mbar_init(&v_full, kProdThreads);
    tc::mbar_init(&v_empty, 1);
    tc::mbar_init(&acc_full, 1);
    tc::mbar_init(&acc_empty, kEpiThreads);
    tc::mbar_init(&e_full, 1);
    tc::mbar_init(&stage_zeroed, kEpiThreads);
    tc::mbar_init(&t_ready, kEpiThreads);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) tc::tmem_alloc(&tmem_slot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  pdl_launch_dependents();

  if (warp < kEpiWarps) {
    // ---- epilogue: TMEM lane quadrant warp % 4 = (plane p, 32-column block of
    // x), columns [32 half, 32 half + 32) ----
    const int quad = warp & 3, half = warp >> 2;
    const int p = quad >> 1, x = ((quad & 1) << 5) + lane;
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    const long long cstride = pg.row_stride();
    const int c_begin = half * 32, c_end = min(half * 32 + 32, pg.rows());
    // the v stage zeroed (the producers write only the groups that hold data),
    // then the T tiles
    for (int e = tid; e < (int)(2 * kPlane / 16); e += kEpiThreads) reinterpret_cast<uint4*>(V)[e] = make_uint4(0u, 0u, 0u, 0u);
    tc::fence_smem_to_async();
    tc::mbar_arrive(&stage_zeroed);
    for (int e = tid; e < a.timage16; e += kEpiThreads) reinterpret_cast<uint4*>(sm)[e] = a.timage[e];
    tc::fence_smem_to_async();
    tc::mbar_arrive(&t_ready);
    pdl_wait();  // the output (and, for z, the values added to) belong to earlier kernels
    for (int it = 0, pair = p_first; pair < npairs; pair += p_stride, ++it) {
      const uint32_t par = (uint32_t)it & 1u;
      const int plane = 2 * pair + p;
      const bool valid = plane < a.nplanes && x < a.nx;
      const long long ob = valid ? pg.base(plane) + x : 0;
      double nxt[4];  // z: the values added to, loaded while the products run
      auto load4 = [&](int c0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) nxt[u] = (valid && c0 + u < c_end) ? a.out[ob + (c0 + u) * cstride] : 0.0;
      };
      if (!kXY) load4(c_begin);
      int ok = 1;
      if (lane == 0) ok = tc::mbar_wait(&acc_full, par) && tc::mbar_wait(&e_full, par);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) {
        failed = 1;
        break;
      }
      tc::mbar_wait(&acc_full, par);
      tc::mbar_wait(&e_full, par);
      tc::fence_after_sync();
      const int e = e_acc[p];
      const int s = e + a.e_t - 16 - 41;
      const uint32_t tbase = tmem + lane_base;
#pragma unroll 1
      for (int c0 = c_begin; c0 < c_end; c0 += 4) {
        double r[4], cur[4];
        if (!kXY) {
#pragma unroll
          for (int u = 0; u < 4; ++u) cur[u] = nxt[u];
          if (c0 + 4 < c_end) load4(c0 + 4);
        }
        combine4(tbase + (uint32_t)c0, s, r);
        if (e == kNonFinite)
#pragma unroll
          for (int u = 0; u < 4; ++u) r[u] = __longlong_as_double(0x7ff8000000000000ll);
        if (valid)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (c0 + u < c_end) a.out[ob + (c0 + u) * cstride] = kXY ? r[u] : r[u] + cur[u];
      }
      tc::fence_before_sync();
      tc::mbar_arrive(&acc_empty);
    }
  } else if (warp < kMmaWarp) {
    // ---- producers: item i = (row, 4-column group) of a plane ----
    const int ptid = tid - kEpiThreads, pw = ptid >> 5;
    const int nrows = pg.rows(), nx = a.nx, ncg = (nx + 3) >> 2, nitems = nrows * ncg;
    const long long rstride = pg.row_stride();
    int goff[kMaxItems], cnt[kMaxItems];
    uint32_t soff[kMaxItems];
#pragma unroll
    for (int t = 0; t < kMaxItems; ++t) {
      const int i = ptid + t * kProdThreads;
      const int j = i / ncg, c = (i - j * ncg) * 4;
      const bool iv = i < nitems;
      goff[t] = iv ? (int)(j * rstride) + c : 0;
      soff[t] = iv ? quad_offset64(j, c) : 0u;
      cnt[t] = iv ? min(4, nx - c) : 0;
    }
    double x[kMaxItems][4];
    auto load_item = [&](int t, const double* src) {  // src null: past the last plane
#pragma unroll
      for (int u = 0; u < 4; ++u) x[t][u] = (src && u < cnt[t]) ? __ldg(src + goff[t] + u) : 0.0;
    };
    auto plane_ptr = [&](int plane) { return plane < a.nplanes ? a.v + pg.base(plane) : nullptr; };
    pdl_wait();  // v is written by an earlier kernel
    {
      const double* src = plane_ptr(2 * p_first);
#pragma unroll
      for (int t = 0; t < kMaxItems; ++t) load_item(t, src);
    }
    int slot = 0;
    for (int it = 0, pair = p_first; pair < npairs; pair += p_stride, ++it) {
      const uint32_t par = (uint32_t)it & 1u;
      if (ptid == 0)
        prod_go = ((it > 0 || tc::mbar_wait(&stage_zeroed, 0u)) && tc::mbar_wait(&v_empty, par ^ 1u)) ? 1 : 0;
      tc::named_sync(1, kProdThreads);
      if (!prod_go) {
        if (ptid == 0) failed = 1;
        break;
      }
#pragma unroll 1
      for (int pl = 0; pl < 2; ++pl) {
        unsigned int mx = 0u;
#pragma unroll
        for (int t = 0; t < kMaxItems; ++t)
#pragma unroll
          for (int u = 0; u < 4; ++u) mx = max(mx, (unsigned int)__double2hiint(x[t][u]) & 0x7fffffffu);
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) red[slot][pw] = mx;
        tc::named_sync(1, kProdThreads);
#pragma unroll
        for (int w = 0; w < kProdWarps; ++w) mx = max(mx, red[slot][w]);
        slot ^= 1;
        // |v| < 2^e over the plane (0 for a plane of zeros and subnormals)
        const int e = mx >= 0x7ff00000u ? kNonFinite : (mx >> 20) ? (int)(mx >> 20) - 1022 : 0;
        if (ptid == 0) e_stage[pl] = e;
        uint8_t* vp = V + pl * kPlane;
        // the next plane's values are loaded item by item as this one's are sliced
        const double* next = plane_ptr(pl == 0 ? 2 * pair + 1 : 2 * (pair + p_stride));
#pragma unroll
        for (int t = 0; t < kMaxItems; ++t) {
          if (cnt[t] > 0) {
            unsigned long long f[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) f[u] = fixed_point(x[t][u], e);
            uint8_t* dst = vp + soff[t];
            // slice k (most significant first) is digit 6 - k
            *reinterpret_cast<uint2*>(dst) = make_uint2(slice2<6>(f[0], f[1]), slice2<6>(f[2], f[3]));
            *reinterpret_cast<uint2*>(dst + kTile) = make_uint2(slice2<5>(f[0], f[1]), slice2<5>(f[2], f[3]));
            *reinterpret_cast<uint2*>(dst + 2 * kTile) = make_uint2(slice2<4>(f[0], f[1]), slice2<4>(f[2], f[3]));
            *reinterpret_cast<uint2*>(dst + 3 * kTile) = make_uint2(slice2<3>(f[0], f[1]), slice2<3>(f[2], f[3]));
            *reinterpret_cast<uint2*>(dst + 4 * kTile) = make_uint2(slice2<2>(f[0], f[1]), slice2<2>(f[2], f[3]));
            *reinterpret_cast<uint2*>(dst + 5 * kTile) = make_uint2(slice2<1>(f[0], f[1]), slice2<1>(f[2], f[3]));
            *reinterpret_cast<uint2*>(dst + 6 * kTile) = make_uint2(slice2<0>(f[0], f[1]), slice2<0>(f[2], f[3]));
          }
          load_item(t, next);
        }
      }
      tc::fence_smem_to_async();
      tc::mbar_arrive(&v_full);
    }
  } else if (lane == 0) {
    // ---- MMA issue ----
    const uint32_t tb = tc::smem_u32(sm), vb = tc::smem_u32(V);
    const uint32_t t0 = tb + (kXY ? kTile : 0u);
    // 16-row steps of the contractions that hold data (the rest is zero padding)
    const int ks_rows = (pg.rows() + 15) / 16, ks_x = (a.nx + 15) / 16;
    if (!tc::mbar_wait(&t_ready, 0u)) failed = 1;
    for (int it = 0, pair = p_first; pair < npairs && !failed; pair += p_stride, ++it) {
      const uint32_t par = (uint32_t)it & 1u;
      if (!tc::mbar_wait(&v_full, par) || !tc::mbar_wait(&acc_empty, par ^ 1u)) {
        failed = 1;
        break;
      }
      tc::fence_after_sync();
      e_acc[0] = e_stage[0];
      e_acc[1] = e_stage[1];
      tc::mbar_arrive(&e_full);
      // Class c accumulates in columns [64 c, 64 c + 64).  An MMA whose B stacks
      // slices l0 .. l0 + n - 1 along N (at most four: N <= 256) and whose D
      // starts at column 64 (k + l0) puts product (k, l) into class k + l.
      // Contraction over the rows of each plane: A = v slice k (M = (p, x),
      // MN-major, the planes kPlane apart), B = T slices.  Slice 0 of v sets
      // every class.
#pragma unroll 1
      for (int k = 0; k < kS; ++k)
#pragma unroll 1
        for (int l0 = 0; l0 < kS - k; l0 += 4) {
          const uint32_t idesc = tc::idesc_f16(128, 64 * min(4, kS - k - l0)) | tc::kIdescAMajorMN;
          for (int s = 0; s < ks_rows; ++s)
            tc::mma_f16(tmem + 64u * (uint32_t)(k + l0),
                        tc::sw128_mn_desc(vb + (uint32_t)k * kTile + (uint32_t)s * 2048u, kPlane, 1024u),
                        tc::sw128_desc(t0 + (uint32_t)l0 * kTile + (uint32_t)s * 32u), idesc,
                        (k == 0 && s == 0) ? 0u : 1u);
        }
      if (kXY) {
        // contraction along x: A = diag(T_l, T_l) over K = (p', q), read MN-major
        // (T is symmetric), B = v slices of plane p' stacked along N
        const uint32_t zlo = tb, zhi = tb + (uint32_t)(kS + 1) * kTile;
#pragma unroll 1
        for (int l = 0; l < kS; ++l) {
          const uint32_t tl = t0 + (uint32_t)l * kTile;
#pragma unroll 1
          for (int k0 = 0; k0 < kS - l; k0 += 4) {
            const uint32_t idesc = tc::idesc_f16(128, 64 * min(4, kS - l - k0)) | tc::kIdescAMajorMN;
            for (uint32_t pp = 0; pp < 2; ++pp)
              for (uint32_t q = 0; q < (uint32_t)ks_x; ++q) {
                const uint64_t adesc = pp ? tc::sw128_mn_desc(zlo + q * 2048u, tl - zlo, 1024u)
                                          : tc::sw128_mn_desc(tl + q * 2048u, zhi - tl, 1024u);
                tc::mma_f16(tmem + 64u * (uint32_t)(l + k0), adesc,
                            tc::sw128_desc(vb + pp * kPlane + (uint32_t)k0 * kTile + q * 32u), idesc, 1u);
              }
          }
        }
      }
      tc::mma_commit(&v_empty);
      tc::mma_commit(&acc_full);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (failed && tid == 0) a.status[3] = 1;
  if (warp == kMmaWarp) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 512);
  }
}

// x and y contractions: out(y, x) = Tx v + Ty v
__global__ void __launch_bounds__(kThreads64, 1) k_kin_xy_tc64(Kin64 a) { kin64_body<true>(a); }
// z contraction added: out(z, x) += Tz v
__global__ void __launch_bounds__(kThreads64, 1) k_kin_z_tc64(Kin64 a) { kin64_body<false>(a); }

constexpr size_t kSmemXY = 1024 + (kS + 2) * kTile + 2 * kPlane;
constexpr size_t kSmemZ = 1024 + kS * kTile + 2 * kPlane;
static_assert(kSmemXY + 512 <= 227 * 1024, "x/y T tiles and the stage must fit in one CTA's shared memory");
static_assert(kAccCols <= 512, "the accumulator must fit in tensor memory");

uint16_t half_bits(int x) {
  const __half h = __float2half_rn((float)x);
  uint16_t u;
  std::memcpy(&u, &h, 2);
  return u;
}

}  // namespace

// The seven 9-bit slices of a symmetric T (62 bits below 2^e_t > max|T|, rounded
// to nearest, digits in [-256, 256]) as the kernels' shared-memory T region.
void kinetic_smem_image64(const std::vector<double>& T, int n, bool with_zero_tiles, std::vector<uint16_t>* image,
                          int* e_t) {
  double m = 0.0;
  for (double x : T) m = std::max(m, std::fabs(x));
  int e = 0;
  if (m > 0.0) std::frexp(m, &e);
  *e_t = e;
  const int first = with_zero_tiles ? 1 : 0;
  image->assign((size_t)(kS + 2 * first) * kTile / 2, half_bits(0));
  for (int i = 0; i < n; ++i)
    for (int q = 0; q < n; ++q) {
      // |T| 2^(62 - e) < 2^62 is exact to the last FP64 bit where |T| >= 2^(e - 10)
      const unsigned long long f = kBias + (unsigned long long)std::llrint(std::ldexp(T[(size_t)i * n + q], 62 - e));
      for (int l = 0; l < kS; ++l) {
        const int digit = kS - 1 - l;
        const int b = (int)((f >> (9 * digit)) & (digit == kS - 1 ? 0x3ffull : 0x1ffull)) - 256;
        const size_t byte = (size_t)(first + l) * kTile + (size_t)i * 128 + (size_t)(((q >> 3) ^ (i & 7)) << 4) +
                            (size_t)(q & 7) * 2;
        (*image)[byte / 2] = half_bits(b);
      }
    }
}

int launch_kin_tc64(bsl_handle* h, const double* v, bool xy, cudaStream_t s) {
  const Tables& t = h->t;
  DeviceState& d = h->d;
  Kin64 a{};
  a.v = v;
  a.out = d.ukin;
  a.nx = t.nx;
  a.ny = t.ny;
  a.nz = t.nz;
  a.status = d.status;
  a.timage = reinterpret_cast<const uint4*>(xy ? d.kxy_slices64 : d.kz_slices64);
  a.timage16 = (int)((xy ? kS + 2 : kS) * kTile / 16);
  a.e_t = xy ? d.e_txy64 : d.e_tz64;
  a.nplanes = (xy ? t.nz : t.ny) * t.nn;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const dim3 grid(std::min((a.nplanes + 1) / 2, std::max(1, sms)));
  if (xy) {
    cudaFuncSetAttribute(k_kin_xy_tc64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemXY);
    BSL_CUDA(launch_pdl(k_kin_xy_tc64, grid, dim3(kThreads64), kSmemXY, s, a));
  } else {
    cudaFuncSetAttribute(k_kin_z_tc64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemZ);
    BSL_CUDA(launch_pdl(k_kin_z_tc64, grid, dim3(kThreads64), kSmemZ, s, a));
  }
  return BSL_OK;
}

}  // namespace bsl
