// FP64 sinc-DVR kinetic contractions on the tensor cores (tcgen05.mma kind::f16,
// FP32 accumulation in tensor memory), sm_103a.
//
// Reference: Tv_5D_oneCompositeIndex / Mv_5D_oneCompositeIndex,
// Hv-calculators/linRotor/cartSphBasis/HvCalc/linRotCartSphHvRoutines.cpp:1807-1969.
//
// The contractions of bsl_kinetic_tc.cu (the same plane pairs, tiles, swizzle
// and accumulator layout) for FP64 vectors: every line of v that is contracted (a
// column of the plane along y or z, a row along x) and T are cut into eight 9-bit
// integer slices (after Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59,
// 2012) and the 36 products of the classes k + l <= 7 are kept.
//
// What that leaves out, of max |T| times the line's largest |v|, for an element of
// the result:
//   * an element of v is cut 71 bits below its own line's largest element (an
//     exponent per line, so that a small line keeps its bits beside a large one);
//     T is cut there too, which is exact down to 2^-18 max |T| (the smallest
//     element of a 64-point axis is 2^-12.7 of the largest);
//   * the classes from 8 on: 2^-69 root mean square for 64 terms of digits without
//     a pattern, at most 2^-63;
//   * the class sums 0-6 are integers below 2^24 and exact (kinetic_smem_image64
//     refuses a T whose slices could pass that), one unit of class 7 is 2^-79;
//   * the classes are put together as integers and rounded once.
// The sum of |T v| along the line is at least 2^-12.7 of the same product, so this
// stays below one FP64 rounding (2^-53) of that sum, and below a dot product's
// n 2^-53 even at its largest: every element is held to its own terms as in FP64,
// whatever the range of v (the tail of a bound state, a column of 1e-20 beside
// one of 1): test_kinetic_f64_lines.py, test_gpu_kinetic_f64.py.  A line with an
// infinity or a NaN is formed by the plain sums.
//
// Why: the FP64 pipe executes 2 lanes a clock and SM, so 3 x 54 multiply-adds
// per coefficient take 0.85 ms at 54^3 and 21 functions.  Measured there, x/y and
// z: 97 and 57 us against 656 and 337 us of plain sums in two launches; 36 and 22
// us at 27^3.  An item (a plane pair and direction) takes its slicing (11,000
// clocks, integer pipe) and its MMAs (8,000) in turn, since the eight slices leave
// room for one stage; the epilogue (13,000, FP64 additions and the
// read-modify-write) runs beside them.
//
// Pipeline: as there, 8 epilogue warps, 8 producer warps and one MMA thread, but
// with one shared-memory stage (128 KiB).  The accumulator has two parts, for
// half of T's rows each, so that the epilogue reads one while the other's MMAs
// run.  The x/y kernel takes a pair of planes as two items, along y and along x,
// since the lines, and so the slices, differ.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "bsl_device.cuh"
#include "bsl_internal.h"
#include "bsl_tc.cuh"

namespace bsl {
namespace {

constexpr int kS = 8;                           // slices of v and of T
constexpr uint32_t kTile = 64 * 128;            // 64 rows x 64 FP16, one 128-byte swizzled row each
constexpr uint32_t kPair = 2 * kTile;           // one slice of a plane pair: 128 rows
constexpr uint32_t kHalfTile = kTile / 2;       // half of the rows of a slice of T
constexpr uint32_t kAccCols = kS * 32;          // classes 0..7 of half of the columns
constexpr int kEpiWarps = 8, kProdWarps = 8, kMmaWarp = kEpiWarps + kProdWarps;
constexpr int kThreads64 = (kMmaWarp + 1) * 32;
constexpr int kProdThreads = kProdWarps * 32, kEpiThreads = kEpiWarps * 32;
constexpr int kMaxItems = 64 * 16 / kProdThreads;  // (row, 4-column group) pieces per producer thread
constexpr int kNonFinite = 1 << 20;                // exponent of a line with an infinity or a NaN

struct Kin64 {
  const uint4* timage;  // the T tiles as laid out in shared memory
  int timage16;
  int e_t;
  const double* t;      // T, for the lines that are not finite
  const double* v;
  double* out;
  int nx, ny, nz, nplanes;
  int* status;
};

// 36 bits of a fixed-point value are four 9-bit digits; 256 in every digit makes
// each digit d stand for d - 256
constexpr long long kBias36 = 256ll * ((1ll << 27) + (1ll << 18) + (1ll << 9) + 1ll);
constexpr unsigned long long kMask36 = (1ull << 36) - 1;

// T's rows (the results' columns) are taken in two halves, of a multiple of 4 and
// at most 32 rows the first, so that the accumulator has two parts
__host__ __device__ __forceinline__ int half_rows(int n) { return (n + 7) / 8 * 4; }

__device__ __forceinline__ uint32_t quad_offset64(int r, int k) {
  return (uint32_t)(r * 128 + (((k >> 3) ^ (r & 7)) << 4) + ((k & 7) << 1));
}

// e of a line whose largest |v| has the upper word hi: |v| < 2^e
__device__ __forceinline__ int line_exponent(unsigned int hi) {
  const int ev = (int)(hi >> 20);
  return ev == 0x7ff ? kNonFinite : max(ev, 1) - 1022;
}

// v 2^(71 - e), truncated, for |v| < 2^e of a line whose largest exponent field
// (at least 1) is top, as eight biased digits, four in each of hi and lo
struct Digits {
  unsigned long long hi, lo;
};
__device__ __forceinline__ Digits digits_of(double v, int top) {
  const long long b = __double_as_longlong(v);
  const int ev = (int)(((unsigned long long)b >> 52) & 0x7ff);
  unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
  if (ev) m |= 1ull << 52;
  const int d = top - max(ev, 1);  // v 2^(71 - e) = m 2^(18 - d)
  const long long mh = (long long)(m >> min(18 + d, 63));
  const long long ml = (long long)((d <= 18 ? m << (18 - d) : m >> min(d - 18, 63)) & kMask36);
  const long long s = kBias36 + (b < 0 ? -ml : ml);
  return Digits{(unsigned long long)(kBias36 + (b < 0 ? -mh : mh) + (s >> 36)), (unsigned long long)s & kMask36};
}

// digit k of two 36-bit groups as FP16 integers in [-256, 256] (the top digit reaches 512 before the bias)
template <int kDigit>
__device__ __forceinline__ uint32_t slice2(unsigned long long a, unsigned long long b) {
  constexpr uint32_t mask = kDigit == 3 ? 0x03ff03ffu : 0x01ff01ffu;
  // 0x6400 + d is 1024 + d in FP16 for d < 1024
  const uint32_t r = (__byte_perm((uint32_t)(a >> (9 * kDigit)), (uint32_t)(b >> (9 * kDigit)), 0x5410) & mask) | 0x64006400u;
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
  __device__ __forceinline__ int row_stride() const { return kXY ? nx : nx * ny; }
  __device__ __forceinline__ int rows() const { return kXY ? ny : nz; }
};

// The CTA's items: one per plane pair first, first + stride, ..., or two (along y,
// then along x) for x/y.
template <bool kXY>
struct Items64 {
  int pair, stride, end;
  bool along_x = false;
  __device__ __forceinline__ bool more() const { return pair < end; }
  __device__ __forceinline__ void next() {
    if (kXY) along_x = !along_x;
    if (!along_x) pair += stride;
  }
};

__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(1023 + e) << 52); }

// What a thread's line scales by: class 3's unit 2^s as 2^b 2^rest, rest 0 unless
// the products with 2^b could leave the normal range, and -(3 2^51 + 3 2^15) 2^b.
struct LineScale {
  int b, rest;
  double unit, shift;
  __device__ __forceinline__ explicit LineScale(int s) : b(min(max(s, -900), 900)) {
    rest = s - b;
    unit = pow2(b);
    shift = __longlong_as_double((long long)(1023 + b + 52) << 52 | 0x8008000000018000ll);
  }
};

// (hi + lo 2^-36) 2^b rounded to nearest: hi and lo placed in the mantissas of
// 3 2^51 + hi and 3 2^15 + lo 2^-36 and added with one rounding.  (The same on the
// integer pipe, about 40 operations, is no faster: 386 against 367 us an iteration
// of 54^3.)
__device__ __forceinline__ double rounded(long long hi, long long lo, const LineScale& q) {
  const double h = __longlong_as_double(hi + (0x4338ll << 48)), l = __longlong_as_double(lo + (0x40f8ll << 48));
  return fma(l, q.unit, fma(h, q.unit, q.shift));
}

// 4 consecutive columns of the eight classes as FP64 values: classes 0-3 and 4-7
// put together as 64-bit integers (below 2^46 and 2^51), the second in units of
// 2^-36 of the first's, and rounded once.
__device__ __forceinline__ void combine4(uint32_t taddr, const LineScale& q, double (&out)[4]) {
  float c[kS][4];
#pragma unroll
  for (int k = 0; k < kS; ++k) tc::tmem_ld4_nowait(taddr + 32u * k, c[k]);
  tc::tmem_wait_ld();
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int c12 = __float2int_rn(c[1][u]) * 512 + __float2int_rn(c[2][u]);
    const long long hi = ((long long)__float2int_rn(c[0][u]) << 27) + ((long long)c12 << 9) + __float2int_rn(c[3][u]);
    const long long lo = ((long long)__float2int_rn(c[4][u]) << 27) + ((long long)__float2int_rn(c[5][u]) << 18) +
                         ((long long)__float2int_rn(c[6][u]) << 9) + __float2int_rn(c[7][u]);
    out[u] = rounded(hi, lo, q);
  }
  for (int rest = q.rest; rest != 0;) {
    const int k = min(max(rest, -1000), 1000);
#pragma unroll
    for (int u = 0; u < 4; ++u) out[u] *= pow2(k);
    rest -= k;
  }
}

// one element by the plain sum (a line with an infinity or a NaN)
__device__ __forceinline__ double plain_sum(const double* trow, const double* v, int stride, int n) {
  double acc = 0.0;
#pragma unroll 1
  for (int q = 0; q < n; ++q) acc += __ldg(trow + q) * __ldg(v + (long long)q * stride);
  return acc;
}

// After a time-out: NaN in the planes of the CTA's items, so that an H v whose
// caller does not read the status words (bsl_hv_apply_device) cannot be taken
// for a result.
template <bool kXY>
__device__ __forceinline__ void poison(const Kin64& a, Items64<kXY> w) {
  pdl_wait();
  const Planes64<kXY> pg{a.nx, a.ny, a.nz};
  for (; w.more(); w.pair += w.stride)
    for (int e = threadIdx.x; e < 2 * pg.rows() * a.nx; e += blockDim.x) {
      const int row = e / a.nx, pl = row >= pg.rows(), plane = 2 * w.pair + pl;
      if (plane < a.nplanes)
        a.out[pg.base(plane) + (long long)(row - pl * pg.rows()) * pg.row_stride() + e % a.nx] =
            __longlong_as_double(0x7ff8000000000000ll);
    }
}

template <bool kXY>
__device__ __forceinline__ void kin64_body(const Kin64& a) {
  extern __shared__ uint8_t smraw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~(uintptr_t)1023);
  uint8_t* V = sm + kS * kTile;  // the T tiles T0 .. T7, then the v stage [slice][plane]
  __shared__ uint64_t v_full, v_empty, acc_full[2], acc_empty[2], e_full[2], y_done, stage_zeroed, t_ready;
  __shared__ uint32_t tmem_slot;
  __shared__ int e_line[2][2][64];          // [item & 1][plane][line]: the lines' exponents
  __shared__ uint4 line_max[3][16];         // upper words of the lines' largest |v|, three planes in turn
  __shared__ int prod_go, failed, skip;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Planes64<kXY> pg{a.nx, a.ny, a.nz};
  const Items64<kXY> first{(int)blockIdx.x, (int)gridDim.x, (a.nplanes + 1) / 2};

  // a time-out recorded before this launch: leave before any allocation or wait
  if (tid == 0) skip = *(volatile int*)(a.status + 3);
  if (tid < 48) line_max[tid >> 4][tid & 15] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  if (skip) {
    poison<kXY>(a, first);
    return;
  }
  if (tid == 0) {
    tc::mbar_init(&v_full, kProdThreads);
    tc::mbar_init(&v_empty, 1);
    for (int h = 0; h < 2; ++h) {
      tc::mbar_init(&acc_full[h], 1);
      tc::mbar_init(&e_full[h], 1);
      tc::mbar_init(&acc_empty[h], kEpiThreads / 2);
    }
    tc::mbar_init(&y_done, kEpiThreads);
    tc::mbar_init(&stage_zeroed, kEpiThreads);
    tc::mbar_init(&t_ready, kEpiThreads);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) tc::tmem_alloc(&tmem_slot, 2 * kAccCols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  pdl_launch_dependents();

  if (warp < kEpiWarps) {
    // ---- epilogue: TMEM lane quadrant warp % 4 = (plane p, 32-line block),
    // half of the columns; a lane is a line: the plane's column x of a
    // contraction over its rows, its row of a contraction along x ----
    const int quad = warp & 3, half = warp >> 2;
    const int p = quad >> 1, line = ((quad & 1) << 5) + lane;
    const uint32_t tbase = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)half * kAccCols;
    const int rstride = pg.row_stride(), rows = pg.rows();
    // the v stage zeroed (the producers write only the groups that hold data),
    // then the T tiles
    for (int e = tid; e < (int)(kS * kPair / 16); e += kEpiThreads) reinterpret_cast<uint4*>(V)[e] = make_uint4(0u, 0u, 0u, 0u);
    tc::fence_smem_to_async();
    tc::mbar_arrive(&stage_zeroed);
    for (int e = tid; e < a.timage16; e += kEpiThreads) reinterpret_cast<uint4*>(sm)[e] = a.timage[e];
    tc::fence_smem_to_async();
    tc::mbar_arrive(&t_ready);
    pdl_wait();  // the output (and, for z, the values added to) belong to earlier kernels
    int it = 0;
    for (Items64<kXY> w = first; w.more(); w.next(), ++it) {
      const uint32_t par = (uint32_t)it & 1u;
      const int plane = 2 * w.pair + p;
      const int nlines = w.along_x ? rows : a.nx, n = w.along_x ? a.nx : rows;
      const bool valid = plane < a.nplanes && line < nlines;
      const long long base = valid ? pg.base(plane) + (w.along_x ? line * rstride : line) : 0;
      const int cstride = w.along_x ? 1 : rstride, mid = half_rows(n);
      const int c_begin = half * mid, c_end = half ? n : min(mid, n);
      double* out = a.out + base;
      const bool add = !kXY || w.along_x;
      double nxt[4];  // the values added to, loaded while the products run
      auto load4 = [&](int c0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) nxt[u] = (valid && c0 + u < c_end) ? out[(c0 + u) * cstride] : 0.0;
      };
      // lane 0 waits (bounded) and the warp leaves together on a time-out; every
      // lane's own wait then returns at once and orders its accesses
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        int ok = lane == 0 ? tc::mbar_wait(bar, parity) : 1;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        return ok && tc::mbar_wait(bar, parity);
      };
      // along x other threads of this CTA wrote the sums along y that are added to
      bool ok = !kXY || !w.along_x || wait(&y_done, (uint32_t)(it >> 1) & 1u);
      if (ok && add) load4(c_begin);
      ok = ok && wait(&acc_full[half], par) && wait(&e_full[half], par);
      if (__any_sync(0xffffffffu, !ok)) {
        failed = 1;
        break;
      }
      tc::fence_after_sync();
      const int e = e_line[par][p][line];
      const LineScale q(e == kNonFinite ? 0 : e + a.e_t - 43);
#pragma unroll 1
      for (int c0 = c_begin; c0 < c_end; c0 += 4) {
        double r[4], cur[4];
        if (add) {
#pragma unroll
          for (int u = 0; u < 4; ++u) cur[u] = nxt[u];
          if (c0 + 4 < c_end) load4(c0 + 4);
        }
        combine4(tbase + (uint32_t)(c0 - c_begin), q, r);
        if (e == kNonFinite && valid)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (c0 + u < c_end) r[u] = plain_sum(a.t + (c0 + u) * n, a.v + base, cstride, n);
        if (valid)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (c0 + u < c_end) out[(c0 + u) * cstride] = add ? r[u] + cur[u] : r[u];
        __syncwarp();
      }
      tc::fence_before_sync();
      tc::mbar_arrive(&acc_empty[half]);
      if (kXY && !w.along_x) tc::mbar_arrive(&y_done);
    }
  } else if (warp < kMmaWarp) {
    // ---- producers: piece i = (row, 4-column group) of a plane ----
    const int ptid = tid - kEpiThreads;
    const int nx = a.nx, rstride = pg.row_stride(), ncg = (nx + 3) >> 2, npieces = pg.rows() * ncg;
    int row[kMaxItems], col[kMaxItems], cnt[kMaxItems];  // cnt 0: no such piece
#pragma unroll
    for (int t = 0; t < kMaxItems; ++t) {
      const int i = ptid + t * kProdThreads;
      const bool iv = i < npieces;
      row[t] = iv ? i / ncg : 0;
      col[t] = iv ? (i - row[t] * ncg) * 4 : 0;
      cnt[t] = iv ? min(4, nx - col[t]) : 0;
    }
    double x[kMaxItems][4];
    auto load_piece = [&](int t, const double* src) {  // src null: past the last plane
      const double* q = src + (row[t] * rstride + col[t]);
#pragma unroll
      for (int u = 0; u < 4; ++u) x[t][u] = (src && u < cnt[t]) ? __ldg(q + u) : 0.0;
    };
    auto plane_ptr = [&](const Items64<kXY>& w, int pl) {
      const int plane = 2 * w.pair + pl;
      return w.more() && plane < a.nplanes ? a.v + pg.base(plane) : nullptr;
    };
    pdl_wait();  // v is written by an earlier kernel
    Items64<kXY> w = first;
    {
      const double* src = plane_ptr(w, 0);
#pragma unroll
      for (int t = 0; t < kMaxItems; ++t) load_piece(t, src);
    }
    int slot = 0;
    for (int it = 0; w.more(); ++it) {
      const uint32_t par = (uint32_t)it & 1u;
      if (ptid == 0)
        prod_go = ((it > 0 || tc::mbar_wait(&stage_zeroed, 0u)) && tc::mbar_wait(&v_empty, par ^ 1u)) ? 1 : 0;
      tc::named_sync(1, kProdThreads);
      if (!prod_go) {
        if (ptid == 0) failed = 1;
        break;
      }
      const bool along_x = w.along_x;
#pragma unroll 1
      for (int pl = 0; pl < 2; ++pl) {
        // the largest |v| of every line (by the upper words), over the plane's pieces
        unsigned int* mx = reinterpret_cast<unsigned int*>(line_max[slot]);
#pragma unroll
        for (int t = 0; t < kMaxItems; ++t)
          if (cnt[t] > 0) {
            unsigned int hi[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) hi[u] = (unsigned int)__double2hiint(x[t][u]) & 0x7fffffffu;
            if (kXY && along_x) {
              atomicMax(mx + row[t], max(max(hi[0], hi[1]), max(hi[2], hi[3])));
            } else {
#pragma unroll
              for (int u = 0; u < 4; ++u) atomicMax(mx + col[t] + u, hi[u]);
            }
          }
        tc::named_sync(1, kProdThreads);
        // the slot of the plane after next: last read before this barrier, next written after the next one
        const int clear = slot == 0 ? 2 : slot - 1;
        if (ptid < 64) {
          reinterpret_cast<unsigned int*>(line_max[clear])[ptid] = 0u;
          e_line[par][pl][ptid] = line_exponent(mx[ptid]);
        }
        slot = slot == 2 ? 0 : slot + 1;
        uint8_t* vp = V + pl * kTile;
        // the next plane's values are loaded piece by piece as this one's are sliced
        if (pl == 1) w.next();
        const double* next = plane_ptr(w, pl ^ 1);
#pragma unroll
        for (int t = 0; t < kMaxItems; ++t) {
          if (cnt[t] > 0) {
            uint4 h;
            if (kXY && along_x) {
              h.x = h.y = h.z = h.w = mx[row[t]];
            } else {
              h = reinterpret_cast<const uint4*>(mx)[col[t] >> 2];
            }
            const unsigned int hs[4] = {h.x, h.y, h.z, h.w};
            Digits f[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) f[u] = digits_of(x[t][u], max((int)(hs[u] >> 20), 1));
            uint8_t* dst = vp + quad_offset64(row[t], col[t]);
            // slice k, the most significant first
            auto put = [&](int k, uint32_t lo, uint32_t hi) {
              *reinterpret_cast<uint2*>(dst + k * kPair) = make_uint2(lo, hi);
            };
            put(0, slice2<3>(f[0].hi, f[1].hi), slice2<3>(f[2].hi, f[3].hi));
            put(1, slice2<2>(f[0].hi, f[1].hi), slice2<2>(f[2].hi, f[3].hi));
            put(2, slice2<1>(f[0].hi, f[1].hi), slice2<1>(f[2].hi, f[3].hi));
            put(3, slice2<0>(f[0].hi, f[1].hi), slice2<0>(f[2].hi, f[3].hi));
            put(4, slice2<3>(f[0].lo, f[1].lo), slice2<3>(f[2].lo, f[3].lo));
            put(5, slice2<2>(f[0].lo, f[1].lo), slice2<2>(f[2].lo, f[3].lo));
            put(6, slice2<1>(f[0].lo, f[1].lo), slice2<1>(f[2].lo, f[3].lo));
            put(7, slice2<0>(f[0].lo, f[1].lo), slice2<0>(f[2].lo, f[3].lo));
          }
          load_piece(t, next);
        }
      }
      tc::fence_smem_to_async();
      tc::mbar_arrive(&v_full);
    }
  } else if (lane == 0) {
    // ---- MMA issue ----
    const uint32_t tb = tc::smem_u32(sm), vb = tc::smem_u32(V);
    // A = a slice of the pair: M = (p, x) over the rows (MN-major, the planes kTile
    // apart) or M = (p, row) along x (K-major, 128 rows); B = T slices stacked along N
    const uint64_t a_rows = tc::sw128_mn_desc(vb, kTile, 1024u), a_x = tc::sw128_desc(vb), b0 = tc::sw128_desc(tb);
    // 16-wide steps of the contractions that hold data (the rest is zero padding)
    const int ks_rows = (pg.rows() + 15) / 16, ks_x = (a.nx + 15) / 16;
    if (!tc::mbar_wait(&t_ready, 0u)) failed = 1;
    int it = 0;
    for (Items64<kXY> w = first; w.more() && !failed; w.next(), ++it) {
      const uint32_t par = (uint32_t)it & 1u;
      if (!tc::mbar_wait(&v_full, par)) {
        failed = 1;
        break;
      }
      // Class c of a half accumulates in its columns [32 c, 32 c + 32).  The MMA of
      // v's slice k stacks T's slices 0 .. 7 - k along N and starts at class k, so
      // that product (k, l) goes into class k + l; slice 0 sets every class.
      const bool x = kXY && w.along_x;
      const uint64_t a0 = x ? a_x : a_rows;
      const uint32_t astep = x ? 32u / 16u : 2048u / 16u, major = x ? 0u : tc::kIdescAMajorMN;
      const int ks = x ? ks_x : ks_rows;
#pragma unroll 1
      for (uint32_t half = 0; half < 2; ++half) {
        if (!tc::mbar_wait(&acc_empty[half], par ^ 1u)) {
          failed = 1;
          break;
        }
        tc::fence_after_sync();
        tc::mbar_arrive(&e_full[half]);
        const uint64_t bd = b0 + half * (kS * kHalfTile / 16u);
#pragma unroll
        for (int k = 0; k < kS; ++k)
          for (int i = 0; i < ks; ++i)
            tc::mma_f16(tmem + half * kAccCols + 32u * k, a0 + (uint32_t)k * (kPair / 16u) + (uint32_t)i * astep,
                        bd + (uint32_t)i * 2u, tc::idesc_f16(128, 32 * (kS - k)) | major, (k == 0 && i == 0) ? 0u : 1u);
        if (half) tc::mma_commit(&v_empty);
        tc::mma_commit(&acc_full[half]);
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (failed && tid == 0) a.status[3] = 1;
  if (warp == kMmaWarp) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 2 * kAccCols);
  }
  if (failed) poison<kXY>(a, first);
}

// x and y contractions: out(y, x) = Ty v, then + Tx v
__global__ void __launch_bounds__(kThreads64, 1) k_kin_xy_tc64(Kin64 a) { kin64_body<true>(a); }
// z contraction added: out(z, x) += Tz v
__global__ void __launch_bounds__(kThreads64, 1) k_kin_z_tc64(Kin64 a) { kin64_body<false>(a); }

constexpr size_t kSmem64 = 1024 + kS * kTile + kS * kPair;
static_assert(kSmem64 + 3072 <= 227 * 1024, "the T tiles and the stage must fit in one CTA's shared memory");
static_assert(2 * kAccCols <= 512, "the accumulator must fit in tensor memory");

uint16_t half_bits(int x) {
  const __half h = __float2half_rn((float)x);
  uint16_t u;
  std::memcpy(&u, &h, 2);
  return u;
}

}  // namespace

// The eight 9-bit slices of a symmetric T, [half][slice] (71 bits below 2^e_t > max|T|, digits in
// [-256, 256]) as the kernels' shared-memory T region.  False when a class sum
// that has to be exact (0-6) could come near 2^24 for some v: 256 times the sum
// of |digit| over a row and the slices up to the class's above 15 2^20.  The
// sinc-DVR matrices up to 64 points reach 0.8 of 2^24, and 2^22 in class 1.
bool kinetic_smem_image64(const std::vector<double>& T, int n, std::vector<uint16_t>* image, int* e_t) {
  double m = 0.0;
  for (double x : T) m = std::max(m, std::fabs(x));
  int e = 0;
  if (m > 0.0) std::frexp(m, &e);
  *e_t = e;
  image->assign((size_t)kS * kTile / 2, half_bits(0));
  const __int128 bias = ((__int128)kBias36 << 36) + kBias36;
  long long most = 0, first = 0;
  for (int i = 0; i < n; ++i) {
    long long row = 0, two = 0;
    for (int q = 0; q < n; ++q) {
      const __int128 f = bias + (__int128)std::nearbyint(std::ldexp(T[(size_t)i * n + q], 71 - e));
      for (int l = 0; l < kS; ++l) {
        const int digit = kS - 1 - l;
        const int b = (int)((f >> (9 * digit)) & (digit == kS - 1 ? 0x3ff : 0x1ff)) - 256;
        if (l < kS - 1) row += std::abs(b);
        if (l < 2) two += std::abs(b);
        const int half = i >= half_rows(n), r = i - half * half_rows(n);
        const size_t byte = (size_t)(half * kS + l) * kHalfTile + (size_t)r * 128 +
                            (size_t)(((q >> 3) ^ (r & 7)) << 4) + (size_t)(q & 7) * 2;
        (*image)[byte / 2] = half_bits(b);
      }
    }
    most = std::max(most, row);
    first = std::max(first, two);
  }
  return 256 * most <= 15ll << 20 && 256 * first < 4000000;
}

int launch_kin_tc64(bsl_handle* h, const double* v, bool xy, cudaStream_t s) {
  const Tables& t = h->t;
  DeviceState& d = h->d;
  Kin64 a{};
  a.t = xy ? d.tx : d.tz;
  a.v = v;
  a.out = d.ukin;
  a.nx = t.nx;
  a.ny = t.ny;
  a.nz = t.nz;
  a.status = d.status;
  a.timage = reinterpret_cast<const uint4*>(xy ? d.kxy_slices64 : d.kz_slices64);
  a.timage16 = (int)(kS * kTile / 16);
  a.e_t = xy ? d.e_txy64 : d.e_tz64;
  a.nplanes = (xy ? t.nz : t.ny) * t.nn;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const dim3 grid(std::min((a.nplanes + 1) / 2, std::max(1, sms)));
  if (xy) {
    cudaFuncSetAttribute(k_kin_xy_tc64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem64);
    BSL_CUDA(launch_pdl(k_kin_xy_tc64, grid, dim3(kThreads64), kSmem64, s, a));
  } else {
    cudaFuncSetAttribute(k_kin_z_tc64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem64);
    BSL_CUDA(launch_pdl(k_kin_z_tc64, grid, dim3(kThreads64), kSmem64, s, a));
  }
  return BSL_OK;
}

}  // namespace bsl
