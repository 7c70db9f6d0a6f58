// Sinc-DVR kinetic contractions on the fifth-generation tensor cores
// (tcgen05.mma kind::f16, accumulators in tensor memory), sm_103a, with
// exact accumulation.
//
// Reference: Tv_5D_oneCompositeIndex / Mv_5D_oneCompositeIndex,
// Hv-calculators/linRotor/cartSphBasis/HvCalc/linRotCartSphHvRoutines.cpp:1807-1969.
//
// Work unit: a pair of planes.  The accumulator D has M = 128 rows (p, x) --
// plane p of the pair, grid column x -- and N = 64 columns (the other in-plane
// index), K = 64 per contraction:
//   x and y, planes (y, x) of fixed (s, z); both directions
//     accumulate into the same D[(p, x)][y]:
//       y:  sum_q v_p(q, x) Ty[y][q]      A = v tile read MN-major, B = T
//       x:  sum_q Tx[x][q] v_p(y, q)      A = diag(Tx, Tx) over K = (p', q), B = v tile
//     (the block-diagonal A is two 128-row tiles [T; 0] and [0; T] made from the
//     T tile and zero tiles laid out around it);
//   z, planes (z, x) of fixed (s, y):
//       sum_q v_p(q, x) Tz[z][q]           A = v tile read MN-major, B = T
// k_kin_tc<kXY> forms the first and k_kin_tc<kZ> adds the second to it; small
// problems take k_kin_tc<kAll>, which forms both in one launch and leaves the z
// part in a buffer of its own for the apply to add (kin_tc_one_launch).
// Every v tile is stored once, row by row as it lies in memory (64 FP16 per
// 128-byte swizzled row), and read by both terms; the output rows of D are
// grid columns, so the epilogue's stores are coalesced along x.
//
// Exactness (error-free slicing after Ozaki, Ogita, Oishi and Rump,
// Numer. Algorithms 59, 2012, here with 9-bit fixed-point slices): each plane
// of the double-float Lanczos vector is scaled by a power of two to below 1 in
// magnitude and cut into four 9-bit signed integer slices,
// v = 2^(e - 8) (a1 + 2^-9 a2 + 2^-18 a3 + 2^-27 a4) (36 bits relative to the
// plane's maximum); T is scaled from its largest element and cut the same way,
// rounded to nearest so that the symmetric T stays exactly symmetric.  The
// slices are integers in [-256, 256], exact in FP16, their products are exact,
// and the products of each scale class k + l <= 3 (10 products) share one
// accumulator.  A class sum is bounded by 2 * sum_{k+l=c} 256 max_x sum_q |b_l[x][q]|,
// below 2^23.6 for the sinc-DVR T (its first slice decays as 1/(x - q)^2), so
// the FP32 accumulation in tensor memory is exact whatever its internal
// rounding.  The four classes are combined on the CUDA cores into a
// double-float pair.
//
// Pipeline: one persistent CTA per SM with three roles.  Eight producer warps
// load a plane pair, find each plane's scale and write the slices into one of
// two 64 KiB shared-memory stages; one thread issues the pair's 72 (x/y) or
// 16 (z) MMAs into one of two 256-column accumulator stages; eight epilogue
// warps read the finished accumulators and store (x/y) or add (z) the
// double-float results.  mbarriers hand the stages over; every wait is bounded
// and a timeout sets status[3].
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "bsl_device.cuh"
#include "bsl_internal.h"
#include "bsl_slices.cuh"
#include "bsl_tc.cuh"

namespace bsl {
namespace {

constexpr uint32_t kTile = 64 * 128;          // 8 KiB: 64 rows x 64 FP16, one 128-byte swizzled row each
constexpr uint32_t kPlaneSlices = kVS * kTile;  // the v slices of one plane, contiguous
constexpr uint32_t kStage = 2 * kPlaneSlices;   // v slices of a plane pair: [plane][slice] tiles
constexpr int kStages = 2;                    // shared-memory stages and accumulator stages
constexpr uint32_t kAccCols = 4 * 64;         // accumulator columns of one pair (classes 0..3)
constexpr int kEpiWarps = 8;                  // warps 0-7
constexpr int kProdWarps = 8;                 // warps 8-15
constexpr int kMmaWarp = kEpiWarps + kProdWarps;  // warp 16: MMA issue and tensor-memory owner
constexpr int kWsThreads = (kMmaWarp + 1) * 32;
constexpr int kProdThreads = kProdWarps * 32;
constexpr int kEpiThreads = kEpiWarps * 32;
constexpr int kMaxItems = 64 * 16 / kProdThreads;  // (row, 4-column group) items per producer thread

struct KinTC {
  const uint4* timage;      // the T tiles as laid out in shared memory: Z T0 .. T3 Z (x/y), then Tz unless it is the same
  int timage16;             // its size in 16-byte units
  int tz_tile;              // first tile of Tz's slices
  int e_txy, e_tz;          // T = 2^(e_t - 8) (b1 + 2^-9 b2 + 2^-18 b3 + 2^-27 b4)
  const float2* v;          // the Lanczos v as double-float pairs
  float2 *out_xy, *out_z;   // Tx v + Ty v; Tz v
  int nx, ny, nz, nn;
  int* status;
  int nslices;              // slices of v and of T kept (1-4; 4 = exact), classes k + l < nslices
  // graph-replayed iterations: the first CTA's epilogue warps finish the previous
  // update's deferred beta (null: nothing deferred)
  double* fin_partials;
  double* scalars;
  double* hist;
  int* jdev;
  int fin_count, hist_stride;
};

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~(uintptr_t)1023);
}

// byte offset of element k (a multiple of 4) of row r in an SW128 tile of 64 FP16 per row
__device__ __forceinline__ uint32_t quad_offset(int r, int k) {
  return (uint32_t)(r * 128 + (((k >> 3) ^ (r & 7)) << 4) + ((k & 7) << 1));
}

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// the four class accumulators of 8 consecutive columns as double-float pairs
// times `scale` (combine_classes).  With fewer than four slices the classes at
// and above `nslices` were never written and are taken as zero.
__device__ __forceinline__ void load_pairs8(uint32_t taddr, float scale, int nslices, float2 (&out)[8]) {
  float c0[8], c1[8], c2[8], c3[8];
  tc::tmem_ld8_nowait(taddr, c0);
  tc::tmem_ld8_nowait(taddr + 64u, c1);
  tc::tmem_ld8_nowait(taddr + 128u, c2);
  tc::tmem_ld8_nowait(taddr + 192u, c3);
  tc::tmem_wait_ld();
  if (nslices < 4) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      c3[u] = 0.f;
      c2[u] = nslices > 2 ? c2[u] : 0.f;
      c1[u] = nslices > 1 ? c1[u] : 0.f;
    }
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) out[u] = combine_classes(c0[u], c1[u], c2[u], c3[u], scale);
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Plane geometry: x/y planes are the contiguous (y, x) planes of fixed (s, z);
// z planes are the (z, x) planes of fixed (s, y), rows nx * ny apart.
struct Planes {
  int nx, ny, nz, nxy, nzx;  // nxy, nzx: planes of x/y and z
  __device__ __forceinline__ int count(int z) const { return z ? nzx : nxy; }
  __device__ __forceinline__ long long base(int z, int plane) const {
    if (!z) return (long long)plane * nx * ny;
    return (long long)(plane / ny) * nz * nx * ny + (long long)(plane % ny) * nx;
  }
  __device__ __forceinline__ int row_stride(int z) const { return z ? nx * ny : nx; }
  __device__ __forceinline__ int rows(int z) const { return z ? nz : ny; }
};

// The CTA's work items: the x/y and the z plane pair p of every p = first, first
// + stride, ... below end, in turn (x/y pairs keep the tensor core busy, z pairs
// the producers).
template <int kKinds>
struct Items {
  int pair, z;  // z: 0 an x/y pair, 1 a z pair
  int stride, end;
  const Planes& pg;
  __device__ __forceinline__ Items(const Planes& g, int first, int st, int e)
      : pair(first),
        z(kKinds == 2),
        stride(st),
        end(min(e, ((kKinds == 3 ? max(g.nxy, g.nzx) : g.count(kKinds == 2)) + 1) / 2)),
        pg(g) {
    skip();
  }
  __device__ __forceinline__ bool more() const { return pair < end; }
  __device__ __forceinline__ void skip() {  // to the next pair that exists
    while (pair < end && 2 * pair >= pg.count(z)) step();
  }
  __device__ __forceinline__ void step() {
    if (kKinds != 3 || z) pair += stride;
    if (kKinds == 3) z ^= 1;
  }
  __device__ __forceinline__ void next() {
    step();
    skip();
  }
};

// What a launch forms: the x/y contractions, the z contraction added to them, or
// all three with the z part in a buffer of its own (the apply adds it).
enum Kinds { kXY = 1, kZ = 2, kAll = 3 };
// T tiles in shared memory: Z T0 T1 T2 T3 Z of x/y, the slices of Tz, or both
__host__ __device__ constexpr int t_tiles(int kinds) { return kinds == kXY ? kTS + 2 : kinds == kZ ? kTS : 2 * kTS + 2; }

// After a time-out: NaN in the planes of the CTA's items, so that an H v whose
// caller does not read the status words (bsl_hv_apply_device) cannot be taken
// for a result.
template <int kKinds>
__device__ __forceinline__ void poison(const KinTC& a) {
  pdl_wait();
  const Planes pg{a.nx, a.ny, a.nz, a.nz * a.nn, a.ny * a.nn};
  for (Items<kKinds> w(pg, blockIdx.x, gridDim.x, 1 << 30); w.more(); w.next())
    for (int e = threadIdx.x; e < 2 * pg.rows(w.z) * a.nx; e += blockDim.x) {
      const int row = e / a.nx, pl = row >= pg.rows(w.z), plane = 2 * w.pair + pl;
      if (plane < pg.count(w.z))
        (w.z ? a.out_z : a.out_xy)[pg.base(w.z, plane) + (long long)(row - pl * pg.rows(w.z)) * pg.row_stride(w.z) +
                                   e % a.nx] = make_float2(__int_as_float(0x7fc00000), 0.f);
    }
}

// whether the CTA did its items (false after a time-out)
template <int kKinds>
__device__ __forceinline__ bool kin_ws_body(const KinTC& a, int p_first, int p_stride, int p_end) {
  extern __shared__ uint8_t smraw[];
  uint8_t* sm = align1024(smraw);
  uint8_t* V = sm + t_tiles(kKinds) * kTile;
  __shared__ uint64_t v_full[kStages], v_empty[kStages], acc_full[kStages], acc_empty[kStages], e_full[kStages];
  __shared__ uint64_t stages_zeroed, t_ready;  // setup by the epilogue warps
  __shared__ uint32_t tmem_slot;
  __shared__ int e_stage[kStages][2], e_acc[kStages][2];
  __shared__ float red[2][kProdWarps];
  __shared__ int prod_go, failed, skip;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Planes pg{a.nx, a.ny, a.nz, a.nz * a.nn, a.ny * a.nn};

  // a kinetic time-out recorded before this launch (an earlier launch of the
  // run, or the host's injection) makes the CTA leave before it allocates
  // tensor memory, loads, issues an MMA or waits; one thread reads the flag so
  // that the whole CTA takes the same branch
  if (tid == 0) skip = *(volatile int*)(a.status + 3);
  __syncthreads();
  if (skip) return false;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(&v_full[s], kProdThreads);
      tc::mbar_init(&v_empty[s], 1);
      tc::mbar_init(&acc_full[s], 1);
      tc::mbar_init(&acc_empty[s], kEpiThreads);
      tc::mbar_init(&e_full[s], 1);
    }
    tc::mbar_init(&stages_zeroed, kEpiThreads);
    tc::mbar_init(&t_ready, kEpiThreads);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) tc::tmem_alloc(&tmem_slot, kStages * kAccCols);
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
    {  // setup while the producers' first planes are in flight: zeroed v stages
       // (the producers write only the rows and 4-column groups that hold data,
       // so the padding of every stage stays zero), then the T tiles (a
       // prebuilt image of that region) for the MMA thread
      for (int e = tid; e < (int)(kStages * kStage / 16); e += kEpiThreads)
        reinterpret_cast<uint4*>(V)[e] = make_uint4(0u, 0u, 0u, 0u);
      tc::fence_smem_to_async();
      tc::mbar_arrive(&stages_zeroed);
      constexpr int kBatch = 6;
      for (int e0 = tid; e0 < a.timage16; e0 += kBatch * kEpiThreads) {
        uint4 img[kBatch];
#pragma unroll
        for (int r = 0; r < kBatch; ++r) {
          const int e = e0 + r * kEpiThreads;
          img[r] = e < a.timage16 ? a.timage[e] : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int r = 0; r < kBatch; ++r) {
          const int e = e0 + r * kEpiThreads;
          if (e < a.timage16) reinterpret_cast<uint4*>(sm)[e] = img[r];
        }
      }
      tc::fence_smem_to_async();
      tc::mbar_arrive(&t_ready);
    }
    pdl_wait();  // the output (and, for z alone, the values added to) belong to earlier kernels
    if (kKinds != kZ && a.fin_partials && p_first == 0) {
      __shared__ double fin8[kEpiWarps];
      finish_deferred_beta(a.fin_partials + kBetaPartials, a.fin_count, a.scalars, a.hist, a.hist_stride, a.jdev,
                           a.status, tid, kEpiThreads, 2, fin8);
    }
    int it = 0;
    for (Items<kKinds> w(pg, p_first, p_stride, p_end); w.more(); w.next(), ++it) {
      const int st = it & 1;
      const uint32_t par = (uint32_t)(it >> 1) & 1u;
      const int plane = 2 * w.pair + p;
      const bool valid = plane < pg.count(w.z) && x < a.nx;
      float2* out = (w.z ? a.out_z : a.out_xy) + (valid ? pg.base(w.z, plane) + x : 0);
      const long long cstride = pg.row_stride(w.z);
      const int c_begin = half * 32, c_end = min(half * 32 + 32, pg.rows(w.z));
      float2 nxt[8];  // z alone: the values added to, the first chunk loaded while the products run
      auto load8 = [&](int c0) {
#pragma unroll
        for (int u = 0; u < 8; ++u) nxt[u] = (valid && c0 + u < c_end) ? out[(c0 + u) * cstride] : make_float2(0.f, 0.f);
      };
      if (kKinds == kZ) load8(c_begin);
      // lane 0 waits (bounded) and the warp leaves together on a timeout; once the
      // phases are complete every lane's own wait returns at once and orders its
      // reads after the producers' and the MMA thread's writes
      int ok = 1;
      if (lane == 0) ok = tc::mbar_wait(&acc_full[st], par) && tc::mbar_wait(&e_full[st], par);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) {
        failed = 1;
        break;
      }
      tc::mbar_wait(&acc_full[st], par);
      tc::mbar_wait(&e_full[st], par);
      tc::fence_after_sync();
      const float scale = pow2f(e_acc[st][p] + (w.z ? a.e_tz : a.e_txy) - 16);
      const uint32_t tbase = tmem + (uint32_t)st * kAccCols + lane_base;
#pragma unroll 1
      for (int c0 = c_begin; c0 < c_end; c0 += 8) {
        float2 v[8], cur[8];
        if (kKinds == kZ) {
#pragma unroll
          for (int u = 0; u < 8; ++u) cur[u] = nxt[u];
          if (c0 + 8 < c_end) load8(c0 + 8);  // the next chunk, in flight meanwhile
        }
        load_pairs8(tbase + (uint32_t)c0, scale, a.nslices, v);
        if (valid)
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (c0 + u < c_end) out[(c0 + u) * cstride] = kKinds == kZ ? df_add_fast(cur[u], v[u]) : v[u];
      }
      tc::fence_before_sync();
      tc::mbar_arrive(&acc_empty[st]);
    }
  } else if (warp < kMmaWarp) {
    // ---- producers: piece i = (row i / ncg, 4-column group i % ncg) of a plane,
    // pieces ptid, ptid + 256, ...; the next plane's pieces are loaded into
    // registers while this one is sliced.  With both kinds the rows run to the longer
    // of y and z: those beyond a plane's own are written as zeros ----
    const int ptid = tid - kEpiThreads, pw = ptid >> 5;
    const int nx = a.nx, ncg = (nx + 3) >> 2, nrows = kKinds == kAll ? max(a.ny, a.nz) : pg.rows(kKinds == kZ);
    const int npieces = nrows * ncg;
    int row[kMaxItems], col[kMaxItems], cnt[kMaxItems];
    uint32_t soff[kMaxItems];
#pragma unroll
    for (int t = 0; t < kMaxItems; ++t) {
      const int i = ptid + t * kProdThreads;
      const int j = i / ncg, c = (i - j * ncg) * 4;
      const bool iv = i < npieces;
      row[t] = iv ? j : 0;
      col[t] = iv ? (kKinds == kAll ? c : j * pg.row_stride(kKinds == kZ) + c) : 0;  // one kind: the whole offset
      soff[t] = iv ? quad_offset(j, c) : 0u;
      cnt[t] = iv ? min(4, nx - c) : 0;
    }
    auto load_plane = [&](const Items<kKinds>& w, int pl, float2 (&x)[kMaxItems][4]) {
      const int plane = 2 * w.pair + pl;
      const bool pv = w.more() && plane < pg.count(w.z);
      const float2* src = a.v + (pv ? pg.base(w.z, plane) : 0);
      const int rs = pg.row_stride(w.z), rows = pg.rows(w.z);
#pragma unroll
      for (int t = 0; t < kMaxItems; ++t) {
        const float2* q = src + (kKinds == kAll ? row[t] * rs + col[t] : col[t]);
        const int n = pv && (kKinds != kAll || row[t] < rows) ? cnt[t] : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) x[t][u] = u < n ? __ldg(q + u) : make_float2(0.f, 0.f);
      }
    };
    float2 x[kMaxItems][4];
    pdl_wait();  // v is written by the previous iteration's update
    Items<kKinds> w(pg, p_first, p_stride, p_end);
    load_plane(w, 0, x);  // in flight during the setup
    int slot = 0;
    for (int it = 0; w.more(); ++it) {
      const int st = it & 1;
      const uint32_t par = (uint32_t)(it >> 1) & 1u;
      if (ptid == 0)
        prod_go = ((it > 0 || tc::mbar_wait(&stages_zeroed, 0u)) && tc::mbar_wait(&v_empty[st], par ^ 1u)) ? 1 : 0;
      tc::named_sync(1, kProdThreads);
      if (!prod_go) {
        if (ptid == 0) failed = 1;
        break;
      }
      if (kKinds != kAll) {  // the pair after next into L2, one 16-value row segment per thread
        const int j = ptid >> 2, i = (ptid & 3) * 16;
#pragma unroll
        for (int pl = 0; pl < 2; ++pl) {
          const int far = 2 * (w.pair + 2 * p_stride) + pl;
          if (far < pg.count(w.z) && j < pg.rows(w.z) && i < nx)
            prefetch_l2(a.v + pg.base(w.z, far) + j * pg.row_stride(w.z) + i);
        }
      }
      uint8_t* vs = V + st * kStage;
#pragma unroll 1
      for (int pl = 0; pl < 2; ++pl) {
        float2 y[kMaxItems][4];  // the next plane, in flight while this one is sliced
        if (pl == 1) w.next();
        load_plane(w, pl ^ 1, y);
        float mx = 0.f;
#pragma unroll
        for (int t = 0; t < kMaxItems; ++t)
#pragma unroll
          for (int u = 0; u < 4; ++u) mx = fmaxf(mx, fabsf(x[t][u].x));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) red[slot][pw] = mx;
        tc::named_sync(1, kProdThreads);
#pragma unroll
        for (int r = 0; r < kProdWarps; ++r) mx = fmaxf(mx, red[slot][r]);
        slot ^= 1;
        const int e = plane_exponent(mx);
        if (ptid == 0) e_stage[st][pl] = e;
        const float sc = pow2f(8 - e);
        uint8_t* vp = vs + pl * kPlaneSlices;
#pragma unroll
        for (int t = 0; t < kMaxItems; ++t) {
          if (cnt[t] > 0) {
            float sl[4][kVS];
#pragma unroll
            for (int u = 0; u < 4; ++u) slice4(__fmul_rn(x[t][u].x, sc), __fmul_rn(x[t][u].y, sc), sl[u]);
#pragma unroll
            for (int k = 0; k < kVS; ++k)
              if (k < a.nslices)
                *reinterpret_cast<uint2*>(vp + k * kTile + soff[t]) =
                  make_uint2(pack_h2(sl[0][k], sl[1][k]), pack_h2(sl[2][k], sl[3][k]));
          }
        }
#pragma unroll
        for (int t = 0; t < kMaxItems; ++t)
#pragma unroll
          for (int u = 0; u < 4; ++u) x[t][u] = y[t][u];
      }
      tc::fence_smem_to_async();
      tc::mbar_arrive(&v_full[st]);
    }
  } else if (lane == 0) {
    // ---- MMA issue ----
    const uint32_t tb = tc::smem_u32(sm);
    if (!tc::mbar_wait(&t_ready, 0u)) failed = 1;
    int it = 0;
    for (Items<kKinds> w(pg, p_first, p_stride, p_end); w.more() && !failed; w.next(), ++it) {
      const int st = it & 1;
      const uint32_t par = (uint32_t)(it >> 1) & 1u;
      if (!tc::mbar_wait(&v_full[st], par) || !tc::mbar_wait(&acc_empty[st], par ^ 1u)) {
        failed = 1;
        break;
      }
      tc::fence_after_sync();
      e_acc[st][0] = e_stage[st][0];
      e_acc[st][1] = e_stage[st][1];
      tc::mbar_arrive(&e_full[st]);
      const uint32_t d0 = tmem + (uint32_t)st * kAccCols;
      const uint32_t vb = tc::smem_u32(V + st * kStage);
      // Class c accumulates in columns [64 c, 64 c + 64).  An MMA whose B stacks
      // the slices l = 0 .. ns - 1 - k of one operand along N (rows 64 l ..) and
      // whose D starts at column 64 k puts product (k, l) into class k + l
      // (ns = 4 slices, the exact default: classes 0..3, 10 products).
      // Contraction over the rows of each plane (y for x/y, z for z): A = v
      // slice k (M = (p, x), MN-major, the planes kPlaneSlices apart), B = T
      // slices 0 .. ns - 1 - k; 16 rows (2 KiB) per K step.  The first MMA
      // (k = 0, N = 64 ns) sets every class.
      const uint32_t t0 = tb + kTile, tr = kKinds == kZ ? tb : w.z ? tb + (uint32_t)a.tz_tile * kTile : t0;
      const int ns = a.nslices;
#pragma unroll 1
      for (int k = 0; k < ns; ++k) {
        const uint32_t idesc = tc::idesc_f16(128, 64 * (ns - k)) | tc::kIdescAMajorMN;
#pragma unroll
        for (int s = 0; s < 4; ++s)
          tc::mma_f16(d0 + (uint32_t)k * 64u,
                      tc::sw128_mn_desc(vb + (uint32_t)k * kTile + (uint32_t)s * 2048u, kPlaneSlices, 1024u),
                      tc::sw128_desc(tr + (uint32_t)s * 32u), idesc, (k == 0 && s == 0) ? 0u : 1u);
      }
      if (kKinds != kZ && !w.z) {
        // contraction along x: A = diag(T_l, T_l) over K = (p', q), read MN-major
        // (T is symmetric) with its two 64-row blocks chosen by the start address
        // and the block stride: [T_l; 0] = (T_l, the zero tile above) and
        // [0; T_l] = (the zero tile below, T_l); B = v slices 0 .. 3 - l of plane p'
        // stacked along N
        const uint32_t zlo = tb, zhi = tb + (uint32_t)(kTS + 1) * kTile;
#pragma unroll 1
        for (int l = 0; l < ns; ++l) {
          const uint32_t tl = t0 + (uint32_t)l * kTile;
          const uint32_t idesc = tc::idesc_f16(128, 64 * (ns - l)) | tc::kIdescAMajorMN;
#pragma unroll
          for (int s = 0; s < 8; ++s) {
            const uint32_t pp = (uint32_t)(s >> 2), q = (uint32_t)(s & 3);
            const uint64_t adesc = pp ? tc::sw128_mn_desc(zlo + q * 2048u, tl - zlo, 1024u)
                                      : tc::sw128_mn_desc(tl + q * 2048u, zhi - tl, 1024u);
            tc::mma_f16(d0 + (uint32_t)l * 64u, adesc, tc::sw128_desc(vb + pp * kPlaneSlices + q * 32u), idesc, 1u);
          }
        }
      }
      tc::mma_commit(&v_empty[st]);
      tc::mma_commit(&acc_full[st]);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (failed && tid == 0) a.status[3] = 1;
  if (warp == kMmaWarp) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, kStages * kAccCols);
  }
  return !failed;
}

template <int kKinds>
__global__ void __launch_bounds__(kWsThreads, 1) k_kin_tc(const __grid_constant__ KinTC a) {
  if (kin_ws_body<kKinds>(a, blockIdx.x, gridDim.x, 1 << 30)) return;
  const KinTC* again = &a;  // read anew: nothing is kept in registers for a time-out
  asm volatile("" : "+l"(again));
  poison<kKinds>(*again);
}

// Grouped launch over several problems (each with its own grid, T image and
// vectors): CTA c works on problem work[c].x, pairs [work[c].y, work[c].z).
template <int kKinds>
__global__ void __launch_bounds__(kWsThreads, 1) k_kin_tc_group(const KinTC* __restrict__ probs,
                                                                 const int4* __restrict__ work) {
  const int4 w = work[blockIdx.x];
  const KinTC a = probs[w.x];
  kin_ws_body<kKinds>(a, w.y, 1, w.z);
}

constexpr size_t smem_bytes(int kinds) { return 1024 + (size_t)t_tiles(kinds) * kTile + kStages * kStage; }
static_assert(smem_bytes(kAll) + 512 <= 227 * 1024, "the T tiles and the stages must fit in one CTA's shared memory");
static_assert(kStages * kAccCols <= 512, "the accumulator stages must fit in tensor memory");

int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return std::max(1, sms);
}

uint16_t half_bits(float x) {  // FP16 bits of a small integer (|x| <= 2048: exact)
  const __half h = __float2half_rn(x);
  uint16_t u;
  std::memcpy(&u, &h, 2);
  return u;
}

}  // namespace

// Fixed-point FP16 slices of an n x n kinetic matrix, T = 2^(e_t - 8) (b1 +
// 2^-9 b2 + 2^-18 b3 + 2^-27 b4) + O(2^(e_t - 36)), each b an integer in
// [-256, 256] rounded to nearest (a symmetric T stays symmetric), as the bytes
// of the kernels' shared-memory T region: tiles of 64 rows (output index) x 64
// FP16 (contraction index), zero padded, 128-byte rows with 16-byte chunk c of
// row r at chunk c ^ (r % 8); with_zero_tiles adds a zero tile before and after
// the four slice tiles (the x/y layout).
void kinetic_smem_image(const std::vector<double>& T, int n, bool with_zero_tiles, std::vector<uint16_t>* image,
                        int* e_t) {
  double m = 0.0;
  for (double x : T) m = std::max(m, std::fabs(x));
  int e = 0;
  if (m > 0.0) std::frexp(m, &e);  // m = f 2^e, f in [0.5, 1)
  *e_t = e;
  const int first = with_zero_tiles ? 1 : 0, ntiles = kTS + 2 * first;
  image->assign((size_t)ntiles * kTile / 2, half_bits(0.f));
  for (int i = 0; i < n; ++i)
    for (int q = 0; q < n; ++q) {
      double r = std::ldexp(T[(size_t)i * n + q], 8 - e);
      for (int l = 0; l < kTS; ++l) {
        const double b = std::nearbyint(r);
        const size_t byte = (size_t)(first + l) * kTile + (size_t)i * 128 + (size_t)(((q >> 3) ^ (i & 7)) << 4) +
                            (size_t)(q & 7) * 2;
        (*image)[byte / 2] = half_bits((float)b);
        r = (r - b) * 512.0;
      }
    }
}

// The same slices as FP32 integers, [slice][i][q], for the small-grid kernel.
void kinetic_slices_f32(const std::vector<double>& T, int n, std::vector<float>* out) {
  double m = 0.0;
  for (double x : T) m = std::max(m, std::fabs(x));
  int e = 0;
  if (m > 0.0) std::frexp(m, &e);
  out->assign((size_t)kTS * n * n, 0.f);
  for (int i = 0; i < n * n; ++i) {
    double r = std::ldexp(T[i], 8 - e);
    for (int l = 0; l < kTS; ++l) {
      const double b = std::nearbyint(r);
      (*out)[(size_t)l * n * n + i] = (float)b;
      r = (r - b) * 512.0;
    }
  }
}

bool kinetic_tc_supported(const Tables& t) { return t.nx <= 64 && t.ny <= 64 && t.nz <= 64 && t.tx == t.ty; }

namespace {
// the kernel arguments of one problem's contractions of v (fin_count > 0: the
// launch finishes a deferred beta of that many block totals)
KinTC kin_tc_args(bsl_handle* h, const float2* v, int kinds, int fin_count) {
  const Tables& t = h->t;
  DeviceState& d = h->d;
  KinTC a{};
  a.v = v;
  a.out_xy = reinterpret_cast<float2*>(d.ukin);
  a.out_z = kinds == kAll ? d.ukin_z : a.out_xy;
  a.nx = t.nx;
  a.ny = t.ny;
  a.nz = t.nz;
  a.nn = t.nn;
  a.status = d.status;
  a.nslices = h->kin_slices;
  const int tile16 = (int)(kTile / 16);
  a.timage = reinterpret_cast<const uint4*>(d.kin_slices) + (kinds == kZ ? d.kin_tz_tile * tile16 : 0);
  a.timage16 = kinds == kAll ? d.kin_image16 : t_tiles(kinds) * tile16;
  a.tz_tile = d.kin_tz_tile;
  a.e_txy = d.e_txy;
  a.e_tz = d.e_tz;
  if (fin_count > 0) {
    a.fin_partials = d.partials;
    a.scalars = d.scalars;
    a.hist = d.hist;
    a.jdev = d.jdev;
    a.fin_count = fin_count;
    a.hist_stride = d.hist_cap;
  }
  return a;
}

long long pairs_of(const Tables& t, int kinds) {
  return ((long long)(kinds == kXY ? t.nz : kinds == kZ ? t.ny : std::max(t.nz, t.ny)) * t.nn + 1) / 2;
}

template <int kKinds>
int launch_kinds(bsl_handle* h, const float2* v, cudaStream_t s) {
  cudaFuncSetAttribute(k_kin_tc<kKinds>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(kKinds));
  const KinTC a = kin_tc_args(h, v, kKinds, kKinds != kZ && h->defer_reductions ? deferred_beta_count(h) : 0);
  BSL_CUDA(launch_pdl(k_kin_tc<kKinds>, dim3((unsigned)std::min<long long>(pairs_of(h->t, kKinds), sm_count())),
                      dim3(kWsThreads), smem_bytes(kKinds), s, a));
  BSL_CUDA(cudaGetLastError());
  return BSL_OK;
}
}  // namespace

// The shared-memory image of both matrices: Z T0 .. T3 Z of x and y, and the
// slices of Tz after it unless Tz is the same matrix (*tz_tile: its first tile).
void kinetic_tc_image(const Tables& t, std::vector<uint16_t>* image, int* tz_tile, int* e_txy, int* e_tz) {
  kinetic_smem_image(t.tx, t.nx, true, image, e_txy);
  if (t.tz == t.tx) {
    *tz_tile = 1;
    *e_tz = *e_txy;
    return;
  }
  *tz_tile = kTS + 2;
  std::vector<uint16_t> z;
  kinetic_smem_image(t.tz, t.nz, false, &z, e_tz);
  image->insert(image->end(), z.begin(), z.end());
}

size_t kin_group_arg_size() { return sizeof(KinTC); }

// the plane pairs of one problem's x/y or z contraction (the work units)
long long kin_tc_pairs(const bsl_handle* h, bool xy) { return pairs_of(h->t, xy ? kXY : kZ); }

// fill args[b] (kin_group_arg_size() bytes each) for the problems' vectors v[b]
void kin_tc_group_args(bsl_handle** hs, int n, const float2* const* v, bool xy, const int* fin_counts, void* args) {
  KinTC* a = static_cast<KinTC*>(args);
  for (int b = 0; b < n; ++b) a[b] = kin_tc_args(hs[b], v[b], xy ? kXY : kZ, fin_counts ? fin_counts[b] : 0);
}

int launch_kin_tc_group(bool xy, const void* d_args, const int4* d_work, int nctas, cudaStream_t s) {
  const auto kernel = xy ? k_kin_tc_group<kXY> : k_kin_tc_group<kZ>;
  const size_t smem = smem_bytes(xy ? kXY : kZ);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  BSL_CUDA(launch_pdl(kernel, dim3(nctas), dim3(kWsThreads), smem, s, static_cast<const KinTC*>(d_args), d_work));
  return BSL_OK;
}

// One launch up to 800,000 coefficients.  There a launch of either kind is a few
// plane pairs a CTA, so that setting up a CTA (tensor memory, the T tiles, the
// zeroed stages) and draining it are most of its 10-22 us, and one launch pays
// for them once; the z part, 8 bytes a coefficient more for the apply to read,
// stays in L2.  An iteration in one launch against two: 20^3 with 21 functions
// 34.2 against 39.3 us, 24^3 with 10 22.9 against 27.6, 27^3 with 21 36.7
// against 42.2, 33^3 with 15 35.1 against 38.7, with 21 45.1 against 50.5.
// Beyond, the z launch's setup is hidden behind the x/y launch's tail and the
// added bytes are not: 41^3 with 21 62.2 against 58.5 us, 54^3 113 against 88.
//
// Where x/y and z planes differ in number their launches overlap, and the apply of
// blocks without the fused iteration hides the added loads worse.  An iteration
// in one launch against two, us: 54x54x12 with 10 functions 32.6 against 31.9 (with 9
// 31.3 against 33.1), 48x48x16 with 21 49.9 against 46.0 and 27x27x41 45.3 against 44.3
// (40x40x10 39.5 against 40.6), 48x48x16 with 16 39.8 against 39.2 (30x30x10 30.9
// against 33.2), 40x40x10 with 28 51.0 against 49.2 (30^3 53.5 against 56.0); with 36
// functions 70.4 against 64.5 at 40x40x10.
bool kin_tc_one_launch(const bsl_handle* h) {
  const Tables& t = h->t;
  if (!h->d.ukin_z || !vstream_apart_supported(h->vformat, t.nn)) return false;
  if (t.nn <= 9 || t.nz == t.ny) return true;
  const long long size = t.npts * t.nn;
  if (fused_update_supported(h->vformat, t.nn)) return 4 * t.nz >= t.ny && size <= 600000;
  return t.nn <= 16 && (3 * t.nz > t.ny || size <= 400000);
}
bool kin_tc_small(const Tables& t) { return t.npts * t.nn <= 800000; }

int launch_kin_xy_tc(bsl_handle* h, const float2* v, cudaStream_t s) {
  return kin_tc_one_launch(h) ? launch_kinds<kAll>(h, v, s) : launch_kinds<kXY>(h, v, s);
}

int launch_kin_z_tc(bsl_handle* h, const float2* v, cudaStream_t s) {
  return kin_tc_one_launch(h) ? BSL_OK : launch_kinds<kZ>(h, v, s);
}

}  // namespace bsl
