// Density with the factored density matrix (sm_100a, tcgen05): P = L L^T of rank r, so that
// rho_i = sum_k (Phi L)_ik^2 needs r output columns instead of N and Phi' never leaves the SM.
//
// Phi' flows through a ring of small K-step slots instead of a whole resident tile, so the basis
// size is not limited by shared memory and nothing waits for a tile to end:
//
//   * the basis functions are grouped into units of 16 columns, one K-step of the MMA: a carbon-like
//     atom (14 functions) fills one, three hydrogen-like atoms (3 x 5) fill one, other shells are
//     packed in order.  The factor's rows are permuted to match (fact_split_kernel);
//   * a work item is one unit at 64 of the tile's 128 rows: a warp evaluates it in registers, two rows
//     per lane (packed FP32 pairs), and stores whole 16-byte units of hi and lo pieces into the slot
//     (32-byte swizzled K-major rows: eight lanes' 16-byte stores cover all 32 banks, so a store has no
//     bank conflict; the 4-byte stores of a layout in function order were 4-way conflicted and a
//     third of the production time);
//   * items are numbered across tiles and taken from one counter: the warps run ahead into the next
//     tiles as far as the ring and the positions allow, with no barrier among them;
//   * one thread streams the factor's K-step blocks (or loads them once when they fit beside the ring), two
//     warps issue the MMAs unit by unit (the large products and the small ones), one warp computes the tiles'
//     sample positions, and four warps run the epilogue of the previous tile from TMEM meanwhile.
//
// Split products: T = A_hi L_hi (main, "H") + A_hi L_lo + A_lo L_hi (small, "S"; with bf16 pieces also
// A_lo L_lo, 2^-16 of the main term), in separate accumulators: the tensor core's FP32 additions round toward
// zero by 2^-24 of the accumulator, so the small terms stay out of the large one's way, and the large ones take
// turns on up to three (fact_mol_desc): without rescaling N = 294 is 4e-7 off FP64 with three, 7e-7 with one, for
// 0.02 of 0.53 ms.
//
// Bound: the hand-over of K-steps (waits, commits, the issuing threads' serial code: ~420 clocks per
// unit with the MMAs, ~340 without production, ~370 without MMAs) and the producers' issue slots; DRAM
// idle, tensor pipe 20-45% busy.  Measured (B200, fp16x3, one call, before -> now; before: a resident
// Phi' tile per CTA for N <= 320 and rank <= 64, Phi' through HBM beyond, no factor past rank 128):
//   N = 294,  rank 59,  128^3 points:  1.48 -> 0.53 ms
//   N = 588,  rank 119, 192^3 points:  11.2 -> 4.0 ms
//   N = 1176, rank 238, 168^3 points:  42.9 -> 6.3 ms (the factor's 1.3 MB per tile from L2: 7.5 TB/s)
// Tried and dropped: pairing hi and lo factor rows in one MMA of N = 2 r16 (overlapping accumulators,
// +8%); one MMA-issuing lane outside a converged warp (~900 clocks per K-step); 16
// producer warps of 80 registers (same); 128-byte swizzled A reads (same).
//
// Replaces the per-voxel pair loop of gpu_densityqube_shmem_subgrid (kernel_density.cu:74-140).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>

#include "density_factored.cuh"
#include "sm100.cuh"

namespace qmt {
using namespace sm100;

namespace {

// Whose tiles a launch walks: one molecule's, several molecules', or one's whose rank only the device knows.
enum { ONE = 0, MANY = 1, ON_DEVICE = 2 };
enum { UNIT_GENERIC = 0, UNIT_S3S1P1 = 1, UNIT_S8S8S1P3P1D1 = 2 };

constexpr int NPW = 12;                        // producer warps
constexpr int FACT_THREADS = (8 + NPW) * 32;   // copy, 2 MMA warps, positions; 4 epilogue warps; producers
constexpr int GROUP = 2;                       // units per ring slot: one wait and one commit for both
constexpr int MIN_SLOTS = 4, MAX_SLOTS = 12;
constexpr int MIN_UNITS = 2;                   // units of a tile (a smaller molecule gets an empty one)
// Phase parities are read one round of the ring ahead at most: the producers hold at most NPW items
// that have not passed their waits (one a warp), and with at least 4 items a tile and 6 in any two
// consecutive groups these span at most NPW / 3 groups and NPW / 4 tiles past the ring.
constexpr int POS_DEPTH = 4;                   // tiles of sample positions in flight
static_assert(NPW <= 3 * MIN_SLOTS && NPW <= 4 * POS_DEPTH, "see above");
constexpr uint32_t PIECE = 4096;               // one piece of a slot: 128 rows x 32 bytes
constexpr float kFarPoint = 1e15f;             // position of a row without a sample point: every
                                               // exponential is zero, every polynomial finite
constexpr float kLog2e = 1.44269504f;
constexpr float kCut2 = kExpCut * kLog2e;

struct FactParams {
  FactMol one;             // the molecule of a single-molecule launch
  const FactMol* mols;     // device array of nmol molecules
  int nmol;
  int64_t ntiles;
  uint32_t fmt;
  FactPlan plan;
  int* err;
  uint64_t wait_ns;
  const FactDecision* decision;   // ON_DEVICE: the device's, in place of the host's shape and plan
};

__host__ __device__ inline FactShape fact_shape(int rank, int nunits) {
  FactShape f;
  f.refused = rank <= 0;
  f.r16 = rank > 16 ? (rank + 15) / 16 * 16 : 16;
  f.sets = 2 * f.r16 <= 256 ? 2 : 1;
  // The tensor core's additions truncate, so every K-step takes about 2^-24 of T away and the squares double that:
  // a uniform loss, which only rescaling hides.  Units in turn on up to three accumulators divide it by as many where
  // two buffers hold them (a third buffer's worth of TMEM is not given up for it).
  int na = f.sets == 2 ? 256 / f.r16 - 1 : 1;
  if (na > 3) na = 3;
  if (na > nunits) na = nunits;
  f.na = na < 1 ? 1 : na;
  return f;
}

template <int WHO>
__device__ __forceinline__ FactShape fact_shape_of(const FactParams& p, const FactMol& m) {
  if (WHO == ON_DEVICE) return p.decision->shape;
  return FactShape{0, m.r16, m.sets, m.na};
}

// The factor stays in shared memory when at least MIN_SLOTS slots fit beside it; else its blocks (blk bytes each) stream
// through the slots.
__host__ __device__ inline FactPlan fact_plan(int64_t avail, int abytes, int blk, int nunits, bool one) {
  const int64_t whole = (int64_t)blk * nunits;
  FactPlan f;
  f.resident = one && whole + MIN_SLOTS * abytes <= avail ? 1 : 0;
  f.slot_bytes = (uint32_t)(abytes + (f.resident ? 0 : GROUP * blk));
  const int64_t fit = (avail - (f.resident ? whole : 0)) / f.slot_bytes;
  f.nslots = fit < MAX_SLOTS ? (uint32_t)fit : (uint32_t)MAX_SLOTS;
  f.slot_magic = f.nslots ? (uint32_t)(((1ull << 32) + f.nslots - 1) / f.nslots) : 0u;
  return f;
}
template <int WHO>
__device__ __forceinline__ FactPlan fact_plan_of(const FactParams& p) {
  return WHO == ON_DEVICE ? p.decision->plan : p.plan;
}

template <bool MULTI>
__device__ __forceinline__ const FactMol& fact_mol(const FactParams& p, int64_t t) {
  if (!MULTI) return p.one;
  int lo = 0, hi = p.nmol - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&p.mols[mid].tile0) <= t) lo = mid;
    else hi = mid - 1;
  }
  return p.mols[lo];
}

// ---- packed FP32 pairs (rows r and r + 64 of an item): one issue slot for both rows -------------
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 dup(float a) { return pk(a, a); }
__device__ __forceinline__ float2 upk(f2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// 2^(na q), na = -alpha log2(e): the exponential of both rows
__device__ __forceinline__ f2 gauss2(float na, f2 q) {
  const float2 x = upk(mul2(dup(na), q));
  return pk(ex2(x.x), ex2(x.y));
}

// ---- stores: NV values (the rest of the 16 columns zero) of the lane's two rows -----------------
template <int FMT>
__device__ __forceinline__ uint32_t cvt2(float x0, float x1) {
  uint32_t r;
  if constexpr (FMT == 0) {
    const __half2 h = __floats2half2_rn(x0, x1);
    r = *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
    r = *reinterpret_cast<const uint32_t*>(&h);
  }
  return r;
}
template <int FMT>
__device__ __forceinline__ float2 widen2(uint32_t w) {
  if constexpr (FMT == 0) return __half22float2(*reinterpret_cast<const __half2*>(&w));
  else return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

// columns 8 u .. 8 u + 7 of both rows (row r0 at `dst`, row r0 + 64 2048 bytes on)
template <int FMT, bool TWO, int N8>
__device__ __forceinline__ void put_unit8(uint8_t* dst, const f2* v) {
  uint32_t h0[4], h1[4], l0[4], l1[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool two = 2 * k + 1 < N8, any = 2 * k < N8;
    h0[k] = h1[k] = l0[k] = l1[k] = 0;
    if (any) {
      const float2 a = upk(v[2 * k]);
      float2 b = make_float2(0.f, 0.f);
      if (two) b = upk(v[2 * k + 1]);
      h0[k] = cvt2<FMT>(a.x, b.x);
      h1[k] = cvt2<FMT>(a.y, b.y);
      if (TWO) {
        const float2 w0 = widen2<FMT>(h0[k]), w1 = widen2<FMT>(h1[k]);
        l0[k] = cvt2<FMT>(a.x - w0.x, b.x - w0.y);
        l1[k] = cvt2<FMT>(a.y - w1.x, b.y - w1.y);
      }
    }
  }
  *reinterpret_cast<uint4*>(dst) = make_uint4(h0[0], h0[1], h0[2], h0[3]);
  *reinterpret_cast<uint4*>(dst + 2048) = make_uint4(h1[0], h1[1], h1[2], h1[3]);
  if (TWO) {
    *reinterpret_cast<uint4*>(dst + PIECE) = make_uint4(l0[0], l0[1], l0[2], l0[3]);
    *reinterpret_cast<uint4*>(dst + PIECE + 2048) = make_uint4(l1[0], l1[1], l1[2], l1[3]);
  }
}
template <int FMT, bool TWO, int NV>
__device__ __forceinline__ void put16(uint8_t* slot, int r0, const f2 (&v)[NV]) {
  const uint32_t sw = (uint32_t)((r0 >> 2) & 1) * 16u;
  uint8_t* row = slot + r0 * 32;
  put_unit8<FMT, TWO, 8>(row + sw, v);
  put_unit8<FMT, TWO, NV - 8>(row + (sw ^ 16u), v + 8);
}
template <bool TWO>
__device__ __forceinline__ void put_zero(uint8_t* slot, int r0) {
  uint8_t* row = slot + r0 * 32;
  const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int k = 0; k < (TWO ? 2 : 1); ++k) {
    uint8_t* d = row + k * PIECE;
    reinterpret_cast<uint4*>(d)[0] = z;
    reinterpret_cast<uint4*>(d)[1] = z;
    reinterpret_cast<uint4*>(d + 2048)[0] = z;
    reinterpret_cast<uint4*>(d + 2048)[1] = z;
  }
}
template <int FMT, bool TWO>
__device__ __forceinline__ void put1(uint8_t* slot, int r0, int col, f2 v) {
  const float2 x = upk(v);
  const uint32_t off = (uint32_t)r0 * 32u + (uint32_t)((((col >> 3) ^ (r0 >> 2)) & 1) << 4) + (uint32_t)(col & 7) * 2u;
  const uint32_t h = cvt2<FMT>(x.x, x.y);
  *reinterpret_cast<uint16_t*>(slot + off) = (uint16_t)h;
  *reinterpret_cast<uint16_t*>(slot + off + 2048) = (uint16_t)(h >> 16);
  if (TWO) {
    const float2 w = widen2<FMT>(h);
    const uint32_t l = cvt2<FMT>(x.x - w.x, x.y - w.y);
    *reinterpret_cast<uint16_t*>(slot + off + PIECE) = (uint16_t)l;
    *reinterpret_cast<uint16_t*>(slot + off + PIECE + 2048) = (uint16_t)(l >> 16);
  }
}

// ---- production ----------------------------------------------------------------------------------
struct Disp {
  f2 x, y, z, q;
};

// Displacement of the lane's two rows from an atom, correct to one FP32 rounding without FP64: the
// positions come as hi + lo with hi a multiple of 2^-12 bohr (split_pos), the nuclear
// coordinate is split the same way (adding and subtracting 3 * 2^10 rounds it to 2^-12), so the
// difference of the hi parts is exact.
__device__ __forceinline__ f2 disp1(const float4 p, float a) {
  const float ah = __fadd_rn(__fadd_rn(a, 3072.f), -3072.f), al = __fsub_rn(a, ah);
  return add2(sub2(pk(p.x, p.y), dup(ah)), sub2(pk(p.z, p.w), dup(al)));
}
__device__ __forceinline__ Disp displace(const float4 (*pos)[64], int r0, const float* __restrict__ c) {
  Disp d;
  d.x = disp1(pos[0][r0], __ldg(c));
  d.y = disp1(pos[1][r0], __ldg(c + 1));
  d.z = disp1(pos[2][r0], __ldg(c + 2));
  d.q = fma2(d.z, d.z, fma2(d.y, d.y, mul2(d.x, d.x)));
  return d;
}
// bit k: primitive k of the class (na < 0 in .x) is above the cut-off at some row of the item
template <int NP>
__device__ __forceinline__ uint32_t live_prims(const float4* __restrict__ cls, f2 q, int lane) {
  const float2 w = upk(q);
  const float qmin = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(fminf(w.x, w.y))));
  const float na = __ldg(&cls[min(lane, NP - 1)].x);
  return __ballot_sync(0xffffffffu, lane < NP && na * qmin > -kCut2);
}
__device__ __forceinline__ void prim1(const float4* __restrict__ cls, f2 q, f2& s) {
  const float4 t = __ldg(cls);
  s = fma2(dup(t.y), gauss2(t.x, q), s);
}
__device__ __forceinline__ void prim2(const float4* __restrict__ cls, f2 q, f2& s, f2& u) {
  const float4 t = __ldg(cls);
  const f2 e = gauss2(t.x, q);
  s = fma2(dup(t.y), e, s);
  u = fma2(dup(t.z), e, u);
}

// Class table of the s8 s8 s1 p3 p1 d1 layout: 14 float4 {-alpha log2 e, c, c of the second s shell, 0}:
// 8 of the contracted s shells, 3 of the p, then s, p, d (exponents descending in each shell; the
// scale 2^s_j and the angular constant are in c).  Steep primitives, which only matter near the
// atom, sit behind a warp-uniform test.
template <int FMT, bool TWO>
__device__ __forceinline__ void unit_heavy(uint8_t* slot, int r0, int lane, const float4 (*pos)[64],
                                           const float* __restrict__ crd, const float4* __restrict__ cls) {
  const Disp d = displace(pos, r0, crd);
  const uint32_t m = live_prims<14>(cls, d.q, lane);
  if (m == 0) {
    put_zero<TWO>(slot, r0);
    return;
  }
  f2 v[14];
  f2 s1 = 0ull, s2 = 0ull;
  if (m & 0x0fu) {
#pragma unroll
    for (int k = 0; k < 4; ++k) prim2(cls + k, d.q, s1, s2);
  }
  if (m & 0x30u) {
    prim2(cls + 4, d.q, s1, s2);
    prim2(cls + 5, d.q, s1, s2);
  }
  prim2(cls + 6, d.q, s1, s2);
  prim2(cls + 7, d.q, s1, s2);
  v[0] = s1;
  v[1] = s2;
  f2 p3 = 0ull, s3 = 0ull, p1 = 0ull;
  if (m & 0x100u) prim1(cls + 8, d.q, p3);
  prim1(cls + 9, d.q, p3);
  prim1(cls + 10, d.q, p3);
  prim1(cls + 11, d.q, s3);
  prim1(cls + 12, d.q, p1);
  v[2] = s3;
  v[3] = mul2(p3, d.z);
  v[4] = mul2(p3, d.x);
  v[5] = mul2(p3, d.y);
  v[6] = mul2(p1, d.z);
  v[7] = mul2(p1, d.x);
  v[8] = mul2(p1, d.y);
  if (m & 0x2000u) {
    f2 r = 0ull;
    prim1(cls + 13, d.q, r);
    const f2 xx = mul2(d.x, d.x), yy = mul2(d.y, d.y), zz = mul2(d.z, d.z);
    const f2 rx = mul2(r, d.x);
    v[9] = mul2(mul2(r, dup((float)(YD0 / YD1))), sub2(add2(zz, zz), add2(xx, yy)));
    v[10] = mul2(rx, d.z);
    v[11] = mul2(mul2(r, d.y), d.z);
    v[12] = mul2(mul2(r, dup((float)(YD2 / YD1))), sub2(xx, yy));
    v[13] = mul2(rx, d.y);
  } else {
#pragma unroll
    for (int k = 9; k < 14; ++k) v[k] = 0ull;
  }
  put16<FMT, TWO, 14>(slot, r0, v);
}

// Up to three atoms of the s3 s1 p1 layout: class tables of 5 float4 (3 s, s, p).
template <int FMT, bool TWO>
__device__ __forceinline__ void unit_light(uint8_t* slot, int r0, int lane, const float4 (*pos)[64],
                                           const float* __restrict__ coords, const float4* __restrict__ tab, int4 u0,
                                           int4 u1) {
  const int count = u0.x >> 8;
  const int cl[3] = {u0.y, u0.z, u0.w}, at[3] = {u1.x, u1.y, u1.z};
  f2 v[15];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int k = 0; k < 5; ++k) v[5 * i + k] = 0ull;
    if (i < count) {
      const float4* cls = tab + cl[i];
      const Disp d = displace(pos, r0, coords + 3 * at[i]);
      const uint32_t m = live_prims<5>(cls, d.q, lane);
      if (m) {
        f2 s = 0ull, u = 0ull, p = 0ull;
        if (m & 1u) prim1(cls, d.q, s);
        prim1(cls + 1, d.q, s);
        prim1(cls + 2, d.q, s);
        prim1(cls + 3, d.q, u);
        prim1(cls + 4, d.q, p);
        v[5 * i] = s;
        v[5 * i + 1] = u;
        v[5 * i + 2] = mul2(p, d.z);
        v[5 * i + 3] = mul2(p, d.x);
        v[5 * i + 4] = mul2(p, d.y);
      }
    }
  }
  put16<FMT, TWO, 15>(slot, r0, v);
}

// Any other shells: records {first primitive, L | nprim << 8 | column << 16, atom, 0}, primitives
// float4 {-alpha log2 e, c, 0, 0}.
template <int FMT, bool TWO>
__device__ __noinline__ void unit_generic(uint8_t* slot, int r0, const float4 (*pos)[64],
                                          const float* __restrict__ coords, const float4* __restrict__ tab, int count,
                                          int first) {
  put_zero<TWO>(slot, r0);
  for (int i = 0; i < count; ++i) {
    const int4 rec = __ldg(reinterpret_cast<const int4*>(tab) + first + i);
    const int L = rec.y & 0xff, np = (rec.y >> 8) & 0xff, col = rec.y >> 16;
    const Disp d = displace(pos, r0, coords + 3 * rec.z);
    f2 r = 0ull;
    for (int k = 0; k < np; ++k) prim1(tab + rec.x + k, d.q, r);
    if (L == 0) {
      put1<FMT, TWO>(slot, r0, col, r);
    } else if (L == 1) {
      put1<FMT, TWO>(slot, r0, col, mul2(r, d.z));
      put1<FMT, TWO>(slot, r0, col + 1, mul2(r, d.x));
      put1<FMT, TWO>(slot, r0, col + 2, mul2(r, d.y));
    } else {
      const f2 xx = mul2(d.x, d.x), yy = mul2(d.y, d.y), zz = mul2(d.z, d.z);
      const f2 rx = mul2(r, d.x);
      put1<FMT, TWO>(slot, r0, col, mul2(mul2(r, dup((float)(YD0 / YD1))), sub2(add2(zz, zz), add2(xx, yy))));
      put1<FMT, TWO>(slot, r0, col + 1, mul2(rx, d.z));
      put1<FMT, TWO>(slot, r0, col + 2, mul2(mul2(r, d.y), d.z));
      put1<FMT, TWO>(slot, r0, col + 3, mul2(mul2(r, dup((float)(YD2 / YD1))), sub2(xx, yy)));
      put1<FMT, TWO>(slot, r0, col + 4, mul2(rx, d.y));
    }
  }
}

// Position of a sample point as hi + lo, hi a multiple of 2^-12 (exact in FP32 within 4096 bohr).
__device__ __forceinline__ float2 split_pos(double x) {
  const float h = (float)(rint(x * 4096.0) * (1.0 / 4096.0));
  return make_float2(h, (float)(x - (double)h));
}

}  // namespace

namespace {
struct FactBars {
  uint64_t a_full[MAX_SLOTS], b_full[MAX_SLOTS], empty[MAX_SLOTS];
  uint64_t pos_full[POS_DEPTH], pos_empty[POS_DEPTH];
  uint64_t t_full[2], t_empty[2], res_bar, drain_bar[2];
  volatile int abort_flag;
};

// MMA issue: the whole warp walks the groups, one lane issues.  MAIN: the H products; else the S ones, by
// a warp of its own: a thread spends about 110 clocks on each MMA with new operands (waits, descriptors,
// issue) whatever its N, more than the 58 to 128 the tensor core takes, and the two accumulator chains
// never meet.
template <int FMT, bool TWO, int WHO, bool MAIN>
__device__ __forceinline__ void issue_mma(const FactParams& p, FactBars& B, uint8_t* smem, uint8_t* res, uint32_t tmem) {
  constexpr bool MULTI = WHO == MANY;
  uint32_t s = 0, ph = 0, tile_it = 0;   // slot and its phase
  int last_sets = 2;
  const bool leader = elect_one();
  const FactPlan plan = fact_plan_of<WHO>(p);
  const bool streamed = MULTI || !plan.resident;
  const uint32_t ring0 = smem_u32(smem);
  constexpr uint32_t UNIT_A = TWO ? 2 * PIECE : PIECE, ABYTES = GROUP * UNIT_A;
  bool ok = true, ready = false;
  FactShape f = fact_shape_of<WHO>(p, p.one);
  if (!streamed) ok = mbar_wait_warp(&B.res_bar, 0u, &B.abort_flag, p.wait_ns);
  for (int64_t t = blockIdx.x; t < p.ntiles && ok; t += gridDim.x, ++tile_it) {
    const FactMol& M = fact_mol<MULTI>(p, t);
    const int nunits = M.nunits;
    if (MULTI) f = fact_shape_of<WHO>(p, M);
    const uint32_t r16 = (uint32_t)f.r16;
    // TMEM: a half per tile in turn, or (sets == 1) all of it; the tiles whose columns this one
    // overwrites must have been read
    const int sets = f.sets;
    const uint32_t set = tile_it & 1u, d0 = tmem + (sets == 2 ? set * 256u : 0u);
    if (tile_it >= 2) ok = mbar_wait_warp(&B.t_empty[set], ((tile_it - 2u) >> 1) & 1u, &B.abort_flag, p.wait_ns);
    if (ok && tile_it >= 1 && (sets == 1 || last_sets == 1))
      ok = mbar_wait_warp(&B.t_empty[set ^ 1u], ((tile_it - 1u) >> 1) & 1u, &B.abort_flag, p.wait_ns);
    if (!ok) break;
    last_sets = sets;
    tc_fence_after();
    const uint32_t na = (uint32_t)f.na, S = d0 + na * r16;
    const uint32_t idesc = make_idesc(p.fmt, 128, r16);
    const uint32_t blk = (uint32_t)(TWO ? 2 : 1) * r16 * 32u, half = r16 * 32u;
    uint32_t acc = 0, ha = 0;   // accumulated before; H accumulator of the next unit (in turn)
    uint32_t bres = smem_u32(res);
    for (int u0 = 0; u0 < nunits; u0 += GROUP) {
      ok = (ready || mbar_wait_warp(&B.a_full[s], ph, &B.abort_flag, p.wait_ns)) &&
           (!streamed || mbar_wait_warp(&B.b_full[s], ph, &B.abort_flag, p.wait_ns));
      if (!ok) break;
      tc_fence_after();
      // the next group's state, read while this one's MMAs are issued
      const uint32_t sn = s + 1 == plan.nslots ? 0 : s + 1, phn = s + 1 == plan.nslots ? ph ^ 1u : ph;
      const bool peek = mbar_test_wait(&B.a_full[sn], phn);
      const uint32_t slot = ring0 + s * plan.slot_bytes;
      uint32_t a = slot, b = streamed ? slot + ABYTES : bres;
#pragma unroll
      for (int k = 0; k < GROUP; ++k) {
        if (u0 + k < nunits) {
          const uint64_t ahi = sw32_kmajor_desc(a), bhi = sw32_kmajor_desc(b);
          if (MAIN) {
            if (leader) mma_f16(d0 + ha * r16, ahi, bhi, idesc, acc);
          } else {
            const uint64_t alo = sw32_kmajor_desc(a + PIECE), blo = sw32_kmajor_desc(b + half);
            if (leader) {
              mma_f16(S, ahi, blo, idesc, acc);
              mma_f16(S, alo, bhi, idesc, 1u);
              if (FMT == 1) mma_f16(S, alo, blo, idesc, 1u);
            }
          }
          if (!MAIN || ++ha == na) {
            acc = 1u;
            ha = 0;
          }
          a += UNIT_A;
          b += blk;
        }
      }
      ready = __all_sync(0xffffffffu, peek);
      bres = b;
      if (leader) tc_commit(&B.empty[s]);
      s = sn;
      ph = phn;
    }
    if (!ok) break;
    if (leader) {
      tc_commit(&B.t_full[set]);
      tc_commit(&B.pos_empty[tile_it % POS_DEPTH]);
    }
  }
  // every MMA issued by this warp has completed once drain_bar flips
  if (leader) {
    tc_commit(&B.drain_bar[MAIN ? 0 : 1]);
    mbar_wait_drain(&B.drain_bar[MAIN ? 0 : 1], 0u, 500000000ull);
  }
  __syncwarp();
}

}  // namespace

// One persistent CTA per SM walks the tiles blockIdx.x, blockIdx.x + gridDim.x, ...
template <int FMT, bool TWO, int WHO>
__global__ void __launch_bounds__(FACT_THREADS, 1) density_factored_kernel(const __grid_constant__ FactParams p) {
  constexpr bool MULTI = WHO == MANY;
  extern __shared__ uint8_t smem_dyn[];
  if (WHO == ON_DEVICE && p.decision->shape.refused) return;   // the unfactored launch of the pair does the work
  __shared__ FactBars B;
  __shared__ __align__(16) float4 pos_s[POS_DEPTH][3][64];   // {hi r, hi r + 64, lo r, lo r + 64}
  __shared__ double rho_s[128];
  __shared__ double red[2][4];
  __shared__ uint32_t tmem_slot;
  __shared__ int item_ctr;

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const FactPlan plan = fact_plan_of<WHO>(p);
  const uint32_t nslots = plan.nslots;
  constexpr uint32_t UNIT_A = TWO ? 2 * PIECE : PIECE, ABYTES = GROUP * UNIT_A;
  constexpr uint32_t NISSUE = TWO ? 2 : 1;   // MMA-issuing warps
  uint8_t* res = smem + (size_t)nslots * plan.slot_bytes;   // the resident factor

  if (threadIdx.x == 0) {
    B.abort_flag = 0;
    item_ctr = 0;
    for (uint32_t s = 0; s < nslots; ++s) {
      mbar_init(&B.a_full[s], 2 * GROUP);   // two items of 64 rows per unit
      mbar_init(&B.b_full[s], 1);
      mbar_init(&B.empty[s], NISSUE);
    }
    for (int k = 0; k < POS_DEPTH; ++k) {
      mbar_init(&B.pos_full[k], 32);
      mbar_init(&B.pos_empty[k], NISSUE);
    }
    for (int k = 0; k < 2; ++k) {
      mbar_init(&B.t_full[k], NISSUE);
      mbar_init(&B.t_empty[k], 128);
    }
    mbar_init(&B.res_bar, 1);
    for (uint32_t k = 0; k < NISSUE; ++k) mbar_init(&B.drain_bar[k], 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    // ---- the factor's K-step blocks ------------------------------------------------------------
    if (lane == 0) {
      if (!MULTI && plan.resident) {
        const uint32_t blk = (uint32_t)(TWO ? 2 : 1) * (uint32_t)fact_shape_of<WHO>(p, p.one).r16 * 32u;
        mbar_expect_tx(&B.res_bar, blk * (uint32_t)p.one.nunits);
        for (int u = 0; u < p.one.nunits; ++u) bulk_load(res + (size_t)u * blk, p.one.B + (size_t)u * blk, blk, &B.res_bar);
        mbar_wait_drain(&B.res_bar, 0u, p.wait_ns < 100000000ull ? 100000000ull : p.wait_ns);
      } else {
        uint32_t s = 0, ph = 0, issued = 0, par = 0;
        bool ok = true;
        FactShape f = fact_shape_of<WHO>(p, p.one);
        for (int64_t t = blockIdx.x; t < p.ntiles && ok; t += gridDim.x) {
          const FactMol& M = fact_mol<MULTI>(p, t);
          const int nunits = M.nunits;
          if (MULTI) f = fact_shape_of<WHO>(p, M);
          const uint32_t blk = (uint32_t)(TWO ? 2 : 1) * (uint32_t)f.r16 * 32u;
          const uint8_t* src = M.B;
          for (int u = 0; u < nunits; u += GROUP, src += GROUP * blk) {
            if (!mbar_wait(&B.empty[s], ph ^ 1u, &B.abort_flag, p.wait_ns)) {
              ok = false;
              break;
            }
            const uint32_t bytes = blk * (uint32_t)min(GROUP, nunits - u);
            mbar_expect_tx(&B.b_full[s], bytes);
            bulk_load(smem + (size_t)s * plan.slot_bytes + ABYTES, src, bytes, &B.b_full[s]);
            issued |= 1u << s;
            par = (par & ~(1u << s)) | (ph << s);
            if (++s == nslots) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
        if (!ok)   // wait for the copies in flight before the CTA exits
          for (uint32_t k = 0; k < nslots; ++k)
            if ((issued >> k) & 1u) mbar_wait_drain(&B.b_full[k], (par >> k) & 1u, 100000000ull);
      }
    }
  } else if (warp == 1) {
    issue_mma<FMT, TWO, WHO, true>(p, B, smem, res, tmem);
  } else if (warp == 2) {
    if (TWO) issue_mma<FMT, TWO, WHO, false>(p, B, smem, res, tmem);
  } else if (warp == 3) {
    // ---- sample positions: a lane writes rows r and r + 64, r = lane and lane + 32 -------------------
    uint32_t tile_it = 0;
    for (int64_t t = blockIdx.x; t < p.ntiles; t += gridDim.x, ++tile_it) {
      const FactMol& M = fact_mol<MULTI>(p, t);
      const uint32_t b = tile_it % POS_DEPTH;
      if (!mbar_wait(&B.pos_empty[b], ((tile_it / POS_DEPTH) & 1u) ^ 1u, &B.abort_flag, p.wait_ns)) break;
#pragma unroll 1
      for (int r = lane; r < 64; r += 32) {
        float2 c[2][3];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          double x, y, z;
          int64_t vox;
          if (tile_point<double>(M.pm, t - M.tile0, r + 64 * k, x, y, z, vox)) {
            c[k][0] = split_pos(x);
            c[k][1] = split_pos(y);
            c[k][2] = split_pos(z);
          } else {
            c[k][0] = c[k][1] = c[k][2] = make_float2(kFarPoint, 0.f);
          }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) pos_s[b][k][r] = make_float4(c[0][k].x, c[1][k].x, c[0][k].y, c[1][k].y);
      }
      mbar_arrive(&B.pos_full[b]);
    }
  } else if (warp < 8) {
    // ---- epilogue: rho = sum_k (2^-h_k T_k)^2, thread = row (TMEM lane) -----------------------------
    const int q = warp & 3, row = q * 32 + lane;
    uint32_t tile_it = 0;
    FactShape f = fact_shape_of<WHO>(p, p.one);
    for (int64_t t = blockIdx.x; t < p.ntiles; t += gridDim.x, ++tile_it) {
      const FactMol& M = fact_mol<MULTI>(p, t);
      if (MULTI) f = fact_shape_of<WHO>(p, M);
      const uint32_t set = tile_it & 1u;
      // the four warps leave together: one of them giving up while the others go on would leave
      // those waiting at the next named barrier
      const bool got = mbar_wait(&B.t_full[set], (tile_it >> 1) & 1u, &B.abort_flag, p.wait_ns);
      if (barrier_any(1, 128, !got)) break;
      tc_fence_after();
      const int r16 = f.r16;
      const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + (f.sets == 2 ? set * 256u : 0u);
      const float4* hs = reinterpret_cast<const float4*>(M.hscale);
      double acc = 0.0;
      // sixteen columns of H and S in flight while the sixteen before them are squared
      uint32_t ha[16], la[16], hb[16], lb[16];
      auto load = [&](int c, uint32_t(&h)[16], uint32_t(&l)[16]) {
        tmem_ld16_issue(base + (uint32_t)c, h);
        if (TWO) tmem_ld16_issue(base + (uint32_t)(f.na * r16 + c), l);
      };
      auto square = [&](int c, uint32_t(&h)[16], uint32_t(&l)[16]) {
        f2 sq = 0ull;
#pragma unroll
        for (int e4 = 0; e4 < 4; ++e4) {
          const float4 h4 = __ldg(hs + (c >> 2) + e4);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = 4 * e4 + 2 * e;
            f2 t2 = pk(__uint_as_float(h[j]), __uint_as_float(h[j + 1]));
            if (TWO) t2 = add2(t2, pk(__uint_as_float(l[j]), __uint_as_float(l[j + 1])));
            t2 = mul2(t2, e == 0 ? pk(h4.x, h4.y) : pk(h4.z, h4.w));
            sq = fma2(t2, t2, sq);   // eight squares per FP32 partial, summed in FP64
          }
        }
        const float2 w = upk(sq);
        acc += (double)w.x + (double)w.y;
      };
      auto arrived = [&](uint32_t(&h)[16], uint32_t(&l)[16]) {
        tmem_ld16_wait(h);
        if (TWO) tmem_ld16_wait(l);
      };
      if (f.na > 1) {
        // several H accumulators: their sum takes the registers of the second block of columns
#pragma unroll 1
        for (int c = 0; c < r16; c += 16) {
          load(c, ha, la);
          tmem_ld16_issue(base + (uint32_t)(r16 + c), hb);
          if (f.na > 2) tmem_ld16_issue(base + (uint32_t)(2 * r16 + c), lb);
          arrived(ha, la);
          tmem_ld16_wait(hb);
#pragma unroll
          for (int j = 0; j < 16; ++j) ha[j] = __float_as_uint(__uint_as_float(ha[j]) + __uint_as_float(hb[j]));
          if (f.na > 2) {
            tmem_ld16_wait(lb);
#pragma unroll
            for (int j = 0; j < 16; ++j) ha[j] = __float_as_uint(__uint_as_float(ha[j]) + __uint_as_float(lb[j]));
          }
          square(c, ha, la);
        }
      } else {
        load(0, ha, la);
#pragma unroll 1
        for (int c = 0; c < r16; c += 32) {
          arrived(ha, la);
          if (c + 16 < r16) load(c + 16, hb, lb);
          square(c, ha, la);
          if (c + 16 < r16) {
            arrived(hb, lb);
            if (c + 32 < r16) load(c + 32, ha, la);
            square(c + 16, hb, lb);
          }
        }
      }
      tc_fence_before();
      mbar_arrive(&B.t_empty[set]);
      double r = acc;
      if (M.pm.s3 > 1) {
        rho_s[row] = r;   // (read by the previous tile before its last barrier)
        named_barrier(2, 128);
        r = 0.0;
        if (row < M.pm.vpt)
          for (int sub = 0; sub < M.pm.s3; ++sub) r += rho_s[row * M.pm.s3 + sub];
      }
      double sum = 0.0;
      int64_t vox, ix, iy, iz;
      const int64_t lt = t - M.tile0;
      if (tile_voxel(M.pm, lt, row, vox, ix, iy, iz)) {
        const float qv = (float)(r * M.outscale);
        M.qube[vox] = qv;
        sum = qv;
      }
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) red[set][q] = sum;
      named_barrier(2, 128);
      if (row == 0) M.partials[lt] = (red[set][0] + red[set][1]) + (red[set][2] + red[set][3]);
    }
  } else {
    // ---- production of Phi' ------------------------------------------------------------------------
    int64_t t = blockIdx.x;
    uint32_t tile_it = 0, kg0 = 0, seen = 0xffffffffu;
    int base = 0;
    const FactMol* M = &fact_mol<MULTI>(p, min(t, p.ntiles - 1));
    int nunits = M->nunits;
    const int4* units = M->units;
    const float* coords = M->coords;
    int nxt = 0;
    if (lane == 0) nxt = atomicAdd(&item_ctr, 1);
    for (;;) {
      const int itm = __shfl_sync(0xffffffffu, nxt, 0);
      while (t < p.ntiles && itm >= base + 2 * nunits) {
        base += 2 * nunits;
        kg0 += (uint32_t)((nunits + GROUP - 1) / GROUP);
        t += gridDim.x;
        ++tile_it;
        if (MULTI && t < p.ntiles) {
          M = &fact_mol<MULTI>(p, t);
          nunits = M->nunits;
          units = M->units;
          coords = M->coords;
        }
      }
      if (t >= p.ntiles) break;
      const int u = (itm - base) >> 1, r0 = ((itm - base) & 1) * 32 + lane;
      const uint32_t kg = kg0 + (uint32_t)(u / GROUP), round = __umulhi(kg, plan.slot_magic), s = kg - round * nslots;
      const uint32_t ph = round & 1u, b = tile_it % POS_DEPTH;
      const int4 u0 = __ldg(units + 2 * u), u1 = __ldg(units + 2 * u + 1);
      if ((seen != tile_it && !mbar_wait_warp(&B.pos_full[b], (tile_it / POS_DEPTH) & 1u, &B.abort_flag, p.wait_ns)) ||
          !mbar_wait_warp(&B.empty[s], ph ^ 1u, &B.abort_flag, p.wait_ns))
        break;
      seen = tile_it;
      // (the next item is taken only now: a warp holds at most one item that has not passed its waits)
      if (lane == 0) nxt = atomicAdd(&item_ctr, 1);
      uint8_t* slot = smem + (size_t)s * plan.slot_bytes + (u % GROUP) * UNIT_A;
      const float4* tab = reinterpret_cast<const float4*>(units);
      const int kind = u0.x & 0xff;
      if (kind == UNIT_S8S8S1P3P1D1)
        unit_heavy<FMT, TWO>(slot, r0, lane, pos_s[b], coords + 3 * u1.x, tab + u0.y);
      else if (kind == UNIT_S3S1P1)
        unit_light<FMT, TWO>(slot, r0, lane, pos_s[b], coords, tab, u0, u1);
      else
        unit_generic<FMT, TWO>(slot, r0, pos_s[b], coords, tab, u0.x >> 8, u0.y);
      // generic-proxy writes of the slot become visible to the tensor core, then one arrival
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      // (the last group of an odd tile has one unit, whose items count double)
      if (lane == 0) mbar_arrive_count(&B.a_full[s], (u % GROUP == 0 && u + 1 == nunits) ? GROUP : 1);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (B.abort_flag && threadIdx.x == 0) atomicExch(p.err, 1);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------
namespace {

// Host copy of the unit tables: per unit two int4 (kind | count << 8 and class indices; atoms), the
// class tables and generic shells behind them (indices in 16-byte words from the start), and the
// function of each column (-1: padding).
struct UnitTables {
  std::vector<int4> words;
  std::vector<int> column;   // 16 per unit
  int nunits = 0;
};

float4 prim_entry(float alpha, float c, float c2 = 0.f) { return make_float4(-(alpha * kLog2e), c, c2, 0.f); }

UnitTables build_units(const qmt_mol* m, const std::vector<float>& fs) {
  struct Unit {
    int4 a, b;
  };
  std::vector<Unit> units;
  std::vector<float4> cls;                       // class tables, shared by atoms with equal ones
  std::vector<std::pair<int, int>> known;        // (first entry, entries)
  std::vector<int4> recs;
  UnitTables out;
  const double ang[3] = {YS, YP, YD1};
  auto is = [&](int sidx, int L, int np, int same) {
    const Shell& x = m->shells[sidx];
    return x.L == L && x.nprim == np && x.same_exp == same;
  };
  // primitives of a shell by descending exponent, coefficients with the column scale and the
  // angular constant
  auto shell_entries = [&](int sidx, int second) {
    const Shell& sh = m->shells[sidx];
    std::vector<int> ord(sh.nprim);
    for (int k = 0; k < sh.nprim; ++k) ord[k] = k;
    std::stable_sort(ord.begin(), ord.end(), [&](int u, int v) { return m->alpha[sh.prim + u] > m->alpha[sh.prim + v]; });
    std::vector<float4> e;
    auto coef = [&](const Shell& x, int k) { return (float)((double)m->coeff[x.prim + k] * fs[x.func] * ang[x.L]); };
    for (int k : ord)
      e.push_back(prim_entry(m->alpha[sh.prim + k], coef(sh, k), second >= 0 ? coef(m->shells[second], k) : 0.f));
    return e;
  };
  auto intern = [&](const std::vector<float4>& e) {
    for (const auto& kn : known)
      if (kn.second == (int)e.size() && !std::memcmp(cls.data() + kn.first, e.data(), e.size() * sizeof(float4)))
        return kn.first;
    known.emplace_back((int)cls.size(), (int)e.size());
    cls.insert(cls.end(), e.begin(), e.end());
    return known.back().first;
  };
  auto append = [](std::vector<float4>& a, const std::vector<float4>& b) { a.insert(a.end(), b.begin(), b.end()); };

  int open_light = -1, open_generic = -1, generic_cols = 0;
  for (int a = 0; a < m->natoms; ++a) {
    const int s0 = m->atom_shell[a], s1 = m->atom_shell[a + 1], ns = s1 - s0;
    if (ns == 6 && is(s0, 0, 8, 0) && is(s0 + 1, 0, 8, 1) && is(s0 + 2, 0, 1, 0) && is(s0 + 3, 1, 3, 0) &&
        is(s0 + 4, 1, 1, 0) && is(s0 + 5, 2, 1, 0)) {
      std::vector<float4> e = shell_entries(s0, s0 + 1);
      append(e, shell_entries(s0 + 3, -1));
      append(e, shell_entries(s0 + 2, -1));
      append(e, shell_entries(s0 + 4, -1));
      append(e, shell_entries(s0 + 5, -1));
      units.push_back({make_int4(UNIT_S8S8S1P3P1D1 | 1 << 8, intern(e), 0, 0), make_int4(a, 0, 0, 0)});
      for (int k = 0; k < 16; ++k) out.column.push_back(k < 14 ? m->shells[s0].func + k : -1);
    } else if (ns == 3 && is(s0, 0, 3, 0) && is(s0 + 1, 0, 1, 0) && is(s0 + 2, 1, 1, 0)) {
      std::vector<float4> e = shell_entries(s0, -1);
      append(e, shell_entries(s0 + 1, -1));
      append(e, shell_entries(s0 + 2, -1));
      if (open_light < 0 || (units[open_light].a.x >> 8) == 3) {
        open_light = (int)units.size();
        units.push_back({make_int4(UNIT_S3S1P1, 0, 0, 0), make_int4(0, 0, 0, 0)});
        for (int k = 0; k < 16; ++k) out.column.push_back(-1);
      }
      Unit& u = units[open_light];
      const int i = u.a.x >> 8;
      (&u.a.y)[i] = intern(e);
      (&u.b.x)[i] = a;
      u.a.x += 1 << 8;
      for (int k = 0; k < 5; ++k) out.column[16 * open_light + 5 * i + k] = m->shells[s0].func + k;
    } else {
      for (int sidx = s0; sidx < s1; ++sidx) {
        const Shell& sh = m->shells[sidx];
        const int nf = 2 * sh.L + 1;
        if (open_generic < 0 || generic_cols + nf > 16) {
          open_generic = (int)units.size();
          generic_cols = 0;
          units.push_back({make_int4(UNIT_GENERIC, (int)recs.size(), 0, 0), make_int4(0, 0, 0, 0)});
          for (int k = 0; k < 16; ++k) out.column.push_back(-1);
        }
        Unit& u = units[open_generic];
        u.a.x += 1 << 8;
        recs.push_back(make_int4(intern(shell_entries(sidx, -1)), sh.L | sh.nprim << 8 | generic_cols << 16, sh.atom, 0));
        for (int k = 0; k < nf; ++k) out.column[16 * open_generic + generic_cols + k] = sh.func + k;
        generic_cols += nf;
      }
    }
  }
  while ((int)units.size() < MIN_UNITS) {
    units.push_back({make_int4(UNIT_GENERIC, 0, 0, 0), make_int4(0, 0, 0, 0)});
    for (int k = 0; k < 16; ++k) out.column.push_back(-1);
  }
  // indices become 16-byte words from the start of the table
  out.nunits = (int)units.size();
  const int cls0 = 2 * out.nunits, rec0 = cls0 + (int)cls.size();
  for (Unit& u : units) {
    const int kind = u.a.x & 0xff;
    if (kind == UNIT_GENERIC) {
      u.a.y += rec0;
    } else {
      for (int i = 0; i < (u.a.x >> 8); ++i) (&u.a.y)[i] += cls0;
    }
    out.words.push_back(u.a);
    out.words.push_back(u.b);
  }
  for (const float4& f : cls) {
    int4 w;
    std::memcpy(&w, &f, sizeof(w));
    out.words.push_back(w);
  }
  for (int4 r : recs) {
    r.x += cls0;
    out.words.push_back(r);
  }
  return out;
}

// ---- pivoted Cholesky factorisation (FP64, one thread-block cluster) ----------------------------------
// Largest remaining diagonal first (compared in FP32, lowest index on a tie: any pivot near the largest
// serves), until it is at most tol times the first, or rmax columns are done.  Each CTA owns a block of
// rows: their remaining diagonal and their rows of L in shared memory (of L2 when they do not fit).  A
// column is a chain of latencies: the CTAs exchange their largest diagonals through distributed shared
// memory (one cluster barrier; none with a single CTA), fetch the pivot's row of L from its owner while
// P's row comes from L2, form their elements, eight lanes a row, and find their next largest diagonal.
// info: [0] the rank, 0 when it exceeds the limit or a remaining diagonal is negative beyond rounding (the matrix is
// indefinite; [1] is set then).
constexpr int PIV_THREADS = 512;
constexpr int PIV_MAX_CTAS = 16;
constexpr int PIV_PRE = 2;                    // rows per thread whose element of P is fetched early
struct PivotArgs {
  const double* P;
  int np, n, rmax, rows;      // rows per CTA
  int rows_in_smem, ld;       // row stride of L in shared memory
  int limit;                  // of the rank (rmax: of the columns formed, at least 16)
  double tol;
  double* L;                  // n x rmax, FP64 (used when the rows do not fit in shared memory)
  float* L0;                  // n x ld0, FP32, zero beyond the rank up to a multiple of 16
  int ld0;                    // (at least rmax rounded up to 16)
  int* info;
  double* dmax;               // the first pivot
  unsigned long long* zero;   // nzero words that the kernel clears first: column maxima, info, dmax, the check's flag
  int nzero;
  int* usable;                // as fact_split_kernel leaves them, here where there is no factor; else the word's
  uint32_t number;            // kMailPending
  volatile unsigned long long* mail;
};
constexpr unsigned kMailPending = 1u << 30;   // there is a rank, the check is to come

struct PivotCand {
  double d;
  int at;
  uint32_t key;   // FP32 bits of d (0 when it is not positive): ordered like the values
};
__device__ __forceinline__ uint32_t pivot_key(double d) { return d > 0.0 ? __float_as_uint((float)d) : 0u; }
// The warp's best candidate, the lowest lane on a tie, on every lane.
__device__ __forceinline__ PivotCand pivot_best(PivotCand c) {
  const uint32_t mx = __reduce_max_sync(0xffffffffu, c.key);
  const int w = __ffs(__ballot_sync(0xffffffffu, c.key == mx)) - 1;
  PivotCand b;
  b.key = mx;
  b.d = __shfl_sync(0xffffffffu, c.d, w);
  b.at = __shfl_sync(0xffffffffu, c.at, w);
  return b;
}

__global__ void __launch_bounds__(PIV_THREADS, 1) fact_pivot_kernel(PivotArgs a) {
  extern __shared__ double piv_s[];
  __shared__ __align__(16) PivotCand cand[2][32];   // per column parity and CTA
  __shared__ PivotCand wbest[PIV_THREADS / 32];
  const uint32_t c = cluster_cta_rank(), ncta = gridDim.x;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, sub = t & 7, r0 = (int)c * a.rows;
  const int nr = max(0, min(a.rows, a.n - r0)), nr4 = (nr + 3) / 4 * 4;   // (whole warps in every round)
  double* d = piv_s;                            // remaining diagonal of the rows
  double* lj = d + a.rows;                      // the pivot's row of L
  double* own = a.rows_in_smem ? lj + a.rmax : a.L + (size_t)r0 * a.rmax;
  const int ld = a.rows_in_smem ? a.ld : a.rmax;
  if (c == 0)   // (info is written behind a barrier, the rest by later kernels)
    for (int i = t; i < a.nzero; i += PIV_THREADS) a.zero[i] = 0ull;
  const PivotCand none{0.0, 0x7fffffff, 0u};
  PivotCand best = none;                        // of this thread's rows (lanes with sub == 0)
  for (int i = t >> 3; i < nr; i += PIV_THREADS / 8)
    if (sub == 0) {
      const double v = a.P[(size_t)(r0 + i) * a.np + r0 + i];
      d[i] = v;
      if (pivot_key(v) > best.key) best = PivotCand{v, r0 + i, pivot_key(v)};
    }
  if (t < 64) cand[t >> 5][t & 31] = none;
  if (ncta > 1) cluster_barrier();              // every CTA's candidates are cleared before the first store
  int q = 0;
  bool high = false;
  double dmax = 0.0;
  for (;; ++q) {
    best = pivot_best(best);
    if (lane == 0) wbest[warp] = best;
    __syncthreads();   // (also: this column's elements are in `own` and d)
    if (warp == 0) {
      best = pivot_best(lane < PIV_THREADS / 32 ? wbest[lane] : none);
      if (lane < (int)ncta) {   // this CTA's candidate to every CTA
        const uint32_t p = cluster_addr(&cand[q & 1][c], (uint32_t)lane);
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(p), "d"(best.d) : "memory");
        asm volatile("st.shared::cluster.v2.b32 [%0], {%1, %2};" ::"r"(p + 8), "r"(best.at), "r"(best.key) : "memory");
      }
    }
    if (ncta > 1) cluster_barrier();
    else __syncthreads();
    best = pivot_best(cand[q & 1][lane]);       // (CTAs in row order)
    if (q == 0) dmax = best.d;
    if (!(best.d > a.tol * dmax)) break;
    if (q == a.rmax) {
      high = true;
      break;
    }
    const int jp = best.at;
    double pij[PIV_PRE];
#pragma unroll
    for (int k = 0; k < PIV_PRE; ++k) {
      const int i = (t >> 3) + k * (PIV_THREADS / 8);
      pij[k] = sub == 0 && i < nr ? __ldg(a.P + (size_t)jp * a.np + r0 + i) : 0.0;
    }
    const uint32_t oc = (uint32_t)(jp / a.rows);
    for (int k = t; k < q; k += PIV_THREADS)
      lj[k] = a.rows_in_smem ? cluster_load_f64(own + (size_t)(jp - (int)oc * a.rows) * ld + k, oc)
                             : __ldcg(a.L + (size_t)jp * a.rmax + k);
    // 1 / sqrt of the pivot to ~1e-14: an FP32 estimate and one Newton step (the library's FP64 rsqrt is a
    // long serial chain, and L0 is kept in FP32)
    const double y0 = (double)rsqrtf((float)best.d);
    const double ipiv = y0 * (1.5 - 0.5 * best.d * y0 * y0), piv = best.d * ipiv;
    __syncthreads();
    best = none;
#pragma unroll 1
    for (int i = t >> 3, k2 = 0; i < nr4; i += PIV_THREADS / 8, ++k2) {
      double s = 0.0;
      const bool in = i < nr;
      const double* li = own + (size_t)(in ? i : 0) * ld;
      for (int k = sub; k < q; k += 8) s = fma(a.rows_in_smem ? li[k] : __ldcg(li + k), lj[k], s);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (in && sub == 0) {
        const bool isp = r0 + i == jp;
        const double p = k2 == 0 ? pij[0] : (k2 == 1 ? pij[1] : __ldg(a.P + (size_t)jp * a.np + r0 + i));
        const double x = isp ? piv : (p - s) * ipiv;
        if (a.rows_in_smem) own[(size_t)i * ld + q] = x;
        else __stcg(own + (size_t)i * ld + q, x);
        a.L0[(size_t)(r0 + i) * a.ld0 + q] = (float)x;
        const double dn = isp ? 0.0 : d[i] - x * x;
        d[i] = dn;
        if (pivot_key(dn) > best.key) best = PivotCand{dn, r0 + i, pivot_key(dn)};
      }
    }
  }
  bool bad = high;
  for (int i = t; i < nr; i += PIV_THREADS) bad |= d[i] < -10.0 * a.tol * dmax;
  if (__syncthreads_or(bad) && t == 0) atomicExch(a.info + 1, 1);
  const int pad = max(16, (q + 15) / 16 * 16) - q;
  for (int i = t; i < nr * pad; i += PIV_THREADS) a.L0[(size_t)(r0 + i / pad) * a.ld0 + q + i % pad] = 0.f;
  if (ncta > 1) cluster_barrier();   // no CTA leaves while another may still read its shared memory; every [1] is in
  if (c == 0 && t == 0) {
    const int r = __ldcg(a.info + 1) || q > a.limit ? 0 : q;
    a.info[0] = r;
    *a.dmax = dmax;
    if (r == 0) *a.usable = 0;
    *a.mail = (unsigned long long)a.number << 32 | (r ? kMailPending | (unsigned)r : 0u);
  }
}

__device__ __forceinline__ int ceil16(int r) { return r > 16 ? (r + 15) / 16 * 16 : 16; }

// ---- refinement of the factor (FP64, device) ----------------------------------------------------
// The float32 input matrix is L L^T only up to its rounding, and a pivoted Cholesky factor takes that
// rounding from the pivot columns alone, amplified: 1.2e-6 relative L2 of the density at 30 atoms, of
// 1.25e-6 in all.  One power step spreads it over every column: with Y = P L0 and M = L0^T Y = C C^T,
// L = Y C^-T is the Nystroem approximation of P on the range of Y (2e-7, as the truncated
// eigendecomposition).  L0 only spans the space, so it comes as float32.
//
// The rank r is read from the device (info of fact_pivot_kernel), so that nothing here waits for the host: the grids are
// sized for the largest one.
__global__ void __launch_bounds__(256) fact_y_kernel(const double* __restrict__ P, int np, const float* __restrict__ L0,
                                                     int ld0, int n, const int* __restrict__ rank,
                                                     double* __restrict__ Y) {
  __shared__ double ps[32][33];
  __shared__ float ls[32][32];
  const int r16 = ceil16(*rank);
  if (*rank == 0 || (int)blockIdx.y * 32 >= r16) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, i0 = blockIdx.x * 32, q = blockIdx.y * 32 + tx;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int j0 = 0; j0 < n; j0 += 32) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = ty + 8 * k;
      ps[r][tx] = i0 + r < n && j0 + tx < n ? P[(size_t)(i0 + r) * np + j0 + tx] : 0.0;
      ls[r][tx] = j0 + r < n && q < r16 ? L0[(size_t)(j0 + r) * ld0 + q] : 0.f;
    }
    __syncthreads();
#pragma unroll 8
    for (int j = 0; j < 32; ++j) {
      const double l = ls[j][tx];
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] = fma(ps[ty + 8 * k][j], l, acc[k]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (i0 + ty + 8 * k < n && q < r16) Y[(size_t)(i0 + ty + 8 * k) * r16 + q] = acc[k];
}

// M = L0^T Y, r16 x r16; one block per 16 x 16 tile.
__global__ void __launch_bounds__(256) fact_m_kernel(const float* __restrict__ L0, int ld0, const double* __restrict__ Y,
                                                     int n, const int* __restrict__ rank, double* __restrict__ M) {
  __shared__ float ls[32][17];
  __shared__ double ys[32][17];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, a = blockIdx.x * 16, b = blockIdx.y * 16;
  const int r16 = ceil16(*rank);
  if (*rank == 0 || a >= r16 || b > a) return;   // the lower triangle is read
  double acc = 0.0;
  for (int i0 = 0; i0 < n; i0 += 32) {
    for (int r = ty; r < 32; r += 16) {
      const bool in = i0 + r < n;
      ls[r][tx] = in ? L0[(size_t)(i0 + r) * ld0 + a + tx] : 0.f;
      ys[r][tx] = in ? Y[(size_t)(i0 + r) * r16 + b + tx] : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int i = 0; i < 32; ++i) acc = fma((double)ls[i][ty], ys[i][tx], acc);
    __syncthreads();
  }
  M[(size_t)(a + ty) * r16 + b + tx] = acc;
}

// Lower Cholesky factor of the leading r x r block of M (one CTA), as its transpose in CT (CT[k * r16 + i] =
// C_ik, i > k; 1 / C_kk for i = k).  Panels of CHOL_NB columns: thread i holds row i of the panel in
// registers (one barrier a column), then all threads update what is right of it from the panel in shared
// memory.  A column whose pivot is lost in rounding (1e-12 of its diagonal element: a pivot of L0 that was
// the input's rounding) is left out, zero in CT; the residual check sees whether that mattered.
constexpr int CHOL_NB = 16, CHOL_THREADS = 1024;
__global__ void __launch_bounds__(CHOL_THREADS) fact_chol_kernel(double* __restrict__ M, const int* __restrict__ rank,
                                                                uint32_t smem, double* __restrict__ CT) {
  extern __shared__ double chol_s[];
  __shared__ double prow[2][CHOL_NB];
  __shared__ double pan[kFactorMaxR16][CHOL_NB + 1];   // the panel, scaled: C_ik
  const int t = threadIdx.x, tx = t & 31, ty = t >> 5;
  const int r = *rank, r16 = ceil16(r);
  if (r == 0) return;
  const bool in_smem = (uint32_t)r * (uint32_t)(r16 + 1) * 8u <= smem;   // (beside the panel)
  double* a = in_smem ? chol_s : M;
  const int ld = in_smem ? r16 + 1 : r16;
  if (in_smem)
    for (int i = ty; i < r; i += 32)
      for (int j = tx; j <= i; j += 32) a[i * ld + j] = M[(size_t)i * r16 + j];
  double least = 0.0;   // thread i: the least pivot of column i
  __syncthreads();
  if (t < r) least = 1e-12 * a[t * ld + t];
  __syncthreads();
  for (int k0 = 0; k0 < r; k0 += CHOL_NB) {
    const int nb = min(CHOL_NB, r - k0);
    double v[CHOL_NB];
    const bool mine = t < r && t >= k0;
#pragma unroll
    for (int j = 0; j < CHOL_NB; ++j) v[j] = mine && j < nb && k0 + j <= t ? a[t * ld + k0 + j] : 0.0;
#pragma unroll
    for (int j = 0; j < CHOL_NB; ++j) {
      if (j < nb) {
        // row k0 + j has its final values of columns <= j: it publishes column j's C of the rows below
        if (t == k0 + j) {
          const double s = v[j] > least ? rsqrt(v[j]) : 0.0;
          prow[j & 1][0] = s;
        }
        __syncthreads();
        const double s = prow[j & 1][0];
        if (mine && t >= k0 + j) {
          v[j] = t == k0 + j ? s : v[j] * s;      // C_ij (the diagonal keeps 1 / C_jj)
          pan[t][j] = v[j];
        }
        __syncthreads();
        if (mine && t > k0 + j) {
          // columns right of j in the panel: a_ic -= C_ij C_cj
#pragma unroll
          for (int c2 = j + 1; c2 < CHOL_NB; ++c2)
            if (c2 < nb && k0 + c2 <= t) v[c2] = fma(-v[j], pan[k0 + c2][j], v[c2]);
        }
      }
    }
    __syncthreads();
    if (mine) {
      for (int j = 0; j < nb; ++j)
        if (k0 + j <= t) CT[(size_t)(k0 + j) * r16 + t] = pan[t][j];
    }
    // what is right of the panel: a_ij -= sum_k C_ik C_jk (the panel's diagonal is above these rows)
    const int k1 = k0 + nb;
    for (int i = k1 + ty; i < r; i += 32) {
      double ci[CHOL_NB];
#pragma unroll
      for (int k = 0; k < CHOL_NB; ++k) ci[k] = k < nb ? pan[i][k] : 0.0;
      for (int j = k1 + tx; j <= i; j += 32) {
        double x = a[i * ld + j];
#pragma unroll
        for (int k = 0; k < CHOL_NB; ++k) x = fma(-ci[k], k < nb ? pan[j][k] : 0.0, x);
        a[i * ld + j] = x;
      }
    }
    __syncthreads();
  }
}

// L = Y C^-T row by row (a warp each; lane l holds columns l, l + 32, ...; 32 rows of C^T at a time in shared
// memory), in place, and the largest |L_iq| 2^-s_i of each column (as ordered bits of a non-negative double).
constexpr int SOLVE_WARPS = 8;
__global__ void __launch_bounds__(32 * SOLVE_WARPS) fact_solve_kernel(double* __restrict__ Y,
                                                                      const double* __restrict__ CT, int n,
                                                                      const int* __restrict__ rank,
                                                                      const double* __restrict__ inv_s,
                                                                      unsigned long long* __restrict__ colmax) {
  extern __shared__ double ct_s[];   // 32 x r16
  const int r = *rank, r16 = ceil16(r);
  if (r == 0) return;
  const int row = blockIdx.x * SOLVE_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const bool in = row < n;
  double y[kFactorMaxR16 / 32];
#pragma unroll
  for (int b = 0; b < kFactorMaxR16 / 32; ++b)
    y[b] = in && 32 * b + lane < r ? Y[(size_t)row * r16 + 32 * b + lane] : 0.0;
#pragma unroll
  for (int b = 0; b < kFactorMaxR16 / 32; ++b) {
    if (32 * b >= r) break;
    const int ne = min(32, r - 32 * b);
    __syncthreads();
    for (int i = threadIdx.x; i < ne * r16; i += 32 * SOLVE_WARPS) ct_s[i] = CT[(size_t)32 * b * r16 + i];
    __syncthreads();
    for (int e = 0; e < ne; ++e) {
      const int k = 32 * b + e;
      const double* c = ct_s + e * r16;
      const double x = __shfl_sync(0xffffffffu, y[b], e) * c[k];   // (the diagonal holds 1 / C_kk)
      if (lane == e) y[b] = x;
#pragma unroll
      for (int b2 = 0; b2 < kFactorMaxR16 / 32; ++b2)
        if (b2 >= b && 32 * b2 + lane > k && 32 * b2 + lane < r) y[b2] = fma(-c[32 * b2 + lane], x, y[b2]);
    }
  }
  if (!in) return;
  const double sc = inv_s[row];
#pragma unroll
  for (int b = 0; b < kFactorMaxR16 / 32; ++b)
    if (32 * b + lane < r16) {
      Y[(size_t)row * r16 + 32 * b + lane] = y[b];
      atomicMax(colmax + 32 * b + lane, (unsigned long long)__double_as_longlong(fabs(y[b]) * sc));
    }
}

// Column scales: 2^h_q brings the column's largest scaled element near 2^14 (h in [-100, 100]); then
// 2^-h_q in FP32 for the squares (0 for the padding columns).  Thread q of one block, q < r16.
__device__ __forceinline__ void column_scale(const unsigned long long* __restrict__ colmax, int q, int r,
                                             double* __restrict__ two_h, float* __restrict__ hscale) {
  const double mx = __longlong_as_double((long long)colmax[q]);
  int h = mx > 0 ? (int)floor(log2(16000.0 / mx)) : 0;
  h = max(-100, min(100, h));
  two_h[q] = q < r ? ldexp(1.0, h) : 0.0;
  hscale[q] = q < r ? ldexpf(1.0f, -h) : 0.f;
}

// Raises *bad when some |P_ij - sum_q L_iq L_jq| (i >= j) exceeds rel * dmax; L row i at L[i * r16].  One block per
// 32 x 32 tile on or below the diagonal.  The first block also forms the column scales.
__global__ void __launch_bounds__(256) fact_residual_kernel(const double* __restrict__ P, int np,
                                                            const double* __restrict__ L, int n,
                                                            const int* __restrict__ rank, double rel,
                                                            const double* __restrict__ dmax, int* bad,
                                                            const unsigned long long* __restrict__ colmax,
                                                            double* __restrict__ two_h, float* __restrict__ hscale) {
  __shared__ double li[32][33], lj[32][33];
  const int r = *rank, ld = ceil16(r);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  if (r == 0 || j0 > i0) return;
  if (i0 == 0 && (int)threadIdx.x < ld) column_scale(colmax, threadIdx.x, r, two_h, hscale);
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int q0 = 0; q0 < r; q0 += 32) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int x = ty + 8 * k;
      const bool q = q0 + tx < r;
      li[x][tx] = q && i0 + x < n ? L[(size_t)(i0 + x) * ld + q0 + tx] : 0.0;
      lj[x][tx] = q && j0 + x < n ? L[(size_t)(j0 + x) * ld + q0 + tx] : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int q = 0; q < 32; ++q) {
      const double b = lj[tx][q];
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] = fma(li[ty + 8 * k][q], b, acc[k]);
    }
    __syncthreads();
  }
  const double tol = rel * *dmax;   // max |P_jk| <= max_j P_jj for a positive semi-definite P
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = i0 + ty + 8 * k, j = j0 + tx;
    if (i < n && j <= i && !(fabs(P[(size_t)i * np + j] - acc[k]) <= tol)) *bad = 1;
  }
}

// The factor as the kernel reads it: block u holds the 16 columns of unit u for every factor column
// q < r16, one row of 32 bytes per q and piece (hi rows then lo rows), the two 16-byte halves of a row
// exchanged when bit 2 of q is set.
// Element: W = L_jq 2^-s_j 2^h_q of the column's function j, split into hi + lo; zero for padding.
// The last kernel of a factorisation also says what it came to: the rank (0 where the check failed) in *usable for the
// kernels and a host that waits, and with the factorisation's number in page-locked host memory for one that does not.
__global__ void fact_split_kernel(const double* __restrict__ L, const int* __restrict__ rank, const int* __restrict__ column,
                                  int nunits, const double* __restrict__ inv_s, const double* __restrict__ two_h, int fmt,
                                  int nsplit, uint8_t* __restrict__ out, const int* __restrict__ bad, int* usable,
                                  uint32_t number, volatile unsigned long long* mail) {
  const int r = *rank, r16 = ceil16(r), ld = r16;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const int u = *bad ? 0 : r;
    *usable = u;
    *mail = (unsigned long long)number << 32 | (unsigned)u;
  }
  if (r == 0) return;
  const int64_t tot = (int64_t)nunits * 16 * r16;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < tot; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i / r16), q = (int)(i - (int64_t)c * r16), u = c >> 4;
    const int j = column[c];
    const double w = (j >= 0 && q < r) ? L[(size_t)j * ld + q] * inv_s[j] * two_h[q] : 0.0;
    const int e = c & 15, pe = ((((e >> 3) ^ (q >> 2)) & 1) << 3) | (e & 7);
    const size_t blk = (size_t)u * nsplit * r16 * 16, row = (size_t)q * 16 + pe, half = (size_t)r16 * 16;
    uint16_t hi, lo;
    if (fmt == 0) {
      const __half h = __float2half_rn((float)w);
      hi = __half_as_ushort(h);
      lo = __half_as_ushort(__float2half_rn((float)(w - (double)__half2float(h))));
    } else {
      const __nv_bfloat16 h = __float2bfloat16_rn((float)w);
      hi = __bfloat16_as_ushort(h);
      lo = __bfloat16_as_ushort(__float2bfloat16_rn((float)(w - (double)__bfloat162float(h))));
    }
    uint16_t* o = reinterpret_cast<uint16_t*>(out) + blk + row;
    o[0] = hi;
    if (nsplit == 2) o[half] = lo;
  }
}

// The device's decision for a call that takes ranks up to `limit`.
__global__ void fact_decide_kernel(const int* __restrict__ usable, int limit, int nunits, int64_t avail, int abytes,
                                   int nsplit, FactDecision* out) {
  const int r = *usable <= limit ? *usable : 0;
  const FactShape f = fact_shape(r, nunits);
  out->shape = f;
  out->plan = fact_plan(avail, abytes, nsplit * f.r16 * 32, nunits, true);
  out->rank = r;
}

constexpr int kBf16MaxRank = 128;
constexpr double kFactorTol = 1e-7;
constexpr double kFactorResid = 2e-7;

}  // namespace

static qmt_status launch_pivot(qmt_mol* m, int rmax, int limit, double* L, float* L0, int ld0, int* info, double* dmax,
                               unsigned long long* zero, int nzero, cudaStream_t s) {
  const int n = m->norbs;
  int maxsm = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  QMT_CUDA(cudaFuncSetAttribute(fact_pivot_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  for (int ncta = n > 320 ? PIV_MAX_CTAS : (n > 128 ? 8 : 1); ncta >= 1; ncta /= 2) {
    PivotArgs a{};
    a.P = m->d_P64.as<double>();
    a.np = m->npad;
    a.n = n;
    a.rmax = rmax;
    a.rows = (n + ncta - 1) / ncta;
    a.ld = rmax + 8;   // (four rows of a warp on two sets of banks)
    a.limit = limit;
    a.tol = kFactorTol;
    a.L = L;
    a.L0 = L0;
    a.ld0 = ld0;
    a.info = info;
    a.dmax = dmax;
    a.zero = zero;
    a.nzero = nzero;
    a.usable = m->fact_usable();
    a.number = m->fact_number;
    a.mail = m->fact_mail;
    const size_t base = (size_t)(a.rows + rmax) * sizeof(double), rows = (size_t)a.rows * a.ld * sizeof(double);
    if (base > (size_t)maxsm - 2048) continue;
    a.rows_in_smem = base + rows <= (size_t)maxsm - 2048 ? 1 : 0;
    const size_t smem = base + (a.rows_in_smem ? rows : 0);
    QMT_CUDA(cudaFuncSetAttribute(fact_pivot_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ncta);
    cfg.blockDim = dim3(PIV_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ncta;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int nclusters = 0;
    if (ncta > 1 &&
        (cudaOccupancyMaxActiveClusters(&nclusters, fact_pivot_kernel, &cfg) != cudaSuccess || nclusters < 1)) {
      cudaGetLastError();   // a smaller cluster
      continue;
    }
    QMT_CUDA(cudaLaunchKernelEx(&cfg, fact_pivot_kernel, a));
    note_launches(1);
    return QMT_OK;
  }
  return fail(QMT_BAD_ARG, "factorisation does not fit in shared memory");
}

qmt_status ensure_unit_tables(qmt_mol* m, const std::vector<float>& fs, cudaStream_t s) {
  const UnitTables t = build_units(m, fs);
  const size_t wb = t.words.size() * sizeof(int4), cb = t.column.size() * sizeof(int);
  qmt_status st = m->d_fact_tab.reserve(wb + cb);
  if (st) return st;
  // pageable uploads return once the data is staged, so the host vectors may go
  QMT_CUDA(cudaMemcpyAsync(m->d_fact_tab.ptr, t.words.data(), wb, cudaMemcpyHostToDevice, s));
  QMT_CUDA(cudaMemcpyAsync(m->d_fact_tab.as<uint8_t>() + wb, t.column.data(), cb, cudaMemcpyHostToDevice, s));
  m->fact_units = t.nunits;
  m->fact_col_off = wb;
  return QMT_OK;
}

static int rank_limit(int n16, int fmt, bool any_rank) {
  if (fmt != 0) return std::min(kBf16MaxRank, n16 / 2);
  return any_rank && n16 <= kFactorMaxR16 ? n16 : std::min(kFactorMaxR16, n16 / 2);
}
int factor_limit(const qmt_mol* m, int fmt, bool any_rank) {
  const int lim = rank_limit((m->norbs + 15) / 16 * 16, fmt, any_rank);
  // a density matrix of N_e electrons whose occupations are at most 2 has rank >= N_e / 2: with
  // the nuclear charge for N_e (ions of up to 16 charges allowed for) a rank above the limit is known
  // without factoring
  return 0.5 * m->qtot > std::max(16, lim) + 8 ? 0 : lim;
}

// What the device has left of the molecule's last factorisation in the page-locked word; with `pending` also a rank that
// is still to be checked.
static bool mail_arrived(const qmt_mol* m, unsigned pending, unsigned* word) {
  const unsigned long long mail = *m->fact_mail;
  *word = (unsigned)mail;
  return (uint32_t)(mail >> 32) == m->fact_number && !(*word & kMailPending & ~pending);
}
// Polled for as long as the stream works: the word is there before a copy of the rank and a synchronisation would have
// been (a first call with a sum, 16^3 points: 218 -> 208 us).
static qmt_status read_mail(qmt_mol* m, unsigned pending, unsigned* word, cudaStream_t s) {
  for (;;) {
    const cudaError_t e = cudaStreamQuery(s);   // (before the look: what the stream has done is then there)
    if (mail_arrived(m, pending, word)) {
      if (e == cudaErrorNotReady) cudaGetLastError();   // (the query leaves its answer there)
      return QMT_OK;
    }
    if (e != cudaErrorNotReady) {
      QMT_CUDA(e);
      return fail(QMT_CUDA_ERR, "the factorisation left no rank");
    }
    cudaGetLastError();
  }
}

// A density matrix of rank r (r = occupied orbitals for an SCF density, P = 2 C_occ C_occ^T) is
// P = L L^T with L n x r.  L comes from a pivoted Cholesky factorisation (fact_pivot_kernel), stopped
// once every remaining diagonal element is at most kFactorTol of the largest one, and is refined; it is
// used when the matrix it leaves out is at most kFactorResid of max |P| (float32 input rounding is
// ~6e-8).  A matrix that is not positive semi-definite, or of high rank, takes the unfactored path.
// The scaled factor W_jk = L_jk 2^(h_k - s_j) (so Phi' W = 2^h_k (Phi L)_k, each column scaled to a
// maximum near 2^14) goes to the blocks of fact_split_kernel.  Unless the call may wait, nothing does: the rank and the
// check stay on the device until factor_rank reads them.
qmt_status ensure_factor(qmt_mol* m, int prec, int fmt, int nsplit, int kpad, bool any_rank, bool wait,
                         cudaStream_t s) {
  qmt_status st;
  // built for this precision (rank -1: the device knows), or refused by at least this rank limit
  int rank = 0;
  if (m->fact_prec == prec && (st = factor_rank(m, false, &rank, s))) return st;
  if (m->fact_prec == prec && (rank > 0 || m->fact_any_rank || !any_rank)) return QMT_OK;
  if ((st = ensure_basis_operands(m, kpad, s))) return st;
  const int n = m->norbs, np = m->npad, n16 = (n + 15) / 16 * 16;
  m->fact_prec = -1;   // (until all of it is enqueued)
  // device scratch: L (FP64), Y (then the refined L), M, C^T, column maxima, info, L0.  The kernels work on whole
  // blocks of 16 columns, so it is sized by the rank limit rounded up to them (n16 / 2 is an odd multiple of 8 for
  // every second n16); for any rank where that may be asked for later, so that a call being captured in a graph
  // allocates nothing.
  const int rmax = std::max(16, rank_limit(n16, fmt, any_rank));
  const int rbuf = (std::max(16, rank_limit(n16, fmt, true)) + 15) / 16 * 16;
  const size_t nr = (size_t)n * rbuf, rr = (size_t)rbuf * rbuf;
  if ((st = m->d_fact_L.reserve((2 * nr + 2 * rr + rbuf + 8) * sizeof(double) + nr * sizeof(float))) ||
      (st = m->d_fact_scale.reserve(kFactorMaxR16 * (sizeof(double) + sizeof(float)))) ||
      (st = m->d_fact_B.reserve((size_t)m->fact_units * nsplit * rbuf * 32)))
    return st;
  const int limit = factor_limit(m, fmt, any_rank);
  if (limit == 0) {
    m->fact_prec = prec;
    m->fact_any_rank = any_rank;
    m->fact_rank = 0;
    return QMT_OK;
  }
  double* Lp = m->d_fact_L.as<double>();
  double* Y = Lp + nr;
  double* M = Y + nr;
  double* CT = M + rr;
  unsigned long long* colmax = reinterpret_cast<unsigned long long*>(CT + rr);
  int* info = reinterpret_cast<int*>(colmax + rbuf);
  double* dmax = reinterpret_cast<double*>(colmax + rbuf + 1);
  int* bad = reinterpret_cast<int*>(colmax + rbuf + 2);
  float* L0 = reinterpret_cast<float*>(colmax + rbuf + 8);
  double* two_h = m->d_fact_scale.as<double>();
  const double* P = m->d_P64.as<double>();
  const int r16max = (rmax + 15) / 16 * 16;   // <= rbuf
  if (++m->fact_number == 0) m->fact_number = 1;
  if ((st = launch_pivot(m, rmax, limit, Lp, L0, rbuf, info, dmax, colmax, rbuf + 8, s))) return st;
  if (wait) {   // the pivots alone may refuse the matrix, and the rest need not run
    unsigned word = 0;
    if ((st = read_mail(m, kMailPending, &word, s))) return st;
    if (word == 0) {
      m->fact_prec = prec;
      m->fact_any_rank = any_rank;
      m->fact_rank = 0;
      return QMT_OK;
    }
  }
  // refined, and what the factor then leaves out, max |P - L L^T|, checked
  fact_y_kernel<<<dim3((n + 31) / 32, (r16max + 31) / 32), 256, 0, s>>>(P, np, L0, rbuf, n, info, Y);
  QMT_CHECK_LAUNCH("fact_y_kernel");
  fact_m_kernel<<<dim3(r16max / 16, r16max / 16), 256, 0, s>>>(L0, rbuf, Y, n, info, M);
  QMT_CHECK_LAUNCH("fact_m_kernel");
  const size_t csm = std::min<size_t>((size_t)rmax * (r16max + 1) * sizeof(double), 180u * 1024u);
  QMT_CUDA(cudaFuncSetAttribute(fact_chol_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 180 * 1024));
  fact_chol_kernel<<<1, CHOL_THREADS, csm, s>>>(M, info, (uint32_t)csm, CT);
  QMT_CHECK_LAUNCH("fact_chol_kernel");
  const size_t ssm = (size_t)32 * r16max * sizeof(double);
  QMT_CUDA(cudaFuncSetAttribute(fact_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                32 * kFactorMaxR16 * (int)sizeof(double)));
  fact_solve_kernel<<<(n + SOLVE_WARPS - 1) / SOLVE_WARPS, 32 * SOLVE_WARPS, ssm, s>>>(
      Y, CT, n, info, m->d_split_scale.as<double>(), colmax);
  QMT_CHECK_LAUNCH("fact_solve_kernel");
  fact_residual_kernel<<<dim3((n + 31) / 32, (n + 31) / 32), 256, 0, s>>>(
      P, np, Y, n, info, kFactorResid, dmax, bad, colmax, two_h, reinterpret_cast<float*>(two_h + kFactorMaxR16));
  QMT_CHECK_LAUNCH("fact_residual_kernel");
  const int64_t tot = (int64_t)m->fact_units * 16 * r16max;
  const int blocks = (int)std::min<int64_t>((tot + 255) / 256, (int64_t)sm_count() * 4);
  fact_split_kernel<<<std::max(blocks, 1), 256, 0, s>>>(
      Y, info, reinterpret_cast<const int*>(m->d_fact_tab.as<uint8_t>() + m->fact_col_off), m->fact_units,
      m->d_split_scale.as<double>(), two_h, fmt, nsplit, m->d_fact_B.as<uint8_t>(), bad, m->fact_usable(), m->fact_number,
      m->fact_mail);
  QMT_CHECK_LAUNCH("fact_split_kernel");
  m->fact_prec = prec;
  m->fact_any_rank = any_rank;
  m->fact_rank = -1;
  return QMT_OK;
}

qmt_status factor_rank(qmt_mol* m, bool wait, int* rank, cudaStream_t s) {
  unsigned word = 0;
  if (m->fact_rank < 0) {
    if (mail_arrived(m, 0, &word)) {
      m->fact_rank = (int)word;
    } else if (wait) {
      qmt_status st = read_mail(m, 0, &word, s);
      if (st) return st;
      m->fact_rank = (int)word;
    }
  }
  *rank = m->fact_rank;
  return QMT_OK;
}

void fact_mol_desc(const qmt_mol* m, int rank, const PointMap& pm, int64_t tile0, int64_t ntiles, float* qube,
                   double outscale, FactMol& d) {
  d = FactMol{};
  d.pm = pm;
  d.tile0 = tile0;
  d.ntiles = ntiles;
  d.nunits = m->fact_units;
  const FactShape f = fact_shape(rank, d.nunits);
  d.r16 = f.r16;
  d.sets = f.sets;
  d.na = f.na;
  d.B = m->d_fact_B.as<uint8_t>();
  d.units = m->d_fact_tab.as<int4>();
  d.coords = m->d_coords.as<float>();
  d.hscale = reinterpret_cast<const float*>(m->d_fact_scale.as<double>() + kFactorMaxR16);
  d.qube = qube;
  d.partials = m->d_partials.as<double>();
  d.outscale = outscale;
}

namespace {

// `blk`: bytes of the largest K-step block of the launch.  ON_DEVICE asks the device to decide for ranks up to `limit`.
template <int FMT, bool TWO, int WHO>
qmt_status launch_as(FactParams& p, int blk, const int* usable, int limit, cudaStream_t s) {
  auto kern = density_factored_kernel<FMT, TWO, WHO>;
  int maxsm = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaFuncAttributes fa;
  QMT_CUDA(cudaFuncGetAttributes(&fa, kern));
  const int64_t avail = (int64_t)maxsm - (int64_t)fa.sharedSizeBytes - 1024;
  const int abytes = GROUP * (TWO ? 2 * (int)PIECE : (int)PIECE);
  // (streamed, the largest rank has the fewest slots)
  if (fact_plan(avail, abytes, blk, p.one.nunits, false).nslots < (uint32_t)MIN_SLOTS)
    return fail(QMT_BAD_ARG, "factored density slots do not fit in shared memory");
  p.plan = fact_plan(avail, abytes, blk, p.one.nunits, WHO == ONE);
  size_t dyn = (size_t)p.plan.slot_bytes * p.plan.nslots + (p.plan.resident ? (size_t)blk * p.one.nunits : 0) + 1024;
  const int grid = (int)std::min<int64_t>(p.ntiles, sm_count());
  if (grid <= 0) return QMT_OK;
  if (WHO == ON_DEVICE) {
    dyn = (size_t)avail + 1024;
    fact_decide_kernel<<<1, 1, 0, s>>>(usable, limit, p.one.nunits, avail, abytes, TWO ? 2 : 1,
                                       const_cast<FactDecision*>(p.decision));
    QMT_CHECK_LAUNCH("fact_decide_kernel");
  }
  QMT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
  kern<<<grid, FACT_THREADS, dyn, s>>>(p);
  QMT_CHECK_LAUNCH("density_factored_kernel");
  return QMT_OK;
}

template <int FMT, bool TWO>
qmt_status launch_whose(FactParams& p, int blk, const int* usable, int limit, cudaStream_t s) {
  if (p.nmol > 1) return launch_as<FMT, TWO, MANY>(p, blk, usable, limit, s);
  if (p.decision) return launch_as<FMT, TWO, ON_DEVICE>(p, blk, usable, limit, s);
  return launch_as<FMT, TWO, ONE>(p, blk, usable, limit, s);
}

qmt_status launch_params(FactParams& p, int r16, int fmt, int nsplit, const int* usable, int limit, int* err,
                         cudaStream_t s) {
  p.fmt = (uint32_t)fmt;
  p.err = err;
  p.wait_ns = wait_limit_ns();
  const int blk = nsplit * r16 * 32;
  if (fmt == 0) return launch_whose<0, true>(p, blk, usable, limit, s);
  return nsplit == 2 ? launch_whose<1, true>(p, blk, usable, limit, s) : launch_whose<1, false>(p, blk, usable, limit, s);
}

}  // namespace

qmt_status launch_factored(const FactMol* host, const FactMol* dev, int nmol, int64_t ntiles, int fmt, int nsplit,
                           int* err, cudaStream_t s) {
  FactParams p{};
  int r16 = 0;
  for (int i = 0; i < nmol; ++i) r16 = std::max(r16, host[i].r16);
  if (nmol == 1) p.one = host[0];
  p.mols = dev;
  p.nmol = nmol;
  p.ntiles = ntiles;
  return launch_params(p, r16, fmt, nsplit, nullptr, 0, err, s);
}

qmt_status launch_factored_on_device(qmt_mol* m, const FactMol& d, int limit, int fmt, int nsplit, int* err,
                                     const FactDecision** decision, cudaStream_t s) {
  FactParams p{};
  p.one = d;
  p.nmol = 1;
  p.ntiles = d.ntiles;
  *decision = p.decision = reinterpret_cast<const FactDecision*>(m->fact_decision());
  return launch_params(p, d.r16, fmt, nsplit, m->fact_usable(), limit, err, s);
}

}  // namespace qmt
