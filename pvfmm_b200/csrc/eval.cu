// FMM evaluation on the device (FMM_Tree::RunFMM, reference
// include/fmm_tree.txx:237-738, evaluation halves of include/fmm_pts.txx).
//
// Data layout in HBM:
//   points     sorted by Morton key; FP64 SoA coordinates relative to the
//              centre of the point's leaf; FP64 densities [n_src][k0]
//   UE, DC     FP64 per node, [n_nodes][ns*ke]: upward equivalent densities
//              and downward check potentials (the reference's upward_equiv
//              and dnward_equiv, fmm_pts.txx:1306-1480)
//   spectra    per V-list parent, [parent][freq][child*ke+comp] complex, in
//              the working precision Real
// Precision forms:
//   plain  Real = double everywhere.
//   mixed  Real = float for the two dominant stages, the V-list (DFTs and
//          Hadamard products) and the near field (U list P2P, W list, D2T
//          target evaluation); FP32 tile sums are promoted to FP64 per
//          tile.  The check->equivalent chain (S2U and X check potentials,
//          the pseudo-inverse GEMMs, U2U, D2D) stays FP64: the SVD
//          pseudo-inverse amplifies check-potential errors by up to 1/(4 eps
//          max S), so FP32 check potentials would need the FP32 cutoff,
//          which alone costs ~8e-7 relative error at m=8.
// Stages:
//   S2U   check-surface evaluation + 2 FP64 tensor-core products (pinv
//         factors, fmm_pts.txx:4390-4426), the second one writing the leaves'
//         rows of UE (translate.cu)
//   U2U   one product per level over the contiguous child blocks, written to
//         the parents' rows (fmm_pts.txx:2017-2271)
//   V     pruned DFT of the 8 children, Hadamard with the 26 parent offsets,
//         pruned inverse DFT onto the children's check surfaces (fmm_pts.txx:2689-3759)
//   X     check-surface evaluation (fmm_pts.txx:4444-4736)
//   D2D   one product per level from the parents' rows into the contiguous
//         child blocks (fmm_pts.txx:3762-3790)
//   D2T   2 products (pinv factors, leaves' rows gathered and scaled by
//         2^-depth in the first), then with W and U one fused near-field
//         kernel per target leaf (fmm_pts.txx:4246-4426, 4746-5022, 5032-5418).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>

#include <cuda_fp16.h>

#include "fmm_context.cuh"

namespace pvfmm_b200 {
namespace {

constexpr int kNT = 128;  // threads per block of the point/surface kernels

template <class Real>
struct Cplx {
  Real re, im;
};

__device__ __forceinline__ void node_geom(const MKey& k, double& cx, double& cy, double& cz, double& half, int& depth) {
  unsigned int X, Y, Z, d;
  decode_key(k, X, Y, Z, d);
  const double h = 1.0 / (double)(1u << d);
  half = 0.5 * h;
  cx = X * (1.0 / kTwo30) + half;
  cy = Y * (1.0 / kTwo30) + half;
  cz = Z * (1.0 / kTwo30) + half;
  depth = (int)d;
}

// Periodic boundaries: moves a source node's centre by the unit-cube image
// shift of its list entry (code (sx+1) + 3(sy+1) + 9(sz+1)).
__device__ __forceinline__ void image_shift(unsigned char code, double& cx, double& cy, double& cz) {
  cx += (double)(code % 3) - 1.0;
  cy += (double)((code / 3) % 3) - 1.0;
  cz += (double)(code / 9) - 1.0;
}

// Target coordinate as (hi, lo) in Real.
template <class Real>
struct Pt {
  Real x, y, z, xl, yl, zl;
};
template <class Real>
__device__ __forceinline__ Pt<Real> make_pt(double x, double y, double z) {
  Pt<Real> p;
  p.x = (Real)x;
  p.y = (Real)y;
  p.z = (Real)z;
  p.xl = (Real)(x - (double)p.x);
  p.yl = (Real)(y - (double)p.y);
  p.zl = (Real)(z - (double)p.z);
  return p;
}

// ---------------------------------------------------------------------------
// Near field of one target leaf: D2T (own downward equivalent surface), W
// (upward equivalent surfaces of the W list) and U (points of the P2P list),
// fused.  One block per target leaf.
//
// The sources of all list entries are packed back to back into tiles of
// kTile records in shared memory (leaves hold a few dozen points, so one tile
// spans many entries), double-buffered so that one barrier per tile suffices.
// A record is one source point relative to the target leaf's centre plus its
// KS densities, stored as 16-byte chunks, chunk-major.  FP32 records also
// carry each coordinate's rounding remainder (hi + lo), so target - source
// keeps FP32 relative accuracy for close pairs.  Every thread evaluates two
// targets per loaded record; when a leaf has fewer than 2*kNF targets the
// source records are split among G groups of threads and the G partial sums
// are added in a fixed order.
// ---------------------------------------------------------------------------
constexpr int kNF = 128;        // threads per near-field block
#ifndef PVFMM_NEAR_MIN_BLOCKS_F32
#define PVFMM_NEAR_MIN_BLOCKS_F32 5  // resident blocks per SM the register budget is sized for
#endif
#ifndef PVFMM_NEAR_MIN_BLOCKS_F32_K1
#define PVFMM_NEAR_MIN_BLOCKS_F32_K1 6  // the same for one source density (Laplace kernels)
#endif
#ifndef PVFMM_NEAR_MIN_BLOCKS_F64
#define PVFMM_NEAR_MIN_BLOCKS_F64 5
#endif
#ifndef PVFMM_NEAR_TILE_MULT
#define PVFMM_NEAR_TILE_MULT 2
#endif
#ifndef PVFMM_NEAR_UNROLL
#define PVFMM_NEAR_UNROLL 1
#endif
#ifndef PVFMM_NEAR_GMAX
#define PVFMM_NEAR_GMAX 16  // most thread groups splitting the source records of a small leaf
#endif

constexpr int kNearUnroll = PVFMM_NEAR_UNROLL;      // unroll of the record loop
constexpr int kTile = PVFMM_NEAR_TILE_MULT * kNF;  // source records per tile
#ifndef PVFMM_NEAR_TILE_MULT_K1
#define PVFMM_NEAR_TILE_MULT_K1 2
#endif
// records per tile of the near-field kernel for Real, Ker (the FP32 kernels
// with one source density have the smallest records)
template <class Real, int Ker>
constexpr int near_tile() {
  return sizeof(Real) == 4 && KerDims<Ker>::KS == 1 ? PVFMM_NEAR_TILE_MULT_K1 * kNF : kTile;
}

template <class Real>
struct Vec16 {
  using type = double2;
};
template <>
struct Vec16<float> {
  using type = float4;
};

template <class Real, int KS>
struct Rec {
  static constexpr bool kLo = sizeof(Real) == 4;
  static constexpr int NV = (kLo ? 6 : 3) + KS;
  static constexpr int PER = 16 / (int)sizeof(Real);
  static constexpr int NC = (NV + PER - 1) / PER;
  static constexpr int NVP = NC * PER;
  // value slots: x y z f0 | xl yl zl f1 f2 (FP32);  x y z f0 f1 f2 (FP64)
  __host__ __device__ static constexpr int F(int i) { return kLo ? (i == 0 ? 3 : 6 + i) : 3 + i; }
};

template <class Real, int KS, int TS = kTile>
__device__ __forceinline__ void rec_store(typename Vec16<Real>::type* tile, int j, double x, double y, double z,
                                          const Real* f) {
  using R = Rec<Real, KS>;
  Real v[R::NVP];
#pragma unroll
  for (int i = 0; i < R::NVP; ++i) v[i] = 0;
  v[0] = (Real)x;
  v[1] = (Real)y;
  v[2] = (Real)z;
  if constexpr (R::kLo) {
    v[4] = (Real)(x - (double)v[0]);
    v[5] = (Real)(y - (double)v[1]);
    v[6] = (Real)(z - (double)v[2]);
  }
#pragma unroll
  for (int i = 0; i < KS; ++i) v[R::F(i)] = f[i];
#pragma unroll
  for (int c = 0; c < R::NC; ++c) {
    typename Vec16<Real>::type w;
    memcpy(&w, &v[c * R::PER], 16);
    tile[c * TS + j] = w;
  }
}

// Adds the records j = j0, j0+js, ... < n to two targets (FP64 accumulators;
// FP32 sums never run over more than one tile).
template <class Real, int Ker, bool Surface1 = false, int TS = kTile>
__device__ __forceinline__ void rec_sum2(const typename Vec16<Real>::type* tile, int n, int j0, int js,
                                         const Pt<Real>& pa, const Pt<Real>& pb, double (&acc)[2][KerDims<Ker>::KT]) {
  constexpr int KS = KerDims<Ker>::KS, KT = KerDims<Ker>::KT;
  using R = Rec<Real, KS>;
  // FP32 partial sums run over 16 records at most before going to FP64
  const int step = sizeof(Real) == 4 ? 16 * js : n;
  for (int jb = j0; jb < n; jb += step) {
  const int jend = sizeof(Real) == 4 ? min(n, jb + step) : n;
  Real ua[KT], ub[KT];
#pragma unroll
  for (int k = 0; k < KT; ++k) ua[k] = ub[k] = 0;
#pragma unroll kNearUnroll
  for (int j = jb; j < jend; j += js) {
    Real v[R::NVP];
#pragma unroll
    for (int c = 0; c < R::NC; ++c) {
      const typename Vec16<Real>::type w = tile[c * TS + j];
      memcpy(&v[c * R::PER], &w, 16);
    }
    Real f[KS];
#pragma unroll
    for (int i = 0; i < KS; ++i) f[i] = v[R::F(i)];
    Real rx, ry, rz;
    if constexpr (R::kLo) {
      rx = (pa.x - v[0]) + (pa.xl - v[4]);
      ry = (pa.y - v[1]) + (pa.yl - v[5]);
      rz = (pa.z - v[2]) + (pa.zl - v[6]);
    } else {
      rx = pa.x - v[0];
      ry = pa.y - v[1];
      rz = pa.z - v[2];
    }
    ker_eval<Ker, Real, Surface1>(rx, ry, rz, f, ua);
    if constexpr (R::kLo) {
      rx = (pb.x - v[0]) + (pb.xl - v[4]);
      ry = (pb.y - v[1]) + (pb.yl - v[5]);
      rz = (pb.z - v[2]) + (pb.zl - v[6]);
    } else {
      rx = pb.x - v[0];
      ry = pb.y - v[1];
      rz = pb.z - v[2];
    }
    ker_eval<Ker, Real, Surface1>(rx, ry, rz, f, ub);
  }
#pragma unroll
  for (int k = 0; k < KT; ++k) {
    acc[0][k] += (double)ua[k];
    acc[1][k] += (double)ub[k];
  }
  }
}

// ---------------------------------------------------------------------------
// Packed FP32 pairs (add/sub/mul/fma .f32x2 of sm_100): the mixed form's near
// field evaluates two sources against a target in the two halves of 64-bit
// registers, one instruction per operation for both (the same
// round-to-nearest FP32 operations as two scalar evaluations).
// ---------------------------------------------------------------------------
typedef unsigned long long f2_t;
__device__ __forceinline__ f2_t f2_pack(float lo, float hi) {
  f2_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) {
  f2_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2_t f2_sub(f2_t a, f2_t b) {
  f2_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) {
  f2_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
  f2_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// Kernels with a packed form (the others evaluate one source at a time).
template <int Ker>
constexpr bool kHasPacked = Ker == kKerLaplace || Ker == kKerLaplaceGrad || Ker == kKerLaplacePG || Ker == kKerStokes;

// ker_eval<Ker, float> for two sources at once: r = target - source per half,
// f the source densities.  1/r: one hardware reciprocal square root per half
// (0 for r2 == 0) and one packed Newton-Raphson step, kept at three
// operations as y (r2 y^2 - 3) = -2/r; the Laplace kernels sum with that
// value, -2 / r and (-2 / r)^3 being powers of two times the terms
// (packed_unit, taken out of the FP64 sums), and Stokes velocity, whose terms
// mix, scales it back.
template <int Ker>
__device__ __forceinline__ void ker_eval_x2(f2_t rx, f2_t ry, f2_t rz, const f2_t* f, f2_t* u) {
  const f2_t r2 = f2_fma(rz, rz, f2_fma(ry, ry, f2_mul(rx, rx)));
  float a, b;
  f2_unpack(r2, a, b);
  float ya, yb;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(ya) : "f"(a));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yb) : "f"(b));
  ya = a > 0.f ? ya : 0.f;
  yb = b > 0.f ? yb : 0.f;
  const f2_t y0 = f2_pack(ya, yb);
  const f2_t e = f2_fma(f2_mul(r2, y0), y0, f2_pack(-3.f, -3.f));
  if constexpr (Ker == kKerLaplace) {
    u[0] = f2_fma(f2_mul(y0, e), f[0], u[0]);
  } else if constexpr (Ker == kKerLaplaceGrad) {
    const f2_t y = f2_mul(y0, e);
    const f2_t fr3 = f2_mul(f2_mul(y, y), f2_mul(y, f[0]));
    u[0] = f2_fma(rx, fr3, u[0]);
    u[1] = f2_fma(ry, fr3, u[1]);
    u[2] = f2_fma(rz, fr3, u[2]);
  } else if constexpr (Ker == kKerLaplacePG) {
    const f2_t y = f2_mul(y0, e);
    const f2_t fr = f2_mul(y, f[0]);
    const f2_t fr3 = f2_mul(f2_mul(y, y), fr);
    u[0] = f2_add(u[0], fr);
    u[1] = f2_fma(rx, fr3, u[1]);
    u[2] = f2_fma(ry, fr3, u[2]);
    u[3] = f2_fma(rz, fr3, u[3]);
  } else {  // Stokes velocity: u += (f + r (f.r) / r^2) / r
    const f2_t y = f2_mul(f2_mul(y0, f2_pack(-0.5f, -0.5f)), e);
    const f2_t ip = f2_mul(f2_fma(f[2], rz, f2_fma(f[1], ry, f2_mul(f[0], rx))), f2_mul(y, y));
    u[0] = f2_fma(y, f2_fma(rx, ip, f[0]), u[0]);
    u[1] = f2_fma(y, f2_fma(ry, ip, f[1]), u[1]);
    u[2] = f2_fma(y, f2_fma(rz, ip, f[2]), u[2]);
  }
}

// The densities of the kernels with 1/r^3 terms are stored divided by 8, so
// that those terms overflow no sooner than the kernel's own.  Component k of
// the packed evaluation is packed_unit times the kernel's.
template <int Ker>
constexpr float kPackedDen = Ker == kKerLaplaceGrad || Ker == kKerLaplacePG ? 0.125f : 1.f;
template <int Ker>
__host__ __device__ constexpr double packed_unit(int k) {
  return !kHasPacked<Ker> || Ker == kKerStokes ? 1.0
         : Ker == kKerLaplace                  ? -2.0
         : Ker == kKerLaplacePG && k == 0      ? -0.25
                                               : -1.0;
}

// Records of the packed evaluation: two consecutive sources share one record
// of pairs (v of the first, v of the second) for v = x y z f0 | xl yl zl f1 f2,
// two pairs per 16-byte chunk, chunk-major.  A chunk loads as two packed
// operands for either target, so no operand is duplicated into a pair in the
// loop (with pairs of targets every source value was).
template <int KS>
struct PairRec {
  static constexpr int NV = 6 + KS;
  static constexpr int NC = (NV + 1) / 2;
  __host__ __device__ static constexpr int F(int i) { return i == 0 ? 3 : 6 + i; }
};

// Sources 2j and 2j+1 (x, y, z, f of each; the densities times `den`).
template <int KS, int TP>
__device__ __forceinline__ void pair_store(float4* tile, int j, const double (&x)[2], const double (&y)[2],
                                           const double (&z)[2], const double (&f)[2][KS], float den) {
  using R = PairRec<KS>;
  float v[2 * R::NC][2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    v[0][u] = (float)x[u];
    v[1][u] = (float)y[u];
    v[2][u] = (float)z[u];
    v[4][u] = (float)(x[u] - (double)v[0][u]);
    v[5][u] = (float)(y[u] - (double)v[1][u]);
    v[6][u] = (float)(z[u] - (double)v[2][u]);
#pragma unroll
    for (int i = 0; i < KS; ++i) v[R::F(i)][u] = (float)f[u][i] * den;
    if (R::NV & 1) v[R::NV][u] = 0.f;
  }
#pragma unroll
  for (int c = 0; c < R::NC; ++c)
    tile[c * TP + j] = make_float4(v[2 * c][0], v[2 * c][1], v[2 * c + 1][0], v[2 * c + 1][1]);
}

// Adds the pairs j = j0, j0+js, ... < n of the tile (TP pairs) to two targets
// (FP64 accumulators, in packed_unit units).
template <int Ker, int TP>
__device__ __forceinline__ void pair_sum2(const float4* tile, int n, int j0, int js, const Pt<float>& pa,
                                          const Pt<float>& pb, double (&acc)[2][KerDims<Ker>::KT]) {
  constexpr int KS = KerDims<Ker>::KS, KT = KerDims<Ker>::KT;
  using R = PairRec<KS>;
  f2_t p[2][6];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const Pt<float>& t = q ? pb : pa;
    const float w[6] = {t.x, t.y, t.z, t.xl, t.yl, t.zl};
#pragma unroll
    for (int i = 0; i < 6; ++i) p[q][i] = f2_pack(w[i], w[i]);
  }
  // FP32 partial sums run over 16 records at most before going to FP64
  const int step = 16 * js;
  for (int jb = j0; jb < n; jb += step) {
    const int jend = min(n, jb + step);
    f2_t u[2][KT];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int k = 0; k < KT; ++k) u[q][k] = 0ull;  // (0.f, 0.f)
#pragma unroll kNearUnroll
    for (int j = jb; j < jend; j += js) {
      f2_t v[2 * R::NC];
#pragma unroll
      for (int c = 0; c < R::NC; ++c) {
        const float4 w = tile[c * TP + j];
        v[2 * c] = f2_pack(w.x, w.y);
        v[2 * c + 1] = f2_pack(w.z, w.w);
      }
      f2_t f[KS];
#pragma unroll
      for (int i = 0; i < KS; ++i) f[i] = v[R::F(i)];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const f2_t rx = f2_add(f2_sub(p[q][0], v[0]), f2_sub(p[q][3], v[4]));
        const f2_t ry = f2_add(f2_sub(p[q][1], v[1]), f2_sub(p[q][4], v[5]));
        const f2_t rz = f2_add(f2_sub(p[q][2], v[2]), f2_sub(p[q][5], v[6]));
        ker_eval_x2<Ker>(rx, ry, rz, f, u[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int k = 0; k < KT; ++k) {
        float a, b;
        f2_unpack(u[q][k], a, b);
        acc[q][k] += (double)a + (double)b;
      }
  }
}

// One list entry of a target leaf as a segment of the packed source stream:
// the points of a leaf (kind 0, `node` = first point), the upward equivalent
// surface of a node (kind 1, `node` = node index) or the leaf's own downward
// equivalent surface (kind 2, `node` = row of the D2T densities).  The offset
// between node centres is a small multiple of a power of two, exact in FP32.
struct NearSeg {
  float ox, oy, oz;
  int node;
  int kind_depth;  // kind | depth << 4
};
constexpr int kSegCap = 128;  // list entries per batch

// kDbl: the double-layer pass, P2P sources only (surface values in `den`),
// added to pot.  with_p2p = 0: no P2P sources (no single-layer densities;
// the W and D2T entries still come from the expansions).
template <class Real, int Ker, bool kDbl = false>
__global__ void __launch_bounds__(kNF, sizeof(Real) == 8       ? PVFMM_NEAR_MIN_BLOCKS_F64
                                       : KerDims<Ker>::KS == 1 ? PVFMM_NEAR_MIN_BLOCKS_F32_K1
                                                               : PVFMM_NEAR_MIN_BLOCKS_F32)
    near_field_kernel(const int* __restrict__ tleaf, const MKey* __restrict__ keys, const int* __restrict__ tlo,
                      const int* __restrict__ thi, const int* __restrict__ slo, const int* __restrict__ shi,
                      const int* __restrict__ p_off, const int* __restrict__ p_list, const int* __restrict__ w_off,
                      const int* __restrict__ w_list, const unsigned char* __restrict__ p_img,
                      const unsigned char* __restrict__ w_img, const double* __restrict__ tx,
                      const double* __restrict__ ty, const double* __restrict__ tz, const double* __restrict__ sx,
                      const double* __restrict__ sy, const double* __restrict__ sz, const double* __restrict__ den,
                      const double* __restrict__ ue, const double* __restrict__ de, const double* __restrict__ usurf,
                      int ns, double scale, int with_p2p, double* __restrict__ pot) {
  constexpr int KS = KerDims<Ker>::KS, KT = KerDims<Ker>::KT;
  constexpr bool kF32 = sizeof(Real) == 4;
  constexpr bool kPacked = kF32 && kHasPacked<Ker>;
  constexpr int TPT = 2;  // targets per thread
  constexpr int TILE = near_tile<Real, Ker>();  // source records per tile
  constexpr int RPT = TILE / kNF;                 // records each thread fetches per tile
  using V = typename Vec16<Real>::type;
  constexpr int TILE_V = kPacked ? PairRec<KS>::NC * (TILE / 2) : Rec<Real, KS>::NC * TILE;
  __shared__ V tiles[2][TILE_V];
  // the FP64 D2T records of the mixed form come first and reuse the tiles
  // (a barrier separates their last read from the first tile store), and so
  // do the partial sums of the final fixed-order reduction
  constexpr int TILE64 = Rec<double, KS>::NC * TILE <= 2 * TILE_V ? TILE : TILE / 2;
  static_assert(Rec<double, KS>::NC * TILE64 <= 2 * TILE_V, "D2T records fit the tiles");
  double2* tile64 = reinterpret_cast<double2*>(&tiles[0][0]);
  static_assert(sizeof(tiles) >= sizeof(double) * kNF * TPT * KT, "reduction buffer larger than the tiles");
  double(*red)[TPT][KT] = reinterpret_cast<double(*)[TPT][KT]>(&tiles[0][0]);
  __shared__ NearSeg seg[kSegCap];
  __shared__ int start[kSegCap + 1];
  const int b = blockIdx.x;
  const int T = tleaf[b];
  double cx, cy, cz, half;
  int dT;
  node_geom(keys[T], cx, cy, cz, half, dT);
  const int t0 = tlo[T], nt = thi[T] - t0;
  const int dim = ns * KS;
  const int wb = kDbl ? 0 : w_off[T], nW = kDbl ? 0 : w_off[T + 1] - wb;
  const int pbeg = p_off[T], nP = with_p2p ? p_off[T + 1] - pbeg : 0;
  const int nD = (!kDbl && de && !kF32) ? 1 : 0;  // plain form: D2T is a segment of the stream
  const int n_ent = nD + nW + nP;
  int buf = 0;
  for (int c0 = 0; c0 < nt; c0 += TPT * kNF) {
    // thread (ti, g): targets ti + q nc (q < TPT) of the chunk, source records
    // g, g + G, ... of every tile
    const int m = min(TPT * kNF, nt - c0);
    const int nc = (m + TPT - 1) / TPT;
    const int G = min(PVFMM_NEAR_GMAX, kNF / nc);
    const int ti = threadIdx.x % nc, g = threadIdx.x / nc;
    const bool active = g < G;
    int tq[TPT];
    Pt<Real> pt[TPT];
#pragma unroll
    for (int q = 0; q < TPT; ++q) {
      tq[q] = t0 + c0 + (ti + q * nc < m ? ti + q * nc : ti);  // a missing target repeats the first
      pt[q] = make_pt<Real>(tx[tq[q]], ty[tq[q]], tz[tq[q]]);
    }
    double acc[TPT][KT];
#pragma unroll
    for (int q = 0; q < TPT; ++q)
#pragma unroll
      for (int k = 0; k < KT; ++k) acc[q][k] = 0;
    // D2T of the mixed form: the downward equivalent densities come from the
    // FP64-cutoff pseudo-inverse, whose large cancelling components only FP64
    // sums resolve, so they are evaluated from FP64 records.
    if constexpr (kF32 && !kDbl) {
      if (de) {
        const double hr = half * kRad1;
        const double* dens = de + (long)b * dim;
        for (int k0 = 0; k0 < ns; k0 += TILE64) {
          const int n = min(TILE64, ns - k0);
          __syncthreads();
          for (int i = threadIdx.x; i < n; i += kNF) {
            const int k = k0 + i;
            double f[KS];
#pragma unroll
            for (int c = 0; c < KS; ++c) f[c] = dens[k * KS + c];
            rec_store<double, KS, TILE64>(tile64, i, hr * usurf[k * 3 + 0], hr * usurf[k * 3 + 1],
                                        hr * usurf[k * 3 + 2], f);
          }
          __syncthreads();
          if (active)
#pragma unroll
            for (int h = 0; h < TPT / 2; ++h) {
              const Pt<double> pa64 = make_pt<double>(tx[tq[2 * h]], ty[tq[2 * h]], tz[tq[2 * h]]);
              const Pt<double> pb64 = make_pt<double>(tx[tq[2 * h + 1]], ty[tq[2 * h + 1]], tz[tq[2 * h + 1]]);
              rec_sum2<double, Ker, true, TILE64>(tile64, n, g, G, pa64, pb64,
                                          *reinterpret_cast<double(*)[2][KT]>(&acc[2 * h][0]));
            }
        }
        if constexpr (kPacked) {
#pragma unroll
          for (int q = 0; q < TPT; ++q)
#pragma unroll
            for (int k = 0; k < KT; ++k) acc[q][k] *= packed_unit<Ker>(k);
        }
      }
    }
    for (int e0 = 0; e0 < n_ent; e0 += kSegCap) {
      const int ne = min(kSegCap, n_ent - e0);
      __syncthreads();  // the previous batch (or chunk) is done with seg, start and the tiles
      for (int i = threadIdx.x; i < ne; i += kNF) {
        const int e = e0 + i;
        NearSeg sg;
        int cnt;
        if (e < nD) {
          sg = {0.f, 0.f, 0.f, b, 2 | (dT << 4)};
          cnt = ns;
        } else {
          const bool is_w = e < nD + nW;
          const int q = is_w ? wb + e - nD : pbeg + e - nD - nW;
          const int S = is_w ? w_list[q] : p_list[q];
          double sxc, syc, szc, sh;
          int dS;
          node_geom(keys[S], sxc, syc, szc, sh, dS);
          if (p_img) image_shift(is_w ? w_img[q] : p_img[q], sxc, syc, szc);
          sg.ox = (float)(sxc - cx);
          sg.oy = (float)(syc - cy);
          sg.oz = (float)(szc - cz);
          if (is_w) {
            sg.node = S;
            sg.kind_depth = 1 | (dS << 4);
            cnt = ns;
          } else {
            sg.node = slo[S];
            sg.kind_depth = 0;
            cnt = shi[S] - slo[S];
          }
        }
        seg[i] = sg;
        start[i] = cnt;
      }
      __syncthreads();
      if (threadIdx.x < 32) {  // exclusive scan of the counts (4 entries per lane)
        const int lane = threadIdx.x;
        int v[4], sum = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int idx = lane * 4 + q;
          v[q] = idx < ne ? start[idx] : 0;
          sum += v[q];
        }
        int inc = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, inc, d);
          if (lane >= d) inc += y;
        }
        int ex = inc - sum;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int idx = lane * 4 + q;
          if (idx < ne) start[idx] = ex;
          ex += v[q];
        }
        if (lane == 31) start[ne] = inc;
      }
      __syncthreads();
      const int total = start[ne];
      const int ntile = (total + TILE - 1) / TILE;
      // records slot(u) of a tile, fetched one tile ahead
      auto slot = [&](int u) { return kPacked ? RPT * (int)threadIdx.x + u : (int)threadIdx.x + u * kNF; };
      double rx_[RPT], ry_[RPT], rz_[RPT], rf_[RPT][KS];
      auto fetch = [&](int t) {
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
          const int r = t * TILE + slot(u);
          if (r >= total) {
            if constexpr (kPacked) {  // a missing second source of a pair: density 0, off the leaf
              rx_[u] = ry_[u] = rz_[u] = 1;
#pragma unroll
              for (int c = 0; c < KS; ++c) rf_[u][c] = 0;
            }
            continue;
          }
          int lo = 0, hi = ne;  // largest s with start[s] <= r
          while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (start[mid] <= r) lo = mid;
            else hi = mid;
          }
          const NearSeg sg = seg[lo];
          const int i = r - start[lo];
          const int kind = sg.kind_depth & 15;
          if (kind == 0) {
            const int p = sg.node + i;
            rx_[u] = sx[p] + (double)sg.ox;
            ry_[u] = sy[p] + (double)sg.oy;
            rz_[u] = sz[p] + (double)sg.oz;
#pragma unroll
            for (int c = 0; c < KS; ++c) rf_[u][c] = den[(long)p * KS + c];
          } else {
            const double hr = ldexp(kind == 1 ? kRad0 : kRad1, -((sg.kind_depth >> 4) + 1));
            const double* dens = (kind == 1 ? ue : de) + (long)sg.node * dim;
            rx_[u] = (double)sg.ox + hr * usurf[i * 3 + 0];
            ry_[u] = (double)sg.oy + hr * usurf[i * 3 + 1];
            rz_[u] = (double)sg.oz + hr * usurf[i * 3 + 2];
#pragma unroll
            for (int c = 0; c < KS; ++c) rf_[u][c] = dens[i * KS + c];
          }
        }
      };
      if (ntile > 0) fetch(0);
      for (int t = 0; t < ntile; ++t) {
        const int n = min(TILE, total - t * TILE);
        if constexpr (kPacked) {
          static_assert(RPT == 2, "a thread stores the two sources of a pair");
          if (slot(0) < n) pair_store<KS, TILE / 2>(tiles[buf], threadIdx.x, rx_, ry_, rz_, rf_, kPackedDen<Ker>);
        } else {
#pragma unroll
          for (int u = 0; u < RPT; ++u) {
            const int j = slot(u);
            if (j < n) {
              Real f[KS];
#pragma unroll
              for (int c = 0; c < KS; ++c) f[c] = (Real)rf_[u][c];
              rec_store<Real, KS, TILE>(tiles[buf], j, rx_[u], ry_[u], rz_[u], f);
            }
          }
        }
        if (t + 1 < ntile) fetch(t + 1);
        __syncthreads();  // tiles[buf] complete; tiles[buf^1] no longer read (its readers passed this barrier)
        if (active) {
          if constexpr (kPacked) pair_sum2<Ker, TILE / 2>(tiles[buf], (n + 1) / 2, g, G, pt[0], pt[1], acc);
          else rec_sum2<Real, Ker, false, TILE>(tiles[buf], n, g, G, pt[0], pt[1], acc);
        }
        buf ^= 1;
      }
    }
    // fixed-order sum of the G partial sums of each target (in the tiles'
    // memory: every thread is done reading them past this barrier)
    __syncthreads();
    if (active)
#pragma unroll
      for (int q = 0; q < TPT; ++q)
#pragma unroll
        for (int k = 0; k < KT; ++k) red[threadIdx.x][q][k] = acc[q][k];
    __syncthreads();
    if (active && g == 0) {
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        if (ti + q * nc >= m) break;
        double sum[KT];
#pragma unroll
        for (int k = 0; k < KT; ++k) sum[k] = red[ti][q][k];
        for (int gg = 1; gg < G; ++gg)
#pragma unroll
          for (int k = 0; k < KT; ++k) sum[k] += red[gg * nc + ti][q][k];
        const long o = (long)(t0 + c0 + ti + q * nc) * KT;
        if constexpr (kPacked) {
#pragma unroll
          for (int k = 0; k < KT; ++k) sum[k] *= 1.0 / packed_unit<Ker>(k);
        }
#pragma unroll
        for (int k = 0; k < KT; ++k) pot[o + k] = kDbl ? pot[o + k] + sum[k] * scale : sum[k] * scale;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Sources -> check surface of a node, FP64.  XList = false (S2U, fmm_pts.txx:
// 2275-2637): node = nodes[b], sources = its own points, output row b of
// `out` scaled by scale*2^(-deg depth) (level factor of the check->equivalent
// operator).  XList = true (X, fmm_pts.txx:4444-4736): sources = the points of
// the X list's leaves, output row = node.  accumulate: added to the row.
//
// One thread per (node, pair of check points k and k + ns/2; ns is even),
// numbered through all nodes, so that every lane has work whatever ns and the
// leaf sizes are.  The lanes of a warp mostly share a node and read its
// sources as broadcasts from L1: four loads for two pairs, no shared memory
// and no barrier.  Bound by the FP64 pipe (12 operations a Laplace pair).
// LPS neighbouring lanes split the sources of one pair and add their sums in
// a fixed order: 4 for X, whose few nodes have long lists, and for S2U when
// one thread per pair would not fill the chip (surface_lanes).
// Against one block per node with the sources in shared memory and two Newton
// steps: 4M clustered points S2U with its products 3.15 -> 2.81 ms, X list
// 0.48 -> 0.33 ms.
// ---------------------------------------------------------------------------
inline int surface_lanes(long n_pairs) { return n_pairs < 148L * 1024 ? 4 : 1; }

template <int Ker, bool XList, int LPS>
__global__ void __launch_bounds__(kNT) surface_check_kernel(
    long n_thr, const int* __restrict__ nodes, const MKey* __restrict__ keys, const int* __restrict__ slo,
    const int* __restrict__ shi, const int* __restrict__ x_off, const int* __restrict__ x_list,
    const unsigned char* __restrict__ x_img, const double* __restrict__ sx, const double* __restrict__ sy,
    const double* __restrict__ sz, const double* __restrict__ den, const double* __restrict__ usurf, int ns,
    double rad, double scale, int deg, bool accumulate, double* __restrict__ out) {
  constexpr int KS = KerDims<Ker>::KS, KT = KerDims<Ker>::KT;
  constexpr int NP = LPS == 1 && KT <= 3 ? 2 : 1;  // partial sums per check point (even and odd sources)
  const int sub = threadIdx.x % LPS;
  const long id = (blockIdx.x * (long)kNT + threadIdx.x) / LPS;
  if (id >= n_thr) return;
  const int nh = ns / 2;
  const long b = id / nh;
  const int k = (int)(id - b * nh);
  const int T = nodes[b];
  double cx, cy, cz, half;
  int dT;
  node_geom(keys[T], cx, cy, cz, half, dT);
  const double hr = half * rad;
  double px[2], py[2], pz[2], acc[2][NP][KT];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    px[h] = hr * usurf[(k + h * nh) * 3 + 0];
    py[h] = hr * usurf[(k + h * nh) * 3 + 1];
    pz[h] = hr * usurf[(k + h * nh) * 3 + 2];
#pragma unroll
    for (int i = 0; i < NP; ++i)
#pragma unroll
      for (int c = 0; c < KT; ++c) acc[h][i][c] = 0;
  }
  // the points [lo, hi) of a leaf whose centre is at (ox, oy, oz)
  auto points = [&](int lo, int hi, double ox, double oy, double oz) {
    auto one = [&](int j, int i) {
      double f[KS];
      double x = __ldg(sx + j), y = __ldg(sy + j), z = __ldg(sz + j);
      if constexpr (XList) {
        x += ox;
        y += oy;
        z += oz;
      }
#pragma unroll
      for (int c = 0; c < KS; ++c) f[c] = __ldg(den + (long)j * KS + c);
#pragma unroll
      for (int h = 0; h < 2; ++h) ker_eval<Ker, double>(px[h] - x, py[h] - y, pz[h] - z, f, acc[h][i]);
    };
    int j = lo + sub;
    for (; j + NP <= hi; j += NP * LPS)
#pragma unroll
      for (int i = 0; i < NP; ++i) one(j + i, i);
    if (NP > 1 && j < hi) one(j, 0);
  };
  if constexpr (XList) {
    for (int q = x_off[T]; q < x_off[T + 1]; ++q) {
      const int S = x_list[q];
      double sxc, syc, szc, sh;
      int dS;
      node_geom(keys[S], sxc, syc, szc, sh, dS);
      if (x_img) image_shift(x_img[q], sxc, syc, szc);
      points(slo[S], shi[S], sxc - cx, syc - cy, szc - cz);
    }
  } else {
    points(slo[T], shi[T], 0, 0, 0);
  }
  if constexpr (LPS > 1) {
    const unsigned grp = ((1u << LPS) - 1) << (threadIdx.x % 32 / LPS * LPS);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < KT; ++c)
#pragma unroll
        for (int d = 1; d < LPS; d <<= 1) acc[h][0][c] += __shfl_xor_sync(grp, acc[h][0][c], d);
    if (sub != 0) return;
  }
  const double oscale = XList ? scale : scale * ldexp(1.0, -deg * dT);
  double* o = out + ((XList ? (long)T : b) * ns + k) * KT;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int c = 0; c < KT; ++c) {
      double v = acc[h][0][c];
      if (NP > 1) v += acc[h][NP - 1][c];
      double* dst = o + (long)h * nh * KT + c;
      *dst = accumulate ? *dst + v * oscale : v * oscale;
    }
}

// ---------------------------------------------------------------------------
// V-list: pruned separable DFTs over the (2m)^3 grid (FFT_UpEquiv /
// FFT_Check2Equiv, fmm_pts.txx:2689-2858) and the Hadamard products
// (VListHadamard, fmm_pts.txx:3249-3344).  Only the m^3 corner holding the
// upward equivalent surface enters the forward transform and only the m^3
// corner holding the check surface is produced by the inverse.  The grid
// size is a compile-time constant.  A block handles G grids (child x
// component) of one parent.
// ---------------------------------------------------------------------------

// ---------------------------------------------------------------------------
// Split-FP16 spectra of the mixed form's Hadamards.  A value v of parent q is
// stored as hi = fp16(v 2^-E), lo = fp16(v 2^-E - hi) (22 bits and lo's sign,
// as a TF32 hi/lo pair), with one exponent E per parent such that no value of
// its spectra exceeds 2^15.  Values down to 2^-18 of that bound keep all 22
// bits; below that the error stays at 2^-25, 2^-40 of the bound.  TF32 halves
// kept 22 bits at any size, so a child much weaker than its strongest sibling
// loses bits here; that sibling's own FP32 rounding (2^-24 of it) is larger
// wherever its field reaches, which is everywhere the weak one's does.
// Rms errors of potentials against the plain form, 100k points, 24 sets each,
// over those of the TF32 form (and its plain DFT sums): m = 8 0.85 to 0.88,
// m = 10 0.99 to 1.00; with densities times 2^0 .. 2^40 per cell of side 1/16
// 0.86 to 0.87 and 0.97 to 1.01.
// ---------------------------------------------------------------------------
// (re, im) as two packed halves: their hi parts and their lo parts.
__device__ __forceinline__ void half_split(float re, float im, unsigned& hi, unsigned& lo) {
  const __half2 h = __floats2half2_rn(re, im);
  const float2 hf = __half22float2(h);
  const __half2 l = __floats2half2_rn(re - hf.x, im - hf.y);
  memcpy(&hi, &h, 4);
  memcpy(&lo, &l, 4);
}
// Row of frequency f, parent q (n_q parents): frequency-major, so that the
// rows which the blocks of one frequency gather lie together (m = 8: 64 bytes
// each, 1 MB for 16k parents).
__device__ __forceinline__ long split_row(int f, long q, long n_q) { return (long)f * n_q + q; }
// Word of element e's hi part in its row (its lo part is 2 words on): elements
// 2k and 2k+1 share one 16-byte piece (hi, hi, lo, lo), the hi and lo A
// fragments of one lane.
__device__ __forceinline__ int split_word(int e) { return (e >> 1) * 4 + (e & 1); }

// Exponents of the parents' spectra: |spectrum value| <= sum |density| of its
// child, so E = (exponent of the largest such sum over the 8 children) - 15,
// but at least -126: below that 2^-E would leave the range of FP64 (densities
// near 1e-304 and less), and lo's step 2^(E-24) is finer there than FP32's
// smallest step 2^-149.  qinv = 2^-E; qscale = 2^(E + op_exp) also carries the
// operators' largest scale, so that the running sums of the products are at
// most as large as the largest output spectra allow.  One block of 8 warps per
// parent, one child per warp; `len` values per child.  A sum that is zero or
// not finite leaves E = 0.
__global__ void __launch_bounds__(256) vsrc_scale_kernel(const int* __restrict__ vsrc, const int* __restrict__ child0,
                                                         const double* __restrict__ ue, int len, int op_exp,
                                                         float* __restrict__ qscale, double* __restrict__ qinv) {
  __shared__ double part[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double* row = ue + (long)(child0[vsrc[blockIdx.x]] + warp) * len;
  double sum = 0;
  for (int i = lane; i < len; i += 32) sum += fabs(row[i]);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  if (lane == 0) part[warp] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double top = 0;
    bool finite = true;
    for (int c = 0; c < 8; ++c) {
      finite = finite && isfinite(part[c]);
      top = fmax(top, part[c]);
    }
    int e = 15;
    if (finite && top > 0) frexp(top, &e);
    e = max(e - 15, -126);
    qscale[blockIdx.x] = (float)ldexp(1.0, e + op_exp);
    qinv[blockIdx.x] = ldexp(1.0, -e);
  }
}

// cos and sin of 2 pi j / N for the DFTs, evaluated by the compiler from their
// Taylor series after reduction to [0, pi/4]: the twiddles of the unrolled
// transforms become literal operands (read from shared memory before).
constexpr double taylor_trig(double x, bool sine) {
  double term = sine ? x : 1.0, sum = term;
  for (int k = sine ? 2 : 1; k < 26; k += 2) {
    term *= -x * x / (k * (k + 1));
    sum += term;
  }
  return sum;
}
constexpr double twiddle_cos(int j, int N) {  // cos(2 pi j / N)
  j %= N;
  if (j < 0) j += N;
  if (2 * j > N) j = N - j;                            // cos is even
  if (4 * j > N) return -twiddle_cos(N - 2 * j, 2 * N);  // cos(pi - x) = -cos x
  if (8 * j > N) return taylor_trig(1.57079632679489661923 * (N - 4 * j) / N, true);
  return taylor_trig(6.28318530717958647693 * j / N, false);
}
constexpr double twiddle_sin(int j, int N) { return twiddle_cos(4 * j - N, 4 * N); }  // cos(x - pi/2)
template <class Real, int N>
struct Twiddles {
  Real c[N] = {}, s[N] = {};
  constexpr Twiddles() {
    for (int j = 0; j < N; ++j) {
      c[j] = (Real)twiddle_cos(j, N);
      s[j] = (Real)twiddle_sin(j, N);
    }
    // exact where a factor is 0 or +-1
    c[0] = 1;
    s[0] = 0;
    if (N % 2 == 0) {
      c[N / 2] = -1;
      s[N / 2] = 0;
    }
    if (N % 4 == 0) {
      c[N / 4] = 0;
      s[N / 4] = 1;
      c[3 * (N / 4)] = 0;
      s[3 * (N / 4)] = -1;
    }
  }
};

// a += v (c + i s) for constants c, s (folded when they are 0 or 1)
template <class Real>
__device__ __forceinline__ void cmac(Cplx<Real>& a, const Cplx<Real>& v, Real c, Real s) {
  if (c == (Real)1) {
    a.re += v.re;
    a.im += v.im;
  } else if (c != (Real)0) {
    a.re += v.re * c;
    a.im += v.im * c;
  }
  if (s == (Real)1) {
    a.re -= v.im;
    a.im += v.re;
  } else if (s == (Real)-1) {
    a.re += v.im;
    a.im -= v.re;
  } else if (s != (Real)0) {
    a.re -= v.im * s;
    a.im += v.re * s;
  }
}
template <class Real>
__device__ __forceinline__ Cplx<Real> cadd(const Cplx<Real>& a, const Cplx<Real>& b) { return {a.re + b.re, a.im + b.im}; }
template <class Real>
__device__ __forceinline__ Cplx<Real> csub(const Cplx<Real>& a, const Cplx<Real>& b) { return {a.re - b.re, a.im - b.im}; }
template <class Real>
__device__ __forceinline__ Cplx<Real> cmuli(const Cplx<Real>& a) { return {-a.im, a.re}; }

// Output z = M + zp of the length-2M inverse DFT as a plain sum (twr, twi:
// cos and sin of 2 pi j / 2M in shared memory).  FP32 keeps this form: the
// rounding of these sums is the largest part of the mixed form's V-list error,
// and position gradients near leaf corners carry it amplified (up to 4e-5 at
// m = 10), so that the radix-4 sums, although their error was a fifth smaller
// (and the inverse 1.37 -> 0.78 ms at 4M clustered points), moved such outputs
// by more than two forms of the other stages differ.
// Literal: the twiddles as literal operands instead, which blocks of whole rows
// take (4M clustered points 1.37 against 1.83 ms; smaller blocks are faster
// from shared memory, 1M Stokes 0.52 against 0.62 ms).
template <class Real, int M, bool Literal>
__device__ __forceinline__ Cplx<Real> idft_plain(const Cplx<Real> (&v)[2 * M], int zp, const Real* twr,
                                                 const Real* twi) {
  constexpr Twiddles<Real, 2 * M> tw{};
  Real re = 0, im = 0;
#pragma unroll
  for (int k = 0; k < 2 * M; ++k) {
    const int w = (k * (M + zp)) % (2 * M);
    const Real c = Literal ? tw.c[w] : twr[w], s = Literal ? tw.s[w] : twi[w];
    re += v[k].re * c - v[k].im * s;
    im += v[k].re * s + v[k].im * c;
  }
  return {re, im};
}

// Four outputs of the length-2M DFT of M values, X[k0 + j M/2], j = 0..3
// (k0 < M/2): the values' classes y mod 4 are summed once, S_r = sum of
// v[y] w^(k0 y) over y = r (mod 4), w = exp(-pi i / M), and since w^(y M/2) =
// (-i)^y, X[k0 + j M/2] = sum_r (-i)^(j r) S_r.  A quarter of the products of
// the plain sums.
template <class Real, int M>
__device__ __forceinline__ void dft_quad(const Cplx<Real> (&v)[M], int k0, Cplx<Real> (&x)[4]) {
  constexpr Twiddles<Real, 2 * M> tw{};
  Cplx<Real> S[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
#pragma unroll
  for (int y = 0; y < M; ++y) cmac(S[y % 4], v[y], tw.c[(k0 * y) % (2 * M)], -tw.s[(k0 * y) % (2 * M)]);
  const Cplx<Real> a = cadd(S[0], S[2]), b = csub(S[0], S[2]), c = cadd(S[1], S[3]), d = cmuli(csub(S[1], S[3]));
  x[0] = cadd(a, c);
  x[1] = csub(b, d);  // S0 - i S1 - S2 + i S3
  x[2] = csub(a, c);
  x[3] = cadd(b, d);
}

// Adds the inputs k0 + j M/2, j = 0..3 (u[j]) of the length-2M inverse DFT to
// its outputs z = M .. 2M-1 (acc[zp], z = M + zp): W^(k z) = (-1)^k W^(k zp)
// and W^(j zp M/2) = i^(j zp), so the four inputs are combined once per class
// of zp mod 4.
template <class Real, int M>
__device__ __forceinline__ void idft_quad(const Cplx<Real> (&u)[4], int k0, Cplx<Real> (&acc)[M]) {
  constexpr Twiddles<Real, 2 * M> tw{};
  const Cplx<Real> a = cadd(u[0], u[2]), b = csub(u[0], u[2]), c = cadd(u[1], u[3]), d = cmuli(csub(u[1], u[3]));
  // (-1)^(k0 + j M/2): M/2 odd flips the inputs j = 1, 3
  constexpr bool kFlip = (M / 2) % 2 != 0;
  const Cplx<Real> B[4] = {kFlip ? csub(a, c) : cadd(a, c), kFlip ? csub(b, d) : cadd(b, d),
                           kFlip ? cadd(a, c) : csub(a, c), kFlip ? cadd(b, d) : csub(b, d)};
#pragma unroll
  for (int zp = 0; zp < M; ++zp) {
    const int w = (k0 * zp) % (2 * M);
    const Real sg = k0 % 2 ? (Real)-1 : (Real)1;
    cmac(acc[zp], B[zp % 4], sg * tw.c[w], sg * tw.s[w]);
  }
}

template <class Real, int M>
struct FftSizes {
  static constexpr int N1 = 2 * M, NH = M + 1, M3 = M * M * M, N3H = N1 * N1 * NH;
  // forward: a1 [M*M][NH] complex, a2 [M][N1][NH] complex (+4 complex of
  // padding per grid, so that the z-lines of 4 neighbouring grids fall into
  // different banks), the real grid [M3] in a2's memory
  static constexpr int A2S = M * N1 * NH + 4;
  static constexpr size_t up_grid_bytes = sizeof(Real) * 2 * (M * M * NH + A2S);
  // inverse: b1 [M][N1][NH] (+4 padding), b2 [M][M][NH] complex, the real
  // result [M3] in b1's memory
  static constexpr int B1S = M * N1 * NH + 4;
  static constexpr size_t dn_grid_bytes = sizeof(Real) * 2 * (B1S + M * M * NH);
  static constexpr int threads(int G) { return ((8 * NH * G + 31) / 32) * 32; }  // one thread per line of the widest stage
  // Grids per block: the largest divisor G of ngrid with G grids in `budget`
  // bytes and at most max_threads threads (at least 1).
  static constexpr int grids_per_block(size_t per_grid, int ngrid, size_t budget, int max_threads) {
    int best = 1;
    for (int G = 1; G <= ngrid; ++G)
      if (ngrid % G == 0 && G * per_grid <= budget && threads(G) <= max_threads) best = G;
    return best;
  }
  // Two blocks of 112 KB share an SM: the FP32 scalar DFTs of m = 8 take all 8
  // children and so write (read) whole 64-byte rows of the spectra; forward,
  // 4M clustered points, 0.99 ms against 1.30 ms with 4 children in 60 KB.
  // The inverse gains only for those (kRows; 1.62 -> 1.37 ms); the others are
  // slower in large blocks.
  static constexpr int up_grids(int ngrid) { return grids_per_block(up_grid_bytes, ngrid, 112 * 1024, 576); }
  static constexpr bool kRows = sizeof(Real) == 4 && 8 * dn_grid_bytes <= 112 * 1024;  // FP32 up to m = 8
  static constexpr int dn_grids(int ngrid) {
    return kRows && ngrid == 8 ? grids_per_block(dn_grid_bytes, ngrid, 112 * 1024, 576)
                               : grids_per_block(dn_grid_bytes, ngrid, 80 * 1024, 288);
  }
  // Launch bound of the forward kernel, for 8 and 24 grids: 576 threads hold it
  // to 96 registers, too few for the lines of m >= 14 in FP64, whose blocks
  // need far fewer threads (200k points, m = 14 1.10 against 1.02 ms, m = 16
  // 1.57 against 1.47).
  static constexpr int up_bound = threads(up_grids(8)) <= 288 && threads(up_grids(24)) <= 288 ? 288 : 576;
};

// Each stage of the separable DFTs: one thread per input line; it loads the
// line into registers once and writes every output along that axis (radix-4
// sums along y and z, paired outputs kx and M - kx along x, literal twiddles;
// plain sums in the FP32 inverse, see idft_plain).
// Against plain sums with the twiddles in shared memory, piece-major FP64
// spectra and 4-byte FP16 stores, 4M clustered points in the mixed form:
// forward 1.73 -> 1.00 ms, inverse 1.62 -> 1.37 ms; 1M in FP64: 1.98 -> 0.64
// and 0.95 -> 0.67 ms.  What bounds the forward one now is its 64-byte row
// stores at the frequency-major stride.
// Output layout: frequency-major rows (split_row) for the scalar FP64
// Hadamards, spec[f][q][child], and for the split-FP16 ones (`qinv` given),
// each value times 2^-E of its parent as FP16 hi + lo in the order of
// split_word; otherwise rows spec[q][f][child*ke+comp].
template <class Real, int M>
__global__ void __launch_bounds__(FftSizes<Real, M>::up_bound) fft_up_kernel(int ke, int G, int ngroups, const int* __restrict__ vsrc,
                                                      const int* __restrict__ child0, const double* __restrict__ ue,
                                                      const int* __restrict__ fft_map, int ns, long n_q, int kz0,
                                                      int nkz, const double* __restrict__ qinv,
                                                      Cplx<Real>* __restrict__ spec) {
  using F = FftSizes<Real, M>;
  constexpr int N1 = F::N1, NH = F::NH, M3 = F::M3, N3H = F::N3H, A2S = F::A2S;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cplx<Real>* a1 = reinterpret_cast<Cplx<Real>*>(smem_raw);  // G * M*M*NH
  Cplx<Real>* a2 = a1 + G * M * M * NH;                      // G * A2S
  Real* g = reinterpret_cast<Real*>(a2);                     // G * M3, before a2 is written
  const int q = blockIdx.x / ngroups;
  const int gb = (blockIdx.x % ngroups) * G;
  const int ngrid = 8 * ke;
  const int gn = min(G, ngrid - gb);
  const int P = vsrc[q];
  const int c0 = child0[P];
  const int dim = ns * ke;
  const double ascale = qinv ? qinv[q] : 1.0;
  for (int i = threadIdx.x; i < gn * M3; i += blockDim.x) g[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < gn * ns; i += blockDim.x) {
    const int gi = i / ns, k = i % ns;
    const int gg = gb + gi, c = gg / ke, comp = gg % ke;
    const int idx = fft_map[k];  // x + N1*y + N1*N1*z, all < M
    const int x = idx % N1, y = (idx / N1) % N1, z = idx / (N1 * N1);
    g[gi * M3 + x + M * (y + M * z)] = (Real)(ue[(long)(c0 + c) * dim + k * ke + comp] * ascale);
  }
  __syncthreads();
  // x -> kx (real input): line = (gi, z, y)
  for (int r = threadIdx.x; r < gn * M * M; r += blockDim.x) {
    const Real* row = g + r * M;
    Real v[M];
#pragma unroll
    for (int x = 0; x < M; ++x) v[x] = row[x];
    // Outputs kx and M - kx share the sums over even and odd x, one rounding
    // more than a chain of FP32 fmas and the same one in both.  m = 10, whose
    // downward operators amplify rounding most, takes the chains: median error
    // of the potentials against the plain form (100k points, 32 seeds) 2.4e-7
    // (clustered) and 2.7e-7 (uniform) in pairs, 2.1e-7 and 2.3e-7 in chains
    // (and in the all-plain sums before), at 0.10 ms for either (200k points).
    // At the other orders the errors are the same or the pairs' smaller.
    constexpr bool kPairs = sizeof(Real) == 8 || M != 10;
    constexpr Twiddles<Real, N1> tw{};
#pragma unroll
    for (int kx = 0; kx <= (kPairs ? M / 2 : M); ++kx) {
      Cplx<Real> S[2] = {{0, 0}, {0, 0}};
#pragma unroll
      for (int x = 0; x < M; ++x) {
        const int w = (kx * x) % N1, h = kPairs ? x % 2 : 0;
        if (tw.c[w] != (Real)0) S[h].re += v[x] * tw.c[w];
        if (tw.s[w] != (Real)0) S[h].im -= v[x] * tw.s[w];
      }
      if constexpr (!kPairs) {
        a1[r * NH + kx] = S[0];
        continue;
      }
      a1[r * NH + kx] = cadd(S[0], S[1]);
      if (kx < M - kx) a1[r * NH + M - kx] = {S[0].re - S[1].re, S[1].im - S[0].im};
    }
  }
  __syncthreads();
  // y -> ky: line = (gi, z, kx), kx fastest
  for (int i = threadIdx.x; i < gn * M * NH; i += blockDim.x) {
    const int kx = i % NH, zg = i / NH;  // zg = gi*M + z
    const int gi = zg / M, z = zg % M;
    const Cplx<Real>* col = a1 + (zg * M) * NH + kx;
    Cplx<Real> v[M];
#pragma unroll
    for (int y = 0; y < M; ++y) v[y] = col[y * NH];
    Cplx<Real>* dst = a2 + gi * A2S + (z * N1) * NH + kx;
#pragma unroll
    for (int k0 = 0; k0 < M / 2; ++k0) {
      Cplx<Real> x[4];
      dft_quad<Real, M>(v, k0, x);
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[(k0 + j * (M / 2)) * NH] = x[j];
    }
  }
  __syncthreads();
  // z -> kz: line = (gi, ky, kx), gi fastest; spectrum index f = kx + NH*(ky + N1*kz);
  // only the slab kz in [kz0, kz0+nkz) is written, at f - N1*NH*kz0
  Cplx<Real>* out = spec + (long)q * (N1 * NH * nkz) * ngrid;
  // (every thread runs every step: neighbouring lanes exchange halves)
  const int n_line = gn * N1 * NH;
  const bool paired = sizeof(Real) == 4 && qinv && gn % 2 == 0 && gb % 2 == 0;
  for (int i0 = 0; i0 < n_line; i0 += blockDim.x) {
    const int i = i0 + threadIdx.x;
    const bool in = i < n_line;
    const int gi = i % gn, l = i / gn;  // l = ky*NH + kx
    const Cplx<Real>* col = a2 + (in ? gi * A2S + l : 0);
    Cplx<Real> v[M];
#pragma unroll
    for (int z = 0; z < M; ++z) v[z] = col[z * N1 * NH];
#pragma unroll
    for (int k0 = 0; k0 < M / 2; ++k0) {
      Cplx<Real> x[4];
      dft_quad<Real, M>(v, k0, x);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kz = k0 + j * (M / 2);
        if (kz < kz0 || kz >= kz0 + nkz) continue;
        const int f = l + N1 * NH * (kz - kz0);
        if (sizeof(Real) == 4 && qinv) {
          unsigned hi, lo;
          half_split((float)x[j].re, (float)x[j].im, hi, lo);
          unsigned* row = reinterpret_cast<unsigned*>(spec) + split_row(f, q, n_q) * (2 * ngrid);
          if (paired) {  // elements e, e + 1 of a 16-byte piece: (hi, hi) from the even lane, (lo, lo) from the odd one
            const bool odd = gi & 1;
            const unsigned got = __shfl_xor_sync(0xffffffffu, odd ? hi : lo, 1);
            if (in)
              *reinterpret_cast<uint2*>(row + split_word((gb + gi) & ~1) + (odd ? 2 : 0)) =
                  odd ? make_uint2(got, lo) : make_uint2(hi, got);
          } else if (in) {
            unsigned* w = row + split_word(gb + gi);
            w[0] = hi;
            w[2] = lo;
          }
        } else if (in) {
          if (sizeof(Real) == 8 && ke == 1) spec[split_row(f, q, n_q) * 8 + gb + gi] = x[j];
          else out[(long)f * ngrid + gb + gi] = x[j];
        }
      }
    }
  }
}

// Literal blocks hold whole rows (kRows) in up to 576 threads, the others up to
// 288.  Above m = 10 the bound is what the blocks have, so that the lines keep
// their registers (FP32: 126 at m = 12 to 153 at m = 16): held to 96 they
// spilled up to 1.1 KB, mixed inverse at 200k points, m = 12 0.427 ms against
// 0.362, m = 16 2.05 against 1.37.  At m = 10 the 96 registers lack 4 bytes and
// are the faster form (0.163 ms against 0.177 with 102).
template <class Real, int M, bool Literal>
__global__ void __launch_bounds__(Literal || M <= 10 ? 576 : 288)
    ifft_dn_kernel(int ke, int G, int ngroups, const int* __restrict__ vtrg, const int* __restrict__ child0,
                   const MKey* __restrict__ keys, const Cplx<Real>* __restrict__ spec,
                   const int* __restrict__ ifft_map, int ns, int deg, int kz0, int nkz, double* __restrict__ dc) {
  using F = FftSizes<Real, M>;
  constexpr int N1 = F::N1, NH = F::NH, M3 = F::M3, N3H = F::N3H;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int B1S = F::B1S;
  Cplx<Real>* b1 = reinterpret_cast<Cplx<Real>*>(smem_raw);  // G * B1S
  Cplx<Real>* b2 = b1 + G * B1S;                             // G * M*M*NH
  Real* o = reinterpret_cast<Real*>(b1);                     // G * M3, once b1 has been read
  Real* twr = reinterpret_cast<Real*>(b2 + G * M * M * NH);  // FP32: twiddles
  Real* twi = twr + N1;
  const int vt = blockIdx.x / ngroups;
  const int gb = (blockIdx.x % ngroups) * G;
  const int ngrid = 8 * ke;
  const int gn = min(G, ngrid - gb);
  const int P = vtrg[vt];
  const int c0 = child0[P];
  unsigned int X, Y, Z, dP;
  decode_key(keys[P], X, Y, Z, dP);
  const double lscale = ldexp(1.0, deg * ((int)dP + 1));  // 2^(trg_scal * level of the children)
  const int dim = ns * ke;
  if constexpr (sizeof(Real) == 4 && !Literal) {
    for (int j = threadIdx.x; j < N1; j += blockDim.x) {
      double sn, cs;
      sincospi(2.0 * j / N1, &sn, &cs);
      twr[j] = (Real)cs;
      twi[j] = (Real)sn;
    }
    __syncthreads();
  }
  const Cplx<Real>* in = spec + (long)vt * (N1 * NH * nkz) * ngrid + gb;
  // kz -> z in [M, 2M): line = (gi, ky, kx) read straight from the spectrum
  // row of the parent (gi fastest: neighbouring threads read neighbouring
  // children of one frequency).  With a slab of kz the transform of the
  // slab's frequencies alone is added into dc (the transform is linear).
  for (int i = threadIdx.x; i < gn * N1 * NH; i += blockDim.x) {
    const int gi = i % gn, l = i / gn;  // l = ky*NH + kx
    if constexpr (sizeof(Real) == 4) {
      Cplx<Real> v[N1];
#pragma unroll
      for (int kz = 0; kz < N1; ++kz)
        v[kz] = (kz >= kz0 && kz < kz0 + nkz) ? in[(long)(l + N1 * NH * (kz - kz0)) * ngrid + gi] : Cplx<Real>{0, 0};
#pragma unroll
      for (int zp = 0; zp < M; ++zp) b1[gi * B1S + zp * N1 * NH + l] = idft_plain<Real, M, Literal>(v, zp, twr, twi);
      continue;
    }
    Cplx<Real> acc[M] = {};
#pragma unroll
    for (int k0 = 0; k0 < M / 2; ++k0) {
      Cplx<Real> u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kz = k0 + j * (M / 2);
        u[j] = (kz >= kz0 && kz < kz0 + nkz) ? in[(long)(l + N1 * NH * (kz - kz0)) * ngrid + gi] : Cplx<Real>{0, 0};
      }
      idft_quad<Real, M>(u, k0, acc);
    }
#pragma unroll
    for (int zp = 0; zp < M; ++zp) b1[gi * B1S + zp * N1 * NH + l] = acc[zp];
  }
  __syncthreads();
  // ky -> y in [M, 2M): line = (gi, zp, kx), kx fastest
  for (int i = threadIdx.x; i < gn * M * NH; i += blockDim.x) {
    const int kx = i % NH, zg = i / NH;  // zg = gi*M + zp
    const Cplx<Real>* col = b1 + (zg / M) * B1S + ((zg % M) * N1) * NH + kx;
    if constexpr (sizeof(Real) == 4) {
      Cplx<Real> v[N1];
#pragma unroll
      for (int ky = 0; ky < N1; ++ky) v[ky] = col[ky * NH];
#pragma unroll
      for (int yp = 0; yp < M; ++yp) b2[(zg * M + yp) * NH + kx] = idft_plain<Real, M, Literal>(v, yp, twr, twi);
      continue;
    }
    Cplx<Real> acc[M] = {};
#pragma unroll
    for (int k0 = 0; k0 < M / 2; ++k0) {
      Cplx<Real> u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) u[j] = col[(k0 + j * (M / 2)) * NH];
      idft_quad<Real, M>(u, k0, acc);
    }
#pragma unroll
    for (int yp = 0; yp < M; ++yp) b2[(zg * M + yp) * NH + kx] = acc[yp];
  }
  __syncthreads();
  // kx -> x in [M, 2M), c2r: line = (gi, zp, yp)
  for (int r = threadIdx.x; r < gn * M * M; r += blockDim.x) {
    const Cplx<Real>* row = b2 + r * NH;
    constexpr Twiddles<Real, N1> tw{};
    if constexpr (sizeof(Real) == 4) {
      Cplx<Real> v[NH];
#pragma unroll
      for (int kx = 0; kx < NH; ++kx) v[kx] = row[kx];
#pragma unroll
      for (int xp = 0; xp < M; ++xp) {
        Real acc = 0;
#pragma unroll
        for (int kx = 0; kx < NH; ++kx) {
          const int w = (kx * (M + xp)) % N1;
          const Real c = Literal ? tw.c[w] : twr[w], sn = Literal ? tw.s[w] : twi[w];
          const Real t = v[kx].re * c - v[kx].im * sn;
          acc += (kx == 0 || 2 * kx == N1) ? t : (Real)2 * t;
        }
        o[r * M + xp] = acc;
      }
      continue;
    }
    // y[xp] = sum over kx of (2 for 0 < kx < M) (-1)^kx Re(v[kx] W^(kx xp));
    // kx and M - kx share cos and sin up to the sign (-1)^xp
    Cplx<Real> even[M / 2], odd[M / 2];
#pragma unroll
    for (int kx = 0; kx < M / 2; ++kx) {
      const Cplx<Real> p = row[kx], m = row[M - kx];
      const Real f = (kx % 2 ? (Real)-1 : (Real)1) * (kx == 0 ? (Real)1 : (Real)2);
      even[kx] = {f * (p.re + m.re), f * (p.im - m.im)};
      odd[kx] = {f * (p.re - m.re), f * (p.im + m.im)};
    }
    const Cplx<Real> mid = row[M / 2];
#pragma unroll
    for (int xp = 0; xp < M; ++xp) {
      // the middle frequency: W^(M xp / 2) = i^xp, (-1)^(M/2), weight 2
      const Real f = ((M / 2) % 2 ? (Real)-1 : (Real)1) * (xp % 4 < 2 ? (Real)2 : (Real)-2);
      Real acc = xp % 2 ? -f * mid.im : f * mid.re;
#pragma unroll
      for (int kx = 0; kx < M / 2; ++kx) {
        const int w = (kx * xp) % N1;
        const Cplx<Real>& t = xp % 2 ? odd[kx] : even[kx];
        if (tw.c[w] != (Real)0) acc += t.re * tw.c[w];
        if (tw.s[w] != (Real)0) acc -= t.im * tw.s[w];
      }
      o[r * M + xp] = acc;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < gn * ns; i += blockDim.x) {
    const int gi = i / ns, k = i % ns;
    const int gg = gb + gi, c = gg / ke, comp = gg % ke;
    const int idx = ifft_map[k];
    const int x = idx % N1 - M, y = (idx / N1) % N1 - M, z = idx / (N1 * N1) - M;
    dc[(long)(c0 + c) * dim + k * ke + comp] += (double)o[gi * M3 + x + M * (y + M * z)] * lscale;
  }
}

// 16-byte asynchronous global->shared copy; src_bytes = 0 zero-fills.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int src_bytes) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Hadamard products (VListHadamard, fmm_pts.txx:3249-3344) for vector
// expansions, organised as a register-tiled SIMT product per frequency f:
//   OUT[P][j1][c] += sum_{offset o, source child j2, i} M[f][o][j1][j2][i][c] * IN[Q_o(P)][f][j2][i]
// (KI equivalent-density components i, KO check-potential components c).  A
// block owns 128 target parents at one frequency and KOC output components
// (blockIdx.z picks the group); a thread owns one parent.  The offset blocks
// of frequency f sit in shared memory (chunks of OC offsets), read by every
// thread at the same address (broadcast).  The neighbour spectra of offset
// o+1 are copied asynchronously into a second shared buffer while offset o is
// computed; a thread only reads the rows it copied itself, so waiting on its
// own copy group is enough.  Missing neighbours are zero-filled and skipped.
template <class Real, int KI, int KO, int KOC, int OC>
__global__ void __launch_bounds__(128) hadamard_kernel(int n3h, long n_vtrg, long vt_stride, const int* __restrict__ vtab,
                                                       const Cplx<Real>* __restrict__ spec_in,
                                                       const Cplx<Real>* __restrict__ vop,
                                                       Cplx<Real>* __restrict__ spec_out) {
  constexpr int NGI = 8 * KI, NGO = 8 * KOC;
  constexpr int BLK = 64 * KI * KO;                               // complex entries per offset
  constexpr int ROW = NGI * sizeof(Cplx<Real>) / 16;              // 16-byte chunks per input row
  constexpr int STRIDE = NGI + 16 / (int)sizeof(Cplx<Real>);      // padded row (complex), breaks bank aliasing
  constexpr int NT = 128;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cplx<Real>* Ms = reinterpret_cast<Cplx<Real>*>(smem_raw);       // OC * BLK
  Cplx<Real>* xb = Ms + OC * BLK;                                 // 2 * NT * STRIDE
  const int f = blockIdx.y;
  const int c0 = blockIdx.z * KOC;
  const long p = (long)blockIdx.x * NT + threadIdx.x;
  Real ar[NGO], ai[NGO];
#pragma unroll
  for (int j = 0; j < NGO; ++j) ar[j] = ai[j] = 0;
  auto issue = [&](int o, int buf) {
    const int q = (o < 26 && p < n_vtrg) ? __ldg(vtab + (long)o * vt_stride + p) : -1;
    const Cplx<Real>* src = spec_in + ((long)(q < 0 ? 0 : q) * n3h + f) * NGI;
    Cplx<Real>* dst = xb + ((long)buf * NT + threadIdx.x) * STRIDE;
#pragma unroll
    for (int c = 0; c < ROW; ++c)
      cp_async16(reinterpret_cast<unsigned char*>(dst) + 16 * c, reinterpret_cast<const unsigned char*>(src) + 16 * c,
                 q >= 0 ? 16 : 0);
    cp_async_commit();
    return q;
  };
  int qc = issue(0, 0), qn = -1;
  for (int oc = 0; oc < 26; oc += OC) {
    const int no = min(OC, 26 - oc);
    __syncthreads();
    const Cplx<Real>* src = vop + ((long)f * 26 + oc) * BLK;
    for (int i = threadIdx.x; i < no * BLK; i += NT) Ms[i] = src[i];
    __syncthreads();
    for (int oo = 0; oo < no; ++oo) {
      const int o = oc + oo;
      qn = issue(o + 1, (o + 1) & 1);   // empty group past the last offset
      cp_async_wait<1>();               // this thread's row of offset o has landed
      const Cplx<Real>* Mo = Ms + oo * BLK;
      if (qc >= 0) {
        const Cplx<Real>* xr = xb + ((long)(o & 1) * NT + threadIdx.x) * STRIDE;
#pragma unroll
        for (int j2 = 0; j2 < 8; ++j2) {
          Cplx<Real> x[KI];
#pragma unroll
          for (int i = 0; i < KI; ++i) x[i] = xr[j2 * KI + i];
#pragma unroll
          for (int j1 = 0; j1 < 8; ++j1)
#pragma unroll
            for (int i = 0; i < KI; ++i)
#pragma unroll
              for (int c = 0; c < KOC; ++c) {
                const Cplx<Real> a = Mo[((j1 * 8 + j2) * KI + i) * KO + c0 + c];
                ar[j1 * KOC + c] += a.re * x[i].re - a.im * x[i].im;
                ai[j1 * KOC + c] += a.re * x[i].im + a.im * x[i].re;
              }
        }
      }
      qc = qn;
    }
  }
  cp_async_wait<0>();
  if (p < n_vtrg) {
    Cplx<Real>* out = spec_out + (p * n3h + f) * (8 * KO);
#pragma unroll
    for (int j1 = 0; j1 < 8; ++j1)
#pragma unroll
      for (int c = 0; c < KOC; ++c) out[j1 * KO + c0 + c] = {ar[j1 * KOC + c], ai[j1 * KOC + c]};
  }
}

// Hadamard products for scalar expansions (ke = 1), register form.  Same
// product as hadamard_kernel,
//   OUT[P][j1] += sum_{offset o, source child j2} M[f][o][j1][j2] * IN[Q_o(P)][f][j2],
// but each thread gathers the neighbour spectra of its PB target parents
// straight from global memory (L2) into registers, one offset ahead of the one
// it multiplies, so shared memory holds only the 26 operator blocks of the
// block's frequency (read as 16-byte broadcasts).  The input spectra are
// frequency-major rows (split_row).  Offsets that none of the thread's
// parents has are skipped.
template <class Real, int PB>
__global__ void __launch_bounds__(128, 4) hadamard_rd_kernel(int n3h, long n_vtrg, long vt_stride, long n_vsrc,
                                                             const int* __restrict__ vtab,
                                                             const unsigned* __restrict__ vmask,
                                                          const Cplx<Real>* __restrict__ spec_in,
                                                          const Cplx<Real>* __restrict__ vop,
                                                          Cplx<Real>* __restrict__ spec_out) {
  constexpr int NT = 128;
  constexpr int BLK = 64;                                       // 8 x 8 complex per offset
  using V = typename Vec16<Real>::type;                         // 16 bytes
  constexpr int CPV = 16 / (int)sizeof(Cplx<Real>);             // complex values per vector (2 or 1)
  constexpr int NV = 8 / CPV;                                   // vectors per spectrum row
  __shared__ V Ms[26 * BLK / CPV];
  const int f = blockIdx.y;
  const long pbase = (long)blockIdx.x * NT * PB + threadIdx.x;
  {
    const V* src = reinterpret_cast<const V*>(vop + (long)f * 26 * BLK);
    for (int i = threadIdx.x; i < 26 * BLK / CPV; i += NT) Ms[i] = __ldg(src + i);
  }
  long prow[PB];
  bool pin[PB];
#pragma unroll
  for (int k = 0; k < PB; ++k) {
    prow[k] = pbase + (long)k * NT;
    pin[k] = prow[k] < n_vtrg;
  }
  Real ar[PB][8], ai[PB][8];
#pragma unroll
  for (int k = 0; k < PB; ++k)
#pragma unroll
    for (int j = 0; j < 8; ++j) ar[k][j] = ai[k][j] = 0;
  V xc[PB][NV], xn[PB][NV];
  unsigned mc = 0, mn = 0;  // bit k: parent k has offset o
  auto load = [&](int o, V (&x)[PB][NV], unsigned& mask) {
    mask = 0;
#pragma unroll
    for (int k = 0; k < PB; ++k) {
      const int q = pin[k] ? __ldg(vtab + (long)o * vt_stride + prow[k]) : -1;
      if (q >= 0) {
        mask |= 1u << k;
        const V* r = reinterpret_cast<const V*>(spec_in) + split_row(f, q, n_vsrc) * NV;
#pragma unroll
        for (int v = 0; v < NV; ++v) x[k][v] = __ldg(r + v);
      } else {
#pragma unroll
        for (int v = 0; v < NV; ++v) memset(&x[k][v], 0, 16);
      }
    }
  };
  auto compute = [&](int o, const V (&x)[PB][NV], unsigned mask) {
    if (!mask) return;
    const V* Mo = Ms + o * (BLK / CPV);
#pragma unroll
    for (int jv = 0; jv < NV; ++jv) {  // source children j2 = jv*CPV .. jv*CPV+CPV-1
      Real xr[PB][CPV], xi[PB][CPV];
#pragma unroll
      for (int k = 0; k < PB; ++k) {
        Real t[2 * CPV];
        memcpy(t, &x[k][jv], 16);
#pragma unroll
        for (int c = 0; c < CPV; ++c) {
          xr[k][c] = t[2 * c];
          xi[k][c] = t[2 * c + 1];
        }
      }
#pragma unroll
      for (int j1 = 0; j1 < 8; ++j1) {
        Real m[2 * CPV];
        const V mv = Mo[(j1 * 8) / CPV + jv];
        memcpy(m, &mv, 16);
#pragma unroll
        for (int c = 0; c < CPV; ++c)
#pragma unroll
          for (int k = 0; k < PB; ++k) {
            ar[k][j1] += m[2 * c] * xr[k][c] - m[2 * c + 1] * xi[k][c];
            ai[k][j1] += m[2 * c] * xi[k][c] + m[2 * c + 1] * xr[k][c];
          }
      }
    }
  };
  __syncthreads();  // Ms staged
  // the offsets occupied for any parent of the warp, in increasing order (the
  // targets are ordered by occupied-offset pattern, so the others are
  // common); two register sets in turn: the gathers of the next offset are in
  // flight while one is multiplied
  unsigned pm = 0;
#pragma unroll
  for (int k = 0; k < PB; ++k) pm |= pin[k] ? __ldg(vmask + prow[k]) : 0u;
  unsigned rem = __reduce_or_sync(0xffffffffu, pm);
  const int nlive = __popc(rem);
  auto take = [&]() {
    const int o = __ffs(rem) - 1;
    rem &= rem - 1;
    return o;
  };
  int oc = nlive > 0 ? take() : 0;
  if (nlive > 0) load(oc, xc, mc);
#pragma unroll 1
  for (int i = 0; i < nlive; i += 2) {
    const int on = i + 1 < nlive ? take() : -1;
    if (on >= 0) load(on, xn, mn);
    compute(oc, xc, mc);
    const int onn = i + 2 < nlive ? take() : -1;
    if (onn >= 0) load(onn, xc, mc);
    if (on >= 0) compute(on, xn, mn);
    oc = onn;
  }
#pragma unroll
  for (int k = 0; k < PB; ++k) {
    if (!pin[k]) continue;
    V* out = reinterpret_cast<V*>(spec_out + (prow[k] * n3h + f) * 8);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      Real t[2 * CPV];
#pragma unroll
      for (int c = 0; c < CPV; ++c) {
        t[2 * c] = ar[k][v * CPV + c];
        t[2 * c + 1] = ai[k][v * CPV + c];
      }
      V w;
      memcpy(&w, t, 16);
      out[v] = w;
    }
  }
}

// ---------------------------------------------------------------------------
// Hadamard products of the mixed form (scalar expansions here, 3-component
// ones below) on the tensor cores: mma.sync m16n8k16 on split-FP16 spectra and
// operators with FP32 accumulation, three products per value (a_lo b_hi +
// a_hi b_lo + a_hi b_hi), which carries the products to ~2^-22 relative.
//
// Per frequency f the product is a real GEMM over parent rows:
//   OUT[P][(e_out, re|im)] += sum_o sum_(e, re|im) IN[Q_o(P)][(e, re|im)] * B_o[(e, re|im)][(e_out, re|im)]
// with elements e = child * ke + component and B_o the real form of the
// complex block M[f][o].  A warp owns 16-row tiles of target parents.  The A
// fragments come straight from the input rows in L2: lane (g, t) loads the
// 16-byte piece t of each 8 elements (elements 2t and 2t+1: hi re|im of both,
// then lo) of rows g and g+8 (four lanes read 64 contiguous bytes), which is
// its hi and lo fragment when the K order of the k-step is chosen as columns
// 2t, 2t+1 -> element 2t (re, im), columns 2t+8, 2t+9 -> element 2t+1.  No
// conversion is left in the loop.  The products of one offset accumulate in a
// fresh fragment that joins the running sum with a rounded FP32 fma, times the
// source parent's 2^E: the tensor cores' own FP32 accumulation is not
// round-to-nearest and, carried over all 26 offsets, left a bias of ~2e-6 in
// the far-field potential.
// Why FP16: the same 11-bit halves as a TF32 hi/lo pair at twice the MMA rate
// (measured 554 against 276 TFLOP/s for mma.sync), with half the operator
// bytes, and the split is done once per spectrum value by the forward DFT
// instead of at each of its up to 26 uses (24 conversions and subtractions
// per 16 rows and offset).  Measured against that TF32 form: 4M clustered
// points (m = 8, 16,037 parents) 10.8 -> 7.05 ms, 2M surface points 13.1 ->
// 7.5 ms, 1M Stokes points (m = 6) 9.5 -> 6.1 ms; outputs 3e-9 to 9e-7 apart.
// What bounds the scalar kernel is the L1 data path (83% of its rate at 1M
// clustered points, tensor pipe 34%, issue slots 59%: 12 wavefronts for the
// two gathers of a tile and offset, 8 for the operator fragments, 4 for scales
// and indices, against 13 cycles of MMA), with 49% of
// the gathered sectors hit in L1; so the kernel keeps its shared memory small:
// operator fragments 27 KB per block, 3 blocks per SM (4 blocks, with a
// smaller L1, took 9.0 ms; two tiles per warp 7.7 ms).  Each warp prefetches
// the index table of its next tile by itself (a block-wide table behind a
// barrier: 7.4 ms, surface 8.6 ms).
// ---------------------------------------------------------------------------
// d = a b (zero accumulator) and d += a b
__device__ __forceinline__ void mma_f16_zero(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                             unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma_f16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                        unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The three products of one k-step: rows g (x) and g+8 (y), b = (hi, hi, lo, lo).
__device__ __forceinline__ void mma_split(float (&d)[4], const uint4& x, const uint4& y, const uint4& b) {
  mma_f16_zero(d, x.z, y.z, x.w, y.w, b.x, b.y);
  mma_f16(d, x.x, y.x, x.y, y.y, b.z, b.w);
  mma_f16(d, x.x, y.x, x.y, y.y, b.x, b.y);
}

constexpr int kTcWarps = 8;    // warps per block of the scalar tensor-core Hadamard
constexpr int kTcBlocks = 3;   // blocks per SM
constexpr int kTcStages = 3;   // register sets of gathered rows
constexpr int kTcChunks = 16;  // tiles per warp (operator fragments staged once)

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}

constexpr int kTcEnt = 26 * 16 + 16;  // words of a tile's table: source parents [26][16], patterns [16]

__global__ void __launch_bounds__(32 * kTcWarps, kTcBlocks)
    hadamard_tc_kernel(int n3h, long n_vtrg, long vt_stride, long n_vsrc, int chunks, const int* __restrict__ vtab,
                       const unsigned* __restrict__ vmask, const uint4* __restrict__ spec_in,
                       const float* __restrict__ qscale, const uint4* __restrict__ bfrag,
                       const float* __restrict__ fscale, float2* __restrict__ spec_out) {
  extern __shared__ uint4 Bs[];  // [26 offsets][2 n-tiles][32 lanes], then two tables per warp
  const int f = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  int* ent = reinterpret_cast<int*>(Bs + 26 * 2 * 32) + warp * 2 * kTcEnt;
  // table of the warp's tile c into buffer c % 2 (rows past the end repeat the
  // last parent; their sums are not stored)
  auto tile_p0 = [&](int c) { return ((long)(blockIdx.x * chunks + c) * kTcWarps + warp) * 16; };
  auto fetch = [&](int c) {
    const long p0 = tile_p0(c);
    if (c < chunks && p0 < n_vtrg) {
      const long p = min(p0 + (lane & 15), n_vtrg - 1);
      int* dst = ent + (c & 1) * kTcEnt + lane;
      const int* src = vtab + (long)(lane >> 4) * vt_stride + p;
#pragma unroll
      for (int o = 0; o < 26; o += 2) cp_async4(dst + o * 16, src + (long)o * vt_stride);
      if (lane < 16) cp_async4(dst + 26 * 16, vmask + p);
    }
    cp_async_commit();
  };
  fetch(0);
  {
    const uint4* src = bfrag + (long)f * 26 * 2 * 32;
    for (int i = threadIdx.x; i < 26 * 2 * 32; i += 32 * kTcWarps) Bs[i] = __ldg(src + i);
  }
  const float fs = fscale[f];
  const uint4* in_f = spec_in + split_row(f, 0, n_vsrc) * 4 + t;  // row q: in_f[q * 4]
  __syncthreads();  // the operator fragments are staged
  for (int c = 0; c < chunks; ++c) {
    const long p0 = tile_p0(c);
    if (p0 >= n_vtrg) break;
    cp_async_wait<0>();
    __syncwarp();  // the tile's table has landed, and the other buffer is no longer read
    fetch(c + 1);
    const int* qs = ent + (c & 1) * kTcEnt + g;
    // offsets without a source parent for any of the tile's parents are
    // neither loaded nor multiplied (their products are zero); the targets
    // are ordered by occupied-offset pattern, so such offsets are common
    unsigned rem = __reduce_or_sync(0xffffffffu, (unsigned)ent[(c & 1) * kTcEnt + 26 * 16 + (lane & 15)]);
    float acc[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[nt][i] = 0.f;
    struct Rows {
      uint4 x[2];
      float s[2];
    };
    auto load = [&](int o, Rows& r) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int q = qs[o * 16 + 8 * h];
        r.x[h] = q >= 0 ? __ldg(in_f + (long)q * 4) : make_uint4(0u, 0u, 0u, 0u);
        r.s[h] = q >= 0 ? __ldg(qscale + q) : 0.f;
      }
    };
    auto compute = [&](int o, const Rows& r) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        float d[4];
        mma_split(d, r.x[0], r.x[1], Bs[(o * 2 + nt) * 32 + lane]);  // consecutive lanes: conflict-free
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[nt][i] = fmaf(d[i], r.s[i >> 1], acc[nt][i]);
      }
    };
    // The tile's occupied offsets in increasing order, one set bit at a time,
    // kStages register sets in turn: the gathers of the next offsets are in
    // flight while one is multiplied.
    constexpr int kStages = kTcStages;
    const int nlive = __popc(rem);
    Rows r[kStages];
    int o[kStages];
#pragma unroll
    for (int k = 0; k < kStages - 1; ++k)
      if (k < nlive) {
        o[k] = __ffs(rem) - 1;
        rem &= rem - 1;
        load(o[k], r[k]);
      }
#pragma unroll 1
    for (int i = 0; i < nlive; i += kStages) {
#pragma unroll
      for (int k = 0; k < kStages; ++k) {
        constexpr int kAhead = kStages - 1;
        const int n = (k + kAhead) % kStages;
        if (i + k + kAhead < nlive) {
          o[n] = __ffs(rem) - 1;
          rem &= rem - 1;
          load(o[n], r[n]);
        }
        if (k == 0 || i + k < nlive) compute(o[k], r[k]);
      }
    }
    // C fragment: (row g, cols 2t, 2t+1) and (row g+8, same cols); column
    // n = nt*8 + 2t (+1) is child j1 = 4nt + t, re (im).
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long p = p0 + g + 8 * h;
      if (p >= n_vtrg) continue;
      float2* out = spec_out + (p * n3h + f) * 8;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) out[4 * nt + t] = make_float2(acc[nt][2 * h] * fs, acc[nt][2 * h + 1] * fs);
    }
  }
}

// ---------------------------------------------------------------------------
// The same for 3-component expansions (Stokes velocity, pressure and velocity
// gradient, Biot-Savart), per group z of KOC output components: K = 48 (24
// elements, 3 k-steps of 8) and N = 16 KOC (2 KOC n-tiles).  A warp owns 16
// target parents; lane (g, t) loads the 16-byte pieces 4u + t, u = 0..2, of
// the 192-byte rows g and g+8.  The B fragments of an offset (9 KB for KOC =
// 3) are too many to stage for all 26 offsets, so the block streams them,
// kTc3Opb offsets at a time, into a double buffer in shared memory
// (cp.async, one barrier per group), shared by its 8 warps; offsets that no
// parent of the block has are skipped, those that no parent of a warp has are
// skipped by that warp.  Each k-step accumulates in a fresh fragment.
// ---------------------------------------------------------------------------
constexpr int kTc3Warps = 8;
constexpr int kTc3Blocks = 2;  // blocks per SM
constexpr int kTc3Opb = 4;  // offsets whose B fragments are staged per barrier (1M Stokes points: 2 6.22, 4 6.14 ms)

template <int KOC>
__global__ void __launch_bounds__(32 * kTc3Warps, kTc3Blocks)
    hadamard_tc3_kernel(int n3h, long n_vtrg, long vt_stride, long n_vsrc, int ko, const int* __restrict__ vtab,
                        const unsigned* __restrict__ vmask, const uint4* __restrict__ spec_in,
                        const float* __restrict__ qscale, const uint4* __restrict__ bfrag,
                        const float* __restrict__ fscale, float2* __restrict__ spec_out) {
  constexpr int NNT = 2 * KOC;        // n-tiles of the group
  constexpr int NB = 3 * NNT;         // (k-step, n-tile) fragment blocks per offset
  constexpr int NP = kTc3Warps * 16;  // target parents of the block
  constexpr int OPB = kTc3Opb;
  extern __shared__ uint4 Bs[];       // [2][OPB][NB][32 lanes]: (b0 hi, b1 hi, b0 lo, b1 lo)
  int* qs = reinterpret_cast<int*>(Bs + 2 * OPB * NB * 32);  // [26][NP] source parent of each (offset, parent)
  unsigned* wl = reinterpret_cast<unsigned*>(qs + 26 * NP);  // [kTc3Warps] occupied offsets of each warp
  const int f = blockIdx.y, z = blockIdx.z, ngroups = gridDim.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const long pb = (long)blockIdx.x * NP;
  for (int i = threadIdx.x; i < 26 * NP; i += 32 * kTc3Warps) {
    const int o = i / NP;
    const long p = pb + i % NP;
    qs[i] = p < n_vtrg ? __ldg(vtab + (long)o * vt_stride + p) : -1;
  }
  {
    const long p = pb + warp * 16 + (lane & 15);
    unsigned m = (lane < 16 && p < n_vtrg) ? __ldg(vmask + p) : 0u;
    m = __reduce_or_sync(0xffffffffu, m);
    if (lane == 0) wl[warp] = m;
  }
  __syncthreads();
  unsigned blive = 0;
#pragma unroll
  for (int w = 0; w < kTc3Warps; ++w) blive |= wl[w];
  const unsigned wlive = wl[warp];
  const float fs = fscale[f];
  const uint4* bsrc = bfrag + ((long)f * 26 * ngroups + z) * NB * 32;  // + o * ngroups * NB * 32
  // the next (up to) OPB block-live offsets of srem into buffer buf
  unsigned srem = blive;
  auto stage_group = [&](int buf) {
#pragma unroll
    for (int j = 0; j < OPB; ++j) {
      if (!srem) break;
      const int o = __ffs(srem) - 1;
      srem &= srem - 1;
      const uint4* src = bsrc + (long)o * ngroups * NB * 32;
      uint4* dst = Bs + (buf * OPB + j) * NB * 32;
      for (int i = threadIdx.x; i < NB * 32; i += 32 * kTc3Warps) cp_async16(dst + i, src + i, 16);
    }
  };
  const int w0 = warp * 16;
  const uint4* in_f = spec_in + split_row(f, 0, n_vsrc) * 12 + t;
  struct Rows {
    uint4 x[3][2];
    float s[2];
  };
  auto load = [&](int o, Rows& r) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int q = qs[o * NP + w0 + g + 8 * h];
      const uint4* row = in_f + (long)(q < 0 ? 0 : q) * 12;
#pragma unroll
      for (int u = 0; u < 3; ++u) r.x[u][h] = q >= 0 ? __ldg(row + 4 * u) : make_uint4(0u, 0u, 0u, 0u);
      r.s[h] = q >= 0 ? __ldg(qscale + q) : 0.f;
    }
  };
  float acc[NNT][4];
#pragma unroll
  for (int nt = 0; nt < NNT; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[nt][i] = 0.f;
  Rows xc, xn;
  unsigned rem = blive;
  int oc = rem ? __ffs(rem) - 1 : 0;
  if (rem) {
    stage_group(0);
    if (wlive >> oc & 1u) load(oc, xn);
  }
  cp_async_commit();
#pragma unroll 1
  for (int k = 0; rem; ++k) {
    rem &= rem - 1;
    const int on = rem ? __ffs(rem) - 1 : -1;
    const int grp = k / OPB, slot = k % OPB;
    if (slot == 0) {
      cp_async_wait<0>();  // this thread's copies of the group's offsets have landed
      __syncthreads();     // everyone's have; every warp is done with the other buffer
      stage_group((grp + 1) & 1);
      cp_async_commit();
    }
    if (wlive >> oc & 1u) {
      xc = xn;
      if (on >= 0 && (wlive >> on & 1u)) load(on, xn);  // the next offset's rows, in flight meanwhile
      const uint4* bq = Bs + ((grp & 1) * OPB + slot) * NB * 32 + lane;
#pragma unroll
      for (int nt = 0; nt < NNT; ++nt)
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          float d[4];
          mma_split(d, xc.x[u][0], xc.x[u][1], bq[(u * NNT + nt) * 32]);
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[nt][i] = fmaf(d[i], xc.s[i >> 1], acc[nt][i]);
        }
    } else if (on >= 0 && (wlive >> on & 1u)) {
      load(on, xn);
    }
    oc = on;
  }
  cp_async_wait<0>();
  // C fragment: (row g, cols 2t, 2t+1) and (row g+8, same cols); columns
  // nt*8 + 2t (+1) are the re (im) part of output element e = 4nt + t =
  // j1 * KOC + c of the group.
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const long p = pb + w0 + g + 8 * h;
    if (p >= n_vtrg) continue;
    float2* out = spec_out + (p * n3h + f) * (8 * ko) + z * KOC;
#pragma unroll
    for (int nt = 0; nt < NNT; ++nt) {
      const int e = 4 * nt + t;
      out[(e / KOC) * ko + e % KOC] = make_float2(acc[nt][2 * h] * fs, acc[nt][2 * h + 1] * fs);
    }
  }
}

template <int KOC>
void launch_hadamard_tc3(Context& ctx, int n3h, long f_base, int ko, const Cplx<float>* sin_, Cplx<float>* sout,
                         long p0, long np) {
  DevTree& T = ctx.tree;
  constexpr int NB = 6 * KOC, NP = kTc3Warps * 16;
  const int ngroups = ko / KOC;
  const size_t sm = (size_t)2 * kTc3Opb * NB * 32 * sizeof(uint4) + (size_t)26 * NP * sizeof(int) +
                    kTc3Warps * sizeof(int);
  PVFMM_CUDA_CHECK(cudaFuncSetAttribute(hadamard_tc3_kernel<KOC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  dim3 grid(ceil_div(np, (long)NP), n3h, ngroups);
  ++ctx.n_launch;
  hadamard_tc3_kernel<KOC><<<grid, 32 * kTc3Warps, sm, ctx.stream>>>(
      n3h, np, T.n_vtrg, T.n_vsrc, ko, T.vtab.get<int>() + p0, T.vmask.get<unsigned>() + p0,
      reinterpret_cast<const uint4*>(sin_), ctx.qscale.get<float>(),
      ctx.dops.vop_frag.get<uint4>() + f_base * 26 * ngroups * NB * 32, ctx.dops.vop_fscale.get<float>() + f_base,
      reinterpret_cast<float2*>(sout));
}

// ---------------------------------------------------------------------------
// Hadamard products of the plain form for 3-component expansions on the FP64
// tensor cores (mma.sync m8n8k4 .f64).  The same real GEMM per frequency f and
// output group z as hadamard_tc3_kernel, K = 48 in 12 k-steps of 4, N = 16 KOC
// in 2 KOC n-tiles of 8, in FP64 with no split.  A warp owns 8 target parents
// (rows); lane (g, t) holds row g, and with the K order k-step s, column
// c -> double 12c + s its A values for all 12 k-steps are the contiguous
// doubles 12t .. 12t+11 of the row (6 16-byte loads).  The B fragments of an
// offset (18 KB for KOC = 3) are streamed offset by offset into a double
// buffer in shared memory (cp.async, one barrier per offset) shared by the
// block's 8 warps; offsets no parent of the block has are skipped, those no
// parent of a warp has are skipped by that warp.
// ---------------------------------------------------------------------------
constexpr int kDmWarps = 8;

template <int KOC>
__global__ void __launch_bounds__(32 * kDmWarps, 2)
    hadamard_dmma3_kernel(int n3h, long n_vtrg, long vt_stride, int ko, const int* __restrict__ vtab,
                          const unsigned* __restrict__ vmask, const double2* __restrict__ spec_in,
                          const double* __restrict__ bfrag, double2* __restrict__ spec_out) {
  constexpr int NNT = 2 * KOC;       // n-tiles of the group
  constexpr int NB = 12 * NNT;       // (k-step, n-tile) fragment blocks per offset
  constexpr int NP = kDmWarps * 8;   // target parents of the block
  extern __shared__ double Bd[];     // [2][NB][32 lanes]
  int* qs = reinterpret_cast<int*>(Bd + 2 * NB * 32);  // [26][NP]
  unsigned* wl = reinterpret_cast<unsigned*>(qs + 26 * NP);  // [kDmWarps]
  const int f = blockIdx.y, z = blockIdx.z, ngroups = gridDim.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const long pb = (long)blockIdx.x * NP;
  for (int i = threadIdx.x; i < 26 * NP; i += 32 * kDmWarps) {
    const int o = i / NP;
    const long p = pb + i % NP;
    qs[i] = p < n_vtrg ? __ldg(vtab + (long)o * vt_stride + p) : -1;
  }
  {
    const long p = pb + warp * 8 + (lane & 7);
    unsigned m = (lane < 8 && p < n_vtrg) ? __ldg(vmask + p) : 0u;
    m = __reduce_or_sync(0xffffffffu, m);
    if (lane == 0) wl[warp] = m;
  }
  __syncthreads();
  unsigned blive = 0;
#pragma unroll
  for (int w = 0; w < kDmWarps; ++w) blive |= wl[w];
  const unsigned wlive = wl[warp];
  const double* bsrc = bfrag + ((long)f * 26 * ngroups + z) * NB * 32;
  auto stage = [&](int o, int buf) {
    const double2* src = reinterpret_cast<const double2*>(bsrc + (long)o * ngroups * NB * 32);
    double2* dst = reinterpret_cast<double2*>(Bd + buf * NB * 32);
    for (int i = threadIdx.x; i < NB * 16; i += 32 * kDmWarps) cp_async16(dst + i, src + i, 16);
  };
  const int w0 = warp * 8;
  auto load = [&](int o, double2 (&x)[6]) {
    const int q = qs[o * NP + w0 + g];
    const double2* row = spec_in + ((long)(q < 0 ? 0 : q) * n3h + f) * 24 + 6 * t;
#pragma unroll
    for (int u = 0; u < 6; ++u) x[u] = q >= 0 ? __ldg(row + u) : make_double2(0.0, 0.0);
  };
  double acc[NNT][2];
#pragma unroll
  for (int nt = 0; nt < NNT; ++nt) acc[nt][0] = acc[nt][1] = 0.0;
  double2 xc[6], xn[6];
  unsigned rem = blive;
  int oc = rem ? __ffs(rem) - 1 : 0;
  if (rem) {
    stage(oc, 0);
    if (wlive >> oc & 1u) load(oc, xn);
  }
  cp_async_commit();
#pragma unroll 1
  for (int k = 0; rem; ++k) {
    rem &= rem - 1;
    const int on = rem ? __ffs(rem) - 1 : -1;
    cp_async_wait<0>();  // this thread's copies of offset oc have landed
    __syncthreads();     // everyone's have; every warp is done with the other buffer
    if (on >= 0) stage(on, (k + 1) & 1);
    cp_async_commit();
    if (wlive >> oc & 1u) {
#pragma unroll
      for (int u = 0; u < 6; ++u) xc[u] = xn[u];
      if (on >= 0 && (wlive >> on & 1u)) load(on, xn);  // the next offset's row, in flight meanwhile
      const double* bq = Bd + (k & 1) * NB * 32 + lane;
#pragma unroll
      for (int sk = 0; sk < 12; ++sk) {
        const double a = sk & 1 ? xc[sk >> 1].y : xc[sk >> 1].x;
#pragma unroll
        for (int nt = 0; nt < NNT; ++nt) dmma(acc[nt], a, bq[(sk * NNT + nt) * 32]);
      }
    } else if (on >= 0 && (wlive >> on & 1u)) {
      load(on, xn);
    }
    oc = on;
  }
  cp_async_wait<0>();
  // C fragment: (row g, cols 2t, 2t+1): the re and im part of output element
  // e = 4 nt + t = j1 * KOC + c of the group
  const long p = pb + w0 + g;
  if (p < n_vtrg) {
    double2* out = spec_out + (p * n3h + f) * (8 * ko) + z * KOC;
#pragma unroll
    for (int nt = 0; nt < NNT; ++nt) {
      const int e = 4 * nt + t;
      out[(e / KOC) * ko + e % KOC] = make_double2(acc[nt][0], acc[nt][1]);
    }
  }
}

// ---------------------------------------------------------------------------
// Hadamard products of the plain form for scalar expansions (ke = 1) on the
// FP64 tensor cores: per frequency the real GEMM OUT[P][(j1, re|im)] +=
// sum_o IN[Q_o(P)][(j2, re|im)] B_o[..][..] with K = N = 16 (4 k-steps, 2
// n-tiles of mma.sync m8n8k4 .f64).  A warp owns MT tiles of 8 target parents;
// with the K order k-step s, column t -> child t + 4 (s/2), re|im = s % 2, lane
// (g, t) needs children t and t+4 of row g: two 16-byte pieces of its 128-byte
// row of the frequency-major input spectra (four lanes read 64 contiguous
// bytes), gathered from L2 two offsets ahead.  A block stages its
// frequency's B fragments (26 offsets, 53 KB) once and walks `chunks` chunks
// of target parents; each warp walks only the offsets occupied for one of its
// parents.  Frequency-major rows instead of one 16-byte piece per child and
// parent: 1M clustered points (m = 8) 6.35 -> 4.43 ms.
// ---------------------------------------------------------------------------
constexpr int kDm1Warps = 8;

template <int MT>
__global__ void __launch_bounds__(32 * kDm1Warps, 2)
    hadamard_dmma1_kernel(int n3h, long n_vtrg, long vt_stride, long n_vsrc, int chunks, const int* __restrict__ vtab,
                          const unsigned* __restrict__ vmask, const double2* __restrict__ spec_in,
                          const double* __restrict__ bfrag, double2* __restrict__ spec_out) {
  extern __shared__ double Bs1[];  // [26 offsets][8 blocks (s, nt)][32 lanes]
  constexpr int NP = kDm1Warps * 8 * MT;  // target parents of a chunk
  int* qs = reinterpret_cast<int*>(Bs1 + 26 * 8 * 32);  // [26][NP]
  unsigned* ms = reinterpret_cast<unsigned*>(qs + 26 * NP);  // [NP]
  const int f = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  {
    const double2* src = reinterpret_cast<const double2*>(bfrag + (long)f * 26 * 8 * 32);
    double2* dst = reinterpret_cast<double2*>(Bs1);
    for (int i = threadIdx.x; i < 26 * 8 * 16; i += 32 * kDm1Warps) dst[i] = __ldg(src + i);
  }
  const double2* in0 = spec_in + split_row(f, 0, n_vsrc) * 8 + t;  // row q: in0[8 q] (child t), in0[8 q + 4]
  for (int c = 0; c < chunks; ++c) {
    const long pb = ((long)blockIdx.x * chunks + c) * NP;
    if (pb >= n_vtrg) break;
    if (c > 0) __syncthreads();  // every warp is done with the previous chunk's qs
    for (int i = threadIdx.x; i < 26 * NP; i += 32 * kDm1Warps) {
      const int o = i / NP;
      const long p = pb + i % NP;
      qs[i] = p < n_vtrg ? __ldg(vtab + (long)o * vt_stride + p) : -1;
    }
    for (int i = threadIdx.x; i < NP; i += 32 * kDm1Warps) ms[i] = pb + i < n_vtrg ? __ldg(vmask + pb + i) : 0u;
    __syncthreads();
    const int w0 = warp * 8 * MT;
    double acc[MT][2][2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = 0.0;
    unsigned live = 0;
    for (int k = lane; k < 8 * MT; k += 32) live |= ms[w0 + k];
    live = __reduce_or_sync(0xffffffffu, live);
    double2 xa[MT][2], xb[MT][2], xc[MT][2];
    auto load = [&](int o, double2 (&x)[MT][2]) {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const int q = qs[o * NP + w0 + mt * 8 + g];
        x[mt][0] = q >= 0 ? __ldg(in0 + (long)q * 8) : make_double2(0.0, 0.0);
        x[mt][1] = q >= 0 ? __ldg(in0 + (long)q * 8 + 4) : make_double2(0.0, 0.0);
      }
    };
    auto compute = [&](int o, const double2 (&x)[MT][2]) {
      double b[4][2];
#pragma unroll
      for (int sk = 0; sk < 4; ++sk)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) b[sk][nt] = Bs1[((o * 4 + sk) * 2 + nt) * 32 + lane];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const double a[4] = {x[mt][0].x, x[mt][0].y, x[mt][1].x, x[mt][1].y};
#pragma unroll
        for (int sk = 0; sk < 4; ++sk)
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) dmma(acc[mt][nt], a[sk], b[sk][nt]);
      }
    };
    unsigned rem = live;
    const int nlive = __popc(live);
    auto take = [&]() {
      const int o = __ffs(rem) - 1;
      rem &= rem - 1;
      return o;
    };
    int oa = 0, ob = 0, oc = 0;
    if (nlive > 0) {
      oa = take();
      load(oa, xa);
    }
    if (nlive > 1) {
      ob = take();
      load(ob, xb);
    }
#pragma unroll 1
    for (int i = 0; i < nlive; i += 3) {
      if (i + 2 < nlive) {
        oc = take();
        load(oc, xc);
      }
      compute(oa, xa);
      if (i + 3 < nlive) {
        oa = take();
        load(oa, xa);
      }
      if (i + 1 < nlive) compute(ob, xb);
      if (i + 4 < nlive) {
        ob = take();
        load(ob, xb);
      }
      if (i + 2 < nlive) compute(oc, xc);
    }
    // C fragment: (row g, cols 2t, 2t+1) of n-tile nt = the re and im part of
    // child j1 = 4 nt + t
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const long p = pb + w0 + mt * 8 + g;
      if (p >= n_vtrg) continue;
      double2* out = spec_out + (p * n3h + f) * 8;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) out[4 * nt + t] = make_double2(acc[mt][nt][0], acc[mt][nt][1]);
    }
  }
}

void launch_hadamard_dmma1(Context& ctx, int n3h, long f_base, const Cplx<double>* sin_, Cplx<double>* sout, long p0,
                           long np) {
  DevTree& T = ctx.tree;
  constexpr int MT = 2;
  const size_t sm = (size_t)26 * 8 * 32 * sizeof(double) + (size_t)27 * kDm1Warps * 8 * MT * sizeof(int);
  PVFMM_CUDA_CHECK(
      cudaFuncSetAttribute(hadamard_dmma1_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  const int chunks = 8;
  dim3 grid(ceil_div(np, (long)8 * MT * kDm1Warps * chunks), n3h);
  ++ctx.n_launch;
  hadamard_dmma1_kernel<MT><<<grid, 32 * kDm1Warps, sm, ctx.stream>>>(
      n3h, np, T.n_vtrg, T.n_vsrc, chunks, T.vtab.get<int>() + p0, T.vmask.get<unsigned>() + p0,
      reinterpret_cast<const double2*>(sin_), ctx.dops.vop_frag.get<double>() + f_base * 26 * 8 * 32,
      reinterpret_cast<double2*>(sout));
}

template <int KOC>
void launch_hadamard_dmma3(Context& ctx, int n3h, long f_base, int ko, const Cplx<double>* sin_, Cplx<double>* sout,
                           long p0, long np) {
  DevTree& T = ctx.tree;
  constexpr int NB = 24 * KOC, NP = kDmWarps * 8;
  const int ngroups = ko / KOC;
  const size_t sm = (size_t)2 * NB * 32 * sizeof(double) + (size_t)26 * NP * sizeof(int) + kDmWarps * sizeof(int);
  PVFMM_CUDA_CHECK(
      cudaFuncSetAttribute(hadamard_dmma3_kernel<KOC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  dim3 grid(ceil_div(np, (long)NP), n3h, ngroups);
  ++ctx.n_launch;
  hadamard_dmma3_kernel<KOC><<<grid, 32 * kDmWarps, sm, ctx.stream>>>(
      n3h, np, T.n_vtrg, ko, T.vtab.get<int>() + p0, T.vmask.get<unsigned>() + p0,
      reinterpret_cast<const double2*>(sin_), ctx.dops.vop_frag.get<double>() + f_base * 26 * ngroups * NB * 32,
      reinterpret_cast<double2*>(sout));
}

// Target parents [p0, p0 + np) of the V-list; sout holds their rows.
void launch_hadamard_tc(Context& ctx, int n3h, long f_base, const Cplx<float>* sin_, Cplx<float>* sout, long p0,
                        long np) {
  DevTree& T = ctx.tree;
  const size_t sm = (size_t)26 * 2 * 32 * sizeof(uint4) + (size_t)kTcWarps * 2 * kTcEnt * sizeof(int);
  PVFMM_CUDA_CHECK(cudaFuncSetAttribute(hadamard_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  const int chunks = kTcChunks;
  dim3 grid(ceil_div(np, (long)16 * kTcWarps * chunks), n3h);
  ++ctx.n_launch;
  hadamard_tc_kernel<<<grid, 32 * kTcWarps, sm, ctx.stream>>>(
      n3h, np, T.n_vtrg, T.n_vsrc, chunks, T.vtab.get<int>() + p0, T.vmask.get<unsigned>() + p0,
      reinterpret_cast<const uint4*>(sin_), ctx.qscale.get<float>(),
      ctx.dops.vop_frag.get<uint4>() + f_base * 26 * 2 * 32, ctx.dops.vop_fscale.get<float>() + f_base,
      reinterpret_cast<float2*>(sout));
}

template <class Real, int PB>
void launch_hadamard_rd(Context& ctx, int n3h, long f_base, const Cplx<Real>* sin_, Cplx<Real>* sout, long p0,
                        long np) {
  DevTree& T = ctx.tree;
  dim3 grid(ceil_div(np, 128 * PB), n3h);
  ++ctx.n_launch;
  hadamard_rd_kernel<Real, PB><<<grid, 128, 0, ctx.stream>>>(n3h, np, T.n_vtrg, T.n_vsrc, T.vtab.get<int>() + p0,
                                                             T.vmask.get<unsigned>() + p0, sin_,
                                                             ctx.dops.vop.get<Cplx<Real>>() + f_base * 26 * 64, sout);
}

// Target parents per thread (register tile) of the FP64 scalar Hadamard.
#ifndef PVFMM_HAD_PB_F64
#define PVFMM_HAD_PB_F64 1
#endif

template <class Real, int KI, int KO, int OC>
size_t hadamard_smem() {
  constexpr int STRIDE = 8 * KI + 16 / (int)sizeof(Cplx<Real>);
  return sizeof(Cplx<Real>) * ((size_t)OC * 64 * KI * KO + 2 * 128 * STRIDE);
}

template <class Real, int KI, int KO, int KOC, int OC>
void launch_hadamard(Context& ctx, int n3h, long f_base, const Cplx<Real>* sin_, Cplx<Real>* sout, long p0,
                     long np) {
  static_assert(KO % KOC == 0, "output components in whole groups");
  DevTree& T = ctx.tree;
  const size_t sm = hadamard_smem<Real, KI, KO, OC>();
  PVFMM_CUDA_CHECK(cudaFuncSetAttribute(hadamard_kernel<Real, KI, KO, KOC, OC>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  dim3 grid(ceil_div(np, 128), n3h, KO / KOC);
  ++ctx.n_launch;
  hadamard_kernel<Real, KI, KO, KOC, OC><<<grid, 128, sm, ctx.stream>>>(
      n3h, np, T.n_vtrg, T.vtab.get<int>() + p0, sin_, ctx.dops.vop.get<Cplx<Real>>() + f_base * 26 * 64 * KI * KO,
      sout);
}

// ---------------------------------------------------------------------------
// Small helpers.
// ---------------------------------------------------------------------------
// Per-component scales of the C interface's rescale (at most 9 components):
// scale_x^src_scal of the densities, scale_x * scale_x^src_scal and 1 of the
// double-layer values, scale_x^trg_scal of the outputs.
struct OutScales {
  double v[9];
};

// Densities (k values per point) in sorted order, each scaled in the input
// precision as the reference scales them (pvfmm-wrapper.cpp:591-599).
template <class Tin>
__global__ void sort_densities(const Tin* __restrict__ in, const int* __restrict__ perm, long n, int k,
                               OutScales sc, double* __restrict__ out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long p = perm[i];
  for (int j = 0; j < k; ++j) out[i * k + j] = (double)((Tin)in[p * k + j] * (Tin)sc.v[j]);
}

// Periodic lattice sum: subtracts from every target value the volume
// potential of the mean source density, taken as the sum of the root's
// upward equivalent density per component (the reference's PostProcessing,
// fmm_pts.txx:5741-5771, with laplace_vol_poten -|x|^2/6 and
// stokes_vol_poten -(|x|^2 - x_l^2)/4 of kernel.txx:1289-1295, 1456-1467) at
// the target's unit-cube position x.  kin = k1 = 1 (Laplace potential) or 3
// (Stokes velocity).  Every block forms the sums itself (ns*kin values).
__global__ void __launch_bounds__(256) periodic_mean_correction(
    long n_trg, const int* __restrict__ trg_leaf, const MKey* __restrict__ keys, const double* __restrict__ tx,
    const double* __restrict__ ty, const double* __restrict__ tz, const double* __restrict__ ue_root, int ns, int kin,
    int k1, double* __restrict__ pot) {
  __shared__ double part[256][3];
  __shared__ double avg[3];
  double a[3] = {0, 0, 0};
  for (int i = threadIdx.x; i < ns; i += blockDim.x)
    for (int k = 0; k < kin && k < 3; ++k) a[k] += ue_root[(long)i * kin + k];
  for (int k = 0; k < 3; ++k) part[threadIdx.x][k] = a[k];
  __syncthreads();
  if (threadIdx.x < 3) {
    double v = 0;
    for (int j = 0; j < (int)blockDim.x; ++j) v += part[j][threadIdx.x];
    avg[threadIdx.x] = v;
  }
  __syncthreads();
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n_trg; t += (long)gridDim.x * blockDim.x) {
    double cx, cy, cz, half;
    int d;
    node_geom(keys[trg_leaf[t]], cx, cy, cz, half, d);
    const double x = tx[t] + cx, y = ty[t] + cy, z = tz[t] + cz;
    if (k1 == 1) {
      pot[t] += avg[0] * (x * x + y * y + z * z) / 6;
    } else {
      pot[t * 3 + 0] += avg[0] * (y * y + z * z) / 4;
      pot[t * 3 + 1] += avg[1] * (x * x + z * z) / 4;
      pot[t * 3 + 2] += avg[2] * (x * x + y * y) / 4;
    }
  }
}

template <class Tout>
__global__ void unsort_values(const double* __restrict__ pot, const int* __restrict__ perm, long n, int k1,
                              OutScales sc, Tout* __restrict__ out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long p = perm[i];
  for (int k = 0; k < k1; ++k) out[p * k1 + k] = (Tout)((Tout)pot[i * k1 + k] * (Tout)sc.v[k]);
}

template <class Real>
void upload_vec(DevBuf& b, const std::vector<double>& v, cudaStream_t s) {
  std::vector<Real> tmp(v.begin(), v.end());
  Real* d = b.as<Real>(tmp.size());
  PVFMM_CUDA_CHECK(cudaMemcpyAsync(d, tmp.data(), tmp.size() * sizeof(Real), cudaMemcpyHostToDevice, s));
  PVFMM_CUDA_CHECK(cudaStreamSynchronize(s));
}

// V-list: forward DFTs of every source parent, then the Hadamard products
// and inverse DFTs of the target parents in chunks of `chunk` parents (the
// output spectra of one chunk at a time; one chunk when device memory
// allows).  With several chunks, stage 4 ends after the first chunk's
// products and stage 5 covers the rest.
// Kernel of the mixed form's scalar Hadamard: the warp-level MMA kernel
// gathering from L2 (hadamard_tc_kernel), or with PVFMM_B200_HADAMARD=tcgen05
// the tcgen05 kernel with TMEM accumulators over tiles of Morton-consecutive
// targets (hadamard_tc.cu).
bool use_tc5(const Context&) {
  const char* e = std::getenv("PVFMM_B200_HADAMARD");
  return e && std::strcmp(e, "tcgen05") == 0;
}
// Hadamard of 3-component expansions: tensor cores (hadamard_tc3_kernel in
// the mixed form, hadamard_dmma3_kernel in the plain form), or with
// PVFMM_B200_HADAMARD3=simt the SIMT kernel (hadamard_kernel).
bool use_simt3() {
  const char* e = std::getenv("PVFMM_B200_HADAMARD3");
  return e && std::strcmp(e, "simt") == 0;
}
// Plain-form Hadamard of scalar expansions: FP64 tensor cores
// (hadamard_dmma1_kernel), or with PVFMM_B200_HADAMARD=simt the FP64 SIMT
// kernel (hadamard_rd_kernel).
bool use_simt1() {
  const char* e = std::getenv("PVFMM_B200_HADAMARD");
  return e && std::strcmp(e, "simt") == 0;
}

template <class Real, int M>
void vlist_fft_t(Context& ctx, const double* ue, double* dc, Cplx<Real>* sin_, Cplx<Real>* sout, int kin, int kout,
                 long chunk, int nslab, const std::function<void(int)>& ev) {
  DevTree& T = ctx.tree;
  auto s = ctx.stream;
  using F = FftSizes<Real, M>;
  const int ngrid_up = 8 * kin, ngrid_dn = 8 * kout;
  const int Gu = F::up_grids(ngrid_up), Gd = F::dn_grids(ngrid_dn);
  const size_t sm_up = Gu * F::up_grid_bytes;
  PVFMM_CUDA_CHECK(cudaFuncSetAttribute(fft_up_kernel<Real, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_up));
  const size_t sm_dn = Gd * F::dn_grid_bytes + 2 * F::N1 * sizeof(Real);
  auto ifft = ifft_dn_kernel<Real, M, false>;
  if constexpr (F::kRows) {
    if (ngrid_dn == 8) ifft = ifft_dn_kernel<Real, M, true>;
  }
  PVFMM_CUDA_CHECK(cudaFuncSetAttribute(ifft, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_dn));
  // split-FP16 input spectra for the mixed form's tensor-core Hadamards
  const double* qinv = nullptr;
  if (sizeof(Real) == 4 && !(kin == 1 ? use_tc5(ctx) : use_simt3())) {
    float* qs = ctx.qscale.as<float>(T.n_vsrc);
    double* qi = ctx.qinv.as<double>(T.n_vsrc);
    ++ctx.n_launch;
    vsrc_scale_kernel<<<T.n_vsrc, 256, 0, s>>>(T.vsrc.get<int>(), T.child0.get<int>(), ue, ctx.ns * kin,
                                             ctx.vop_exp, qs, qi);
    qinv = qi;
  }
  // slabs of kz (the slowest frequency index): each slab's forward DFT rows,
  // products and inverse DFT contribution in turn (nslab = 1: all at once)
  for (int sl = 0; sl < nslab; ++sl) {
    const int kz0 = F::N1 * sl / nslab, nkz = F::N1 * (sl + 1) / nslab - kz0;
    const int n3h = F::N1 * F::NH * nkz;           // the slab's frequencies
    const long f_base = (long)F::N1 * F::NH * kz0;  // its first frequency
    ++ctx.n_launch;
    fft_up_kernel<Real, M><<<T.n_vsrc * (ngrid_up / Gu), F::threads(Gu), sm_up, s>>>(
        kin, Gu, ngrid_up / Gu, T.vsrc.get<int>(), T.child0.get<int>(), ue, ctx.dops.fft_map.get<int>(), ctx.ns,
        T.n_vsrc, kz0, nkz, qinv, sin_);
    if (sl == 0) ev(4);
    for (long p0 = 0; p0 < T.n_vtrg; p0 += chunk) {
      const long np = std::min(chunk, T.n_vtrg - p0);
      if (kin == 1 && kout == 1) {
        if constexpr (sizeof(Real) == 8) {
          if (use_simt1()) launch_hadamard_rd<Real, PVFMM_HAD_PB_F64>(ctx, n3h, f_base, sin_, sout, p0, np);
          else launch_hadamard_dmma1(ctx, n3h, f_base, sin_, sout, p0, np);
        }
        else if (use_tc5(ctx)) launch_hadamard_tc5(ctx, n3h, f_base, sin_, sout, p0, np);
        else launch_hadamard_tc(ctx, n3h, f_base, sin_, sout, p0, np);
      } else if (!use_simt3()) {  // 3-component expansions: tensor cores (split FP16 or FP64)
        if constexpr (sizeof(Real) == 4) {
          if (kout == 1) launch_hadamard_tc3<1>(ctx, n3h, f_base, 1, sin_, sout, p0, np);
          else launch_hadamard_tc3<3>(ctx, n3h, f_base, kout, sin_, sout, p0, np);
        } else {
          if (kout == 1) launch_hadamard_dmma3<1>(ctx, n3h, f_base, 1, sin_, sout, p0, np);
          else launch_hadamard_dmma3<3>(ctx, n3h, f_base, kout, sin_, sout, p0, np);
        }
      } else if (kout == 3) {  // Stokes velocity, Biot-Savart
        launch_hadamard<Real, 3, 3, 3, 4>(ctx, n3h, f_base, sin_, sout, p0, np);
      } else if (kout == 1) {  // Stokes pressure
        launch_hadamard<Real, 3, 1, 1, 4>(ctx, n3h, f_base, sin_, sout, p0, np);
      } else {  // Stokes velocity gradient: 9 outputs in 3 groups of 3
        launch_hadamard<Real, 3, 9, 3, 2>(ctx, n3h, f_base, sin_, sout, p0, np);
      }
      if (p0 == 0 && sl == 0) ev(5);
      ++ctx.n_launch;
      ifft<<<np * (ngrid_dn / Gd), F::threads(Gd), sm_dn, s>>>(
          kout, Gd, ngrid_dn / Gd, T.vtrg.get<int>() + p0, T.child0.get<int>(), T.key.get<MKey>(), sout,
          ctx.dops.ifft_map.get<int>(), ctx.ns, ctx.ki.deg, kz0, nkz, dc);
    }
  }
}

// V-list of equivalent densities with kin components onto check potentials
// with kout components.
template <class Real>
void vlist(Context& ctx, const double* ue, double* dc, int kin, int kout, const std::function<void(int)>& ev) {
  DevTree& T = ctx.tree;
  const int m = ctx.m, n1 = 2 * m, n3h_all = 4 * m * m * (m + 1);
  // input spectra of all source parents for a slab of kz: the whole spectrum
  // (one slab) when it takes at most 45% of the free device memory (counting
  // this buffer's current allocation), else the fewest slabs that do
  const size_t in_all = (size_t)T.n_vsrc * n3h_all * 8 * kin * sizeof(Cplx<Real>);
  int nslab = 1;
  if (in_all > ctx.spec_in.cap) {
    size_t free_b = 0, total_b = 0;
    PVFMM_CUDA_CHECK(cudaMemGetInfo(&free_b, &total_b));
    const double avail = 0.45 * (double)(free_b + ctx.spec_in.cap + ctx.spec_out.cap);
    while (nslab < n1 && (double)in_all / nslab > avail) ++nslab;
  }
  // PVFMM_B200_VLIST_SLABS sets the slab count (to exercise the slab path)
  if (const char* e = std::getenv("PVFMM_B200_VLIST_SLABS")) {
    const int v = std::atoi(e);
    if (v > 0) nslab = std::min(v, n1);
  }
  const int n3h = n1 * (m + 1) * ((n1 + nslab - 1) / nslab);  // frequencies of the largest slab
  Cplx<Real>* sin_ = ctx.spec_in.as<Cplx<Real>>((size_t)T.n_vsrc * n3h * 8 * kin);
  // output spectra: all target parents at once when they fit in 90% of the
  // free device memory (counting this buffer's current allocation), else
  // chunks of that size
  const size_t row = (size_t)n3h * 8 * kout * sizeof(Cplx<Real>);
  long chunk = T.n_vtrg;
  if ((size_t)T.n_vtrg * row > ctx.spec_out.cap) {  // query the device only when the buffer must grow
    size_t free_b = 0, total_b = 0;
    PVFMM_CUDA_CHECK(cudaMemGetInfo(&free_b, &total_b));
    const double avail = 0.9 * (double)(free_b + ctx.spec_out.cap);
    if ((double)T.n_vtrg * row > avail) chunk = std::max(256L, (long)(avail / row));
  }
  // PVFMM_B200_VLIST_CHUNK caps the chunk (to exercise the chunked path)
  if (const char* e = std::getenv("PVFMM_B200_VLIST_CHUNK")) {
    const long c = std::atol(e);
    if (c > 0) chunk = std::min(chunk, c);
  }
  // the tcgen05 Hadamard walks tiles of Morton-consecutive targets, which stay
  // inside windows of 2048 positions: its chunks are whole windows
  if (sizeof(Real) == 4 && kin == 1 && kout == 1 && use_tc5(ctx) && chunk < T.n_vtrg)
    chunk = std::max(2048L, chunk / 2048 * 2048);
  Cplx<Real>* sout = ctx.spec_out.as<Cplx<Real>>((size_t)std::min(chunk, T.n_vtrg) * n3h * 8 * kout);
  switch (m) {
    case 2: vlist_fft_t<Real, 2>(ctx, ue, dc, sin_, sout, kin, kout, chunk, nslab, ev); break;
    case 4: vlist_fft_t<Real, 4>(ctx, ue, dc, sin_, sout, kin, kout, chunk, nslab, ev); break;
    case 6: vlist_fft_t<Real, 6>(ctx, ue, dc, sin_, sout, kin, kout, chunk, nslab, ev); break;
    case 8: vlist_fft_t<Real, 8>(ctx, ue, dc, sin_, sout, kin, kout, chunk, nslab, ev); break;
    case 10: vlist_fft_t<Real, 10>(ctx, ue, dc, sin_, sout, kin, kout, chunk, nslab, ev); break;
    case 12: vlist_fft_t<Real, 12>(ctx, ue, dc, sin_, sout, kin, kout, chunk, nslab, ev); break;
    case 14: vlist_fft_t<Real, 14>(ctx, ue, dc, sin_, sout, kin, kout, chunk, nslab, ev); break;
    case 16: vlist_fft_t<Real, 16>(ctx, ue, dc, sin_, sout, kin, kout, chunk, nslab, ev); break;
    default: throw std::runtime_error("unsupported multipole order");
  }
}

// S2U check potentials of all source leaves from the values `den` per point.
template <int Ker>
void launch_s2u(Context& ctx, const double* den, double scale, bool accumulate, double* uc) {
  DevTree& T = ctx.tree;
  const long n = T.n_sleaf * (ctx.ns / 2);
  auto run = [&](auto kernel, int lanes) {
    kernel<<<ceil_div(n * lanes, kNT), kNT, 0, ctx.stream>>>(
        n, T.sleaf.get<int>(), T.key.get<MKey>(), T.src_lo.get<int>(), T.src_hi.get<int>(), nullptr, nullptr, nullptr,
        T.sx.get<double>(), T.sy.get<double>(), T.sz.get<double>(), den, ctx.dops.usurf.get<double>(), ctx.ns, kRad1,
        scale, ctx.ki.deg, accumulate, uc);
  };
  if (surface_lanes(n) == 4) run(surface_check_kernel<Ker, false, 4>, 4);
  else run(surface_check_kernel<Ker, false, 1>, 1);
}

template <class Real, int KerS2T, int KerExp>
void evaluate_impl(Context& ctx, const void* den_in, const void* dl_in, bool den_float, void* out, bool out_float) {
  DevTree& T = ctx.tree;
  // double-layer kernels of the source -> check and source -> target
  // sub-kernels (Laplace potential: laplace_dbl_poten; Stokes velocity:
  // stokes_sym_dip; kernel.txx:1334-1340, 1470-1473)
  constexpr int KerDblExp = KerExp == kKerLaplace ? kKerLaplaceDbl : KerExp == kKerStokes ? kKerStokesDbl : -1;
  constexpr int KerDblS2T = KerS2T == kKerLaplace ? kKerLaplaceDbl : KerS2T == kKerStokes ? kKerStokesDbl : -1;
  const bool has_sl = den_in != nullptr, has_dl = dl_in != nullptr;
  if (has_dl && (KerDblExp < 0 || KerDblS2T < 0))
    throw std::runtime_error("this kernel has no double-layer kernel (dl_den must be NULL)");
  if (T.src_counted && T.layers != ((int)has_sl | (int)has_dl << 1))
    throw std::runtime_error("setup=0 requires the same densities (sl_den, dl_den) passed or NULL as at setup");
  auto s = ctx.stream;
  // expansion dims: equivalent densities din = ns*kin, check potentials
  // dout = ns*kout (kin = kout for Laplace and Stokes velocity); the
  // pseudo-inverse factors pass through r = min(din, dout) values
  const int ns = ctx.ns, kin = KerDims<KerExp>::KS, kout = KerDims<KerExp>::KT;
  const int din = ns * kin, dout = ns * kout, deg = ctx.ki.deg;
  // inner widths of the upward and downward check -> equivalent products
  // (the kept singular directions, padded to even)
  const int ru = ctx.ru, rd = ctx.rd;
  const int k0 = ctx.ki.k0, k1 = ctx.ki.k1;
  const long N = T.n_nodes;
  const MKey* keys = T.key.get<MKey>();
  // periodic boundaries: image codes of the list entries (null: free space)
  const unsigned char* pimg = ctx.periodic ? T.p_img.get<unsigned char>() : nullptr;
  const unsigned char* wimg = ctx.periodic ? T.w_img.get<unsigned char>() : nullptr;
  const unsigned char* ximg = ctx.periodic ? T.x_img.get<unsigned char>() : nullptr;
  const std::function<void(int)> ev = [&](int i) {
    if (ctx.events_ready) PVFMM_CUDA_CHECK(cudaEventRecord(ctx.ev[i], s));
  };
  ev(0);
  if (ctx.den_pending) {  // densities uploaded on the side stream during the tree build
    PVFMM_CUDA_CHECK(cudaStreamWaitEvent(s, ctx.den_ev, 0));
    ctx.den_pending = false;
  }
  // densities (sorted, scaled by scale_x^src_scal: pvfmm-wrapper.cpp:522-541, 591-595)
  double* den = ctx.den.as<double>(std::max(T.n_src, 1L) * k0);
  // double-layer values (sorted, scaled by surf_scal: scale_x * scale_x^src_scal
  // for the k0 densities, 1 for the normal; pvfmm-wrapper.cpp:528-535, 596-599)
  double* surf = has_dl ? ctx.surf.as<double>(std::max(T.n_src, 1L) * (k0 + 3)) : nullptr;
  OutScales ss, sf, ts;
  for (int j = 0; j < 9; ++j) {
    ss.v[j] = den_float ? (double)std::pow((float)T.scale_x, (float)ctx.ki.src_scal[j % 3])
                        : std::pow(T.scale_x, ctx.ki.src_scal[j % 3]);
    ts.v[j] = out_float ? (double)std::pow((float)T.scale_x, (float)ctx.ki.trg_scal[j])
                        : std::pow(T.scale_x, ctx.ki.trg_scal[j]);
  }
  for (int j = 0; j < 9; ++j)
    sf.v[j] = j >= k0 ? 1.0 : den_float ? (double)((float)T.scale_x * (float)ss.v[j]) : T.scale_x * ss.v[j];
  auto sort_vals = [&](const void* in, int k, const OutScales& sc, double* o) {
    ++ctx.n_launch;
    if (den_float)
      sort_densities<float><<<ceil_div(T.n_src, 256), 256, 0, s>>>((const float*)in, T.src_perm.get<int>(), T.n_src,
                                                                   k, sc, o);
    else
      sort_densities<double><<<ceil_div(T.n_src, 256), 256, 0, s>>>((const double*)in, T.src_perm.get<int>(),
                                                                    T.n_src, k, sc, o);
  };
  if (T.src_counted && has_sl) sort_vals(den_in, k0, ss, den);
  if (T.src_counted && has_dl) sort_vals(dl_in, k0 + 3, sf, surf);
  double* ue = ctx.ue.as<double>((size_t)N * din);
  double* dc = ctx.dc.as<double>((size_t)N * dout);
  PVFMM_CUDA_CHECK(cudaMemsetAsync(ue, 0, (size_t)N * din * sizeof(double), s));
  PVFMM_CUDA_CHECK(cudaMemsetAsync(dc, 0, (size_t)N * dout * sizeof(double), s));
  // mixed form, Stokes kernel: the FP32 stages (V-list input, W list) read
  // the upward equivalent densities projected onto the directions above the
  // FP32 cutoff (ue32 = ue U_k U_k^T); the FP64 stages keep ue.  (2M-point
  // m=10 Stokes error 3.3e-4 without, 2.8e-5 with; no change for Laplace.)
  // The leaves' rows come from the first r32 columns of the S2U
  // intermediate, the internal nodes' from ue after U2U; leaves without
  // sources keep zero rows.
  const bool proj32 = sizeof(Real) == 4 && kin == 3 && T.src_counted && N > 0 && ctx.r32 > 0;
  double* ue32 = nullptr;
  if (proj32) {
    ue32 = ctx.ue_c.as<double>((size_t)N * din);
    PVFMM_CUDA_CHECK(cudaMemsetAsync(ue32, 0, (size_t)N * din * sizeof(double), s));
  }
  const double* usurf = ctx.dops.usurf.get<double>();
  const double* sx = T.sx.get<double>();
  const double* sy = T.sy.get<double>();
  const double* sz = T.sz.get<double>();
  const int* slo = T.src_lo.get<int>();
  const int* shi = T.src_hi.get<int>();
  const double kscale_exp = ker_scale(KerExp);
  ev(1);
  // ---- S2U
  if (T.src_counted && T.n_sleaf > 0) {
    double* uc = ctx.uc_c.as<double>((size_t)T.n_sleaf * dout);
    double* t1 = ctx.tmp_c.as<double>((size_t)T.n_sleaf * ru);
    ++ctx.n_launch;
    // full FP64 rsqrt here in both forms: the check potentials feed the
    // FP64-cutoff pseudo-inverse, which amplifies their rounding into
    // near-null components of the equivalent densities; the mixed form's FP32
    // V-list does not cancel those (one Newton step here raised the 4M-point
    // potential error from 3e-7 to 2.5e-6)
    if (has_sl)
      launch_s2u<KerExp>(ctx, den, kscale_exp, false, uc);
    if constexpr (KerDblExp >= 0) {
      if (has_dl) {
        ++ctx.n_launch;
        launch_s2u<KerDblExp>(ctx, surf, ker_scale(KerDblExp), has_sl, uc);
      }
    }
    // equivalent densities (uc UC2UE0) UC2UE1 straight into the leaves' rows of UE
    ++ctx.n_launch;
    translate_gemm(s, T.n_sleaf, ru, dout, uc, dout, nullptr, ctx.dops.uc2ue0.get<double>(), ru, t1, ru, nullptr,
                   nullptr, false);
    if (!proj32) {
      ++ctx.n_launch;
      translate_gemm(s, T.n_sleaf, din, ru, t1, ru, nullptr, ctx.dops.uc2ue1.get<double>(), din, ue, din,
                     T.sleaf.get<int>(), nullptr, false);
    } else {
      // the first r32 directions give the leaves' projected rows, ue U_k U_k^T
      // = (t1 columns 0..r32) (UC2UE1 rows 0..r32); ue adds the other
      // directions to a copy of them (both arrays are zero outside the
      // leaves' rows here)
      const int r32 = ctx.r32;
      ++ctx.n_launch;
      translate_gemm(s, T.n_sleaf, din, r32, t1, ru, nullptr, ctx.dops.uc2ue1.get<double>(), din, ue32, din,
                     T.sleaf.get<int>(), nullptr, false);
      PVFMM_CUDA_CHECK(cudaMemcpyAsync(ue, ue32, (size_t)N * din * sizeof(double), cudaMemcpyDeviceToDevice, s));
      if (ru > r32) {
        ++ctx.n_launch;
        translate_gemm(s, T.n_sleaf, din, ru - r32, t1 + r32, ru, nullptr,
                       ctx.dops.uc2ue1.get<double>() + (size_t)r32 * din, din, ue, din, T.sleaf.get<int>(), nullptr,
                       true);
      }
    }
  }
  ev(2);
  // ---- U2U, bottom-up
  if (T.src_counted) {
    for (int d = T.depth - 1; d >= 0; --d) {
      const long ni = T.n_internal[d];
      if (ni == 0) continue;
      // the 8 children of the level's k-th internal node are the k-th block
      // of 8 rows of the next level: one row of 8*din values per parent.  The
      // long K (8 children) is split per child, so that the coarse levels
      // with few parents still fill the GPU; the 8 pieces are added in order.
      ctx.n_launch += 2;
      double* part = ctx.tmp_c.as<double>((size_t)8 * ni * din);
      if (T.up_lists) {  // the children with sources only
        const ChildRows up{T.up_rows.get<int>() + T.int_off[d], T.up_counts.get<int>() + 8 * d, T.int_off[T.depth],
                           T.up_mask.get<unsigned char>() + T.int_off[d]};
        translate_up(s, ni, din, ue + (size_t)T.level_off[d + 1] * din, ctx.dops.u2u.get<double>(), ue,
                     T.int_idx.get<int>() + T.int_off[d], part, up);
        continue;
      }
      translate_gemm(s, ni, din, 8 * din, ue + (size_t)T.level_off[d + 1] * din, 8 * din, nullptr,
                     ctx.dops.u2u.get<double>(), din, ue, din, T.int_idx.get<int>() + T.int_off[d], nullptr, false, 8,
                     part);
    }
  }
  // the internal nodes' projected rows: (ue U_k) U_k^T through a compact
  // n_internal x r32 intermediate
  if (proj32) {
    long nint = 0;
    for (int d = 0; d < T.depth; ++d) nint += T.n_internal[d];
    if (nint > 0) {
      const int r32 = ctx.r32;
      double* tp = ctx.tmp_c.as<double>((size_t)nint * r32);
      ctx.n_launch += 2;
      translate_gemm(s, nint, r32, din, ue, din, T.int_idx.get<int>(), ctx.dops.ue_basis.get<double>(), r32, tp, r32,
                     nullptr, nullptr, false);
      translate_gemm(s, nint, din, r32, tp, r32, nullptr, ctx.dops.uc2ue1.get<double>(), din, ue32, din,
                     T.int_idx.get<int>(), nullptr, false);
    }
  }
  if (!proj32) ue32 = ue;
  // periodic boundaries (PeriodicBC, fmm_pts.txx:2642-2676): the root's
  // downward check potential of the images beyond its 3x3x3 block
  if (ctx.periodic && T.src_counted && N > 0) {
    ++ctx.n_launch;
    translate_gemm(s, 1, dout, din, ue, din, nullptr, ctx.dops.bc.get<double>(), dout, dc, dout, nullptr, nullptr,
                   true);
  }
  ev(3);
  // ---- V-list
  if (T.src_counted && T.n_vtrg > 0 && T.n_vsrc > 0) {
    vlist<Real>(ctx, ue32, dc, kin, kout, ev);
  } else {
    ev(4);
    ev(5);
  }
  if (ctx.tc5_err) {  // the tensor-core Hadamard's error word, checked by the caller after synchronising
    PVFMM_CUDA_CHECK(cudaMemcpyAsync(ctx.tc5_err_host, ctx.tc5_err, sizeof(int), cudaMemcpyDeviceToHost, s));
    ctx.tc5_err = nullptr;
  }
  ev(6);
  // ---- X-list
  if (T.src_counted && T.n_xtrg > 0) {
    ++ctx.n_launch;
    const long n_thr = T.n_xtrg * (ns / 2);
    if (has_sl)
      surface_check_kernel<KerExp, true, 4><<<ceil_div(4 * n_thr, kNT), kNT, 0, s>>>(
          n_thr, T.xtrg.get<int>(), keys, slo, shi, T.x_off.get<int>(), T.x_list.get<int>(), ximg, sx, sy, sz, den,
          usurf, ns, kRad0, kscale_exp, deg, true, dc);
    if constexpr (KerDblExp >= 0) {
      if (has_dl) {
        ++ctx.n_launch;
        surface_check_kernel<KerDblExp, true, 4><<<ceil_div(4 * n_thr, kNT), kNT, 0, s>>>(
            n_thr, T.xtrg.get<int>(), keys, slo, shi, T.x_off.get<int>(), T.x_list.get<int>(), ximg, sx, sy, sz, surf,
            usurf, ns, kRad0, ker_scale(KerDblExp), deg, true, dc);
      }
    }
  }
  ev(7);
  // ---- D2D, top-down
  for (int d = 0; d < T.depth; ++d) {
    const long ni = T.n_internal[d];
    if (ni == 0) continue;
    // the children with targets only, where many leaves are empty
    const ChildRows dn{T.dn_rows.get<int>() + T.int_off[d], T.dn_counts.get<int>() + 8 * d, T.int_off[T.depth],
                       nullptr};
    double* children = dc + (size_t)T.level_off[d + 1] * dout;
    if (ctx.d2d_factored) {  // (parents' dc DC2DE0) over the kept directions, then DC2DE1 M_pe2c
      double* tp = ctx.tmp_c.as<double>((size_t)ni * rd);
      ctx.n_launch += 2;
      translate_gemm(s, ni, rd, dout, dc, dout, T.int_idx.get<int>() + T.int_off[d], ctx.dops.dc2de0.get<double>(),
                     rd, tp, rd, nullptr, nullptr, false);
      if (T.dn_lists)
        translate_down(s, ni, dout, rd, tp, rd, nullptr, ctx.dops.d2d_f2.get<double>(), children, dn);
      else
        translate_gemm(s, ni, 8 * dout, rd, tp, rd, nullptr, ctx.dops.d2d_f2.get<double>(), 8 * dout, children,
                       8 * dout, nullptr, nullptr, true);
    } else {
      ++ctx.n_launch;
      if (T.dn_lists)
        translate_down(s, ni, dout, dout, dc, dout, T.int_idx.get<int>() + T.int_off[d], ctx.dops.d2d.get<double>(),
                       children, dn);
      else
        translate_gemm(s, ni, 8 * dout, dout, dc, dout, T.int_idx.get<int>() + T.int_off[d],
                       ctx.dops.d2d.get<double>(), 8 * dout, children, 8 * dout, nullptr, nullptr, true);
    }
  }
  ev(8);
  // ---- D2T equivalent densities, then the fused near field
  double* pot = ctx.pot.as<double>(std::max(T.n_trg, 1L) * k1);
  if (T.n_tleaf > 0) {
    double* de = ctx.de_c.as<double>((size_t)T.n_tleaf * din);
    double* t1 = ctx.uc_c.as<double>((size_t)T.n_tleaf * rd);
    // (2^(-deg depth) DC[leaf] DC2DE0) DC2DE1, the check potentials gathered
    // from the leaves' rows of DC
    ctx.n_launch += 2;
    translate_gemm(s, T.n_tleaf, rd, dout, dc, dout, T.tleaf.get<int>(), ctx.dops.dc2de0.get<double>(), rd, t1, rd,
                   nullptr, keys, false, 1, nullptr, deg);
    translate_gemm(s, T.n_tleaf, din, rd, t1, rd, nullptr, ctx.dops.dc2de1.get<double>(), din, de, din, nullptr,
                   nullptr, false);
    ev(12);
    ++ctx.n_launch;
    near_field_kernel<Real, KerS2T><<<T.n_tleaf, kNF, 0, s>>>(
        T.tleaf.get<int>(), keys, T.trg_lo.get<int>(), T.trg_hi.get<int>(), slo, shi, T.p_off.get<int>(),
        T.p_list.get<int>(), T.w_off.get<int>(), T.w_list.get<int>(), pimg, wimg, T.tx.get<double>(),
        T.ty.get<double>(), T.tz.get<double>(), sx, sy, sz, den, ue32, T.src_counted ? de : nullptr, usurf, ns,
        ker_scale(KerS2T), has_sl ? 1 : 0, pot);
    if constexpr (KerDblS2T >= 0) {
      if (has_dl) {  // the double layer's P2P sources, added
        ++ctx.n_launch;
        near_field_kernel<Real, KerDblS2T, true><<<T.n_tleaf, kNF, 0, s>>>(
            T.tleaf.get<int>(), keys, T.trg_lo.get<int>(), T.trg_hi.get<int>(), slo, shi, T.p_off.get<int>(),
            T.p_list.get<int>(), T.w_off.get<int>(), T.w_list.get<int>(), pimg, wimg, T.tx.get<double>(),
            T.ty.get<double>(), T.tz.get<double>(), sx, sy, sz, surf, nullptr, nullptr, usurf, ns,
            ker_scale(KerDblS2T), 1, pot);
      }
    }
  } else {
    ev(12);
  }
  // periodic lattice sum of a kernel with a volume potential: the potential
  // of the mean density is taken out (PostProcessing, fmm_pts.txx:5741-5771)
  if (ctx.periodic && ctx.periodic_axes == 7 && ctx.bc_lattice && T.src_counted && T.n_trg > 0 &&
      (ctx.kernel == kLaplacePot || ctx.kernel == kStokesVel)) {
    ++ctx.n_launch;
    periodic_mean_correction<<<592, 256, 0, s>>>(T.n_trg, T.trg_leaf.get<int>(), keys, T.tx.get<double>(),
                                                 T.ty.get<double>(), T.tz.get<double>(), ue, ns, kin, k1, pot);
  }
  ev(9);
  // ---- output in input order, scaled by scale_x^trg_scal
  ++ctx.n_launch;
  if (out_float)
    unsort_values<float><<<ceil_div(T.n_trg, 256), 256, 0, s>>>(pot, T.trg_perm.get<int>(), T.n_trg, k1, ts,
                                                                (float*)out);
  else
    unsort_values<double><<<ceil_div(T.n_trg, 256), 256, 0, s>>>(pot, T.trg_perm.get<int>(), T.n_trg, k1, ts,
                                                                 (double*)out);
  ev(10);
  PVFMM_CUDA_CHECK(cudaGetLastError());
}

}  // namespace

// Exponents of the operators per frequency: fscale[f] = 2^(E - 14) with every
// |re|, |im| of frequency f below 2^E, so that the fragments stay below 2^14.
// (upload_vop_fragments then moves the largest of them to the parents' scales.)
__global__ void __launch_bounds__(256) vop_scale_kernel(int n, const float2* __restrict__ vop,
                                                        float* __restrict__ fscale) {
  __shared__ float part[256];
  float top = 0;
  for (int i = threadIdx.x; i < n; i += 256) {
    const float2 v = vop[(long)blockIdx.x * n + i];
    top = fmaxf(top, fmaxf(fabsf(v.x), fabsf(v.y)));
  }
  part[threadIdx.x] = top;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 256; ++i) top = fmaxf(top, part[i]);
    int e = 14;
    if (top > 0) frexpf(top, &e);
    fscale[blockIdx.x] = ldexpf(1.f, e - 14);
  }
}

// B fragments of hadamard_tc_kernel and hadamard_tc3_kernel: for frequency f,
// offset o, output group z (KOC components), block (k-step u, n-tile nt) and
// lane (g, t), the operator entries of the input elements e = 8u + 2t (b0) and
// e + 1 (b1), e = j2 * ki + i, onto column 8 nt + g (output element
// e_out = 4 nt + g / 2 = j1 * KOC + c, component z KOC + c, re|im = g % 2):
// b0 = (B[(e, re)], B[(e, im)]) with B[(e, re)][(e_out, re)] = Re M,
// B[(e, im)][(e_out, re)] = -Im M, B[(e, re)][(e_out, im)] = Im M,
// B[(e, im)][(e_out, im)] = Re M; divided by fscale[f] and stored as
// [f][o][z][block][lane] uint4 = (b0 hi, b1 hi, b0 lo, b1 lo).  Built on the
// device from the FP32 operator blocks vop[f][o][j1][j2][i][c].
__global__ void vop_fragments_kernel(long n, int ki, int ko, int koc, const float2* __restrict__ vop,
                                     const float* __restrict__ fscale, uint4* __restrict__ frag) {
  const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const int nnt = 2 * koc, nb = ki * nnt, ngroups = ko / koc;
  const int lane = (int)(idx % 32);
  const int blk = (int)(idx / 32 % nb);
  const int z = (int)(idx / 32 / nb % ngroups);
  const long fo = idx / 32 / nb / ngroups;  // f * 26 + o
  const int u = blk / nnt, nt = blk % nnt;
  const int g = lane >> 2, t = lane & 3;
  const int e_out = 4 * nt + g / 2, pout = g & 1;
  const int j1 = e_out / koc, c = z * koc + e_out % koc;
  const float inv = 1.f / fscale[fo / 26];  // a power of two
  unsigned hi[2], lo[2];
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const int e = 8 * u + 2 * t + w, j2 = e / ki, i = e % ki;
    const float2 mv = vop[(((fo * 8 + j1) * 8 + j2) * ki + i) * ko + c];
    half_split((pout == 0 ? mv.x : mv.y) * inv, (pout == 0 ? -mv.y : mv.x) * inv, hi[w], lo[w]);
  }
  frag[idx] = make_uint4(hi[0], hi[1], lo[0], lo[1]);
}

// B fragments of hadamard_dmma3_kernel: for frequency f, offset o, output
// group z, block (k-step s, n-tile nt) and lane (g, t): b = B[k][n] with
// k = double 12t + s of the input row (element e_in = k / 2 = j2 * 3 + i,
// re|im = k % 2) and n = 8 nt + g (element e_out = n / 2 = j1 * KOC + c,
// re|im = g % 2); stored as [f][o][z][block][lane] doubles.  Built on the
// device from the FP64 operator blocks.
__global__ void vop_dmma3_fragments_kernel(long n, int ko, int koc, const double2* __restrict__ vop,
                                           double* __restrict__ frag) {
  const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const int nnt = 2 * koc, nb = 12 * nnt, ngroups = ko / koc;
  const int lane = (int)(idx % 32);
  const int blk = (int)(idx / 32 % nb);
  const int z = (int)(idx / 32 / nb % ngroups);
  const long fo = idx / 32 / nb / ngroups;  // f * 26 + o
  const int sk = blk / nnt, nt = blk % nnt;
  const int g = lane >> 2, t = lane & 3;
  const int k = 12 * t + sk, e_in = k / 2, pin = k % 2;
  const int e_out = 4 * nt + g / 2, pout = g & 1;
  const int j2 = e_in / 3, i = e_in % 3, j1 = e_out / koc, c = z * koc + e_out % koc;
  const double2 mv = vop[((fo * 8 + j1) * 8 + j2) * 3 * ko + i * ko + c];
  // real form of the complex product: [re; im] of the input times
  // [[Re, Im], [-Im, Re]] gives [re; im] of the output
  frag[idx] = pin == 0 ? (pout == 0 ? mv.x : mv.y) : (pout == 0 ? -mv.y : mv.x);
}

// B fragments of hadamard_dmma1_kernel: for frequency f, offset o, block
// (k-step s, n-tile nt) and lane (g, t): b = B[k][n] with k = (child
// t + 4 (s/2), re|im s % 2) and n = 8 nt + g (child 4 nt + g/2, re|im g % 2);
// stored as [f][o][s][nt][lane] doubles.
__global__ void vop_dmma1_fragments_kernel(long n, const double2* __restrict__ vop, double* __restrict__ frag) {
  const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const int lane = (int)(idx % 32), nt = (int)(idx / 32 % 2), sk = (int)(idx / 64 % 4);
  const long fo = idx / 256;  // f * 26 + o
  const int g = lane >> 2, t = lane & 3;
  const int j2 = t + 4 * (sk >> 1), pin = sk & 1, j1 = 4 * nt + g / 2, pout = g & 1;
  const double2 mv = vop[(fo * 8 + j1) * 8 + j2];
  frag[idx] = pin == 0 ? (pout == 0 ? mv.x : mv.y) : (pout == 0 ? -mv.y : mv.x);
}

static void upload_vop_dmma1_fragments(Context& ctx) {
  const int m = ctx.m, n3h = 4 * m * m * (m + 1);
  const long n = (long)n3h * 26 * 8 * 32;
  double* dev = ctx.dops.vop_frag.as<double>(n);
  ++ctx.n_launch;
  vop_dmma1_fragments_kernel<<<ceil_div(n, 256L), 256, 0, ctx.stream>>>(n, ctx.dops.vop.get<double2>(), dev);
  PVFMM_CUDA_CHECK(cudaGetLastError());
  PVFMM_CUDA_CHECK(cudaStreamSynchronize(ctx.stream));
}

static void upload_vop_dmma3_fragments(Context& ctx) {
  const HostOperators& h = ctx.hops;
  const int m = ctx.m, n3h = 4 * m * m * (m + 1);
  const int ko = h.kout, koc = ko == 1 ? 1 : 3;
  const long n = (long)n3h * 26 * (ko / koc) * (24 * koc) * 32;
  double* dev = ctx.dops.vop_frag.as<double>(n);
  ++ctx.n_launch;
  vop_dmma3_fragments_kernel<<<ceil_div(n, 256L), 256, 0, ctx.stream>>>(n, ko, koc, ctx.dops.vop.get<double2>(),
                                                                         dev);
  PVFMM_CUDA_CHECK(cudaGetLastError());
  PVFMM_CUDA_CHECK(cudaStreamSynchronize(ctx.stream));
}

static void upload_vop_fragments(Context& ctx) {
  const HostOperators& h = ctx.hops;
  const int m = ctx.m, n3h = 4 * m * m * (m + 1);
  const int ki = h.kin, ko = h.kout, koc = ko == 1 ? 1 : 3;
  const long n = (long)n3h * 26 * (ko / koc) * (ki * 2 * koc) * 32;
  uint4* dev = ctx.dops.vop_frag.as<uint4>(n);
  float* fs = ctx.dops.vop_fscale.as<float>(n3h);
  ctx.n_launch += 2;
  vop_scale_kernel<<<n3h, 256, 0, ctx.stream>>>(26 * 64 * ki * ko, ctx.dops.vop.get<float2>(), fs);
  vop_fragments_kernel<<<ceil_div(n, 256L), 256, 0, ctx.stream>>>(n, ki, ko, koc, ctx.dops.vop.get<float2>(), fs, dev);
  PVFMM_CUDA_CHECK(cudaGetLastError());
  // The largest scale 2^vop_exp goes to the source parents (vsrc_scale_kernel):
  // the Hadamards' sums before fscale[f] <= 1 then stay within the bound of the
  // largest output spectra.  Summed in units of the scaled operators they left
  // the FP32 range at densities 2^18 to 2^20 smaller (about 1e31).  -23 keeps the
  // smallest parent scale, 2^(-126 + vop_exp), representable.
  std::vector<float> hfs(n3h);
  PVFMM_CUDA_CHECK(cudaMemcpyAsync(hfs.data(), fs, n3h * sizeof(float), cudaMemcpyDeviceToHost, ctx.stream));
  PVFMM_CUDA_CHECK(cudaStreamSynchronize(ctx.stream));
  std::frexp(*std::max_element(hfs.begin(), hfs.end()), &ctx.vop_exp);
  ctx.vop_exp = std::max(ctx.vop_exp - 1, -23);
  for (float& v : hfs) v = std::ldexp(v, -ctx.vop_exp);
  PVFMM_CUDA_CHECK(cudaMemcpyAsync(fs, hfs.data(), n3h * sizeof(float), cudaMemcpyHostToDevice, ctx.stream));
  PVFMM_CUDA_CHECK(cudaStreamSynchronize(ctx.stream));
}

// Check -> equivalent factors C2E0 (rows x r) and C2E1 (r x cols) without the
// directions the cutoff dropped: a zero column of C2E0 multiplies its row of
// C2E1 by zero, so the product is unchanged when both are left out.  The
// directions listed in `first` come first (padded to an even count with a
// zero direction, *n_first), then the other kept ones; the inner width *rc is
// padded to even as well (the translation products take 16-byte rows).
void compact_factors(const std::vector<double>& c0, const std::vector<double>& c1, int rows, int r, int cols,
                     const std::vector<int>& first, std::vector<double>& o0, std::vector<double>& o1, int* rc,
                     int* n_first, std::vector<int>* order_out = nullptr) {
  std::vector<int> order(first);
  if (order.size() & 1) order.push_back(-1);
  *n_first = (int)order.size();
  std::vector<char> taken(r, 0);
  for (int j : first) taken[j] = 1;
  for (int j = 0; j < r; ++j) {
    if (taken[j]) continue;
    bool kept = false;
    for (int i = 0; i < rows && !kept; ++i) kept = c0[(size_t)i * r + j] != 0.0;
    if (kept) order.push_back(j);
  }
  if (order.size() & 1) order.push_back(-1);
  if (order.empty()) order.assign(2, -1);
  const int n = (int)order.size();
  *rc = n;
  o0.assign((size_t)rows * n, 0.0);
  o1.assign((size_t)n * cols, 0.0);
  for (int k = 0; k < n; ++k) {
    const int j = order[k];
    if (j < 0) continue;
    for (int i = 0; i < rows; ++i) o0[(size_t)i * n + k] = c0[(size_t)i * r + j];
    std::copy(c1.begin() + (size_t)j * cols, c1.begin() + (size_t)(j + 1) * cols, o1.begin() + (size_t)k * cols);
  }
  if (order_out) *order_out = std::move(order);
}

void upload_operators(Context& ctx) {
  const HostOperators& h = ctx.hops;
  auto s = ctx.stream;
  {
    const int din = h.ns * h.kin, dout = h.ns * h.kout, rk = std::min(din, dout);
    const bool proj32 = ctx.precision == 1 && ctx.ki.ke == 3;
    std::vector<double> a0, a1, b0, b1;
    int nf = 0;
    compact_factors(h.uc2ue0, h.uc2ue1, dout, rk, din, proj32 ? h.ue32_dirs : std::vector<int>(), a0, a1, &ctx.ru,
                    &ctx.r32);
    std::vector<int> dorder;
    compact_factors(h.dc2de0, h.dc2de1, dout, rk, din, std::vector<int>(), b0, b1, &ctx.rd, &nf, &dorder);
    upload_vec<double>(ctx.dops.uc2ue0, a0, s);
    upload_vec<double>(ctx.dops.uc2ue1, a1, s);
    upload_vec<double>(ctx.dops.dc2de0, b0, s);
    upload_vec<double>(ctx.dops.dc2de1, b1, s);
    // D2D = DC2DE0 (DC2DE1 M_pe2c): through the rd kept downward directions
    // the two products take 2 rd dout (1 + 8) flops per parent against
    // 16 dout^2 for the formed operator (mixed Stokes form: rd = 520 of
    // 1464); taken when that saves a quarter of the flops, since the split
    // adds a launch and an intermediate per level
    ctx.d2d_factored = !h.d2d_f2.empty() && 3L * ctx.rd < 2L * dout;
    if (ctx.d2d_factored) {
      std::vector<double> f2((size_t)ctx.rd * 8 * dout, 0.0);
      for (int k = 0; k < ctx.rd; ++k)
        if (dorder[k] >= 0)
          std::copy(h.d2d_f2.begin() + (size_t)dorder[k] * 8 * dout,
                    h.d2d_f2.begin() + (size_t)(dorder[k] + 1) * 8 * dout, f2.begin() + (size_t)k * 8 * dout);
      upload_vec<double>(ctx.dops.d2d_f2, f2, s);
    }
    if (proj32) {
      // U_k (din x r32): the transpose of the first r32 rows of the compacted
      // UC2UE1, so that ue U_k U_k^T is the projection onto those directions
      std::vector<double> ub((size_t)din * std::max(ctx.r32, 1), 0.0);
      for (int k = 0; k < ctx.r32; ++k)
        for (int a = 0; a < din; ++a) ub[(size_t)a * ctx.r32 + k] = a1[(size_t)k * din + a];
      upload_vec<double>(ctx.dops.ue_basis, ub, s);
    }
    PVFMM_CUDA_CHECK(cudaStreamSynchronize(s));  // the host vectors go out of scope
  }
  upload_vec<double>(ctx.dops.u2u, h.u2u, s);
  upload_vec<double>(ctx.dops.d2d, h.d2d, s);
  upload_vec<double>(ctx.dops.usurf, h.usurf, s);
  if (ctx.precision == 0) upload_vec<double>(ctx.dops.vop, h.vop, s);
  else upload_vec<float>(ctx.dops.vop, h.vop, s);
  if (ctx.precision == 1 && ctx.ki.ke == 1) {
    std::vector<float> lay;
    hadamard_tc5_operator_layout(h.vop, 4 * ctx.m * ctx.m * (ctx.m + 1), lay);
    float* dev = ctx.dops.vop_tc5.as<float>(lay.size());
    PVFMM_CUDA_CHECK(cudaMemcpyAsync(dev, lay.data(), lay.size() * sizeof(float), cudaMemcpyHostToDevice, s));
    PVFMM_CUDA_CHECK(cudaStreamSynchronize(s));
    if (!ctx.tc5_err_host) PVFMM_CUDA_CHECK(cudaMallocHost((void**)&ctx.tc5_err_host, sizeof(int)));
    *ctx.tc5_err_host = 0;
  }
  int* fm = ctx.dops.fft_map.as<int>(h.fft_map.size());
  int* im = ctx.dops.ifft_map.as<int>(h.ifft_map.size());
  PVFMM_CUDA_CHECK(cudaMemcpyAsync(fm, h.fft_map.data(), h.fft_map.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  PVFMM_CUDA_CHECK(cudaMemcpyAsync(im, h.ifft_map.data(), h.ifft_map.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  PVFMM_CUDA_CHECK(cudaStreamSynchronize(s));
  if (ctx.precision == 1) upload_vop_fragments(ctx);  // from the uploaded FP32 vop
  if (ctx.precision == 0 && ctx.ki.ke == 3) upload_vop_dmma3_fragments(ctx);  // from the uploaded FP64 vop
  if (ctx.precision == 0 && ctx.ki.ke == 1) upload_vop_dmma1_fragments(ctx);
}

void evaluate(Context& ctx, const void* den_in, const void* dl_in, bool den_float, void* out, bool out_float) {
  const bool f32 = ctx.precision == 1;
  switch (ctx.kernel) {
    case kLaplacePot:
      if (f32) evaluate_impl<float, kKerLaplace, kKerLaplace>(ctx, den_in, dl_in, den_float, out, out_float);
      else evaluate_impl<double, kKerLaplace, kKerLaplace>(ctx, den_in, dl_in, den_float, out, out_float);
      break;
    case kLaplaceGrad:
      if (f32) evaluate_impl<float, kKerLaplaceGrad, kKerLaplace>(ctx, den_in, dl_in, den_float, out, out_float);
      else evaluate_impl<double, kKerLaplaceGrad, kKerLaplace>(ctx, den_in, dl_in, den_float, out, out_float);
      break;
    case kLaplacePotGrad:
      if (f32) evaluate_impl<float, kKerLaplacePG, kKerLaplace>(ctx, den_in, dl_in, den_float, out, out_float);
      else evaluate_impl<double, kKerLaplacePG, kKerLaplace>(ctx, den_in, dl_in, den_float, out, out_float);
      break;
    case kStokesVel:
      if (f32) evaluate_impl<float, kKerStokes, kKerStokes>(ctx, den_in, dl_in, den_float, out, out_float);
      else evaluate_impl<double, kKerStokes, kKerStokes>(ctx, den_in, dl_in, den_float, out, out_float);
      break;
    // the kernels that expand themselves (kernel.txx:894-901)
    case kStokesPress:
      if (f32) evaluate_impl<float, kKerStokesPress, kKerStokesPress>(ctx, den_in, dl_in, den_float, out, out_float);
      else evaluate_impl<double, kKerStokesPress, kKerStokesPress>(ctx, den_in, dl_in, den_float, out, out_float);
      break;
    case kStokesVelGrad:
      if (f32) evaluate_impl<float, kKerStokesGrad, kKerStokesGrad>(ctx, den_in, dl_in, den_float, out, out_float);
      else evaluate_impl<double, kKerStokesGrad, kKerStokesGrad>(ctx, den_in, dl_in, den_float, out, out_float);
      break;
    case kBiotSavart:
      if (f32) evaluate_impl<float, kKerBiotSavart, kKerBiotSavart>(ctx, den_in, dl_in, den_float, out, out_float);
      else evaluate_impl<double, kKerBiotSavart, kKerBiotSavart>(ctx, den_in, dl_in, den_float, out, out_float);
      break;
    default:
      throw std::runtime_error("unsupported kernel");
  }
}

}  // namespace pvfmm_b200

namespace {
template <class Real, int M>
void dft_local_bytes(int* up, int* dn) {
  using namespace pvfmm_b200;
  cudaFuncAttributes a{};
  PVFMM_CUDA_CHECK(cudaFuncGetAttributes(&a, fft_up_kernel<Real, M>));
  *up = (int)a.localSizeBytes;
  PVFMM_CUDA_CHECK(cudaFuncGetAttributes(&a, ifft_dn_kernel<Real, M, false>));
  *dn = (int)a.localSizeBytes;
  if constexpr (FftSizes<Real, M>::kRows) {
    PVFMM_CUDA_CHECK(cudaFuncGetAttributes(&a, ifft_dn_kernel<Real, M, true>));
    *dn = std::max(*dn, (int)a.localSizeBytes);
  }
}
}  // namespace

// Local memory per thread of the V-list DFT kernels of a form (0 plain, 1
// mixed) and order, forward and inverse: what of a line did not fit the
// registers (internal entry point used by the GPU tests; no counterpart in the
// reference).  Returns 0 on success.
extern "C" int PVFMMB200DftLocalBytes(int precision, int m, int* up, int* dn) {
  using pvfmm_b200::set_last_error;
  try {
    auto get = [&](auto order) {
      constexpr int M = decltype(order)::value;
      if (precision == 0) dft_local_bytes<double, M>(up, dn);
      else dft_local_bytes<float, M>(up, dn);
    };
    switch (m) {
      case 2: get(std::integral_constant<int, 2>()); break;
      case 4: get(std::integral_constant<int, 4>()); break;
      case 6: get(std::integral_constant<int, 6>()); break;
      case 8: get(std::integral_constant<int, 8>()); break;
      case 10: get(std::integral_constant<int, 10>()); break;
      case 12: get(std::integral_constant<int, 12>()); break;
      case 14: get(std::integral_constant<int, 14>()); break;
      case 16: get(std::integral_constant<int, 16>()); break;
      default: throw std::runtime_error("unsupported multipole order");
    }
    set_last_error("");
    return 0;
  } catch (const std::exception& e) {
    set_last_error(e.what());
    return 1;
  }
}
