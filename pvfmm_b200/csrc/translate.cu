// FP64 translation products of the FMM on the FP64 tensor cores
// (mma.sync m8n8k4 .f64, the only FP64 MMA of sm_100): the check ->
// equivalent pseudo-inverse products of S2U and D2T, U2U and D2D
// (reference: the per-interaction-block GEMMs of FMM_Pts::EvalList,
// include/fmm_pts.txx:2017-2271, and the surface GEMMs of EvalListPts,
// :4246-4302 and :4390-4426).
//
// Every translation here has the same shape: a tall matrix of node rows
// (one row = the ns*ke values of one node's surface) times one small operator
// shared by all rows,
//   C[crow(i)][:] (+)= s(i) * A[arow(i)][:] * B,
// where the rows of A may be gathered through an index list (the nodes of a
// level, the target leaves), the rows of C may be scattered through one, and
// s(i) is 1 or the level factor 2^-depth of the node.  B (at most
// 8*ns*ke x ns*ke) stays in L2 across the whole launch; the rows of A are
// read once per column tile.
//
// Tiling: a block computes a 128 x 64 tile of C with 8 warps (4 x 2), each
// warp a 32 x 32 tile = 4 x 4 MMA tiles of 8 x 8, FP64 accumulators in
// registers (each A and B fragment feeds four MMAs); few rows take 32 x 64
// tiles (2 x 4 warps of 16 x 16).  Every sum runs over k in order, whatever
// the tile, so the choice changes no value.
// K advances in steps of 16; the A and B tiles of the next steps are copied
// into shared memory with 16-byte cp.async behind the current step's first
// MMAs, one barrier per step (4M clustered points, D2T products: 1.37 ms,
// against 1.41 with a second barrier and the copies issued first, and 1.41
// with three steps in shared memory).
// Row lengths are even (ns = 6(m-1)^2+2), so every row of A, B and C starts
// on a 16-byte boundary.
#include <algorithm>

#include "fmm_context.cuh"

namespace pvfmm_b200 {
namespace {

constexpr int kBN = 64, kBK = 16;
constexpr int kAStride = kBK + 4;  // doubles per A row in shared memory
constexpr int kBStride = kBN + 4;  // doubles per B row in shared memory (B fragment loads conflict-free)
constexpr int kThreadsG = 256;

// A block tile of BM x 64: 8 warps in WM x (8 / WM), each MI x NJ MMA tiles of
// 8 x 8; STAGES K-steps in shared memory.
template <int BM_, int WM_, int STAGES_>
struct GemmTile {
  static constexpr int BM = BM_, WM = WM_, WN = 8 / WM_, STAGES = STAGES_;
  static constexpr int MI = BM / WM / 8, NJ = kBN / WN / 8;
  static constexpr int smem =
      (int)sizeof(double) * STAGES * (BM * kAStride + kBK * kBStride) + (int)sizeof(long) * BM;
};
using LargeTile = GemmTile<128, 4, 2>;
using SmallTile = GemmTile<32, 2, 4>;

__device__ __forceinline__ void cp16(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(valid ? 16 : 0));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}


struct RowMap {
  const int* rows;  // nullptr: identity
  __device__ __forceinline__ long operator()(long i) const { return rows ? (long)rows[i] : i; }
};

// Over parents and children (kUp, kDown; see ChildRows): blockIdx.z is the
// child octant, the rows are the listed parents' indices k.
// kUp: A's rows are the parents' blocks of 8 child rows, of which octant z is
// the K range [z kchunk, (z + 1) kchunk); kDown: B's and C's columns
// [z N, (z + 1) N).
enum GemmMode { kPlainRows, kUp, kDown };

template <class Tile, GemmMode Mode>
__global__ void __launch_bounds__(kThreadsG, 2)
    translate_gemm_kernel(int M, int N, int K, const double* __restrict__ A, long lda, const int* __restrict__ arows,
                          const double* __restrict__ B, long ldb, double* __restrict__ C, long ldc,
                          const int* __restrict__ crows, const MKey* __restrict__ keys, int deg, int accumulate,
                          long m_base, int kchunk, double* __restrict__ partial, ChildRows lists) {
  constexpr int BM = Tile::BM, MI = Tile::MI, NJ = Tile::NJ, STAGES = Tile::STAGES;
  extern __shared__ __align__(16) double tsm[];
  double(*As)[BM * kAStride] = reinterpret_cast<double(*)[BM * kAStride]>(tsm);
  double(*Bs)[kBK * kBStride] = reinterpret_cast<double(*)[kBK * kBStride]>(tsm + STAGES * BM * kAStride);
  long* arow_s = reinterpret_cast<long*>(tsm + STAGES * (BM * kAStride + kBK * kBStride));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int wm = warp / Tile::WN, wn = warp % Tile::WN;  // warp tile (8 MI rows) x (8 NJ cols)
  const long m0 = m_base + (long)blockIdx.y * BM;
  const int n0 = blockIdx.x * kBN;
  const RowMap amap{arows};
  const int* listed = Mode == kPlainRows ? nullptr : lists.rows + blockIdx.z * lists.stride;
  const int rows = Mode == kPlainRows ? M : lists.counts[blockIdx.z];
  if (Mode != kPlainRows && m0 >= rows) return;
  if (Mode == kDown) {
    B += (long)blockIdx.z * N;
    C += (long)blockIdx.z * N;
  }
  // split K: this block sums k in [kbeg, kend) (the whole of K without a split)
  const int kbeg = Mode == kDown ? 0 : blockIdx.z * kchunk, kend = min(K, kbeg + kchunk);
  if (tid < BM) arow_s[tid] = m0 + tid < rows ? amap(listed ? listed[m0 + tid] : m0 + tid) : -1;
  __syncthreads();
  // copy plan: A tile BM rows x 16 doubles in 16-byte chunks, B tile 16 rows x
  // 64 doubles = 512 chunks, 2 per thread.  One group per K-step (empty past
  // the last one).
  const int nk = (kend - kbeg + kBK - 1) / kBK;
  auto issue = [&](int ks) {
    const int k0 = kbeg + ks * kBK, buf = ks % STAGES;
    if (ks < nk) {
#pragma unroll
      for (int u = 0; u < BM * 8 / kThreadsG; ++u) {
        const int c = tid + u * kThreadsG;
        const int r = c >> 3, kc = (c & 7) * 2;  // row, first double of the chunk
        const long ar = arow_s[r];
        const bool v = ar >= 0 && k0 + kc < kend;
        const double* src = v ? A + ar * lda + k0 + kc : A;
        cp16(&As[buf][r * kAStride + kc], src, v);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c = tid + u * kThreadsG;
        const int r = c >> 5, nc = (c & 31) * 2;
        const bool v = k0 + r < kend && n0 + nc < N;
        const double* src = v ? B + (long)(k0 + r) * ldb + n0 + nc : B;
        cp16(&Bs[buf][r * kBStride + nc], src, v);
      }
    }
    cp_commit();
  };
  double acc[MI][NJ][2];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
  for (int ks = 0; ks < STAGES - 1; ++ks) issue(ks);
  for (int ks = 0; ks < nk; ++ks) {
    cp_wait<STAGES - 2>();  // this thread's copies of step ks have landed
    __syncthreads();        // everyone's have; everyone is done with step ks - 1, whose buffer is refilled
    const double* as = As[ks % STAGES] + (wm * 8 * MI) * kAStride;
    const double* bs = Bs[ks % STAGES] + wn * 8 * NJ;
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 4) {
      double a[MI], b[NJ];
#pragma unroll
      for (int i = 0; i < MI; ++i) a[i] = as[(i * 8 + g) * kAStride + kk + t];
#pragma unroll
      for (int j = 0; j < NJ; ++j) b[j] = bs[(kk + t) * kBStride + j * 8 + g];
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) dmma(acc[i][j], a[i], b[j]);
      if (kk == 0) issue(ks + STAGES - 1);  // behind the step's first MMAs
    }
  }
  // epilogue: rows g (+8i), columns 2t, 2t+1 of each 8x8 tile
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const long mi = m0 + wm * 8 * MI + i * 8 + g;
    if (mi >= rows) continue;
    const long out_row = listed ? listed[mi] : mi;
    if (partial) {  // split K: plain partial sums, reduced by translate_reduce
      double* prow = partial + ((long)blockIdx.z * M + out_row) * N;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int n = n0 + wn * 8 * NJ + j * 8 + 2 * t;
        if (n < N) *reinterpret_cast<double2*>(prow + n) = make_double2(acc[i][j][0], acc[i][j][1]);
      }
      continue;
    }
    double s = 1.0;
    if (keys) s = ldexp(1.0, -deg * (int)(keys[arow_s[mi - m0]].lo & 31u));
    const long cr = crows ? (long)crows[out_row] : out_row;
    double* crow = C + cr * ldc;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int n = n0 + wn * 8 * NJ + j * 8 + 2 * t;
      if (n >= N) continue;  // N is even: n < N implies n + 1 < N
      double2 v = make_double2(acc[i][j][0] * s, acc[i][j][1] * s);
      double2* p = reinterpret_cast<double2*>(crow + n);
      if (accumulate) {
        const double2 o = *p;
        v.x += o.x;
        v.y += o.y;
      }
      *p = v;
    }
  }
}

// C[crow(i)][n] (+)= s(i) * sum_z partial[z][i][n], the K pieces added in order.
__global__ void translate_reduce(long M, int N, int ksplit, const double* __restrict__ partial,
                                 const int* __restrict__ arows, const int* __restrict__ crows,
                                 const MKey* __restrict__ keys, int deg, int accumulate, double* __restrict__ C,
                                 long ldc, const unsigned char* __restrict__ mask) {
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e >= M * N) return;
  const long i = e / N;
  const int n = (int)(e % N);
  double v = 0;
  const unsigned m = mask ? mask[i] : ~0u;  // (the pieces of a child without a row were not formed)
  for (int z = 0; z < ksplit; ++z)
    if (m >> z & 1u) v += partial[((long)z * M + i) * N + n];
  if (keys) v *= ldexp(1.0, -deg * (int)(keys[arows ? arows[i] : i].lo & 31u));
  double* c = C + (crows ? (long)crows[i] : i) * ldc + n;
  *c = accumulate ? *c + v : v;
}

}  // namespace

// Rows per block tile: 128, or 32 when the 128-row tiles would not fill the
// two blocks that an SM holds; a product of few rows lasts as long as one tile,
// most of whose rows are padding on the coarse levels.  With the 32-row tiles
// up to 296 blocks (against none, and up to 148): 2k Laplace points U2U 0.089
// -> 0.052 ms and D2D 0.085 -> 0.040; 200k Stokes-gradient points U2U 0.38 ->
// 0.23 (0.25) and D2D 1.22 -> 0.60 (0.80).
constexpr long kSmallTileBlocks = 296;
template <GemmMode Mode>
static void launch_gemm(cudaStream_t s, long M, int N, int K, const double* A, long lda, const int* arows,
                        const double* B, long ldb, double* C, long ldc, const int* crows, const MKey* scale_keys,
                        bool accumulate, int nz, int kchunk, double* partial, int deg, const ChildRows& lists) {
  if ((N & 1) || (K & 1) || (kchunk & 1) || (lda & 1) || (ldb & 1) || (ldc & 1))
    throw std::runtime_error("translate_gemm: row lengths must be even (16-byte rows)");
  if (M >= (1L << 31)) throw std::runtime_error("translate_gemm: too many rows");
  const long cols = (N + kBN - 1) / kBN;
  auto run = [&](auto kernel, int bm, int smem) {
    PVFMM_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    // the column tiles of one row tile are consecutive blocks (they share the
    // A rows in L2); row tiles in launches of at most 65535
    const long tiles = (M + bm - 1) / bm;
    for (long t0 = 0; t0 < tiles; t0 += 65535) {
      dim3 grid((unsigned)cols, (unsigned)std::min(65535L, tiles - t0), (unsigned)nz);
      kernel<<<grid, kThreadsG, smem, s>>>((int)M, N, K, A, lda, arows, B, ldb, C, ldc, crows, scale_keys, deg,
                                           accumulate ? 1 : 0, t0 * bm, kchunk, partial, lists);
      PVFMM_CUDA_CHECK(cudaGetLastError());
    }
  };
  if ((M + LargeTile::BM - 1) / LargeTile::BM * cols * nz <= kSmallTileBlocks)
    run(translate_gemm_kernel<SmallTile, Mode>, SmallTile::BM, SmallTile::smem);
  else
    run(translate_gemm_kernel<LargeTile, Mode>, LargeTile::BM, LargeTile::smem);
}

void translate_gemm(cudaStream_t s, long M, int N, int K, const double* A, long lda, const int* arows,
                    const double* B, long ldb, double* C, long ldc, const int* crows, const MKey* scale_keys,
                    bool accumulate, int ksplit, double* partial, int deg) {
  if (M <= 0 || N <= 0) return;
  if (ksplit < 1 || (ksplit > 1 && (!partial || K % ksplit != 0 || (K / ksplit) % 2 != 0)))
    throw std::runtime_error("translate_gemm: bad K split");
  launch_gemm<kPlainRows>(s, M, N, K, A, lda, arows, B, ldb, C, ldc, crows, scale_keys, accumulate, ksplit, K / ksplit,
                          ksplit > 1 ? partial : nullptr, deg, ChildRows{});
  if (ksplit > 1) {
    translate_reduce<<<(unsigned)((M * N + 255) / 256), 256, 0, s>>>(M, N, ksplit, partial, arows, crows, scale_keys,
                                                                     deg, accumulate ? 1 : 0, C, ldc, nullptr);
    PVFMM_CUDA_CHECK(cudaGetLastError());
  }
}

void translate_up(cudaStream_t s, long M, int din, const double* children, const double* B, double* C,
                  const int* crows, double* partial, const ChildRows& lists) {
  if (M <= 0) return;
  launch_gemm<kUp>(s, M, din, 8 * din, children, 8L * din, nullptr, B, din, C, din, nullptr, nullptr, false, 8, din,
                   partial, 1, lists);
  translate_reduce<<<(unsigned)((M * din + 255) / 256), 256, 0, s>>>(M, din, 8, partial, nullptr, crows, nullptr, 1, 0,
                                                                     C, din, lists.mask);
  PVFMM_CUDA_CHECK(cudaGetLastError());
}

void translate_down(cudaStream_t s, long M, int dout, int K, const double* A, long lda, const int* arows,
                    const double* B, double* children, const ChildRows& lists) {
  if (M <= 0) return;
  launch_gemm<kDown>(s, M, dout, K, A, lda, arows, B, 8L * dout, children, 8L * dout, nullptr, nullptr, true, 8, K,
                     nullptr, 1, lists);
}

bool translate_down_pays(long occupied, long all, int dout) {
  const double padded = (double)((dout + kBN - 1) / kBN * kBN) / dout;
  return occupied * padded < 0.85 * all;
}

}  // namespace pvfmm_b200

// Self-check of the FP64 translation product on random data (internal entry
// point used by the GPU tests; no counterpart in the reference): computes
// C[crow(i)] (+)= s(i) A[arow(i)] B on device copies of the host arrays (K
// split into `ksplit` pieces when > 1) and copies C back.  arows / crows /
// depth may be NULL.  Returns 0 on success.
extern "C" int PVFMMB200TranslateGemmCheck(long M, int N, int K, const double* A, long a_rows, const int* arows,
                                           const double* B, double* C, long c_rows, const int* crows,
                                           const int* depth_of_arow_target, int accumulate, int ksplit) {
  using namespace pvfmm_b200;
  void* buf = nullptr;
  try {
    const size_t nA = (size_t)a_rows * K, nB = (size_t)K * N, nC = (size_t)c_rows * N;
    const size_t nP = ksplit > 1 ? (size_t)ksplit * M * N : 0;
    const size_t bytes = (nA + nB + nC + nP) * 8 + (size_t)M * 4 * 2 + (size_t)a_rows * sizeof(MKey) + 256;
    PVFMM_CUDA_CHECK(cudaMalloc(&buf, bytes));
    double* dA = (double*)buf;
    double* dB = dA + nA;
    double* dC = dB + nB;
    double* dP = dC + nC;
    int* dar = (int*)(dP + nP);
    int* dcr = dar + M;
    MKey* dk = (MKey*)(((uintptr_t)(dcr + M) + 15) & ~(uintptr_t)15);
    PVFMM_CUDA_CHECK(cudaMemcpy(dA, A, nA * 8, cudaMemcpyHostToDevice));
    PVFMM_CUDA_CHECK(cudaMemcpy(dB, B, nB * 8, cudaMemcpyHostToDevice));
    PVFMM_CUDA_CHECK(cudaMemcpy(dC, C, nC * 8, cudaMemcpyHostToDevice));
    if (arows) PVFMM_CUDA_CHECK(cudaMemcpy(dar, arows, M * 4, cudaMemcpyHostToDevice));
    if (crows) PVFMM_CUDA_CHECK(cudaMemcpy(dcr, crows, M * 4, cudaMemcpyHostToDevice));
    if (depth_of_arow_target) {
      std::vector<MKey> k(a_rows);
      for (long i = 0; i < a_rows; ++i) k[i] = make_key(0, 0, 0, (unsigned)depth_of_arow_target[i]);
      PVFMM_CUDA_CHECK(cudaMemcpy(dk, k.data(), a_rows * sizeof(MKey), cudaMemcpyHostToDevice));
    }
    translate_gemm(nullptr, M, N, K, dA, K, arows ? dar : nullptr, dB, N, dC, N, crows ? dcr : nullptr,
                   depth_of_arow_target ? dk : nullptr, accumulate != 0, ksplit, dP);
    PVFMM_CUDA_CHECK(cudaMemcpy(C, dC, nC * 8, cudaMemcpyDeviceToHost));
    cudaFree(buf);
    set_last_error("");
    return 0;
  } catch (const std::exception& e) {
    if (buf) cudaFree(buf);
    set_last_error(e.what());
    return 1;
  }
}

// Self-check of the parent-child products (internal entry point used by the
// GPU tests; no counterpart in the reference): with the children of parent k
// in the bits of mask[k], up[k] = sum over those children z of children[8k + z]
// B_z (B: 8 dim x dim) and down[8k + z] += up_in[k] D_z (D: dim x 8 dim), on
// device copies of the host arrays.  Returns 0 on success.
extern "C" int PVFMMB200ChildProductsCheck(long M, int dim, const unsigned char* mask, const double* children,
                                           const double* B, double* up, const double* up_in, const double* D,
                                           double* down) {
  using namespace pvfmm_b200;
  DevBuf b[8];
  try {
    std::vector<int> rows(8 * M, -1), counts(8, 0);
    for (long k = 0; k < M; ++k)
      for (int z = 0; z < 8; ++z)
        if (mask[k] >> z & 1) rows[z * M + counts[z]++] = (int)k;
    auto put = [&](DevBuf& d, const void* h, size_t bytes) {
      d.ensure(bytes);
      PVFMM_CUDA_CHECK(cudaMemcpy(d.ptr, h, bytes, cudaMemcpyHostToDevice));
    };
    const size_t n1 = (size_t)M * dim * 8, n8 = 8 * n1, nb = (size_t)64 * dim * dim;
    put(b[0], rows.data(), rows.size() * sizeof(int));
    put(b[1], counts.data(), 8 * sizeof(int));
    put(b[2], mask, M);
    put(b[3], children, n8);
    put(b[4], B, nb);
    put(b[5], up, n1);
    const ChildRows lists{b[0].get<int>(), b[1].get<int>(), M, b[2].get<unsigned char>()};
    translate_up(nullptr, M, dim, b[3].get<double>(), b[4].get<double>(), b[5].get<double>(), nullptr,
                 b[6].as<double>(n8 / 8), lists);
    PVFMM_CUDA_CHECK(cudaMemcpy(up, b[5].ptr, n1, cudaMemcpyDeviceToHost));
    put(b[5], up_in, n1);
    put(b[4], D, nb);
    put(b[7], down, n8);
    translate_down(nullptr, M, dim, dim, b[5].get<double>(), dim, nullptr, b[4].get<double>(), b[7].get<double>(),
                   lists);
    PVFMM_CUDA_CHECK(cudaMemcpy(down, b[7].ptr, n8, cudaMemcpyDeviceToHost));
    for (DevBuf& d : b) d.release();
    set_last_error("");
    return 0;
  } catch (const std::exception& e) {
    for (DevBuf& d : b) d.release();
    set_last_error(e.what());
    return 1;
  }
}
