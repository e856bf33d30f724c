// GPU octree construction for the particle FMM.
//
// Reproduces, on the device, the tree PVFMM builds on one rank:
//   * bounding-box map into [0,1)^3        src/pvfmm-wrapper.cpp:458-590
//   * Morton ids + stable sort              include/mortonid.txx:25-53,107-118,
//                                           include/parUtils.txx:527 (ties keep input order)
//   * refinement: a leaf splits while depth < MAX_DEPTH-1 and either the
//     context's seed grid (pvfmm-wrapper.cpp:416-432) or src+trg counts exceed
//     max_pts                               include/fmm_node.txx:63-98, mpi_tree.txx:403-492
//   * 2:1 balance as the closure of the internal-node set under
//     X -> parent(NbrList(X))              include/mpi_tree.txx:745-943
//   * colleagues                            include/mpi_tree.txx:1136-1256
//   * U/V/W/X lists with the Nsrf rule      include/interac_list.txx:98-279,
//                                           include/fmm_pts.txx:4629, 4929, 5295, 5325
// Each level is a Morton-sorted array; children of an internal node are the
// 8 consecutive nodes of the next level.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>

#include "fmm_context.cuh"

namespace pvfmm_b200 {
namespace {

constexpr int kThreads = 256;

// ------------------------------------------------------------------ bbox
template <class T>
__global__ void bbox_partial(const T* __restrict__ pos, long n, double* __restrict__ part) {
  __shared__ double smin[3][kThreads], smax[3][kThreads];
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    for (int d = 0; d < 3; ++d) {
      const double v = (double)pos[i * 3 + d];
      mn[d] = fmin(mn[d], v);
      mx[d] = fmax(mx[d], v);
    }
  for (int d = 0; d < 3; ++d) {
    smin[d][threadIdx.x] = mn[d];
    smax[d][threadIdx.x] = mx[d];
  }
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int d = 0; d < 3; ++d) {
        smin[d][threadIdx.x] = fmin(smin[d][threadIdx.x], smin[d][threadIdx.x + s]);
        smax[d][threadIdx.x] = fmax(smax[d][threadIdx.x], smax[d][threadIdx.x + s]);
      }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int d = 0; d < 3; ++d) {
      part[blockIdx.x * 6 + d] = smin[d][0];
      part[blockIdx.x * 6 + 3 + d] = smax[d][0];
    }
}

__global__ void bbox_final(const double* __restrict__ part, int nb, double* __restrict__ out) {
  __shared__ double smin[3][kThreads], smax[3][kThreads];
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
    for (int d = 0; d < 3; ++d) {
      mn[d] = fmin(mn[d], part[b * 6 + d]);
      mx[d] = fmax(mx[d], part[b * 6 + 3 + d]);
    }
  for (int d = 0; d < 3; ++d) {
    smin[d][threadIdx.x] = mn[d];
    smax[d][threadIdx.x] = mx[d];
  }
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st)
      for (int d = 0; d < 3; ++d) {
        smin[d][threadIdx.x] = fmin(smin[d][threadIdx.x], smin[d][threadIdx.x + st]);
        smax[d][threadIdx.x] = fmax(smax[d][threadIdx.x], smax[d][threadIdx.x + st]);
      }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int d = 0; d < 3; ++d) {
      out[d] = smin[d][0];
      out[3 + d] = smax[d][0];
    }
}

// ------------------------------------------------------------------ keys
// c = pos*scale + shift in the input precision, without fused multiply-add
// (pvfmm-wrapper.cpp:582-586), wrapped into [0,1); Morton coordinate
// floor(c*2^30) (mortonid.txx:39-53).  The reference wraps by adding or
// subtracting 1 until c lies in [0,1); every step but the last is exact, so
// c - floor(c) (one rounding, then 1 -> 0) is the same value and takes no
// loop for coordinates far outside a periodic box.
template <class T>
__device__ __forceinline__ T map_coord(T x, T s, T sh);
template <>
__device__ __forceinline__ double map_coord<double>(double x, double s, double sh) {
  double c = __dadd_rn(__dmul_rn(x, s), sh);
  if (!(c >= 0.0 && c < 1.0) && c == c) {
    c = __dadd_rn(c, -floor(c));
    if (c >= 1.0) c = __dadd_rn(c, -1.0);
  }
  return c;
}
template <>
__device__ __forceinline__ float map_coord<float>(float x, float s, float sh) {
  float c = __fadd_rn(__fmul_rn(x, s), sh);
  if (!(c >= 0.f && c < 1.f) && c == c) {
    c = __fadd_rn(c, -floorf(c));
    if (c >= 1.f) c = __fadd_rn(c, -1.f);
  }
  return c;
}

template <class T>
__global__ void map_and_key(const T* __restrict__ pos, long n, T scale, T sh0, T sh1, T sh2,
                            double* __restrict__ mapped, unsigned long long* __restrict__ hi,
                            unsigned int* __restrict__ lo, int* __restrict__ idx) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const T sh[3] = {sh0, sh1, sh2};
  unsigned int q[3];
  for (int d = 0; d < 3; ++d) {
    const T c = map_coord<T>(pos[i * 3 + d], scale, sh[d]);
    mapped[i * 3 + d] = (double)c;
    q[d] = (unsigned int)floor((double)c * (double)kTwo30);
  }
  const MKey k = make_key(q[0], q[1], q[2], kMaxDepth);
  hi[i] = k.hi;
  lo[i] = k.lo;
  idx[i] = (int)i;
}

__global__ void gather_u64(const unsigned long long* __restrict__ in, const int* __restrict__ perm, long n,
                           unsigned long long* __restrict__ out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[perm[i]];
}

__global__ void assemble_keys(const unsigned long long* __restrict__ hi, const unsigned int* __restrict__ lo_unsorted,
                              const int* __restrict__ perm, long n, MKey* __restrict__ keys) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  MKey k;
  k.hi = hi[i];
  k.lo = lo_unsorted[perm[i]];
  k.pad = 0;
  keys[i] = k;
}

// ------------------------------------------------------------------ refine
// sw: point sets the source positions stand for (1 per density passed)
__global__ void refine_level(const MKey* __restrict__ cur, long n_cur, int d, const MKey* __restrict__ sk, long n_s,
                             int sw, const MKey* __restrict__ tk, long n_t, const MKey* __restrict__ gk, long n_g,
                             long max_pts, int max_depth, int* __restrict__ split) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n_cur) return;
  unsigned int X, Y, Z, dd;
  decode_key(cur[i], X, Y, Z, dd);
  int s = 0;
  if (d < max_depth - 1) {
    const MKey b = cur[i], e = node_end_key(X, Y, Z, d);
    const long g = lower_bound_key(gk, n_g, e) - lower_bound_key(gk, n_g, b);
    long c = 0;
    if (sk) c += sw * (lower_bound_key(sk, n_s, e) - lower_bound_key(sk, n_s, b));
    c += lower_bound_key(tk, n_t, e) - lower_bound_key(tk, n_t, b);
    s = (g > max_pts || c > max_pts) ? 1 : 0;
  }
  split[i] = s;
}

__global__ void make_children(const MKey* __restrict__ cur, const int* __restrict__ flag, const int* __restrict__ offs,
                              long n_cur, int d, MKey* __restrict__ next, MKey* __restrict__ internal_out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n_cur || !flag[i]) return;
  const long k = offs[i];
  if (internal_out) internal_out[k] = cur[i];
  if (next) {
    unsigned int X, Y, Z, dd;
    decode_key(cur[i], X, Y, Z, dd);
    const unsigned int w = kTwo30 >> (d + 1);
    for (int c = 0; c < 8; ++c)
      next[k * 8 + c] = make_key(X + ((c & 1) ? w : 0), Y + ((c & 2) ? w : 0), Z + ((c & 4) ? w : 0), d + 1);
  }
}

// ------------------------------------------------------------------ balance
// For internal node X at level d: parents (level d-1) of its 3^3 neighbours
// clipped to the unit box; per axis these are parent(x) and the parent on the
// side of x within its parent.  Invalid candidates get the sentinel key.
// periodic: the mask of periodic axes (bit 0 x, bit 1 y, bit 2 z; 0 = free space)
__device__ __forceinline__ void parent_candidates(const MKey& key, int d, int periodic, MKey (&out)[8]) {
  unsigned int q[3], dd;
  decode_key(key, q[0], q[1], q[2], dd);
  const unsigned int w = kTwo30 >> d;
  const unsigned int pmask = ~((kTwo30 >> (d - 1)) - 1u);
  long cand[3][2];
  for (int a = 0; a < 3; ++a) {
    const long p0 = (long)(q[a] & pmask);
    cand[a][0] = p0;
    // the neighbour parent across the near face; outside the unit cube it
    // wraps around for periodic boundaries (NbrList, mortonid.cpp:15-55)
    long c = (q[a] & w) ? p0 + 2L * w : p0 - 2L * w;
    if (c < 0 || c >= (long)kTwo30) c = ((periodic >> a) & 1) ? (c + (long)kTwo30) % (long)kTwo30 : -1;
    cand[a][1] = c;
  }
  for (int c = 0; c < 8; ++c) {
    const long x = cand[0][c & 1], y = cand[1][(c >> 1) & 1], z = cand[2][(c >> 2) & 1];
    out[c] = (x < 0 || y < 0 || z < 0) ? MKey{~0ULL, ~0u, 0}
                                       : make_key((unsigned int)x, (unsigned int)y, (unsigned int)z, d - 1);
  }
}

__global__ void nbr_parents(const MKey* __restrict__ S, long n, int d, int periodic, MKey* __restrict__ out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  MKey c[8];
  parent_candidates(S[i], d, periodic, c);
  for (int k = 0; k < 8; ++k) out[i * 8 + k] = c[k];
}

__global__ void split_keys(const MKey* __restrict__ k, long n, unsigned long long* __restrict__ hi,
                           unsigned int* __restrict__ lo, int* __restrict__ idx) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  hi[i] = k[i].hi;
  lo[i] = k[i].lo;
  idx[i] = (int)i;
}

__global__ void unique_flags(const unsigned long long* __restrict__ hi, const unsigned int* __restrict__ lo, long n,
                             int* __restrict__ flag) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bool sentinel = hi[i] == ~0ULL && lo[i] == ~0u;
  const bool first = i == 0 || hi[i] != hi[i - 1] || lo[i] != lo[i - 1];
  flag[i] = (first && !sentinel) ? 1 : 0;
}

__global__ void compact_keys(const unsigned long long* __restrict__ hi, const unsigned int* __restrict__ lo,
                             const int* __restrict__ flag, const int* __restrict__ offs, long n, MKey* __restrict__ out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n || !flag[i]) return;
  MKey k;
  k.hi = hi[i];
  k.lo = lo[i];
  k.pad = 0;
  out[offs[i]] = k;
}

// The balance candidates of level d - 1 <= 21 as the hi words of their keys
// (see sort_unique): R of that level, then the nbr_parents of S, where a
// neighbour outside the box repeats the node's own parent.
__global__ void candidate_hi(const MKey* __restrict__ R, long nR, const MKey* __restrict__ S, long nS, int d,
                             int periodic, unsigned long long* __restrict__ hi) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < nR) {
    hi[i] = R[i].hi;
    return;
  }
  const long j = i - nR;
  if (j >= nS) return;
  MKey c[8];
  parent_candidates(S[j], d, periodic, c);
  for (int k = 0; k < 8; ++k) hi[nR + j * 8 + k] = c[k].hi == ~0ULL ? c[0].hi : c[k].hi;
}

__global__ void keys_from_hi(const unsigned long long* __restrict__ hi, long n, unsigned int lo,
                             MKey* __restrict__ out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) out[i] = MKey{hi[i], lo, 0};
}

// ------------------------------------------------------------------ final tree
// Levels of the final tree: S[d] the sorted keys of the internal nodes of
// level d (n[d] of them), whose children, eight in a row, are level d + 1
// (nodes off[d + 1] ..); ioff[d] numbers the internal nodes through all levels.
struct LevelTab {
  const MKey* S[kMaxDepth];
  long n[kMaxDepth + 1], off[kMaxDepth + 2], ioff[kMaxDepth + 1];
  int depth;  // levels with internal nodes
};

// One thread per internal node of any level: its place in its level is 8 times
// its parent's rank (a search of the level above) plus its octant; it writes
// its own links and its children's keys and parents.  Leaves keep what the
// arrays are preset to (leaf 1, child0 -1, parent 0).  A parent missing from
// the level above (the set is not closed) is reported in *bad and linked to
// the root, so that nothing is read or written out of range.
__global__ void link_nodes(LevelTab lt, long n_int, MKey* __restrict__ keys, unsigned char* __restrict__ leaf,
                           int* __restrict__ child0, int* __restrict__ parent, int* __restrict__ int_idx,
                           int* __restrict__ bad) {
  const long j = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (j == 0) {
    keys[0] = make_key(0, 0, 0, 0);
    parent[0] = -1;
  }
  if (j >= n_int) return;
  int d = 0;
  while (d + 1 < lt.depth && j >= lt.ioff[d + 1]) ++d;
  const long k = j - lt.ioff[d];
  unsigned int q[3], dd;
  const MKey key = lt.S[d][k];
  decode_key(key, q[0], q[1], q[2], dd);
  long g = 0;
  if (d > 0) {
    const unsigned int w = kTwo30 >> d, m = ~(2 * w - 1);
    const MKey pk = make_key(q[0] & m, q[1] & m, q[2] & m, d - 1);
    const long r = lower_bound_key(lt.S[d - 1], lt.n[d - 1], pk);
    if (r < lt.n[d - 1] && key_eq(lt.S[d - 1][r], pk))
      g = lt.off[d] + 8 * r + ((q[0] & w ? 1 : 0) | (q[1] & w ? 2 : 0) | (q[2] & w ? 4 : 0));
    else
      *bad = 1;
  }
  const long c0 = lt.off[d + 1] + 8 * k;
  leaf[g] = 0;
  child0[g] = (int)c0;
  int_idx[j] = (int)g;
  const unsigned int w = kTwo30 >> (d + 1);
  for (int c = 0; c < 8; ++c) {
    keys[c0 + c] = make_key(q[0] + ((c & 1) ? w : 0), q[1] + ((c & 2) ? w : 0), q[2] + ((c & 4) ? w : 0), d + 1);
    parent[c0 + c] = (int)g;
  }
}

__global__ void node_ranges(const MKey* __restrict__ keys, long n, const MKey* __restrict__ sk, long n_s,
                            const MKey* __restrict__ tk, long n_t, int* __restrict__ slo, int* __restrict__ shi,
                            int* __restrict__ tlo, int* __restrict__ thi) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned int X, Y, Z, d;
  decode_key(keys[i], X, Y, Z, d);
  const MKey e = node_end_key(X, Y, Z, d);
  if (sk) {
    slo[i] = (int)lower_bound_key(sk, n_s, keys[i]);
    shi[i] = (int)lower_bound_key(sk, n_s, e);
  } else {
    slo[i] = shi[i] = 0;
  }
  tlo[i] = (int)lower_bound_key(tk, n_t, keys[i]);
  thi[i] = (int)lower_bound_key(tk, n_t, e);
}

// Colleague index ((z+1)*3+(y+1))*3+(x+1) (mpi_tree.txx:1143-1145).
// Colleagues (the 27 same-level cells around a node, itself included; slot
// ci = (dx+1) + 3(dy+1) + 9(dz+1)), from the parent's colleagues: the cell at
// offset d from octant c of parent P is octant (c + d) mod 2 of P's colleague
// at offset floor((c + d) / 2), which exists at this level iff that colleague
// is internal (every internal node has all 8 children in the level arrays).
// Same result as searching the level's sorted keys (interac_list.txx:98-130).
// Periodic boundaries: every colleague of the root along the periodic axes
// (mask `periodic`: bit 0 x, bit 1 y, bit 2 z) is the root itself (one image
// per slot, mpi_tree.txx:1142-1168), and the rule above then wraps the
// colleagues of every level around the unit cube along those axes.
__global__ void colleagues_kernel(long base, long n_level, const int* __restrict__ parent,
                                  const int* __restrict__ child0, int periodic, int* __restrict__ coll) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n_level) return;
  const long v = base + i;
  if (v == 0) {
    for (int ci = 0; ci < 27; ++ci) {
      const int dx = ci % 3 - 1, dy = (ci / 3) % 3 - 1, dz = ci / 9 - 1;
      const bool img = periodic && (dx == 0 || (periodic & 1)) && (dy == 0 || (periodic & 2)) &&
                       (dz == 0 || (periodic & 4));
      coll[ci] = (ci == 13 || img) ? 0 : -1;
    }
    return;
  }
  const int P = parent[v];
  const int oc = (int)(v - child0[P]);
  const int ox = oc & 1, oy = (oc >> 1) & 1, oz = (oc >> 2) & 1;
  for (int ci = 0; ci < 27; ++ci) {
    const int cx = ox + ci % 3 - 1, cy = oy + (ci / 3) % 3 - 1, cz = oz + ci / 9 - 1;  // in [-1, 2]
    const int pci = ((cx >> 1) + 1) + 3 * ((cy >> 1) + 1) + 9 * ((cz >> 1) + 1);
    const int pc = coll[(long)P * 27 + pci];
    int r = -1;
    if (pc >= 0) {
      const int c0 = child0[pc];
      if (c0 >= 0) r = c0 + ((cx & 1) | ((cy & 1) << 1) | ((cz & 1) << 2));
    }
    coll[v * 27 + ci] = r;
  }
}

// Point -> leaf map and coordinates relative to the leaf centre.
template <class Real>
__global__ void localize(const int* __restrict__ leaves, long n_leaves, const MKey* __restrict__ keys,
                         const int* __restrict__ lo, const int* __restrict__ hi, const double* __restrict__ coord,
                         Real* __restrict__ x, Real* __restrict__ y, Real* __restrict__ z, int* __restrict__ pt_leaf) {
  const long li = blockIdx.x * (long)(blockDim.x / 32) + threadIdx.x / 32;  // a warp per leaf
  if (li >= n_leaves) return;
  const int node = leaves[li];
  unsigned int X, Y, Z, d;
  decode_key(keys[node], X, Y, Z, d);
  const double h = 1.0 / (double)(1u << d);
  const double c[3] = {X * (1.0 / kTwo30) + 0.5 * h, Y * (1.0 / kTwo30) + 0.5 * h, Z * (1.0 / kTwo30) + 0.5 * h};
  for (int p = lo[node] + threadIdx.x % 32; p < hi[node]; p += 32) {
    x[p] = (Real)(coord[p * 3 + 0] - c[0]);
    y[p] = (Real)(coord[p * 3 + 1] - c[1]);
    z[p] = (Real)(coord[p * 3 + 2] - c[2]);
    pt_leaf[p] = node;
  }
}

__global__ void gather_coords(const double* __restrict__ in, const int* __restrict__ perm, long n,
                              double* __restrict__ out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long p = perm[i];
  out[i * 3 + 0] = in[p * 3 + 0];
  out[i * 3 + 1] = in[p * 3 + 1];
  out[i * 3 + 2] = in[p * 3 + 2];
}

// Rows of the parent-child products (ChildRows): internal node j (index k in
// its level) joins, for every octant z whose child has points [lo, hi), the
// list of its level and octant.  The order within a list is the order of
// arrival; every row's product is formed by itself, so it changes no value.
__global__ void child_rows(LevelTab lt, long n_int, const int* __restrict__ int_idx, const int* __restrict__ child0,
                           const int* __restrict__ lo, const int* __restrict__ hi, int* __restrict__ rows,
                           int* __restrict__ counts, unsigned char* __restrict__ mask) {
  const long j = blockIdx.x * (long)blockDim.x + threadIdx.x;
  int d = 0;
  const bool in = j < n_int;
  while (in && d + 1 < lt.depth && j >= lt.ioff[d + 1]) ++d;
  const int lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(0xffffffffu, in ? d : -1);
  const int c0 = in ? child0[int_idx[j]] : 0;
  unsigned m = 0;
  for (int z = 0; z < 8; ++z) {
    const bool has = in && hi[c0 + z] > lo[c0 + z];
    const unsigned vote = __ballot_sync(0xffffffffu, has) & same;  // the lanes of this level with a row
    int base = 0;
    const int leader = __ffs(vote) - 1;
    if (has && lane == leader) base = atomicAdd(&counts[d * 8 + z], __popc(vote));
    base = __shfl_sync(0xffffffffu, base, vote ? leader : 0);
    if (has) {
      m |= 1u << z;
      rows[z * n_int + lt.ioff[d] + base + __popc(vote & ((1u << lane) - 1))] = (int)(j - lt.ioff[d]);
    }
  }
  if (in) mask[j] = (unsigned char)m;
}

// ------------------------------------------------------------------ lists
// Image of colleague c at slot ci of node v (periodic boundaries): the
// shift, in units of the unit cube, that moves c to the slot's position next
// to v, coded (sx+1) + 3(sy+1) + 9(sz+1) with s in {-1, 0, 1}; 13 = none.
// The reference stores the same shifts as coord_shift per interaction
// (fmm_pts.txx:2490-2500, 4646-4656, 4932-4942).
__device__ __forceinline__ unsigned char image_code(const MKey* keys, long v, int ci, long c) {
  unsigned int X[3], Y[3], dv, dc;
  decode_key(keys[v], X[0], X[1], X[2], dv);
  decode_key(keys[c], Y[0], Y[1], Y[2], dc);
  const long w = (long)(kTwo30 >> dv);
  const int off[3] = {ci % 3 - 1, (ci / 3) % 3 - 1, ci / 9 - 1};
  int code = 0, mul = 1;
  for (int a = 0; a < 3; ++a) {
    const long e = (long)X[a] + off[a] * w - (long)Y[a];  // a multiple of 2^30
    const int sh = e < 0 ? -1 : (e > 0 ? 1 : 0);
    code += (sh + 1) * mul;
    mul *= 3;
  }
  return (unsigned char)code;
}

// Memberships (0 or 1) and list lengths of a node, summed together.
enum { kSleaf, kTleaf, kVsrc, kP2P, kX, kW, kXtrg, kVtrg, kLeaf, kNodeCounts };
struct NodeCounts {
  int v[kNodeCounts];
};
struct SumCounts {
  __host__ __device__ NodeCounts operator()(const NodeCounts& a, const NodeCounts& b) const {
    NodeCounts c;
    for (int i = 0; i < kNodeCounts; ++i) c.v[i] = a.v[i] + b.v[i];
    return c;
  }
};

// One pass per target node (n_trg > 0); `mode` 0 counts, 1 fills.
// Relative coordinates follow InteracList::BuildList (interac_list.txx:98-279).
// With image arrays (periodic boundaries) every entry also gets the image
// code of its source (U1 / U2 / W: of the node's colleague; U0 / X: of the
// parent's colleague).
__global__ void build_lists(long n_nodes, const unsigned char* __restrict__ leaf, const int* __restrict__ parent,
                            const int* __restrict__ child0, const int* __restrict__ coll, const int* __restrict__ slo,
                            const int* __restrict__ shi, const int* __restrict__ tlo, const int* __restrict__ thi,
                            long nsrf, int sw, int mode, NodeCounts* __restrict__ counts,
                            const int* __restrict__ p_off, const int* __restrict__ x_off,
                            const int* __restrict__ w_off, int* __restrict__ p_list, int* __restrict__ x_list,
                            int* __restrict__ w_list, const MKey* __restrict__ keys, unsigned char* __restrict__ p_img,
                            unsigned char* __restrict__ x_img, unsigned char* __restrict__ w_img) {
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= n_nodes) return;
  const int nt = thi[t] - tlo[t];
  int np = 0, nx = 0, nw = 0, nv = 0;
  if (nt > 0) {
    const bool tleaf = leaf[t];
    const bool img = mode && p_img;
    int* pl = mode ? p_list + p_off[t] : nullptr;
    int* xl = mode ? x_list + x_off[t] : nullptr;
    int* wl = mode ? w_list + w_off[t] : nullptr;
    unsigned char* pi = img ? p_img + p_off[t] : nullptr;
    unsigned char* xi = img ? x_img + x_off[t] : nullptr;
    unsigned char* wi = img ? w_img + w_off[t] : nullptr;
    unsigned char code = 13;
#define ADD(list, cnt, v)      \
  do {                         \
    if (mode) {                \
      list[cnt] = (v);         \
      if (img) list##_img_[cnt] = code; \
    }                          \
    ++cnt;                     \
  } while (0)
    unsigned char* pl_img_ = pi;
    unsigned char* xl_img_ = xi;
    unsigned char* wl_img_ = wi;
    if (tleaf) {
      for (int ci = 0; ci < 27; ++ci) {
        const int c = coll[t * 27 + ci];
        if (c < 0) continue;
        if (img) code = image_code(keys, t, ci, c);
        if (leaf[c]) {
          if (shi[c] > slo[c]) ADD(pl, np, c);  // U1
        } else {
          for (int j = 0; j < 8; ++j) {
            const int ch = child0[c] + j;
            const int rx = (ci % 3) * 4 - 4 + ((j & 1) ? 2 : 0) - 1;
            const int ry = ((ci / 3) % 3) * 4 - 4 + ((j & 2) ? 2 : 0) - 1;
            const int rz = (ci / 9) * 4 - 4 + ((j & 4) ? 2 : 0) - 1;
            const int ns_ch = shi[ch] - slo[ch];
            if (ns_ch <= 0) continue;
            if (max(abs(rx), max(abs(ry), abs(rz))) <= 3) {
              ADD(pl, np, ch);  // U2
            } else if (leaf[ch] && (long)ns_ch * sw <= nsrf) {  // pt_cnt[0] counts each layer
              ADD(pl, np, ch);  // W handled as P2P (fmm_pts.txx:5325)
            } else {
              ADD(wl, nw, ch);  // W (fmm_pts.txx:4929)
            }
          }
        }
      }
    }
    const int p = parent[t];
    if (p >= 0) {
      int p2n = 0;
      {
        const int c0 = child0[p];
        p2n = (int)(t - c0);
      }
      for (int ci = 0; ci < 27; ++ci) {
        const int c = coll[(long)p * 27 + ci];
        if (c < 0 || !leaf[c]) continue;
        if (shi[c] <= slo[c]) continue;
        if (img) code = image_code(keys, p, ci, c);
        const int rx = (ci % 3) * 4 - 4 - ((p2n & 1) ? 2 : 0) + 1;
        const int ry = ((ci / 3) % 3) * 4 - 4 - ((p2n & 2) ? 2 : 0) + 1;
        const int rz = (ci / 9) * 4 - 4 - ((p2n & 4) ? 2 : 0) + 1;
        if (max(abs(rx), max(abs(ry), abs(rz))) <= 3) {
          if (tleaf) ADD(pl, np, c);  // U0
        } else if (tleaf && nt <= nsrf) {
          ADD(pl, np, c);  // X handled as P2P (fmm_pts.txx:5295)
        } else {
          ADD(xl, nx, c);  // X (fmm_pts.txx:4629)
        }
      }
    }
    if (!tleaf) {
      for (int ci = 0; ci < 27; ++ci) {
        if (ci == 13) continue;
        const int c = coll[t * 27 + ci];
        if (c >= 0 && !leaf[c] && shi[c] > slo[c]) ++nv;
      }
    }
#undef ADD
  }
  if (!mode) {
    const bool lf = leaf[t], src = shi[t] > slo[t];
    NodeCounts c;
    c.v[kSleaf] = lf && src;
    c.v[kTleaf] = lf && nt > 0;
    c.v[kVsrc] = !lf && src;
    c.v[kP2P] = np;
    c.v[kX] = nx;
    c.v[kW] = nw;
    c.v[kXtrg] = nx > 0;
    c.v[kVtrg] = nv > 0;
    c.v[kLeaf] = lf;
    counts[t] = c;
  }
}

struct NodeLists {
  int *sleaf, *tleaf, *vsrc, *xtrg, *vtrg;
};

// Places every node in the lists it belongs to, from the prefix sums of the
// counts; ranks >= cap (the capacity of the lists) are skipped.  The last node
// closes the CSR offsets and writes the totals to the pinned slots.
__global__ void scatter_lists(long n, long cap, const NodeCounts* __restrict__ counts,
                              const NodeCounts* __restrict__ offs, NodeLists l, int* __restrict__ node2vsrc,
                              int* __restrict__ po, int* __restrict__ xo, int* __restrict__ wo,
                              int* __restrict__ totals) {
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const NodeCounts c = counts[t], o = offs[t];
  if (c.v[kSleaf] && o.v[kSleaf] < cap) l.sleaf[o.v[kSleaf]] = (int)t;
  if (c.v[kTleaf] && o.v[kTleaf] < cap) l.tleaf[o.v[kTleaf]] = (int)t;
  const bool vs = c.v[kVsrc] && o.v[kVsrc] < cap;
  if (vs) l.vsrc[o.v[kVsrc]] = (int)t;
  node2vsrc[t] = vs ? o.v[kVsrc] : -1;
  if (c.v[kXtrg] && o.v[kXtrg] < cap) l.xtrg[o.v[kXtrg]] = (int)t;
  if (c.v[kVtrg] && o.v[kVtrg] < cap) l.vtrg[o.v[kVtrg]] = (int)t;
  po[t] = o.v[kP2P];
  xo[t] = o.v[kX];
  wo[t] = o.v[kW];
  if (t == n - 1) {
    const NodeCounts sum = SumCounts()(o, c);
    po[n] = sum.v[kP2P];
    xo[n] = sum.v[kX];
    wo[n] = sum.v[kW];
    for (int i = 0; i < kNodeCounts; ++i) totals[i] = sum.v[i];
  }
}

// V-list targets are ordered by their pattern of occupied offsets within
// windows of kVsortWindow consecutive (Morton-ordered) targets: bit o of the
// pattern is set when the target has a source parent at colleague offset o
// (the offsets of vlist_order).  key[i] = window << 26 | pattern.
#ifndef PVFMM_VSORT_WINDOW
#define PVFMM_VSORT_WINDOW 2048
#endif
constexpr long kVsortWindow = PVFMM_VSORT_WINDOW;
__global__ void vlist_keys(const int* __restrict__ vtrg, long n_vtrg, const int* __restrict__ coll,
                           const int* __restrict__ node2vsrc, unsigned long long* __restrict__ key,
                           int* __restrict__ rank) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n_vtrg) return;
  rank[i] = (int)i;
  const long t = vtrg[i];
  unsigned m = 0;
  for (int ci = 0, o = 0; ci < 27; ++ci) {
    if (ci == 13) continue;
    const int c = coll[t * 27 + ci];
    if (c >= 0 && node2vsrc[c] >= 0) m |= 1u << o;
    ++o;
  }
  key[i] = (unsigned long long)(i / kVsortWindow) << 26 | m;
}
// Pattern order from the sorted Morton ranks: position p takes the node of
// rank rank_sorted[p], with its pattern and its row of source parents per
// offset (offset-major: coalesced); vmorton[rank] = p.
__global__ void vlist_order(const int* __restrict__ vtrg_morton, const int* __restrict__ rank_sorted,
                            const unsigned long long* __restrict__ key_sorted, long n, const int* __restrict__ coll,
                            const int* __restrict__ node2vsrc, int* __restrict__ vtrg, int* __restrict__ vmorton,
                            unsigned* __restrict__ mask, int* __restrict__ vtab) {
  const long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int r = rank_sorted[p];
  const long t = vtrg_morton[r];
  vtrg[p] = (int)t;
  vmorton[r] = (int)p;
  mask[p] = (unsigned)(key_sorted[p] & ((1u << 26) - 1));
  for (int ci = 0, o = 0; ci < 27; ++ci) {
    if (ci == 13) continue;
    const int c = coll[t * 27 + ci];
    vtab[(long)o * n + p] = c >= 0 ? node2vsrc[c] : -1;
    ++o;
  }
}

__global__ void gather_u32(const unsigned int* __restrict__ in, const int* __restrict__ perm, long n,
                           unsigned int* __restrict__ out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[perm[i]];
}

__global__ void iota_kernel(int* __restrict__ a, long n) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) a[i] = (int)i;
}

// Pinned host slots of a tree build (ctx.chk): the list totals, the error word
// of link_nodes, the last scan's total, and 12 doubles of bounding boxes.
constexpr int kChkLists = 0, kChkLinks = 16, kChkScan = 17, kChkSlots = 32;
constexpr size_t kChkBytes = kChkSlots * sizeof(int) + 12 * sizeof(double);
inline double* chk_bbox(Context& ctx) { return reinterpret_cast<double*>(ctx.chk + kChkSlots); }

// The total out[n-1] + in[n-1] of an exclusive scan, into a pinned slot.
__global__ void scan_total(const int* __restrict__ in, const int* __restrict__ out, long n, int* __restrict__ slot) {
  *slot = out[n - 1] + in[n - 1];
}

// Exclusive prefix sum of n ints; returns the total (read through a pinned
// slot after a synchronisation).
long exclusive_scan(Context& ctx, const int* in, int* out, long n) {
  if (n <= 0) return 0;
  size_t bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, (int)n, ctx.stream);
  void* tmp = ctx.scratch2.ensure(bytes);
  cub::DeviceScan::ExclusiveSum(tmp, bytes, in, out, (int)n, ctx.stream);
  int* slot = ctx.chk + kChkScan;
  ++ctx.n_launch;
  scan_total<<<1, 1, 0, ctx.stream>>>(in, out, n, slot);
  PVFMM_CUDA_CHECK(cudaStreamSynchronize(ctx.stream));
  return *(volatile int*)slot;
}

// Stable sort of 96-bit keys (hi, lo): by lo, then stably by hi.  On return
// perm[i] is the input position of the i-th smallest key and hs/ls hold the
// sorted halves.  Uses temporaries t[base..base+2].
void sort_hilo(Context& ctx, long n, const unsigned long long* hi, const unsigned int* lo, unsigned long long* hs,
               unsigned int* ls, int* perm, int base) {
  auto& s = ctx.stream;
  int* idx = ctx.t[base].as<int>(n);
  int* p1 = ctx.t[base + 1].as<int>(n);
  unsigned long long* hg = ctx.t[base + 2].as<unsigned long long>(n);
  ++ctx.n_launch;
  iota_kernel<<<ceil_div(n, kThreads), kThreads, 0, s>>>(idx, n);
  size_t b1 = 0, b2 = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, b1, lo, ls, idx, p1, (int)n, 0, 32, s);
  cub::DeviceRadixSort::SortPairs(nullptr, b2, hg, hs, p1, perm, (int)n, 0, 64, s);
  void* tmp = ctx.scratch.ensure(std::max(b1, b2));
  cub::DeviceRadixSort::SortPairs(tmp, b1, lo, ls, idx, p1, (int)n, 0, 32, s);
  ++ctx.n_launch;
  gather_u64<<<ceil_div(n, kThreads), kThreads, 0, s>>>(hi, p1, n, hg);
  cub::DeviceRadixSort::SortPairs(tmp, b2, hg, hs, p1, perm, (int)n, 0, 64, s);
  ++ctx.n_launch;
  gather_u32<<<ceil_div(n, kThreads), kThreads, 0, s>>>(lo, perm, n, ls);
}

// The sorted, unique keys of the level's internal nodes after balance: R (the
// refined ones, nR) with the neighbours' parents of S, the balanced level d
// below (nS nodes); returns their count.  A node of depth L = d - 1 <= 21 has
// zero coordinate bits below 30 - L, so its key is hi (top 3L bits of the
// 63-bit interleave) with lo = L: one keys-only radix sort over those bits
// orders them.
long balance_level(Context& ctx, const MKey* R, long nR, const MKey* S, long nS, int d, DevBuf& out) {
  auto& s = ctx.stream;
  const long n = nR + 8 * nS;
  const int depth = d - 1;
  unsigned long long* h = ctx.t[10].as<unsigned long long>(n);
  unsigned long long* hs = ctx.t[13].as<unsigned long long>(n);
  ++ctx.n_launch;
  candidate_hi<<<ceil_div(nR + nS, kThreads), kThreads, 0, s>>>(R, nR, S, nS, d, ctx.periodic ? ctx.periodic_axes : 0,
                                                               h);
  const int begin_bit = 3 * (21 - depth);
  size_t b1 = 0, b2 = 0;
  int* slot = ctx.chk + kChkScan;
  cub::DeviceRadixSort::SortKeys(nullptr, b1, h, hs, (int)n, begin_bit, 63, s);
  cub::DeviceSelect::Unique(nullptr, b2, hs, h, slot, (int)n, s);
  void* tmp = ctx.scratch.ensure(std::max(b1, b2));
  // (a root-only level has no key bits: every candidate is the root)
  const unsigned long long* sorted = h;
  unsigned long long* uniq = hs;
  if (begin_bit < 63) {
    cub::DeviceRadixSort::SortKeys(tmp, b1, h, hs, (int)n, begin_bit, 63, s);
    sorted = hs;
    uniq = h;
  }
  cub::DeviceSelect::Unique(tmp, b2, sorted, uniq, slot, (int)n, s);
  PVFMM_CUDA_CHECK(cudaStreamSynchronize(s));
  const long cnt = *(volatile int*)slot;
  MKey* o = out.as<MKey>(std::max(cnt, 1L));
  ++ctx.n_launch;
  keys_from_hi<<<ceil_div(std::max(cnt, 1L), kThreads), kThreads, 0, s>>>(uniq, cnt, (unsigned int)depth, o);
  return cnt;
}

// Sorts node keys (of levels deeper than 21: full 96-bit keys) and removes
// duplicates and sentinels; returns the count.
long sort_unique(Context& ctx, const MKey* in, long n, DevBuf& out) {
  auto& s = ctx.stream;
  if (n == 0) return 0;
  unsigned long long* h = ctx.t[10].as<unsigned long long>(n);
  unsigned int* l = ctx.t[11].as<unsigned int>(n);
  int* ix = ctx.t[12].as<int>(n);
  ++ctx.n_launch;
  split_keys<<<ceil_div(n, kThreads), kThreads, 0, s>>>(in, n, h, l, ix);
  unsigned long long* hs = ctx.t[13].as<unsigned long long>(n);
  unsigned int* ls = ctx.t[14].as<unsigned int>(n);
  int* perm = ctx.t[15].as<int>(n);
  sort_hilo(ctx, n, h, l, hs, ls, perm, 16);
  int* fl = ctx.t[19].as<int>(n);
  int* of = ctx.t[20].as<int>(n);
  ++ctx.n_launch;
  unique_flags<<<ceil_div(n, kThreads), kThreads, 0, s>>>(hs, ls, n, fl);
  const long cnt = exclusive_scan(ctx, fl, of, n);
  MKey* o = out.as<MKey>(std::max(cnt, 1L));
  ++ctx.n_launch;
  compact_keys<<<ceil_div(n, kThreads), kThreads, 0, s>>>(hs, ls, fl, of, n, o);
  return cnt;
}

// Sorts mapped points: perm (sorted -> input), sorted keys, sorted coords.
void sort_point_set(Context& ctx, long n, const unsigned long long* hi, const unsigned int* lo, const double* mapped,
                    DevBuf& perm_out, DevBuf& keys_out, DevBuf& coord_out) {
  auto& s = ctx.stream;
  unsigned long long* hs = ctx.t[5].as<unsigned long long>(n);
  unsigned int* ls = ctx.t[6].as<unsigned int>(n);
  int* perm = perm_out.as<int>(n);
  sort_hilo(ctx, n, hi, lo, hs, ls, perm, 16);
  MKey* keys = keys_out.as<MKey>(n);
  ++ctx.n_launch;
  assemble_keys<<<ceil_div(n, kThreads), kThreads, 0, s>>>(hs, lo, perm, n, keys);
  double* c = coord_out.as<double>(n * 3);
  ++ctx.n_launch;
  gather_coords<<<ceil_div(n, kThreads), kThreads, 0, s>>>(mapped, perm, n, c);
}

// Reference bounding-box rule (pvfmm-wrapper.cpp:469-520) in precision Real.
template <class Real>
void bbox_scale_shift(const double* bs, const double* bt, double& scale_out, double* shift_out) {
  const Real eps = std::numeric_limits<Real>::epsilon() * (Real)64;
  auto one = [&](const double* b, Real& sc, Real* sh) {
    const double* mn = b;
    const double* mx = b + 3;
    sc = (Real)1 / (Real)(mx[0] - mn[0] + 2 * (double)eps);
    for (int k = 0; k < 3; ++k) sc = std::min(sc, (Real)(1.0 / (mx[k] - mn[k] + 2 * (double)eps)));
    if (sc * (Real)0 != (Real)0) sc = (Real)1;
    for (int k = 0; k < 3; ++k) sh[k] = (Real)(-mn[k]) * sc + eps;
  };
  Real s0, x0[3], s1, x1[3];
  one(bs, s0, x0);
  one(bt, s1, x1);
  Real c0[3], c1[3];
  for (int k = 0; k < 3; ++k) {
    c0[k] = (Real)(0.5 - (double)x0[k]) / s0;
    c1[k] = (Real)(0.5 - (double)x1[k]) / s1;
  }
  Real sc = 0;
  for (int k = 0; k < 3; ++k) sc = std::max(sc, (Real)std::fabs(c0[k] - c1[k]));
  sc = (Real)1 / (sc + (Real)1 / s0 + (Real)1 / s1);
  scale_out = (double)sc;
  for (int k = 0; k < 3; ++k) shift_out[k] = (double)((Real)0.5 - (c0[k] + c1[k]) * sc / (Real)2);
}

template <class T>
void point_bbox(Context& ctx, const T* pos, long n, double* host6) {
  const int nb = (int)std::min<long>(1024, std::max<long>(1, ceil_div(n, kThreads)));
  double* part = ctx.t[0].as<double>((size_t)nb * 6 + 6);
  ++ctx.n_launch;
  bbox_partial<T><<<nb, kThreads, 0, ctx.stream>>>(pos, n, part);
  ++ctx.n_launch;
  bbox_final<<<1, kThreads, 0, ctx.stream>>>(part, nb, part + (size_t)nb * 6);
  // host6: pinned; the caller synchronises
  PVFMM_CUDA_CHECK(cudaMemcpyAsync(host6, part + (size_t)nb * 6, 6 * sizeof(double), cudaMemcpyDeviceToHost, ctx.stream));
}

template <class T>
void map_points(Context& ctx, const T* pos, long n, double scale, const double* shift, DevBuf& mapped,
                DevBuf& hi, DevBuf& lo) {
  double* mp = mapped.as<double>(n * 3);
  unsigned long long* h = hi.as<unsigned long long>(n);
  unsigned int* l = lo.as<unsigned int>(n);
  int* idx = ctx.t[4].as<int>(n);
  ++ctx.n_launch;
  map_and_key<T><<<ceil_div(n, kThreads), kThreads, 0, ctx.stream>>>(pos, n, (T)scale, (T)shift[0], (T)shift[1],
                                                                      (T)shift[2], mp, h, l, idx);
}

}  // namespace

// Seed grid of the context's initial tree (pvfmm-wrapper.cpp:416-432), as
// sorted Morton keys, in the precision of the context.
static std::vector<MKey> seed_grid_keys(int max_pts, bool real_float) {
  std::vector<MKey> keys;
  long NN;
  if (real_float) NN = (long)std::ceil(std::pow((float)max_pts, 1.0 / 3.0));
  else NN = (long)std::ceil(std::pow((double)max_pts, 1.0 / 3.0));
  keys.reserve(NN * NN * NN);
  for (long i = 0; i < NN * NN * NN; ++i) {
    unsigned int q[3];
    const long comp[3] = {i % NN, (i / NN) % NN, (i / (NN * NN)) % NN};
    for (int d = 0; d < 3; ++d) {
      if (real_float) {
        const float c = (float)((float)comp[d] + 0.5f) / (float)NN;
        q[d] = (unsigned int)std::floor((double)c * (double)kTwo30);
      } else {
        const double c = ((double)comp[d] + 0.5) / (double)NN;
        q[d] = (unsigned int)std::floor(c * (double)kTwo30);
      }
    }
    keys.push_back(make_key(q[0], q[1], q[2], kMaxDepth));
  }
  std::sort(keys.begin(), keys.end(), [](const MKey& a, const MKey& b) { return key_less(a, b); });
  return keys;
}

void build_tree(Context& ctx, const void* src_pos, long n_src, const void* trg_pos, long n_trg, bool pos_float,
                int src_weight, bool trg_alias) {
  if (n_src < 1 || n_trg < 1) throw std::runtime_error("build_tree needs at least one source and one target");
  if (!ctx.chk) PVFMM_CUDA_CHECK(cudaMallocHost((void**)&ctx.chk, kChkBytes));
  DevTree& T = ctx.tree;
  auto& s = ctx.stream;
  T.valid = false;
  T.n_src = n_src;
  T.n_trg = n_trg;
  T.src_weight = n_src > 0 ? src_weight : 0;
  T.src_counted = T.src_weight > 0;
  // 1. bounding box and map (both boxes read back with one synchronisation)
  double* bs = chk_bbox(ctx);
  double* bt = bs + 6;
  if (pos_float) {
    point_bbox<float>(ctx, (const float*)src_pos, n_src, bs);
    if (!trg_alias) point_bbox<float>(ctx, (const float*)trg_pos, n_trg, bt);
  } else {
    point_bbox<double>(ctx, (const double*)src_pos, n_src, bs);
    if (!trg_alias) point_bbox<double>(ctx, (const double*)trg_pos, n_trg, bt);
  }
  PVFMM_CUDA_CHECK(cudaStreamSynchronize(ctx.stream));
  if (trg_alias) std::copy(bs, bs + 6, bt);
  if (!ctx.unit_box && !ctx.periodic) {
    if (pos_float) bbox_scale_shift<float>(bs, bt, T.scale_x, T.shift_x);
    else bbox_scale_shift<double>(bs, bt, T.scale_x, T.shift_x);
  }
  if (ctx.periodic) {
    // periodic boundaries (pvfmm-wrapper.cpp:512-517): scale 1 / box_size in
    // the interface precision, no shift; the mapping wraps into [0,1)
    T.scale_x = pos_float ? (double)(1.0f / (float)ctx.box_size) : 1.0 / ctx.box_size;
    T.shift_x[0] = T.shift_x[1] = T.shift_x[2] = 0.0;
  } else if (ctx.unit_box) {
    // C++ interface (include/pvfmm.txx:216-244): coordinates are used as
    // given, so they must lie in the unit cube.
    for (const double* b : {bs, bt})
      for (int k = 0; k < 3; ++k)
        if (!(b[k] >= 0.0) || !(b[3 + k] < 1.0))
          throw std::runtime_error("coordinates must lie in [0,1)^3 for a unit-box tree");
    T.scale_x = 1.0;
    T.shift_x[0] = T.shift_x[1] = T.shift_x[2] = 0.0;
  }
  DevBuf& src_mapped = ctx.t[1];
  DevBuf& trg_mapped = ctx.t[2];
  DevBuf& hi = ctx.t[7];
  DevBuf& lo = ctx.t[8];
  DevBuf& coords_s = ctx.t[21];
  DevBuf& coords_t = ctx.t[22];
  // 2. sources
  if (pos_float) map_points<float>(ctx, (const float*)src_pos, n_src, T.scale_x, T.shift_x, src_mapped, hi, lo);
  else map_points<double>(ctx, (const double*)src_pos, n_src, T.scale_x, T.shift_x, src_mapped, hi, lo);
  sort_point_set(ctx, n_src, hi.get<unsigned long long>(), lo.get<unsigned int>(), src_mapped.get<double>(),
                 T.src_perm, T.src_key, coords_s);
  // 3. targets
  if (trg_alias) {
    PVFMM_CUDA_CHECK(cudaMemcpyAsync(T.trg_perm.as<int>(n_src), T.src_perm.get<int>(), n_src * sizeof(int),
                                     cudaMemcpyDeviceToDevice, s));
    PVFMM_CUDA_CHECK(cudaMemcpyAsync(T.trg_key.as<MKey>(n_src), T.src_key.get<MKey>(), n_src * sizeof(MKey),
                                     cudaMemcpyDeviceToDevice, s));
    PVFMM_CUDA_CHECK(cudaMemcpyAsync(coords_t.as<double>(n_src * 3), coords_s.get<double>(), n_src * 3 * sizeof(double),
                                     cudaMemcpyDeviceToDevice, s));
  } else {
    if (pos_float) map_points<float>(ctx, (const float*)trg_pos, n_trg, T.scale_x, T.shift_x, trg_mapped, hi, lo);
    else map_points<double>(ctx, (const double*)trg_pos, n_trg, T.scale_x, T.shift_x, trg_mapped, hi, lo);
    sort_point_set(ctx, n_trg, hi.get<unsigned long long>(), lo.get<unsigned int>(), trg_mapped.get<double>(),
                   T.trg_perm, T.trg_key, coords_t);
  }
  // 4. the tree's point set: the seed grid of the C interface, or the
  //    targets for a unit-box tree (pt_coord = trg_coord, pvfmm.txx:238)
  const MKey* sk = T.src_counted ? T.src_key.get<MKey>() : nullptr;
  const MKey* tk = T.trg_key.get<MKey>();
  const MKey* d_gk = tk;
  long n_gk = n_trg;
  if (!ctx.unit_box) {
    // the same for every tree of the context (max_pts and the coordinates'
    // precision): uploaded once
    if (ctx.n_seed == 0 || ctx.seed_float != pos_float) {
      const std::vector<MKey> gk = seed_grid_keys(ctx.max_pts, pos_float);
      ctx.n_seed = 0;
      MKey* g = ctx.seed.as<MKey>(gk.size());
      PVFMM_CUDA_CHECK(cudaMemcpyAsync(g, gk.data(), gk.size() * sizeof(MKey), cudaMemcpyHostToDevice, s));
      PVFMM_CUDA_CHECK(cudaStreamSynchronize(s));  // gk goes out of scope
      ctx.n_seed = (long)gk.size();
      ctx.seed_float = pos_float;
    }
    d_gk = ctx.seed.get<MKey>();
    n_gk = ctx.n_seed;
  }
  // 5. refinement, level by level
  std::vector<long> nR;
  {
    // two persistent level buffers (no allocation in steady state)
    DevBuf* cur_b = &ctx.t[16];
    DevBuf* next_b = &ctx.t[17];
    MKey root = make_key(0, 0, 0, 0);
    PVFMM_CUDA_CHECK(cudaMemcpyAsync(cur_b->as<MKey>(1), &root, sizeof(MKey), cudaMemcpyHostToDevice, s));
    long n_cur = 1;
    int d = 0;
    while (n_cur > 0) {
      int* split = ctx.t[3].as<int>(n_cur);
      int* offs = ctx.t[23].as<int>(n_cur);
      ++ctx.n_launch;
      refine_level<<<ceil_div(n_cur, kThreads), kThreads, 0, s>>>(cur_b->get<MKey>(), n_cur, d, sk, T.n_src,
                                                                   T.src_weight, tk, T.n_trg, d_gk, n_gk,
                                                                   ctx.max_pts, kMaxDepth, split);
      const long n_split = exclusive_scan(ctx, split, offs, n_cur);
      if (n_split == 0) break;
      if ((long)ctx.lvlR.size() <= d) ctx.lvlR.resize(d + 1);
      MKey* R = ctx.lvlR[d].as<MKey>(n_split);
      MKey* next = next_b->as<MKey>(n_split * 8);
      ++ctx.n_launch;
      make_children<<<ceil_div(n_cur, kThreads), kThreads, 0, s>>>(cur_b->get<MKey>(), split, offs, n_cur, d, next, R);
      nR.push_back(n_split);
      std::swap(cur_b, next_b);
      n_cur = n_split * 8;
      ++d;
    }
  }
  const int dint = (int)nR.size() - 1;  // deepest level with internal nodes (-1: root is a leaf)
  // 6. 2:1 balance closure
  std::vector<long> nS(std::max(dint + 1, 0), 0);
  if ((long)ctx.lvlS.size() < dint + 1) ctx.lvlS.resize(dint + 1);
  if (dint >= 0) {
    PVFMM_CUDA_CHECK(cudaMemcpyAsync(ctx.lvlS[dint].as<MKey>(nR[dint]), ctx.lvlR[dint].get<MKey>(),
                                     nR[dint] * sizeof(MKey), cudaMemcpyDeviceToDevice, s));
    nS[dint] = nR[dint];
    for (int d = dint; d >= 1; --d) {
      if (d - 1 <= 21) {
        nS[d - 1] = balance_level(ctx, ctx.lvlR[d - 1].get<MKey>(), nR[d - 1], ctx.lvlS[d].get<MKey>(), nS[d], d,
                                  ctx.lvlS[d - 1]);
        continue;
      }
      const long nc = nR[d - 1] + 8 * nS[d];
      MKey* cand = ctx.t[9].as<MKey>(nc);
      PVFMM_CUDA_CHECK(cudaMemcpyAsync(cand, ctx.lvlR[d - 1].get<MKey>(), nR[d - 1] * sizeof(MKey),
                                       cudaMemcpyDeviceToDevice, s));
      ++ctx.n_launch;
      nbr_parents<<<ceil_div(nS[d], kThreads), kThreads, 0, s>>>(ctx.lvlS[d].get<MKey>(), nS[d], d,
                                                                 ctx.periodic ? ctx.periodic_axes : 0,
                                                                 cand + nR[d - 1]);
      nS[d - 1] = sort_unique(ctx, cand, nc, ctx.lvlS[d - 1]);
    }
  }
  // 7. final node arrays
  const int D = dint + 1;  // deepest level
  T.depth = D;
  T.level_off.assign(D + 2, 0);
  T.n_internal.assign(D + 1, 0);
  T.level_off[0] = 0;
  T.level_off[1] = 1;
  for (int d = 1; d <= D; ++d) T.level_off[d + 1] = T.level_off[d] + 8 * nS[d - 1];
  const long N = T.level_off[D + 1];
  T.n_nodes = N;
  MKey* keys = T.key.as<MKey>(N);
  unsigned char* leaf = T.leaf.as<unsigned char>(N);
  int* parent = T.parent.as<int>(N);
  int* child0 = T.child0.as<int>(N);
  long n_int_total = 0;
  for (int d = 0; d < D; ++d) n_int_total += nS[d];
  int* int_idx = T.int_idx.as<int>(std::max(n_int_total, 1L));
  T.int_off.assign(D + 1, 0);
  LevelTab lt{};
  lt.depth = D;
  long int_base = 0;
  for (int d = 0; d <= D; ++d) {
    const long nint = d < D ? nS[d] : 0;
    T.n_internal[d] = nint;
    T.int_off[d] = int_base;
    if (d < D) lt.S[d] = ctx.lvlS[d].get<MKey>();
    lt.n[d] = nint;
    lt.off[d] = T.level_off[d];
    lt.ioff[d] = int_base;
    int_base += nint;
  }
  lt.off[D + 1] = N;
  ctx.chk[kChkLinks] = 0;  // (nothing in flight writes it)
  PVFMM_CUDA_CHECK(cudaMemsetAsync(leaf, 1, N, s));
  PVFMM_CUDA_CHECK(cudaMemsetAsync(child0, 0xff, N * sizeof(int), s));
  PVFMM_CUDA_CHECK(cudaMemsetAsync(parent, 0, N * sizeof(int), s));
  ++ctx.n_launch;
  link_nodes<<<ceil_div(std::max(n_int_total, 1L), 128), 128, 0, s>>>(lt, n_int_total, keys, leaf, child0, parent,
                                                                       int_idx, ctx.chk + kChkLinks);
  // 8. point ranges and colleagues
  int* slo = T.src_lo.as<int>(N);
  int* shi = T.src_hi.as<int>(N);
  int* tlo = T.trg_lo.as<int>(N);
  int* thi = T.trg_hi.as<int>(N);
  ++ctx.n_launch;
  node_ranges<<<ceil_div(N, kThreads), kThreads, 0, s>>>(keys, N, sk, T.n_src, tk, T.n_trg, slo, shi, tlo, thi);
  int* coll = T.colleague.as<int>(N * 27);
  for (int d = 0; d <= D; ++d) {
    const long base = T.level_off[d], nl = T.level_off[d + 1] - base;
    ++ctx.n_launch;
    colleagues_kernel<<<ceil_div(nl, kThreads), kThreads, 0, s>>>(base, nl, parent, child0,
                                                                   ctx.periodic ? ctx.periodic_axes : 0, coll);
  }
  // 9. compact node lists.  Every node's memberships and list lengths are one
  //    record of counts (NodeCounts), prefix-summed together; the compacted
  //    lists are sized for all N nodes, so that their counts are read back at
  //    one synchronisation.
  {
    NodeCounts* nc = ctx.t[4].as<NodeCounts>(N);
    NodeCounts* no = ctx.t[5].as<NodeCounts>(N);
    int* cnt = ctx.chk + kChkLists;
    const long nsrf = ctx.ns;
    ++ctx.n_launch;
    build_lists<<<ceil_div(N, 128), 128, 0, s>>>(N, leaf, parent, child0, coll, slo, shi, tlo, thi, nsrf,
                                                 T.src_weight, 0, nc, nullptr, nullptr, nullptr, nullptr, nullptr,
                                                 nullptr, keys, nullptr, nullptr, nullptr);
    size_t bytes = 0;
    cub::DeviceScan::ExclusiveScan(nullptr, bytes, nc, no, SumCounts(), NodeCounts{}, (int)N, s);
    void* stmp = ctx.scratch2.ensure(bytes);
    cub::DeviceScan::ExclusiveScan(stmp, bytes, nc, no, SumCounts(), NodeCounts{}, (int)N, s);
    int* po = T.p_off.as<int>(N + 1);
    int* xo = T.x_off.as<int>(N + 1);
    int* wo = T.w_off.as<int>(N + 1);
    int* n2v = T.node2vsrc.as<int>(N);
    int* vtrg_morton = ctx.t[0].as<int>(N);
    ++ctx.n_launch;
    scatter_lists<<<ceil_div(N, kThreads), kThreads, 0, s>>>(
        N, N, nc, no, NodeLists{T.sleaf.as<int>(N), T.tleaf.as<int>(N), T.vsrc.as<int>(N), T.xtrg.as<int>(N), vtrg_morton},
        n2v, po, xo, wo, cnt);
    PVFMM_CUDA_CHECK(cudaStreamSynchronize(s));
    T.n_sleaf = cnt[kSleaf];
    T.n_tleaf = cnt[kTleaf];
    T.n_vsrc = cnt[kVsrc];
    T.n_p2p = cnt[kP2P];
    T.n_x = cnt[kX];
    T.n_w = cnt[kW];
    T.n_xtrg = cnt[kXtrg];
    T.n_vtrg = cnt[kVtrg];
    if (cnt[kLeaf] != (int)(N - n_int_total) || ctx.chk[kChkLinks] != 0)
      throw std::runtime_error("octree build: balanced internal set is not closed");
    int* pl = T.p_list.as<int>(std::max(T.n_p2p, 1L));
    int* xl = T.x_list.as<int>(std::max(T.n_x, 1L));
    int* wl = T.w_list.as<int>(std::max(T.n_w, 1L));
    unsigned char* pim = ctx.periodic ? T.p_img.as<unsigned char>(std::max(T.n_p2p, 1L)) : nullptr;
    unsigned char* xim = ctx.periodic ? T.x_img.as<unsigned char>(std::max(T.n_x, 1L)) : nullptr;
    unsigned char* wim = ctx.periodic ? T.w_img.as<unsigned char>(std::max(T.n_w, 1L)) : nullptr;
    ++ctx.n_launch;
    build_lists<<<ceil_div(N, 128), 128, 0, s>>>(N, leaf, parent, child0, coll, slo, shi, tlo, thi, nsrf,
                                                 T.src_weight, 1, nullptr, po, xo, wo, pl,
                                                 xl, wl, keys, pim, xim, wim);
    int* vt = T.vtab.as<int>(std::max(T.n_vtrg, 1L) * 26);
    unsigned* vm = T.vmask.as<unsigned>(std::max(T.n_vtrg, 1L));
    if (T.n_vtrg > 0) {
      // V-list targets ordered by their pattern of occupied offsets within
      // windows of Morton order (stable: Morton order within a pattern), so
      // that the Hadamard kernels can skip the offsets that are empty for all
      // the parents of a tile while a block's parents stay close in space.
      // Every target is computed independently: the order changes no value.
      // The sort carries each target's Morton rank: vmorton[rank] is the
      // target's position in the pattern order (ranks and positions stay
      // within the same window, so windows of Morton order are contiguous
      // ranges of positions too).
      unsigned long long* key = ctx.t[10].as<unsigned long long>(T.n_vtrg);
      unsigned long long* keys_sorted = ctx.t[13].as<unsigned long long>(T.n_vtrg);
      int* rank_in = ctx.t[12].as<int>(T.n_vtrg);
      int* rank_sorted = ctx.t[14].as<int>(T.n_vtrg);
      ++ctx.n_launch;
      vlist_keys<<<ceil_div(T.n_vtrg, kThreads), kThreads, 0, s>>>(vtrg_morton, T.n_vtrg, coll, n2v, key, rank_in);
      int end_bit = 27;
      while (end_bit < 64 && ((T.n_vtrg - 1) / kVsortWindow) >> (end_bit - 26)) ++end_bit;
      size_t bytes = 0;
      cub::DeviceRadixSort::SortPairs(nullptr, bytes, key, keys_sorted, rank_in, rank_sorted, (int)T.n_vtrg, 0,
                                      end_bit, s);
      void* tmp = ctx.scratch.ensure(bytes);
      cub::DeviceRadixSort::SortPairs(tmp, bytes, key, keys_sorted, rank_in, rank_sorted, (int)T.n_vtrg, 0, end_bit,
                                      s);
      int* vmorton = T.vmorton.as<int>(T.n_vtrg);
      ++ctx.n_launch;
      vlist_order<<<ceil_div(T.n_vtrg, kThreads), kThreads, 0, s>>>(vtrg_morton, rank_sorted, keys_sorted, T.n_vtrg, coll,
                                                                    n2v, T.vtrg.as<int>(N), vmorton, vm, vt);
      T.vtiles_valid = false;
    }
  }
  // 10. point -> leaf and local coordinates, over the leaves with points
  {
    double* sx = T.sx.as<double>(std::max(T.n_src, 1L));
    double* sy = T.sy.as<double>(std::max(T.n_src, 1L));
    double* sz = T.sz.as<double>(std::max(T.n_src, 1L));
    double* tx = T.tx.as<double>(std::max(T.n_trg, 1L));
    double* ty = T.ty.as<double>(std::max(T.n_trg, 1L));
    double* tz = T.tz.as<double>(std::max(T.n_trg, 1L));
    int* sl = T.src_leaf.as<int>(std::max(T.n_src, 1L));
    int* tl = T.trg_leaf.as<int>(std::max(T.n_trg, 1L));
    if (T.n_sleaf > 0) {
      ++ctx.n_launch;
      localize<double><<<ceil_div(T.n_sleaf, 4), 128, 0, s>>>(T.sleaf.get<int>(), T.n_sleaf, keys, slo, shi,
                                                             coords_s.get<double>(), sx, sy, sz, sl);
    }
    if (T.n_tleaf > 0) {
      ++ctx.n_launch;
      localize<double><<<ceil_div(T.n_tleaf, 4), 128, 0, s>>>(T.tleaf.get<int>(), T.n_tleaf, keys, tlo, thi,
                                                             coords_t.get<double>(), tx, ty, tz, tl);
    }
  }
  // 11. rows of the parent-child products where enough leaves are empty and
  //     the tree is large enough for the products to outlast their launches
  //     (2M surface points, 38k internal nodes, 62% of the leaves empty: U2U
  //     2.19 -> 1.14 ms, D2D 2.08 -> 1.10; 150k surface points with 2k internal
  //     nodes: U2U 0.127 -> 0.122, D2D 0.101 -> 0.117, and 0.02 for the lists)
  T.up_lists = T.dn_lists = false;
  if (n_int_total >= 4096) {
    const long leaves = N - n_int_total;
    auto lists = [&](const int* lo, const int* hi, DevBuf& rows, DevBuf& counts, DevBuf& mask) {
      int* r = rows.as<int>(8 * n_int_total);
      int* c = counts.as<int>(8 * kMaxDepth);
      unsigned char* m = mask.as<unsigned char>(n_int_total);
      PVFMM_CUDA_CHECK(cudaMemsetAsync(c, 0, 8 * kMaxDepth * sizeof(int), s));
      ++ctx.n_launch;
      child_rows<<<ceil_div(n_int_total, 128), 128, 0, s>>>(lt, n_int_total, int_idx, child0, lo, hi, r, c, m);
    };
    // U2U's products have no padding to pay for: a list at 15% empty leaves
    T.up_lists = T.src_counted && T.n_sleaf < 0.85 * leaves;
    if (T.up_lists) lists(slo, shi, T.up_rows, T.up_counts, T.up_mask);
    T.dn_lists = translate_down_pays(T.n_tleaf, leaves, ctx.ns * ctx.hops.kout);
    if (T.dn_lists) lists(tlo, thi, T.dn_rows, T.dn_counts, T.dn_mask);
  }
  PVFMM_CUDA_CHECK(cudaGetLastError());
  T.valid = true;  // the evaluation is queued behind the last kernels
}

}  // namespace pvfmm_b200

// Runs link_nodes on the internal nodes of `levels` (sorted keys per level) in
// arrays followed by guard bands and compares every array, guards included,
// with links found by searching all node keys on the host.  A node whose
// parent is missing is expected at the root, and reported.
static void check_link_nodes(const std::vector<std::vector<pvfmm_b200::MKey>>& levels) {
  using namespace pvfmm_b200;
  constexpr long kGuard = 64;
  LevelTab lt{};
  lt.depth = (int)levels.size();
  long n_int = 0, N = 1;
  for (int d = 0; d < lt.depth; ++d) {
    lt.n[d] = (long)levels[d].size();
    lt.ioff[d] = n_int;
    lt.off[d + 1] = N;
    n_int += lt.n[d];
    N += 8 * lt.n[d];
  }
  lt.off[lt.depth + 1] = N;
  // expected arrays (guards: bytes 0x5a)
  const int g4 = 0x5a5a5a5a;
  std::vector<MKey> keys(N + kGuard, MKey{0x5a5a5a5a5a5a5a5aULL, 0x5a5a5a5au, 0x5a5a5a5au});
  std::vector<unsigned char> leaf(N + kGuard, 0x5a);
  std::vector<int> child0(N + kGuard, g4), parent(N + kGuard, g4), int_idx(n_int + kGuard, g4);
  std::map<std::pair<unsigned long long, unsigned int>, long> where;  // node of a key
  for (long i = 0; i < N; ++i) {
    leaf[i] = 1;
    child0[i] = -1;
    parent[i] = 0;
  }
  keys[0] = make_key(0, 0, 0, 0);
  parent[0] = -1;
  where[{keys[0].hi, keys[0].lo}] = 0;
  bool bad = false;
  for (int d = 0; d < lt.depth; ++d)
    for (long k = 0; k < lt.n[d]; ++k) {
      const MKey& key = levels[d][k];
      const auto it = where.find({key.hi, key.lo});
      const long g = it == where.end() ? 0 : it->second;
      bad = bad || it == where.end();
      leaf[g] = 0;
      child0[g] = (int)(lt.off[d + 1] + 8 * k);
      int_idx[lt.ioff[d] + k] = (int)g;
      unsigned int X, Y, Z, dd;
      decode_key(key, X, Y, Z, dd);
      const unsigned int w = kTwo30 >> (d + 1);
      for (int c = 0; c < 8; ++c) {
        const long i = lt.off[d + 1] + 8 * k + c;
        keys[i] = make_key(X + (c & 1) * w, Y + (c >> 1 & 1) * w, Z + (c >> 2) * w, d + 1);
        parent[i] = (int)g;
        where[{keys[i].hi, keys[i].lo}] = i;
      }
    }
  DevBuf b[7];
  try {
    MKey* S = b[0].as<MKey>(n_int);
    MKey* dk = b[1].as<MKey>(keys.size());
    unsigned char* dl = b[2].as<unsigned char>(leaf.size());
    int* dc = b[3].as<int>(child0.size());
    int* dp = b[4].as<int>(parent.size());
    int* di = b[5].as<int>(int_idx.size());
    int* db = b[6].as<int>(1);
    for (int d = 0; d < lt.depth; ++d) {
      lt.S[d] = S + lt.ioff[d];
      PVFMM_CUDA_CHECK(cudaMemcpy(S + lt.ioff[d], levels[d].data(), lt.n[d] * sizeof(MKey), cudaMemcpyHostToDevice));
    }
    PVFMM_CUDA_CHECK(cudaMemset(dk, 0x5a, keys.size() * sizeof(MKey)));
    PVFMM_CUDA_CHECK(cudaMemset(dl, 0x5a, leaf.size()));
    PVFMM_CUDA_CHECK(cudaMemset(dl, 1, N));
    PVFMM_CUDA_CHECK(cudaMemset(dc, 0x5a, child0.size() * sizeof(int)));
    PVFMM_CUDA_CHECK(cudaMemset(dc, 0xff, N * sizeof(int)));
    PVFMM_CUDA_CHECK(cudaMemset(dp, 0x5a, parent.size() * sizeof(int)));
    PVFMM_CUDA_CHECK(cudaMemset(dp, 0, N * sizeof(int)));
    PVFMM_CUDA_CHECK(cudaMemset(di, 0x5a, int_idx.size() * sizeof(int)));
    PVFMM_CUDA_CHECK(cudaMemset(db, 0, sizeof(int)));
    link_nodes<<<ceil_div(n_int, 128), 128>>>(lt, n_int, dk, dl, dc, dp, di, db);
    PVFMM_CUDA_CHECK(cudaGetLastError());
    auto same = [](const auto& want, const auto* dev, const char* name, size_t from) {
      auto got = want;
      const size_t es = sizeof(want[0]);
      PVFMM_CUDA_CHECK(cudaMemcpy(got.data(), dev, want.size() * es, cudaMemcpyDeviceToHost));
      for (size_t i = from; i < want.size(); ++i)
        if (std::memcmp(&got[i], &want[i], es) != 0)
          throw std::runtime_error(std::string("link_nodes: entry ") + std::to_string(i) + " of " + name);
    };
    same(std::vector<int>{bad}, db, "the error word", 0);
    same(keys, dk, "keys", 0);
    same(leaf, dl, "leaf", 0);
    same(child0, dc, "child0", bad ? 1 : 0);  // (nodes without a parent share the root's entry)
    same(parent, dp, "parent", 0);
    same(int_idx, di, "int_idx", 0);
  } catch (...) {
    for (DevBuf& d : b) d.release();
    throw;
  }
  for (DevBuf& d : b) d.release();
}

// Self-check of the bounded writes of the tree build (internal entry point,
// used by the GPU tests; no counterpart in the reference).  Runs scatter_lists
// with `n` nodes in every list against a capacity of `cap` < n, and link_nodes
// on a set that is not closed (n nodes of level 2 whose parents are missing)
// and on closed ones of five levels (about n nodes), in buffers followed by
// guard bands, and checks that what is in range is written as a host
// computation has it and nothing beyond it.  Returns 0 when that holds, 1
// otherwise (message in PVFMMGetLastError).
extern "C" int PVFMMB200CheckBoundedWrites(long n, long cap) {
  using namespace pvfmm_b200;
  constexpr long kGuard = 64;
  void* buf = nullptr;
  try {
    if (n <= 0 || cap < 0 || cap > n || n > (1L << 24)) throw std::runtime_error("bad sizes");
    // records, then 5 lists of cap, node2vsrc (n), 3 offset arrays (n + 1) and
    // the totals, each followed by a guard band
    const long n_list = cap + kGuard, n_map = n + 1 + kGuard;
    const long n_int = 5 * n_list + 4 * n_map + kNodeCounts + kGuard;
    const size_t rec = (size_t)2 * n * sizeof(NodeCounts);
    PVFMM_CUDA_CHECK(cudaMalloc(&buf, rec + n_int * sizeof(int)));
    NodeCounts* nc = (NodeCounts*)buf;
    int* w = (int*)(nc + 2 * n);
    std::vector<NodeCounts> hr(2 * n);
    for (long i = 0; i < n; ++i)
      for (int k = 0; k < kNodeCounts; ++k) {
        hr[i].v[k] = 1;
        hr[n + i].v[k] = (int)i;
      }
    std::vector<int> h(n_int, -7);
    PVFMM_CUDA_CHECK(cudaMemcpy(nc, hr.data(), rec, cudaMemcpyHostToDevice));
    PVFMM_CUDA_CHECK(cudaMemcpy(w, h.data(), n_int * sizeof(int), cudaMemcpyHostToDevice));
    int* map = w + 5 * n_list;
    scatter_lists<<<ceil_div(n, kThreads), kThreads>>>(
        n, cap, nc, nc + n, NodeLists{w, w + n_list, w + 2 * n_list, w + 3 * n_list, w + 4 * n_list}, map, map + n_map,
        map + 2 * n_map, map + 3 * n_map, map + 4 * n_map);
    PVFMM_CUDA_CHECK(cudaGetLastError());
    PVFMM_CUDA_CHECK(cudaMemcpy(h.data(), w, n_int * sizeof(int), cudaMemcpyDeviceToHost));
    for (int l = 0; l < 5; ++l)
      for (long k = 0; k < n_list; ++k)
        if (h[l * n_list + k] != (k < cap ? (int)k : -7))
          throw std::runtime_error("scatter_lists wrote rank " + std::to_string(k) + " wrongly");
    for (int l = 0; l < 4; ++l)
      for (long k = 0; k < n_map; ++k) {
        const int want = l == 0 ? (k < cap ? (int)k : k < n ? -1 : -7) : (k <= n ? (int)k : -7);
        if (h[5 * n_list + l * n_map + k] != want)
          throw std::runtime_error("scatter_lists wrote entry " + std::to_string(k) + " of an offset array wrongly");
      }
    for (long k = 0; k < kNodeCounts + kGuard; ++k)
      if (h[5 * n_list + 4 * n_map + k] != (k < kNodeCounts ? (int)n : -7))
        throw std::runtime_error("scatter_lists wrote the totals wrongly");
    cudaFree(buf);
    buf = nullptr;
    const MKey root = make_key(0, 0, 0, 0), far = make_key(kTwo30 / 2, kTwo30 / 2, kTwo30 / 2, 1);
    check_link_nodes({{root}, {far}, std::vector<MKey>(n, make_key(0, 0, 0, 2))});
    // closed sets: of each level's children every third, and the last two
    std::vector<std::vector<MKey>> levels{{root}};
    while (levels.size() < 5) {
      const unsigned int d = (unsigned int)levels.size(), w = kTwo30 >> d;
      std::vector<MKey> next;
      long i = 0;
      for (const MKey& key : levels.back()) {
        unsigned int X, Y, Z, dd;
        decode_key(key, X, Y, Z, dd);
        for (unsigned int c = 0; c < 8 && (long)next.size() < n; ++c, ++i)
          if (i % 3 == 0 || c >= 6) next.push_back(make_key(X + (c & 1) * w, Y + (c >> 1 & 1) * w, Z + (c >> 2) * w, d));
      }
      levels.push_back(next);
      check_link_nodes(levels);
    }
    set_last_error("");
    return 0;
  } catch (const std::exception& e) {
    if (buf) cudaFree(buf);
    set_last_error(e.what());
    return 1;
  }
}
