// Octree of one system for the far-field surrogate (no PAWAN counterpart:
// PAWAN only has the O(N^2) direct sum).
//
// Build, all on the device:
//   1. bounding cube of the system (bbox_kernel)
//   2. 63-bit Morton codes, 21 bits per axis (morton_kernel), sorted with CUB
//   3. sorted copies of the source records (gather_sorted_kernel)
//   4. top-down adaptive split, one level per launch: a cell with more than
//      `leaf` particles is split into its non-empty octants, found by binary
//      search of the sorted codes (split_count_kernel / split_write_kernel;
//      child offsets from an exclusive scan, so the layout is deterministic)
//   5. per-cell moments about the particle centroid, FP64: the leaves from their
//      particles (leaf_moments_kernel), the other cells from their children's,
//      level by level (parent_moments_kernel); each leaf raises the spread radii
//      of its ancestors (spread_kernel), and cell_data_kernel stores the cells
//   6. per target leaf, the interaction lists (lists_kernel): a source cell
//      whose centroid is at least `near_widths` cube widths beyond the target
//      leaf's bounding sphere, and whose particles are all at least 4 sigma_ij
//      from the leaf's, is far (evaluated from its moments); a leaf that is not
//      far is near (exact pair sum).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pgpu {

constexpr int kTreeLevels = 21;
constexpr int kCellFloats = 72;
constexpr int kListStack = 256;
// Smallest u = rho^2 / sigma_ij^2 between any particle of a far cell and any
// of the target leaf (rho >= 4 sigma_ij).  At 4M particles on the coaxial
// rings, u >= 16 / 25 / 36 give the same sampled error (1.4-1.8e-5) and cost
// 846 / 1022 / 1168 ms per evaluation with 256-particle leaves; without the
// test, 128-particle leaves put cells within ~2 sigma in the far field and the
// error grows to 7.5e-3.
constexpr float kFarAccept = 16.f;  // default of pgpu_surrogate_config.far_u

struct TreeCell {
  int start, end;       // sorted particle range
  int first_child;      // index of the first child cell (children are contiguous), -1 for leaves
  int nchild;
  int level;
  int parent;           // -1 for the root
  unsigned long long prefix;  // Morton prefix of the cell (3 * level bits)
};

// Per-cell data (floats), about the cell's particle centroid c, y = x - c:
//   0-2 c, 3-5 A = sum alpha, 6-14 M[a][b] = sum alpha_a y_b,
//   15-32 Q[a][bc] = sum alpha_a y_b y_c for bc in (00,01,02,11,12,22),
//   33 R = max |y|, 34 w = cube width, 35-37 cube centre, 38 mean sigma^2/2,
//   39 largest sigma^2/2,
//   40-69 T[a][bcd] = sum alpha_a y_b y_c y_d for bcd in (000,001,002,011,012,
//   022,111,112,122,222) (the third moments of the order-3 expansion), 70-71 0.
struct CellData { float v[kCellFloats]; };

__device__ __forceinline__ unsigned f2ord(float f) {
  const unsigned b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// box[0..2] = ordered min, box[3..5] = ordered max (initialised by the host to
// 0xffffffff / 0).
__global__ void bbox_kernel(const float4 *P, int64_t off, int64_t n, unsigned *box) {
  float mn[3] = {3e38f, 3e38f, 3e38f}, mx[3] = {-3e38f, -3e38f, -3e38f};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float4 p = P[off + i];
    mn[0] = fminf(mn[0], p.x); mn[1] = fminf(mn[1], p.y); mn[2] = fminf(mn[2], p.z);
    mx[0] = fmaxf(mx[0], p.x); mx[1] = fmaxf(mx[1], p.y); mx[2] = fmaxf(mx[2], p.z);
  }
  for (int o = 16; o > 0; o >>= 1)
    for (int k = 0; k < 3; ++k) {
      mn[k] = fminf(mn[k], __shfl_down_sync(0xffffffffu, mn[k], o));
      mx[k] = fmaxf(mx[k], __shfl_down_sync(0xffffffffu, mx[k], o));
    }
  if ((threadIdx.x & 31) == 0)
    for (int k = 0; k < 3; ++k) {
      atomicMin(&box[k], f2ord(mn[k]));
      atomicMax(&box[3 + k], f2ord(mx[k]));
    }
}

__device__ __forceinline__ unsigned long long spread21(unsigned long long v) {
  v &= 0x1fffffULL;
  v = (v | (v << 32)) & 0x1f00000000ffffULL;
  v = (v | (v << 16)) & 0x1f0000ff0000ffULL;
  v = (v | (v << 8)) & 0x100f00f00f00f00fULL;
  v = (v | (v << 4)) & 0x10c30c30c30c30c3ULL;
  v = (v | (v << 2)) & 0x1249249249249249ULL;
  return v;
}
__device__ __forceinline__ unsigned compact21(unsigned long long v) {
  v &= 0x1249249249249249ULL;
  v = (v ^ (v >> 2)) & 0x10c30c30c30c30c3ULL;
  v = (v ^ (v >> 4)) & 0x100f00f00f00f00fULL;
  v = (v ^ (v >> 8)) & 0x1f0000ff0000ffULL;
  v = (v ^ (v >> 16)) & 0x1f00000000ffffULL;
  v = (v ^ (v >> 32)) & 0x1fffffULL;
  return (unsigned)v;
}

// geo[0..2] = cube origin, geo[3] = cube edge.
__global__ void morton_kernel(const float4 *P, int64_t off, int64_t n, const float *geo, unsigned long long *code,
                              int *idx) {
  const float s = (float)(1 << 21) / geo[3];
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float4 p = P[off + i];
    const unsigned long long ix = (unsigned long long)min(max((p.x - geo[0]) * s, 0.f), 2097151.f);
    const unsigned long long iy = (unsigned long long)min(max((p.y - geo[1]) * s, 0.f), 2097151.f);
    const unsigned long long iz = (unsigned long long)min(max((p.z - geo[2]) * s, 0.f), 2097151.f);
    code[i] = spread21(ix) | (spread21(iy) << 1) | (spread21(iz) << 2);
    idx[i] = (int)i;
  }
}

__global__ void gather_sorted_kernel(const float4 *P, const float4 *Q, int64_t off, int64_t n, const int *idx,
                                     float4 *Ps, float4 *Qs) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int j = idx[i];
    Ps[i] = P[off + j];
    Qs[i] = Q[off + j];
  }
}

// First index in [lo, hi) whose code >> shift is >= key.
__device__ __forceinline__ int lower_bound_prefix(const unsigned long long *code, int lo, int hi, int shift,
                                                  unsigned long long key) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if ((code[mid] >> shift) < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ bool splittable(const TreeCell &c, int leaf) {
  return c.end - c.start > leaf && c.level < kTreeLevels;
}

// The octants of every cell of the frontier [f0, f1), eight threads per cell:
// thread o finds where octant o ends, so the searches of a cell run side by
// side (the first levels are a handful of cells, and eight searches one after
// another took 60 us of latency per level).  Returns the octant's particle
// range, and in `mask` the non-empty octants of the cell.
__device__ __forceinline__ int2 octant_range(const TreeCell &c, int o, int leaf, const unsigned long long *code,
                                             unsigned &mask) {
  int lo = c.start, hi = c.start;
  const bool split = splittable(c, leaf);
  if (split)
    hi = lower_bound_prefix(code, c.start, c.end, 3 * (kTreeLevels - c.level - 1),
                            (c.prefix << 3) + (unsigned long long)(o + 1));
  const int prev = __shfl_up_sync(0xffffffffu, hi, 1, 8);
  if (split && o > 0) lo = prev;
  mask = (__ballot_sync(0xffffffffu, hi > lo) >> (threadIdx.x & 24)) & 0xffu;
  return make_int2(lo, hi);
}

__global__ void split_count_kernel(const TreeCell *cells, int f0, int f1, const unsigned long long *code, int leaf,
                                   int *nchild) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, i = f0 + (t >> 3), o = t & 7;
  const TreeCell c = cells[min(i, f1 - 1)];
  unsigned mask;
  octant_range(c, o, leaf, code, mask);
  if (i < f1 && o == 0) nchild[i - f0] = __popc(mask);
}

// Writes the children of every frontier cell at base + offs[i] (exclusive scan of nchild).
__global__ void split_write_kernel(TreeCell *cells, int f0, int f1, const unsigned long long *code, int leaf,
                                   const int *offs, int base) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, i = f0 + (t >> 3), o = t & 7;
  const TreeCell c = cells[min(i, f1 - 1)];
  unsigned mask;
  const int2 r = octant_range(c, o, leaf, code, mask);
  if (i >= f1) return;
  const int w = base + offs[i - f0];
  if (r.y > r.x) {
    TreeCell ch;
    ch.start = r.x; ch.end = r.y; ch.first_child = -1; ch.nchild = 0; ch.level = c.level + 1; ch.parent = i;
    ch.prefix = (c.prefix << 3) | (unsigned long long)o;
    cells[w + __popc(mask & ((1u << o) - 1u))] = ch;
  }
  if (o == 0) {
    cells[i].first_child = mask ? w : -1;
    cells[i].nchild = __popc(mask);
  }
}

// FP64 sums of a cell: particle positions, strength and sigma^2/2, the
// moments about the centroid in the order of CellData (M 9, Q 18, T 30), the
// spread radius (bits of a float, for atomicMax) and the largest sigma^2/2.
// T only for expansions of order 3 (nm = kMoments), else nm = kMoments2.
constexpr int kMoments = 57, kMoments2 = 27;
struct CellSums {
  double x[3], a[3], h;
  double m[kMoments];
  unsigned spread;
  float hmax;
};

// What the interaction lists read of a cell, in one place.
struct TreeNode {
  float c[3], R;  // centroid, spread radius
  float w, H;     // cube width, largest sigma^2/2
  int start, end;
  int first_child, nchild;
  int pad[2];
};

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// A leaf is one warp's work, four warps per CTA.  Only leaves at the last level
// hold more than the leaf size (at most 512): particles that no cube separates,
// any number of them.  Those above kWarpLeaf take a CTA of kLeafWarps warps in a
// launch of their own, made when the tree has that level (100,000 particles in
// one point of 300,000: tree 22.8 ms with one warp for them and their 21
// ancestors in turn).
constexpr int kWarpLeaf = 1024, kLeafWarps = 8, kLeafGrid = 1024;

// Sum and maximum over the W warps of a leaf; all threads get the sum in the
// same order.
template <int W> __device__ __forceinline__ double leaf_sum_d(double v, double *red) {
  v = warp_sum_d(v);
  if constexpr (W > 1) {
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.0;
#pragma unroll
    for (int k = 0; k < W; ++k) v += red[k];
  }
  return v;
}
template <int W> __device__ __forceinline__ float leaf_max_f(float v, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if constexpr (W > 1) {
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < W; ++k) v = fmaxf(v, (float)red[k]);
  }
  return v;
}

template <int NM, int W>
__device__ __forceinline__ void leaf_moments(int ci, int start, int end, const float4 *Ps, const float4 *Qs,
                                             CellSums *out, double *red) {
  const int t = threadIdx.x % (32 * W);
  double s[7] = {0, 0, 0, 0, 0, 0, 0};
  float H = 0.f;
  for (int i = start + t; i < end; i += 32 * W) {
    const float4 p = Ps[i], q = Qs[i];
    s[0] += p.x; s[1] += p.y; s[2] += p.z; s[3] += q.x; s[4] += q.y; s[5] += q.z; s[6] += p.w;
    H = fmaxf(H, p.w);
  }
#pragma unroll
  for (int k = 0; k < 7; ++k) s[k] = leaf_sum_d<W>(s[k], red);
  const double cnt = (double)(end - start);
  const double cx = s[0] / cnt, cy = s[1] / cnt, cz = s[2] / cnt;
  double m[NM];
#pragma unroll
  for (int k = 0; k < NM; ++k) m[k] = 0.0;
  float R = 0.f;
  for (int i = start + t; i < end; i += 32 * W) {
    const float4 p = Ps[i], q = Qs[i];
    const double y[3] = {p.x - cx, p.y - cy, p.z - cz};
    const double a[3] = {q.x, q.y, q.z};
    R = fmaxf(R, (float)sqrt(y[0] * y[0] + y[1] * y[1] + y[2] * y[2]));
#pragma unroll
    for (int aa = 0; aa < 3; ++aa) {
      int k2 = 9 + 6 * aa, k3 = 27 + 10 * aa;
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const double ab = a[aa] * y[b];
        m[3 * aa + b] += ab;
#pragma unroll
        for (int c = b; c < 3; ++c) {
          const double abc = ab * y[c];
          m[k2++] += abc;
          if constexpr (NM > kMoments2) {
#pragma unroll
            for (int d = c; d < 3; ++d) m[k3++] += abc * y[d];
          }
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < NM; ++k) m[k] = leaf_sum_d<W>(m[k], red);
  R = leaf_max_f<W>(R, red);
  H = leaf_max_f<W>(H, red);
  if (t == 0) {
    CellSums &c = out[ci];
#pragma unroll
    for (int k = 0; k < 3; ++k) { c.x[k] = s[k]; c.a[k] = s[3 + k]; }
    c.h = s[6];
#pragma unroll
    for (int k = 0; k < NM; ++k) c.m[k] = m[k];
    c.spread = __float_as_uint(R);
    c.hmax = H;
  }
}

template <int NM>
__global__ void __launch_bounds__(128) leaf_moments_kernel(const TreeCell *cells, const int *leaves, int nleaves,
                                                           const float4 *Ps, const float4 *Qs, CellSums *out) {
  const int li = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (li >= nleaves) return;
  const int ci = leaves[li], start = cells[ci].start, end = cells[ci].end;
  if (end - start <= kWarpLeaf) leaf_moments<NM, 1>(ci, start, end, Ps, Qs, out, nullptr);
}
// The leaves above kWarpLeaf among the cells [c0, c1) of the last level.
template <int NM>
__global__ void __launch_bounds__(32 * kLeafWarps) big_leaf_moments_kernel(const TreeCell *cells, int c0, int c1,
                                                                           const float4 *Ps, const float4 *Qs,
                                                                           CellSums *out) {
  __shared__ double red[kLeafWarps];
  for (int ci = c0 + blockIdx.x; ci < c1; ci += gridDim.x) {
    const int start = cells[ci].start, end = cells[ci].end;
    if (end - start > kWarpLeaf) leaf_moments<NM, kLeafWarps>(ci, start, end, Ps, Qs, out, red);
  }
}

// Packed index of a symmetric pair (b <= c) and triple.
__device__ __forceinline__ int sym2(int b, int c) {
  if (b > c) { const int t = b; b = c; c = t; }
  return b == 0 ? c : b == 1 ? 2 + c : 5;
}

// The split cells of [f0, f1) from their children, one warp per cell: with
// s = c_child - c and y = y_child + s,
//   M += A s;  Q_bc += M_b s_c + M_c s_b + A s_b s_c;
//   T_bcd += Q_bc s_d + Q_bd s_c + Q_cd s_b + M_b s_c s_d + M_c s_b s_d + M_d s_b s_c + A s_b s_c s_d
// (one strength component at a time).  Lane e forms moments e and 32 + e.
__global__ void __launch_bounds__(128) parent_moments_kernel(const TreeCell *cells, int f0, int f1, int nm,
                                                             CellSums *sums) {
  const int lane = threadIdx.x & 31;
  const int ci = f0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (ci >= f1) return;
  const TreeCell c = cells[ci];
  if (c.nchild == 0) return;
  double x[3] = {0, 0, 0}, a[3] = {0, 0, 0}, h = 0;
  float H = 0.f;
  for (int k = 0; k < c.nchild; ++k) {
    const CellSums &ch = sums[c.first_child + k];
    for (int m = 0; m < 3; ++m) { x[m] += ch.x[m]; a[m] += ch.a[m]; }
    h += ch.h;
    H = fmaxf(H, ch.hmax);
  }
  const double cnt = (double)(c.end - c.start);
  for (int e = lane; e < nm; e += 32) {
    // strength component and indices of moment e
    int aa, b, cc = -1, d = -1;
    if (e < 9) {
      aa = e / 3; b = e % 3;
    } else if (e < 27) {
      aa = (e - 9) / 6;
      const int k = (e - 9) % 6;
      b = k < 3 ? 0 : k < 5 ? 1 : 2;
      cc = k < 3 ? k : k < 5 ? k - 2 : 2;
    } else {
      aa = (e - 27) / 10;
      const int k = (e - 27) % 10;
      b = k < 6 ? 0 : k < 9 ? 1 : 2;
      cc = k < 3 ? 0 : k < 5 ? 1 : k < 6 ? 2 : k < 8 ? 1 : 2;
      d = k < 3 ? k : k < 5 ? k - 2 : k < 6 ? 2 : k < 8 ? k - 5 : 2;
    }
    double v = 0.0;
    for (int k = 0; k < c.nchild; ++k) {
      const int chi = c.first_child + k;
      const CellSums &ch = sums[chi];
      const double n = (double)(cells[chi].end - cells[chi].start);
      const double sb = ch.x[b] / n - x[b] / cnt;
      const double A = ch.a[aa];
      if (cc < 0) {
        v += ch.m[e] + A * sb;
      } else {
        const double sc = ch.x[cc] / n - x[cc] / cnt;
        const double Mb = ch.m[3 * aa + b], Mc = ch.m[3 * aa + cc];
        if (d < 0) {
          v += ch.m[e] + Mb * sc + Mc * sb + A * sb * sc;
        } else {
          const double sd = ch.x[d] / n - x[d] / cnt;
          const double *Q = ch.m + 9 + 6 * aa;
          v += ch.m[e] + Q[sym2(b, cc)] * sd + Q[sym2(b, d)] * sc + Q[sym2(cc, d)] * sb + Mb * sc * sd +
               Mc * sb * sd + ch.m[3 * aa + d] * sb * sc + A * sb * sc * sd;
        }
      }
    }
    sums[ci].m[e] = v;
  }
  if (lane == 0) {
    CellSums &o = sums[ci];
    for (int m = 0; m < 3; ++m) { o.x[m] = x[m]; o.a[m] = a[m]; }
    o.h = h;
    o.hmax = H;
    o.spread = 0u;
  }
}

// Spread radii of the split cells: every leaf takes its particles' largest
// distance from each ancestor's centroid; the large ones with a CTA per ancestor
// (blockIdx.y).
template <int W>
__device__ __forceinline__ void leaf_spread(const TreeCell *cells, const TreeCell &l, int ci, const float4 *Ps,
                                            CellSums *sums, double *red) {
  const int t = threadIdx.x % (32 * W);
  const double cnt = (double)(cells[ci].end - cells[ci].start);
  const double cx = sums[ci].x[0] / cnt, cy = sums[ci].x[1] / cnt, cz = sums[ci].x[2] / cnt;
  float R = 0.f;
  for (int i = l.start + t; i < l.end; i += 32 * W) {
    const float4 p = Ps[i];
    const double y[3] = {p.x - cx, p.y - cy, p.z - cz};
    R = fmaxf(R, (float)sqrt(y[0] * y[0] + y[1] * y[1] + y[2] * y[2]));
  }
  R = leaf_max_f<W>(R, red);
  // non-negative floats order as their bits
  if (t == 0) atomicMax(&sums[ci].spread, __float_as_uint(R));
}
__global__ void __launch_bounds__(128) spread_kernel(const TreeCell *cells, const int *leaves, int nleaves,
                                                     const float4 *Ps, CellSums *sums) {
  const int li = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (li >= nleaves) return;
  const TreeCell l = cells[leaves[li]];
  if (l.end - l.start > kWarpLeaf) return;
  for (int ci = l.parent; ci >= 0; ci = cells[ci].parent) leaf_spread<1>(cells, l, ci, Ps, sums, nullptr);
}
__global__ void __launch_bounds__(32 * kLeafWarps) big_spread_kernel(const TreeCell *cells, int c0, int c1,
                                                                     const float4 *Ps, CellSums *sums) {
  __shared__ double red[kLeafWarps];
  for (int k = c0 + blockIdx.x; k < c1; k += gridDim.x) {
    const TreeCell l = cells[k];
    if (l.end - l.start <= kWarpLeaf) continue;
    int ci = l.parent;
    for (int up = 0; up < (int)blockIdx.y; ++up) ci = cells[ci].parent;
    leaf_spread<kLeafWarps>(cells, l, ci, Ps, sums, red);
  }
}

__global__ void cell_data_kernel(const TreeCell *cells, int ncells, int nm, const CellSums *sums, const float *geo,
                                 CellData *out, TreeNode *nodes) {
  const int ci = blockIdx.x * blockDim.x + threadIdx.x;
  if (ci >= ncells) return;
  const TreeCell c = cells[ci];
  const CellSums &s = sums[ci];
  const double cnt = (double)(c.end - c.start);
  CellData &d = out[ci];
  TreeNode n;
  for (int m = 0; m < 3; ++m) {
    d.v[m] = n.c[m] = (float)(s.x[m] / cnt);
    d.v[3 + m] = (float)s.a[m];
  }
  for (int k = 0; k < 27; ++k) d.v[6 + k] = (float)s.m[k];
  d.v[33] = n.R = __uint_as_float(s.spread);
  const float w = geo[3] / (float)(1u << c.level);
  d.v[34] = n.w = w;
  const unsigned long long pre = c.prefix;
  const unsigned ix = compact21(pre), iy = compact21(pre >> 1), iz = compact21(pre >> 2);
  d.v[35] = geo[0] + (ix + 0.5f) * w;
  d.v[36] = geo[1] + (iy + 0.5f) * w;
  d.v[37] = geo[2] + (iz + 0.5f) * w;
  d.v[38] = (float)(s.h / cnt);
  d.v[39] = n.H = s.hmax;
  if (nm > kMoments2)
    for (int k = 0; k < 30; ++k) d.v[40 + k] = (float)s.m[27 + k];
  d.v[70] = 0.f;
  d.v[71] = 0.f;
  n.start = c.start; n.end = c.end; n.first_child = c.first_child; n.nchild = c.nchild;
  n.pad[0] = n.pad[1] = 0;
  nodes[ci] = n;
}

// Interaction lists of every leaf, one warp per leaf.  pass 0 counts, pass 1
// writes at the offsets of an exclusive scan of the counts.  A cell that is not
// far is opened by testing its children side by side (one dependent load per
// opened cell instead of one per visited cell); the far ones go to the list at
// once, the others to the warp's stack, first child on top, so that near leaves
// come up in sorted order.  Near leaves are emitted as runs of the sorted
// particle order: consecutive near leaves whose ranges touch are merged (children
// are in octant order, which is sorted order, so runs are long).  The stack is
// bounded (kListStack); overflow sets *err, and the caller treats a non-zero
// *err as a failed build.
constexpr int kListWarps = 4;

__global__ void __launch_bounds__(32 * kListWarps) lists_kernel(const TreeNode *nodes, const int *leaves, int nleaves,
                                                                float near_widths, float far_u, int pass, int *far_cnt,
                                                                int *near_cnt, const int *far_off, const int *near_off,
                                                                int *far_list, int2 *near_runs, int *err) {
  // entries: (first child, number of children), or of a near leaf (start, -end)
  __shared__ int2 stacks[kListWarps][kListStack];
  const int lane = threadIdx.x & 31;
  const int li = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (li >= nleaves) return;
  int2 *stack = stacks[threadIdx.x >> 5];
  const TreeNode t = nodes[leaves[li]];
  int sp = 0, nf = 0, nn = 0, run_s = -1, run_e = -1;
  const int fo = pass ? far_off[li] : 0, no = pass ? near_off[li] : 0;
  const TreeNode root = nodes[0];  // holds every leaf: never far
  if (lane == 0) stack[0] = root.nchild ? make_int2(root.first_child, root.nchild) : make_int2(root.start, -root.end);
  sp = 1;
  __syncwarp();
  while (sp > 0) {
    const int2 e = stack[--sp];
    __syncwarp();
    if (e.y < 0) {  // a near leaf
      if (e.x != run_e) {
        if (run_s >= 0) {
          if (pass && lane == 0) near_runs[no + nn] = make_int2(run_s, run_e);
          ++nn;
        }
        run_s = e.x;
      }
      run_e = -e.y;
      continue;
    }
    TreeNode c;
    bool far = false;
    const int ci = e.x + lane;
    if (lane < e.y) {
      c = nodes[ci];
      const bool contains = c.start <= t.start && t.end <= c.end;
      const float dx = c.c[0] - t.c[0], dy = c.c[1] - t.c[1], dz = c.c[2] - t.c[2];
      const float d = sqrtf(dx * dx + dy * dy + dz * dz) - t.R;
      // far: beyond near_widths cube widths, and every pair of the two cells at
      // u = rho^2 / sigma_ij^2 >= far_u, so that the Gaussian regularisation
      // the singular-kernel expansion leaves out stays small
      const float gap = d - c.R;
      far = !contains && d >= near_widths * c.w && gap > 0.f && gap * gap >= far_u * (t.H + c.H);
    }
    const unsigned below = (1u << lane) - 1u;
    const unsigned fm = __ballot_sync(0xffffffffu, far);
    const unsigned nm = __ballot_sync(0xffffffffu, lane < e.y && !far);
    if (far && pass) far_list[fo + nf + __popc(fm & below)] = ci;
    nf += __popc(fm);
    if (sp + __popc(nm) > kListStack) {
      if (lane == 0) atomicExch(err, 1);
      break;
    }
    if (lane < e.y && !far)
      stack[sp + __popc(nm) - 1 - __popc(nm & below)] =
          c.nchild ? make_int2(c.first_child, c.nchild) : make_int2(c.start, -c.end);
    sp += __popc(nm);
    __syncwarp();
  }
  if (run_s >= 0) {
    if (pass && lane == 0) near_runs[no + nn] = make_int2(run_s, run_e);
    ++nn;
  }
  if (!pass && lane == 0) {
    far_cnt[li] = nf;
    near_cnt[li] = nn;
  }
}

__global__ void leaf_flags_kernel(const TreeCell *cells, int ncells, int *flag) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ncells) flag[i] = cells[i].nchild == 0;
}
__global__ void positive_flags_kernel(const int *cnt, int n, int *flag) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) flag[i] = cnt[i] > 0;
}
__global__ void leaf_scatter_kernel(const int *flag, const int *pos, int ncells, int *leaves) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ncells && flag[i]) leaves[pos[i]] = i;
}

}  // namespace pgpu
