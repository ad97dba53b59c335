// Device kernels of the B200 vortex-particle path.
//
//   pair_kernel     all-pairs velocity / stretching / diffusion rates
//                   (PAWAN __parallel::interact, src/interaction/parallel.cpp:14-86,
//                   per-pair INTERACT, interaction_utils.h:523-576)
//   stage_kernel    RK3 / RK4 / Euler stage updates on the FP64 state, fused with
//                   the reduction of the per-chunk partial rates and the repack of
//                   the next stage's source records (src/integration/rk4.cpp:12-77,
//                   rk3.cpp:12-65, integration.cpp:198-208)
//   diag_pair_kernel / diag_wake_kernel
//                   conserved-quantity diagnostics (interaction.cpp:64-194,
//                   parallel.cpp:140-401)
//   scatter / gather / pack kernels for the host row-major <-> device SoA layout.
//
// Work decomposition of the O(N^2) kernels.  Each system (one PAWAN
// __interaction: all of its particles interact) is cut into target tiles of
// TT = BLOCK * TPT particles and NCH source chunks.  A work item is one
// (system, tile, chunk); items of all systems form one list ordered by
// decreasing system size, and a persistent grid (a few CTAs per SM) takes items
// from an atomic counter.  Every item writes compensated per-target partial
// sums for its chunk to partial[chunk][component][particle] (FP64); the next
// stage kernel adds the NCH partials in a fixed order, so results are
// bit-reproducible run to run.
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "pair_math.cuh"

namespace pgpu {

constexpr int kMaxChunks = 16;
// Sources per compensation group of the FP32 pair kernel: plain FP32 partial
// sums over this many sources, then one error-free two-sum per component.
constexpr int kPairCG = 128;
constexpr int kDiagFields = 23;
// FP64 far regime: u = rho^2 / sigma^2 >= 100, where erfc(sqrt(u/2)) and the
// e^{-u/2} terms of q and F vanish at double precision (the closed form and
// the far limit agree to the last bit from u ~ 90 on).
constexpr double kFarU64 = 100.0;

// One system in the work list (sorted by decreasing work).
struct PlanEntry {
  int64_t off;         // first particle slot of the system
  int64_t n;           // particles in the system (all of them are sources)
  int64_t item_start;  // first work item of the system
  int64_t tiles;       // target tiles
  int64_t chunk;       // sources per chunk (multiple of the source tile)
  int64_t toff;        // targets: particles [off + toff, off + toff + tn) of the system
  int64_t tn;
  // Slices kernel (pair_slices.cuh): items are rows, chunk is the rows per
  // target tile, mult the step of their order; the sentinel's chunk is the
  // rows per CTA.
  int64_t mult;
};

template <typename T> struct PairArgs {
  const v4_t<T> *P;  // (x, y, z, sigma^2/2)
  const v4_t<T> *Q;  // (alpha, volume)
  double *partial;   // [nch][6][cap]
  const PlanEntry *plan;
  int nsys;
  int nch;
  int64_t cap;
  T nu2;  // 2 nu
  unsigned int *counters;  // [0] next item, [1] finished CTAs
  unsigned long long *nfull;  // accumulated count of full-formula pairs
  // Bounding boxes of the source records in blocks of kBoxGran slots
  // (box_kernel): box[2b] = (min x, min y, min z, max sigma^2/2), box[2b+1] =
  // (max x, max y, max z, 0) over the particles of slots [kBoxGran b,
  // kBoxGran (b + 1)).  Systems start at multiples of kBoxGran, so every
  // source tile is a run of whole blocks.  nullptr: the FP32 kernel reduces
  // each tile's box itself.
  const float4 *box = nullptr;
  // Split positions (FP32C, pgpu_config.split_positions): the FP32 rounding
  // residuals (x - (float)x, y - (float)y, z - (float)z, 0) of every
  // particle, added to the pair differences in tiles with near pairs.
  const float4 *L = nullptr;
  // Slices kernel: targets t of the plan are the particles off + targets[t]
  // of the system, and their sums go to partial rows t (a plan with toff =
  // -off, and cap the number of targets).  nullptr: the particles themselves.
  const int *targets = nullptr;
};

// Slots per precomputed source box (divides every pair-kernel tile).
constexpr int kBoxGran = 64;

// ---------------------------------------------------------------- helpers
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

template <typename T> __device__ __forceinline__ v4_t<T> make_v4(T a, T b, T c, T d);
template <> __device__ __forceinline__ float4 make_v4<float>(float a, float b, float c, float d) {
  return make_float4(a, b, c, d);
}
template <> __device__ __forceinline__ double4 make_v4<double>(double a, double b, double c, double d) {
  return make_double4(a, b, c, d);
}

// Copy one packed record (16 B for FP32, 32 B for FP64) with cp.async.
template <typename T> __device__ __forceinline__ void cp_record(v4_t<T> *dst, const v4_t<T> *src) {
  if constexpr (sizeof(v4_t<T>) == 16) {
    cp_async16(dst, src);
  } else {
    cp_async16(dst, src);
    cp_async16(reinterpret_cast<char *>(dst) + 16, reinterpret_cast<const char *>(src) + 16);
  }
}

// A padding source: far away, zero strength, zero volume.  Every term it adds
// is an exact zero and no term overflows (rho^2 ~ 3e36 < FLT_MAX).
template <typename T> __device__ __forceinline__ v4_t<T> pad_P() { return make_v4<T>(T(1e18), T(1e18), T(1e18), T(1)); }
template <typename T> __device__ __forceinline__ v4_t<T> pad_Q() { return make_v4<T>(T(0), T(0), T(0), T(0)); }

__device__ __forceinline__ int find_plan(const PlanEntry *plan, int nsys, int64_t item) {
  int lo = 0, hi = nsys - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (plan[mid].item_start <= item) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Persistent CTA item loop shared by the O(N^2) kernels.  Returns false when
// the list is exhausted; the last CTA to leave resets the counters so the
// kernel can be relaunched (or replayed from a CUDA graph) with no memset.
__device__ __forceinline__ bool next_item(unsigned int *counters, int64_t total, int64_t &item, int *s_item) {
  __syncthreads();
  if (threadIdx.x == 0) *s_item = (int)atomicAdd(&counters[0], 1u);
  __syncthreads();
  item = *s_item;
  if (item < total) return true;
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned done = atomicAdd(&counters[1], 1u);
    if (done == gridDim.x - 1) {
      counters[0] = 0u;
      counters[1] = 0u;
      __threadfence();
    }
  }
  return false;
}

// ---------------------------------------------------------------- pair kernel
// Axis-aligned box of points held by the lanes of a warp, with the largest
// sigma^2/2 among them; after reduce() every lane holds the warp's box.
struct WarpBox {
  float lo[3], hi[3], hs;
  __device__ __forceinline__ void init() {
#pragma unroll
    for (int m = 0; m < 3; ++m) { lo[m] = 3.0e38f; hi[m] = -3.0e38f; }
    hs = 0.f;
  }
  __device__ __forceinline__ void add(float x, float y, float z, float h) {
    lo[0] = fminf(lo[0], x); hi[0] = fmaxf(hi[0], x);
    lo[1] = fminf(lo[1], y); hi[1] = fmaxf(hi[1], y);
    lo[2] = fminf(lo[2], z); hi[2] = fmaxf(hi[2], z);
    hs = fmaxf(hs, h);
  }
  // A box of FP64 points rounded to FP32, widened by more than the rounding:
  // without it, cores next to each other far from the origin could be one FP32
  // step (1 at a coordinate of 1e7) apart and pass for far.  Once per box:
  // rounding keeps the order, so the smallest rounded value is that of the
  // smallest point (widening every point cost the vorticity field of 30,000
  // particles 5%).
  __device__ __forceinline__ void widen() {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      lo[m] = fmaf(fabsf(lo[m]), -0x1p-22f, lo[m]);
      hi[m] = fmaf(fabsf(hi[m]), 0x1p-22f, hi[m]);
    }
    hs = fmaf(hs, 0x1p-22f, hs);
  }
  __device__ __forceinline__ void reduce() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        lo[m] = fminf(lo[m], __shfl_xor_sync(0xffffffffu, lo[m], o));
        hi[m] = fmaxf(hi[m], __shfl_xor_sync(0xffffffffu, hi[m], o));
      }
      hs = fmaxf(hs, __shfl_xor_sync(0xffffffffu, hs, o));
    }
  }
};

// True when every (target, source) pair of the two boxes has u = r^2 /
// (hs_t + hs_s) >= kFarU: the squared gap between the boxes is a lower bound
// of every pair's r^2.  A zero gap (touching or overlapping boxes, coincident
// particles) is never far.
__device__ __forceinline__ bool all_far(const WarpBox &t, const WarpBox &s, float far_u = kFarU) {
  float d2 = 0.f;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const float gap = fmaxf(fmaxf(s.lo[m] - t.hi[m], t.lo[m] - s.hi[m]), 0.f);
    d2 = fmaf(gap, gap, d2);
  }
  return d2 > 0.f && d2 >= far_u * (t.hs + s.hs);
}

// BLOCK threads, TPT targets per thread, TILE sources per shared-memory tile
// (TILE == BLOCK: each thread stages one record), CG sources per compensation
// group (plain FP32 partial sums over CG sources, then an error-free two-sum
// into the per-target (hi, lo) accumulators).
// This generic body serves the asked-for and tuned shapes of the FP64 mode and
// of both modes of the high-order kernel (KER = kHighOrder: every pair takes
// pair_terms_ho, which has no far regime to skip), whose default is the row list
// (pair_slices.cuh, pair_slices64.cuh); the FP32 Gaussian mode uses
// pair_body_f32 (pair_f32.cuh), the same decomposition with packed FP32.
template <typename T, int BLOCK, int TPT, int CG, int KER>
__device__ __forceinline__ void pair_body_generic(const PairArgs<T> &a) {
  // Gaussian kernel: tiles whose sources are all far from the warp's targets
  // take the far limit with no per-pair test (u >= 50 in FP32, u >= 100 in
  // FP64, where the limit equals the closed form to the precision).  The
  // boxes are kept in FP32: a pair misjudged by their rounding sits at
  // u = 100 (1 - 1e-6) or so, where the far limit is still exact in FP64.
  constexpr bool kTiled = KER == kGaussian;
  constexpr float kTileFarU = sizeof(T) == 4 ? kFarU : (float)kFarU64;
  // Stretching q (a_t x a_s): summed as alpha_t x (sum q alpha_s) per
  // compensation group, except for the FP32 high-order kernel, which forms
  // a_t x a_s per pair.  Along a vortex tube a_t and the group sum are nearly
  // parallel, so the cross product of the sum cancels and keeps the sum's
  // FP32 rounding; the high-order q is ~9x larger than the Gaussian one near
  // rho = 0, which lifts that error to ~1e-5 of max |dalpha| on a ring.
  constexpr bool kPairCross = sizeof(T) == 4 && KER == kHighOrder;
  constexpr int TILE = BLOCK;
  constexpr int TT = BLOCK * TPT;
  static_assert(TILE % CG == 0, "compensation group must divide the tile");
  __shared__ __align__(16) v4_t<T> sP[2][TILE];
  __shared__ __align__(16) v4_t<T> sQ[2][TILE];
  // far tiles: n_s = (x_s - ref) x alpha_s, ref the tile's first source (as in
  // the FP32 far loop, pair_f32.cuh): alpha_s x d = alpha_s x X' + n_s with
  // X' = x_t - ref, so the velocity is (sum q alpha_s) x X' + sum q n_s and
  // alpha_t . w = alpha_s . (X' x alpha_t) + n_s . alpha_t
  __shared__ __align__(16) v4_t<T> sN[kTiled ? TILE : 1];
  __shared__ int s_item;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int64_t total = a.plan[a.nsys].item_start;
  int64_t item;
  while (next_item(a.counters, total, item, &s_item)) {
    const int si = find_plan(a.plan, a.nsys, item);
    const PlanEntry pe = a.plan[si];
    const int64_t local = item - pe.item_start;
    const int64_t tile = local / a.nch;
    const int c = (int)(local - tile * a.nch);
    const int64_t t0 = pe.off + pe.toff + tile * TT;
    const int64_t tend = pe.off + pe.toff + pe.tn;  // end of the targets
    const int64_t s0 = pe.off + (int64_t)c * pe.chunk;
    const int64_t s1 = min(s0 + pe.chunk, pe.off + pe.n);

    T xt[TPT][3], at[TPT][3], hst[TPT], vt[TPT], h50[TPT];
    T vh[TPT][3], vl[TPT][3], dh[TPT][3], dl[TPT][3];
    unsigned nfull = 0;  // pairs evaluated with the full (non-far) formula, self pairs included
#pragma unroll
    for (int k = 0; k < TPT; ++k) {
      int64_t ti = t0 + tid + k * BLOCK;
      ti = ti < tend ? ti : tend - 1;
      const v4_t<T> p = a.P[ti];
      const v4_t<T> q = a.Q[ti];
      xt[k][0] = p.x; xt[k][1] = p.y; xt[k][2] = p.z; hst[k] = p.w;
      h50[k] = T(kFarU) * p.w;
      at[k][0] = q.x; at[k][1] = q.y; at[k][2] = q.z; vt[k] = q.w;
#pragma unroll
      for (int m = 0; m < 3; ++m) { vh[k][m] = 0; vl[k][m] = 0; dh[k][m] = 0; dl[k][m] = 0; }
    }
    // -3 alpha_t: the far limit's F' = -3 r^5 with the constant folded in
    T at3[TPT][3];
#pragma unroll
    for (int k = 0; k < TPT; ++k) {
#pragma unroll
      for (int m = 0; m < 3; ++m) at3[k][m] = T(-3) * at[k][m];
    }
    // bounding box of this warp's targets and their largest sigma^2/2, for the
    // per-tile all-far test below
    WarpBox tb;
    if constexpr (kTiled) {
      tb.init();
#pragma unroll
      for (int k = 0; k < TPT; ++k) tb.add(xt[k][0], xt[k][1], xt[k][2], hst[k]);
      tb.reduce();
      if constexpr (sizeof(T) == 8) tb.widen();
    }

    // Stage the first tile.
    int buf = 0;
    if (s0 < s1) {
      const int64_t j = s0 + tid;
      if (j < s1) { cp_record<T>(&sP[0][tid], a.P + j); cp_record<T>(&sQ[0][tid], a.Q + j); }
      else { sP[0][tid] = pad_P<T>(); sQ[0][tid] = pad_Q<T>(); }
    }
    cp_async_commit();

    for (int64_t sb = s0; sb < s1; sb += TILE) {
      const int64_t nb = sb + TILE;
      if (nb < s1) {
        const int64_t j = nb + tid;
        if (j < s1) { cp_record<T>(&sP[buf ^ 1][tid], a.P + j); cp_record<T>(&sQ[buf ^ 1][tid], a.Q + j); }
        else { sP[buf ^ 1][tid] = pad_P<T>(); sQ[buf ^ 1][tid] = pad_Q<T>(); }
      }
      cp_async_commit();
      cp_async_wait<1>();
      __syncthreads();

      // Every pair of this warp's targets with this tile's sources is far
      // (u >= kTileFarU) when the boxes are at least sqrt(kTileFarU (hs_t +
      // hs_s)) apart; such tiles take the far limit with no per-pair test.
      // The boxes' distance is a lower bound of every pair's, so a far pair
      // is never misclassified near; a pair within rounding of the threshold
      // may take the far limit, whose dropped terms are below 2e-9 at u = 50
      // (FP32) and below double rounding at u = 100 (FP64).
      bool far_tile = false;
      if constexpr (kTiled) {
        WarpBox sb_box;
        sb_box.init();
        for (int r = lane; r < TILE; r += 32) {
          const v4_t<T> p = sP[buf][r];
          sb_box.add(p.x, p.y, p.z, p.w);
        }
        sb_box.reduce();
        if constexpr (sizeof(T) == 8) sb_box.widen();
        far_tile = all_far(tb, sb_box, kTileFarU);
      }
      // reference point of far tiles and n_s of the source this thread staged
      // (far_tile is uniform over the warp, not over the CTA: every thread
      // stages its n_s, and the barrier below is unconditional)
      T rx = 0, ry = 0, rz = 0;
      if constexpr (kTiled) {
        rx = sP[buf][0].x; ry = sP[buf][0].y; rz = sP[buf][0].z;
        const v4_t<T> p = sP[buf][tid];
        const v4_t<T> q = sQ[buf][tid];
        const T px = p.x - rx, py = p.y - ry, pz = p.z - rz;
        sN[tid] = make_v4<T>(py * q.z - pz * q.y, pz * q.x - px * q.z, px * q.y - py * q.x, T(0));
        __syncthreads();
      }

#pragma unroll 1
      for (int g = 0; g < TILE; g += CG) {
        T sv[TPT][3], sd[TPT][3], sp[TPT][3], sdv[TPT][3];
#pragma unroll
        for (int k = 0; k < TPT; ++k) {
#pragma unroll
          for (int m = 0; m < 3; ++m) { sv[k][m] = 0; sd[k][m] = 0; sp[k][m] = 0; sdv[k][m] = 0; }
        }
        if (far_tile) {
          // B3 = X' x (-3 alpha_t)
          T b3[TPT][3];
#pragma unroll
          for (int k = 0; k < TPT; ++k) {
            const T xr0 = xt[k][0] - rx, xr1 = xt[k][1] - ry, xr2 = xt[k][2] - rz;
            b3[k][0] = xr1 * at3[k][2] - xr2 * at3[k][1];
            b3[k][1] = xr2 * at3[k][0] - xr0 * at3[k][2];
            b3[k][2] = xr0 * at3[k][1] - xr1 * at3[k][0];
          }
#pragma unroll 4
          for (int jj = 0; jj < CG; ++jj) {
            const v4_t<T> p = sP[buf][g + jj];
            const v4_t<T> q = sQ[buf][g + jj];
            const v4_t<T> n = sN[g + jj];
#pragma unroll
            for (int k = 0; k < TPT; ++k) {
              const T dx = xt[k][0] - p.x, dy = xt[k][1] - p.y, dz = xt[k][2] - p.z;
              const T r2 = dx * dx + dy * dy + dz * dz;
              // far limit: q' = r^3, F' = -3 r^5 (the -3 is in at3 and b3), no diffusion
              const T ir = fast_rsqrt(r2);
              const T A = ir * ir;
              const T qq = A * ir;
              sp[k][0] += qq * q.x; sp[k][1] += qq * q.y; sp[k][2] += qq * q.z;
              sv[k][0] += qq * n.x; sv[k][1] += qq * n.y; sv[k][2] += qq * n.z;
              const T fd = (qq * A) * (q.x * b3[k][0] + q.y * b3[k][1] + q.z * b3[k][2] +
                                       n.x * at3[k][0] + n.y * at3[k][1] + n.z * at3[k][2]);
              sd[k][0] += fd * dx; sd[k][1] += fd * dy; sd[k][2] += fd * dz;
            }
          }
        } else {
#pragma unroll 4
        for (int jj = 0; jj < CG; ++jj) {
          const v4_t<T> p = sP[buf][g + jj];
          const v4_t<T> q = sQ[buf][g + jj];
#pragma unroll
          for (int k = 0; k < TPT; ++k) {
            const T dx = xt[k][0] - p.x, dy = xt[k][1] - p.y, dz = xt[k][2] - p.z;
            const T r2 = dx * dx + dy * dy + dz * dz;
            T qq, FF;
            if constexpr (KER == kHighOrder) {
              const PairTerms<T> pt = pair_terms_ho(r2, hst[k] + p.w);
              qq = pt.q; FF = pt.F;
              sdv[k][0] += pt.zd * (vt[k] * q.x - q.w * at[k][0]);
              sdv[k][1] += pt.zd * (vt[k] * q.y - q.w * at[k][1]);
              sdv[k][2] += pt.zd * (vt[k] * q.z - q.w * at[k][2]);
            } else if constexpr (sizeof(T) == 4) {
              // far test r^2 >= 50 (hs_t + hs_s) as one FMA against the
              // target's precomputed 50 hs_t
              const bool near = fmaf(-kFarU, p.w, r2) < h50[k];
              // far limit for every lane: q' = r^3, F' = -3 r^5, no diffusion
              const float ir = fast_rsqrt(r2);
              const float A = ir * ir;
              qq = A * ir;
              FF = -3.0f * qq * A;
              // the full formula only when some lane of the warp needs it:
              // the vote keeps the common all-far case free of divergence
              if (__any_sync(0xffffffffu, near)) {
                if (near) {
                  const PairTerms<float> pt = pair_terms_near(r2, hst[k] + p.w);
                  qq = pt.q; FF = pt.F;
                  // v_t a_s - v_s a_t per pair, so nearly equal strengths cancel
                  // before they are summed (as in DIFFUSION, interaction_utils.h:358-369)
                  sdv[k][0] += pt.zd * (vt[k] * q.x - q.w * at[k][0]);
                  sdv[k][1] += pt.zd * (vt[k] * q.y - q.w * at[k][1]);
                  sdv[k][2] += pt.zd * (vt[k] * q.z - q.w * at[k][2]);
                  nfull += TPT == 1 || t0 + tid + k * BLOCK < tend;
                }
              }
            } else {
              // FP64: for u >= kFarU64 the far limit equals the closed form to
              // double rounding (erfc(sqrt(u/2)) and the e^{-u/2} terms are
              // below 1e-16 of q and F); the closed form runs under a vote
              const T s2 = hst[k] + p.w;
              const bool near = r2 < T(kFarU64) * s2;
              const T ir = fast_rsqrt(r2);
              const T A = ir * ir;
              qq = A * ir;
              FF = T(-3) * qq * A;
              if (__any_sync(0xffffffffu, near)) {
                if (near) {
                  const PairTerms<T> pt = pair_terms(r2, s2, ir, fast_rsqrt(s2));
                  qq = pt.q; FF = pt.F;
                  sdv[k][0] += pt.zd * (vt[k] * q.x - q.w * at[k][0]);
                  sdv[k][1] += pt.zd * (vt[k] * q.y - q.w * at[k][1]);
                  sdv[k][2] += pt.zd * (vt[k] * q.z - q.w * at[k][2]);
                  if constexpr (KER == kGaussian) nfull += TPT == 1 || t0 + tid + k * BLOCK < tend;
                }
              }
            }
            // w = alpha_s x d
            const T wx = q.y * dz - q.z * dy;
            const T wy = q.z * dx - q.x * dz;
            const T wz = q.x * dy - q.y * dx;
            sv[k][0] += qq * wx; sv[k][1] += qq * wy; sv[k][2] += qq * wz;
            // d . (alpha_t x alpha_s) = alpha_t . w
            const T fd = FF * (at[k][0] * wx + at[k][1] * wy + at[k][2] * wz);
            sd[k][0] += fd * dx; sd[k][1] += fd * dy; sd[k][2] += fd * dz;
            if constexpr (kPairCross) {
              // sp holds sum q (alpha_t x alpha_s) itself
              sp[k][0] += qq * (at[k][1] * q.z - at[k][2] * q.y);
              sp[k][1] += qq * (at[k][2] * q.x - at[k][0] * q.z);
              sp[k][2] += qq * (at[k][0] * q.y - at[k][1] * q.x);
            } else {
              sp[k][0] += qq * q.x; sp[k][1] += qq * q.y; sp[k][2] += qq * q.z;
            }
          }
        }
        }
#pragma unroll
        for (int k = 0; k < TPT; ++k) {
          if (far_tile) {
            // velocity = (sum q alpha_s) x X' + sum q n_s
            const T xr0 = xt[k][0] - rx, xr1 = xt[k][1] - ry, xr2 = xt[k][2] - rz;
            const T n0 = sv[k][0], n1 = sv[k][1], n2 = sv[k][2];
            sv[k][0] = sp[k][1] * xr2 - sp[k][2] * xr1 + n0;
            sv[k][1] = sp[k][2] * xr0 - sp[k][0] * xr2 + n1;
            sv[k][2] = sp[k][0] * xr1 - sp[k][1] * xr0 + n2;
          }
          // da = alpha_t x (sum q alpha_s) + sum F (d.c) d + 2 nu sum z (v_t a_s - v_s a_t)
          T cx, cy, cz;
          if constexpr (kPairCross) {
            cx = sp[k][0]; cy = sp[k][1]; cz = sp[k][2];
          } else {
            cx = at[k][1] * sp[k][2] - at[k][2] * sp[k][1];
            cy = at[k][2] * sp[k][0] - at[k][0] * sp[k][2];
            cz = at[k][0] * sp[k][1] - at[k][1] * sp[k][0];
          }
          const T ex = cx + sd[k][0] + a.nu2 * sdv[k][0];
          const T ey = cy + sd[k][1] + a.nu2 * sdv[k][1];
          const T ez = cz + sd[k][2] + a.nu2 * sdv[k][2];
          two_sum_acc(vh[k][0], vl[k][0], sv[k][0]);
          two_sum_acc(vh[k][1], vl[k][1], sv[k][1]);
          two_sum_acc(vh[k][2], vl[k][2], sv[k][2]);
          two_sum_acc(dh[k][0], dl[k][0], ex);
          two_sum_acc(dh[k][1], dl[k][1], ey);
          two_sum_acc(dh[k][2], dl[k][2], ez);
        }
      }
      __syncthreads();
      buf ^= 1;
    }
    cp_async_wait<0>();
    if constexpr (KER == kGaussian) {
      // threads past the end repeat the last target: none of their pairs counts
      const unsigned wsum = __reduce_add_sync(0xffffffffu, TPT > 1 || t0 + tid < tend ? nfull : 0u);
      if ((tid & 31) == 0 && wsum) atomicAdd(a.nfull, (unsigned long long)wsum);
      nfull = 0;
    }

#pragma unroll
    for (int k = 0; k < TPT; ++k) {
      const int64_t ti = t0 + tid + k * BLOCK;
      if (ti < tend) {
        double *o = a.partial + (int64_t)c * 6 * a.cap + ti;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          o[m * a.cap] = ((double)vh[k][m] + (double)vl[k][m]) * kInv4Pi;
          o[(3 + m) * a.cap] = ((double)dh[k][m] + (double)dl[k][m]) * kInv4Pi;
        }
      }
    }
  }
}

}  // namespace pgpu

#include "pair_f32.cuh"
#include "pair_slices.cuh"
#include "pair_slices64.cuh"

namespace pgpu {

// FP64 shapes with one target per thread are held to 128 registers (a few
// bytes of spill), which fits two 256-thread CTAs per SM instead of one: per
// evaluation of the 1M ring 3196 ms instead of 3632 ms (Gaussian) and
// 4505 ms instead of 5743 ms (high-order), both with CUDA's erf and roots.  With more targets per thread the
// same cap spills hundreds of bytes, so those shapes keep the registers they
// need.
template <typename T, int BLOCK, int TPT, int KER>
constexpr int pair_min_blocks() {
  return sizeof(T) == 4 && KER == kGaussian ? pair_f32_min_blocks<BLOCK, TPT>()
         : (sizeof(T) == 8 && TPT == 1) ? (65536 / (BLOCK * 128) > 0 ? 65536 / (BLOCK * 128) : 1)
                                                            : 1;
}

// SPLIT: the FP32 Gaussian body with split positions (PairArgs::L).
template <typename T, int BLOCK, int TPT, int CG, int KER = kGaussian, bool SPLIT = false>
__global__ void __launch_bounds__(BLOCK, (pair_min_blocks<T, BLOCK, TPT, KER>())) pair_kernel(PairArgs<T> a) {
  constexpr int kCG = CG < BLOCK ? CG : BLOCK;  // a group never spans more than one tile
  if constexpr (sizeof(T) == 4 && KER == kGaussian) pair_body_f32<BLOCK, TPT, kCG, SPLIT>(a);
  else pair_body_generic<T, BLOCK, TPT, kCG, KER>(a);
}

// ---------------------------------------------------------------- stage kernel
// FP32 residuals of a position after rounding to FP32: x - (float)x exactly
// (Sterbenz), then rounded to FP32, so (float)x + residual carries ~48 bits.
__device__ __forceinline__ float4 split_low(double x, double y, double z) {
  return make_float4((float)(x - (double)(float)x), (float)(y - (double)(float)y), (float)(z - (double)(float)z), 0.f);
}

struct StageArgs {
  float4 *L = nullptr;  // split-position residuals, rewritten with the records (FP32C, split positions)
  double *x0;          // [6][cap] FP64 state (x, y, z, ax, ay, az) at the step start
  double *acc;         // [6][cap] RK accumulator
  double *rates;       // [6][cap] last evaluated rates (velocity, dalpha)
  const double *sig;   // [cap]
  const double *vol;   // [cap]
  const double *partial;
  void *P;
  void *Q;
  const int64_t *sys_off;  // [nsys + 1] ascending slot offsets (capacity layout)
  const int64_t *sys_n;    // [nsys]
  const int64_t *sys_t;    // [2 nsys] owned particles [sys_t[2s], sys_t[2s+1]) of each system
  int nsys;
  int nch;
  int64_t cap;
  int scheme;  // 0 Euler, 1 RK3, 2 RK4, -1 rates only (solve)
  int stage;
  double dt;
  double vinf[3];  // operator-split uniform inflow, applied after the final stage
  int *flag;       // set to 1 if a non-finite value is produced
};

__device__ __forceinline__ int find_sys(const int64_t *off, int nsys, int64_t i) {
  int lo = 0, hi = nsys - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= i) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Source boxes for the FP32 pair kernel's per-tile all-far test (PairArgs::
// box): one warp per block of kBoxGran slots, over the particles of its
// system (slots past a system's particle count are left out; a block with
// none gets an empty box).  O(N) over the FP32 records, run before every pair
// launch, so appended particles and exchanged records are always covered.
static __global__ void __launch_bounds__(256) box_kernel(const float4 *P, const int64_t *sys_off, const int64_t *sys_n,
                                                  int nsys, int64_t cap, int64_t nblocks, float4 *box) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t b = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); b < nblocks; b += warps) {
    const int64_t s0 = b * kBoxGran;
    const int si = find_sys(sys_off, nsys, s0);
    const int64_t end = min(sys_off[si] + sys_n[si], cap);
    WarpBox w;
    w.init();
#pragma unroll
    for (int k = 0; k < kBoxGran / 32; ++k) {
      const int64_t j = s0 + lane + 32 * k;
      if (j < end) {
        const float4 p = P[j];
        w.add(p.x, p.y, p.z, p.w);
      }
    }
    w.reduce();
    if (lane == 0) {
      box[2 * b] = make_float4(w.lo[0], w.lo[1], w.lo[2], w.hs);
      box[2 * b + 1] = make_float4(w.hi[0], w.hi[1], w.hi[2], 0.f);
    }
  }
}

// One RK stage: the chunk partials summed into the rates, the stage update of
// the FP64 state, and the next stage's source records.  Bound by latency below
// about 1e5 particles and by HBM above: a CTA takes 32 particles with one warp
// per component, so a small system still spreads over the SMs, and the loads
// of four chunks are in flight together.  The components meet in shared memory for the records.
constexpr int kStageParticles = 32;
constexpr int kStageBlock = 6 * kStageParticles;

template <typename T>
__global__ void __launch_bounds__(kStageBlock) stage_kernel(StageArgs a) {
  __shared__ double sy[6][kStageParticles];
  const int m = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t nb = (a.cap + kStageParticles - 1) / kStageParticles;
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const int64_t i = b * kStageParticles + lane;
    bool live = i < a.cap;
    if (live) {
      const int s = find_sys(a.sys_off, a.nsys, i);
      const int64_t li = i - a.sys_off[s];
      live = li < a.sys_n[s] && li >= a.sys_t[2 * s] && li < a.sys_t[2 * s + 1];
    }
    if (live) {
      const int64_t e = m * a.cap + i;
      const double *p = a.partial + e;
      const int64_t step = 6 * a.cap;
      double k = 0.0;
      int c = 0;
      for (; c + 4 <= a.nch; c += 4) {
        const double p0 = p[c * step], p1 = p[(c + 1) * step], p2 = p[(c + 2) * step], p3 = p[(c + 3) * step];
        k += p0;
        k += p1;
        k += p2;
        k += p3;
      }
      for (; c < a.nch; ++c) k += p[c * step];
      a.rates[e] = k;
      if (a.scheme >= 0) {
        const double dt = a.dt, x = a.x0[e];
        double yy;
        bool final_stage = false;
        if (a.scheme == 2) {  // classical RK4
          if (a.stage == 0) { a.acc[e] = k; yy = x + 0.5 * dt * k; }
          else if (a.stage == 1) { a.acc[e] += 2.0 * k; yy = x + 0.5 * dt * k; }
          else if (a.stage == 2) { a.acc[e] += 2.0 * k; yy = x + dt * k; }
          else { yy = x + (dt / 6.0) * (a.acc[e] + k); final_stage = true; }
        } else if (a.scheme == 1) {  // Kutta RK3
          if (a.stage == 0) { a.acc[e] = k; yy = x + 0.5 * dt * k; }
          else if (a.stage == 1) { const double acc = a.acc[e]; yy = x + dt * (2.0 * k - acc); a.acc[e] = acc + 4.0 * k; }
          else { yy = x + (dt / 6.0) * (a.acc[e] + k); final_stage = true; }
        } else {  // explicit Euler
          yy = x + dt * k;
          final_stage = true;
        }
        if (final_stage) {
          if (m < 3) yy += a.vinf[m] * dt;
          a.x0[e] = yy;
        }
        if (!isfinite(yy)) *a.flag = 1;
        sy[m][lane] = yy;
      }
    }
    if (a.scheme < 0) continue;
    __syncthreads();
    if (live) {
      if (m == 0) {
        const double sg = a.sig[i];
        static_cast<v4_t<T> *>(a.P)[i] =
            make_v4<T>((T)sy[0][lane], (T)sy[1][lane], (T)sy[2][lane], (T)(0.5 * sg * sg));
      } else if (m == 1) {
        static_cast<v4_t<T> *>(a.Q)[i] = make_v4<T>((T)sy[3][lane], (T)sy[4][lane], (T)sy[5][lane], (T)a.vol[i]);
      } else if (m == 2 && a.L) {
        a.L[i] = split_low(sy[0][lane], sy[1][lane], sy[2][lane]);
      }
    }
    __syncthreads();
  }
}

// Pack the FP64 state at the step start into the source records (and the
// split-position residuals when L is set).
template <typename T>
__global__ void pack_kernel(const double *x0, const double *sig, const double *vol, void *P, void *Q, float4 *L,
                            int64_t lo, int64_t hi, int64_t cap) {
  for (int64_t i = lo + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < hi; i += (int64_t)gridDim.x * blockDim.x) {
    const double sg = sig[i];
    static_cast<v4_t<T> *>(P)[i] = make_v4<T>((T)x0[i], (T)x0[cap + i], (T)x0[2 * cap + i], (T)(0.5 * sg * sg));
    static_cast<v4_t<T> *>(Q)[i] =
        make_v4<T>((T)x0[3 * cap + i], (T)x0[4 * cap + i], (T)x0[5 * cap + i], (T)vol[i]);
    if (L) L[i] = split_low(x0[i], x0[cap + i], x0[2 * cap + i]);
  }
}

// Host row-major layout <-> SoA.  A CTA takes kIoRows rows through shared
// memory, so that both sides are read and written in whole segments: the
// row-major side may be pinned host memory, mapped (uploads and downloads of a
// few thousand particles need no copy of their own then).
constexpr int kIoRows = 256;

// Row-major (n, 3) positions and strengths, (n) radii and volumes, one after
// another in `stage` -> SoA state at slot offset `off`, and the rows' source
// records (and split-position residuals when L is set).
template <typename T>
__global__ void __launch_bounds__(kIoRows) upload_kernel(const double *stage, int64_t n, int64_t off, int64_t cap,
                                                         double *x0, double *sig, double *vol, void *P, void *Q,
                                                         float4 *L) {
  __shared__ double s[6 * kIoRows];
  for (int64_t b = blockIdx.x * (int64_t)kIoRows; b < n; b += (int64_t)gridDim.x * kIoRows) {
    const int rows = (int)min((int64_t)kIoRows, n - b);
    for (int t = threadIdx.x; t < 3 * rows; t += kIoRows) {
      s[t] = stage[3 * b + t];
      s[3 * kIoRows + t] = stage[3 * n + 3 * b + t];
    }
    __syncthreads();
    if ((int)threadIdx.x < rows) {
      const int64_t j = b + threadIdx.x, i = off + j;
      double y[6];
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        y[m] = s[3 * threadIdx.x + m];
        y[3 + m] = s[3 * kIoRows + 3 * threadIdx.x + m];
      }
#pragma unroll
      for (int m = 0; m < 6; ++m) x0[m * cap + i] = y[m];
      const double sg = stage[6 * n + j], v = stage[7 * n + j];
      sig[i] = sg;
      vol[i] = v;
      static_cast<v4_t<T> *>(P)[i] = make_v4<T>((T)y[0], (T)y[1], (T)y[2], (T)(0.5 * sg * sg));
      static_cast<v4_t<T> *>(Q)[i] = make_v4<T>((T)y[3], (T)y[4], (T)y[5], (T)v);
      if (L) L[i] = split_low(y[0], y[1], y[2]);
    }
    __syncthreads();
  }
}

// SoA [3 parts][cap] (from slot offset `off`) -> row-major (n, 3) x parts, parts
// 1 or 2.
static __global__ void __launch_bounds__(kIoRows) gather_kernel(const double *src, int64_t n, int64_t off, int64_t cap,
                                                                int parts, double *stage) {
  __shared__ double s[6 * kIoRows];
  for (int64_t b = blockIdx.x * (int64_t)kIoRows; b < n; b += (int64_t)gridDim.x * kIoRows) {
    const int rows = (int)min((int64_t)kIoRows, n - b);
    if ((int)threadIdx.x < rows) {
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        s[3 * threadIdx.x + m] = src[m * cap + off + b + threadIdx.x];
        if (parts > 1) s[3 * kIoRows + 3 * threadIdx.x + m] = src[(3 + m) * cap + off + b + threadIdx.x];
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 3 * rows; t += kIoRows) {
      stage[3 * b + t] = s[t];
      if (parts > 1) stage[3 * n + 3 * b + t] = s[3 * kIoRows + t];
    }
    __syncthreads();
  }
}

// Flat PAWAN state vector (per wake [x (maxN x 3) ; alpha (maxN x 3)] at offset
// sum of 6 maxN, __interaction::setStates/getStates, interaction.cpp:337-365,
// wake.cpp:856-893) <-> SoA state.  dir = 0: flat -> SoA, 1: SoA -> flat.
static __global__ void flat_kernel(double *flat, int64_t n, int64_t maxn, int64_t off, int64_t cap, double *soa, int dir) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (dir == 0) {
        soa[m * cap + off + i] = flat[3 * i + m];
        soa[(3 + m) * cap + off + i] = flat[3 * maxn + 3 * i + m];
      } else {
        flat[3 * i + m] = soa[m * cap + off + i];
        flat[3 * maxn + 3 * i + m] = soa[(3 + m) * cap + off + i];
      }
    }
  }
}

// ---------------------------------------------------------------- diagnostics
template <typename T> struct DiagArgs {
  const v4_t<T> *P;
  const v4_t<T> *Q;
  double *partial;  // [nch][6][cap]: components 0..4 = helicity, KE, KEF, enstrophy, enstrophyF row sums
  const PlanEntry *plan;
  int nsys;
  int nch;
  int64_t cap;
  unsigned int *counters;
};

// Quadratic diagnostics: per target t and chunk, sums over sources s != t of
//   helicity  q(rho, s_ts) (x_s - x_t).(a_t x a_s)            (HELICITY, interaction_utils.h:214-242)
//   KE        [(rho^2 + 2 s^2) a_t.a_s + (d.a_t)(d.a_s)] / (16 pi (rho^2 + s^2)^1.5)   (:278-306)
//   KEF       (rho^2 + 1.5 s^2) a_t.a_s / (8 pi (rho^2 + s^2)^1.5)                    (:308-331)
// and, for the high-order kernel only (the Gaussian ENST / ENSTF are zero,
// gaussian.h:69-92), with R = rho^2 + s^2 (ENSTROPHY[F], interaction_utils.h:
// 141-201; ENST / ENSTF, highorder.h:71-95):
//   enstrophy  [(2 rho^4 + 7 s^2 rho^2 + 20 s^4) a_t.a_s
//               - (6 rho^4 + 27 s^2 rho^2 + 21 s^4) (d.a_t)(d.a_s) / R] / (8 pi R^3.5)
//   enstrophyF 15 s^4 a_t.a_s / (8 pi R^3.5)
// All terms are symmetric in (t, s), so each unordered pair is
// evaluated once, from its lower index (sources s > t only), and the row sums
// are doubled: they then equal sums over ordered pairs, PAWAN's 2 x sum over
// unordered pairs.  In FP32 the Gaussian helicity's q takes the far limit
// 1/rho^3 for u >= 50 (as in the rate kernel) and the mid/series terms only
// when some lane of the warp needs them.
template <typename T, int BLOCK, int KER>
__device__ __forceinline__ void diag_body_generic(const DiagArgs<T> &a) {
  __shared__ __align__(16) v4_t<T> sP[BLOCK];
  __shared__ __align__(16) v4_t<T> sQ[BLOCK];
  __shared__ int s_item;
  const int tid = threadIdx.x;
  const int64_t total = a.plan[a.nsys].item_start;
  int64_t item;
  while (next_item(a.counters, total, item, &s_item)) {
    const int si = find_plan(a.plan, a.nsys, item);
    const PlanEntry pe = a.plan[si];
    const int64_t local = item - pe.item_start;
    const int64_t tile = local / a.nch;
    const int c = (int)(local - tile * a.nch);
    const int64_t tend = pe.off + pe.toff + pe.tn;   // end of the (owned) targets
    const int64_t tlo = pe.off + pe.toff + tile * BLOCK;  // first target of the tile
    const int64_t t = min(tlo + tid, tend - 1);
    const bool valid = tlo + tid < tend;
    // sources above the tile's first target only (s > t is tested per pair
    // while a tile can still hold s <= t), up to the end of the system
    const int64_t s0 = max(pe.off + (int64_t)c * pe.chunk, tlo);
    const int64_t s1 = min(pe.off + (int64_t)c * pe.chunk + pe.chunk, pe.off + pe.n);
    const v4_t<T> pt = a.P[t], qt = a.Q[t];
    const T h50 = T(kFarU) * pt.w;
    double h = 0, ke = 0, kef = 0, en = 0, enf = 0;
    for (int64_t sb = s0; sb < s1; sb += BLOCK) {
      __syncthreads();
      const int64_t j = sb + tid;
      if (j < s1) { sP[tid] = a.P[j]; sQ[tid] = a.Q[j]; }
      else { sP[tid] = pad_P<T>(); sQ[tid] = pad_Q<T>(); }
      __syncthreads();
      T hh = 0, kk = 0, kf = 0, ee = 0, ef = 0;
      const int cnt = (int)min((int64_t)BLOCK, s1 - sb);
      const bool diag = sb <= tlo + BLOCK - 1;  // the tile may still see s <= t
      for (int jj = 0; jj < cnt; ++jj) {
        const bool use = !diag || sb + jj > t;
        const v4_t<T> p = sP[jj], q = sQ[jj];
        const T dx = pt.x - p.x, dy = pt.y - p.y, dz = pt.z - p.z;
        const T r2 = dx * dx + dy * dy + dz * dz;
        const T s2 = pt.w + p.w;
        T kq;
        if constexpr (KER == kHighOrder) {
          kq = pair_terms_ho(r2, s2).q;
        } else if constexpr (sizeof(T) == 4) {
          const bool near = fmaf(-kFarU, p.w, r2) < h50;
          const float ir = fast_rsqrt(r2);
          kq = ir * ir * ir;
          if (__any_sync(0xffffffffu, near && use)) {
            if (near && use) kq = pair_terms_near(r2, s2).q;
          }
        } else {
          const bool near = r2 < T(kFarU64) * s2;
          const T ir = fast_rsqrt(r2);
          kq = ir * ir * ir;
          if (__any_sync(0xffffffffu, near && use)) {
            if (near && use) kq = pair_terms(r2, s2, ir, fast_rsqrt(s2)).q;
          }
        }
        const T cx = qt.y * q.z - qt.z * q.y, cy = qt.z * q.x - qt.x * q.z, cz = qt.x * q.y - qt.y * q.x;
        const T aa = qt.x * q.x + qt.y * q.y + qt.z * q.z;
        const T dat = dx * qt.x + dy * qt.y + dz * qt.z;
        const T das = dx * q.x + dy * q.y + dz * q.z;
        const T rs = r2 + s2;
        T ir;
        // the enstrophy terms carry R^-4.5: a refined root keeps their FP32 error at rounding level
        if constexpr (sizeof(T) == 4) ir = KER == kHighOrder ? rsqrt_nr(rs) : fast_rsqrt(rs);
        else ir = fast_rsqrt(rs);
        const T ir3 = ir * ir * ir;
        if (use) {
          hh -= kq * (dx * cx + dy * cy + dz * cz);
          kk += ((r2 + T(2) * s2) * aa + dat * das) * ir3;
          kf += (r2 + T(1.5) * s2) * aa * ir3;
          if constexpr (KER == kHighOrder) {
            const T ir7 = ir3 * ir3 * ir;
            const T r4 = r2 * r2, s4 = s2 * s2, rs2 = r2 * s2;
            const T f1 = T(2) * r4 + T(7) * rs2 + T(20) * s4;
            const T f2 = T(6) * r4 + T(27) * rs2 + T(21) * s4;
            ee += (f1 * aa - f2 * (ir * ir) * (dat * das)) * ir7;
            ef += s4 * aa * ir7;
          }
        }
      }
      h += (double)hh;
      ke += (double)kk;
      kef += (double)kf;
      en += (double)ee;
      enf += (double)ef;
    }
    if (valid) {
      // doubled: each unordered pair was summed once
      double *o = a.partial + (int64_t)c * 6 * a.cap + t;
      o[0] = h * (2.0 * kInv4Pi);
      o[a.cap] = ke * (2.0 * kInv4Pi * 0.25);      // 1/(16 pi)
      o[2 * a.cap] = kef * (2.0 * kInv4Pi * 0.5);  // 1/(8 pi)
      if constexpr (KER == kHighOrder) {
        o[3 * a.cap] = en * (2.0 * kInv4Pi * 0.5);          // 1/(8 pi)
        o[4 * a.cap] = enf * (2.0 * kInv4Pi * 0.5 * 15.0);  // 15/(8 pi)
      }
    }
  }
}

}  // namespace pgpu

#include "diag_f32.cuh"

namespace pgpu {

// The FP32 Gaussian diagnostics take the packed body of diag_f32.cuh.
template <typename T, int BLOCK, int KER = kGaussian>
__global__ void __launch_bounds__(BLOCK) diag_pair_kernel(DiagArgs<T> a) {
  if constexpr (sizeof(T) == 4 && KER == kGaussian) diag_body_f32<BLOCK>(a);
  else diag_body_generic<T, BLOCK, KER>(a);
}

// Vorticity field at every particle, PAWAN's influence() (interaction.cpp:
// 212-260; INFLUENCE and SELFINFLUENCE, interaction_utils.h:626-703):
//   k_t = sum_s zeta(rho_ts, sigma_ts) alpha_s,  the self term s = t included,
//   zeta = exp(-rho^2 / (2 sigma^2)) / (sigma^3 (2 pi)^1.5)   (ZETASIG, gaussian.h:20-23)
//   sigma_ts^2 = (sigma_t^2 + sigma_s^2) / 2.
// Always FP64, from the FP64 state (x0, sig) rather than the mode's source
// records: PAWAN's strength solve (resolve.cpp:12-63) LU-solves a matrix of
// these fields, whose conditioning (~1e6 for its vortex rings) turns FP32
// rounding into percent-level strength errors.  Per target and source chunk,
// row sums go to partial[c][0..2][t]; field_reduce_kernel adds the chunks.
// e^{-u/2} is below the smallest double from u = 1491 on, so a pair at
// u >= 1500 adds exactly zero.  A position, radius or strength that is not a
// number reaches every target, as in the sum without the test.
//
// Bound by the FP64 pipe: about 30 operations per pair of one radius, half of
// them the exponential.  Rows of 32 targets by eight slices (pair_slices.cuh);
// a slice whose box puts every pair at u >= 1510 is left out (three quarters
// of the pairs on a ring of unit radius with sigma = 0.02), and where one
// radius serves the slice, 1/sigma leaves the loop.  30,000 particles: 1.02 ms
// per call against 2.84 ms with a square root, a division and the exponential
// for every pair of 256-target tiles.  The high-order kernel (KER = kHighOrder)
// takes its own ZETASIG (highorder.h:20-24), zeta = 1.875 / (pi sigma^3
// (rho^2/sigma^2 + 1)^3.5) = 1.875 / pi sigma^4 (rho^2 + sigma^2)^-3.5, for
// every pair.
struct FieldArgs {
  const double *x0;   // [6][cap] state
  const double *sig;  // [cap]
  double *partial;    // [nch][6][cap]
  const PlanEntry *plan;
  int nsys;
  int nch;
  int64_t cap;
};

template <int SL> struct FieldStage {
  double2 xy[32 * SL], zh[32 * SL], axy[32 * SL];
  double az[32 * SL];
};

template <int SL, int KER>
__global__ void __launch_bounds__(32 * kSliceWarps) field_kernel(FieldArgs a) {
  constexpr int W = kSliceWarps, S = 32 * SL;
  __shared__ __align__(16) FieldStage<SL> stage[W];
  __shared__ double red[W * 3 * 32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  FieldStage<SL> &st = stage[w];
  const int64_t cap = a.cap;
  const int64_t rpc = a.plan[a.nsys].chunk;
  const int64_t row1 = min((blockIdx.x + 1) * rpc, a.plan[a.nsys].item_start);
  for (int64_t row = blockIdx.x * rpc; row < row1;) {
    const RowRun run = row_run(a.plan, a.nsys, rpc, row, row1);
    const int64_t s1 = run.s1;
    int64_t g = run.g;
    const int64_t ti = min(run.t0 + lane, run.tend - 1);
    const double xt = a.x0[ti], yt = a.x0[cap + ti], zt = a.x0[2 * cap + ti];
    const double hst = 0.5 * a.sig[ti] * a.sig[ti];
    WarpBox tb;
    tb.init();
    tb.add((float)xt, (float)yt, (float)zt, (float)hst);
    reduce_box(tb);
    tb.widen();
    const double hst0 = __shfl_sync(0xffffffffu, hst, 0);
    const bool one_t = __all_sync(0xffffffffu, hst == hst0);
    const bool number_t = __all_sync(0xffffffffu, !isnan(xt + yt + zt + hst));  // the boxes pass over NaN
    double k0 = 0, k1 = 0, k2 = 0;
    for (int r = 0; r < run.nrows; ++r) {
      const int64_t cur = run.pe.off + (g * W + w) * S;
      g += run.pe.mult;
      if (g >= run.pe.chunk) g -= run.pe.chunk;
      if (cur >= s1) continue;
      __syncwarp();
      WarpBox sbox;
      sbox.init();
      bool finite = number_t, one = one_t;
      double hs0 = 0;
#pragma unroll
      for (int j = 0; j < SL; ++j) {
        const int64_t i = min(cur + lane + 32 * j, s1 - 1);  // past the end: the last source again, not summed
        const double x = a.x0[i], y = a.x0[cap + i], z = a.x0[2 * cap + i], sg = a.sig[i], hs = 0.5 * sg * sg;
        const double ax = a.x0[3 * cap + i], ay = a.x0[4 * cap + i], az = a.x0[5 * cap + i];
        const int e = lane + 32 * j;
        st.xy[e] = make_double2(x, y);
        st.zh[e] = make_double2(z, hs);
        st.axy[e] = make_double2(ax, ay);
        st.az[e] = az;
        sbox.add((float)x, (float)y, (float)z, (float)hs);
        if (j == 0) hs0 = __shfl_sync(0xffffffffu, hs, 0);
        finite = finite && isfinite(ax) && isfinite(ay) && isfinite(az) && !isnan(x + y + z + hs);
        one = one && hs == hs0;
      }
      reduce_box(sbox);
      sbox.widen();
      // slices that add exactly zero (a strength that is not finite, or a NaN position or radius, would not)
      if (KER == kGaussian && all_far(tb, sbox, 1510.f) && bounded(tb) && bounded(sbox) &&
          __all_sync(0xffffffffu, finite))
        continue;
      one = __all_sync(0xffffffffu, one);
      __syncwarp();
      const int cnt = (int)min((int64_t)S, s1 - cur);
      if constexpr (KER == kHighOrder) {
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
          const double2 xy = st.xy[j], zh = st.zh[j], axy = st.axy[j];
          const double dx = xt - xy.x, dy = yt - xy.y, dz = zt - zh.x;
          const double s2 = hst + zh.y;
          const double iR = fast_rsqrt(dx * dx + dy * dy + dz * dz + s2);
          const double iR2 = iR * iR;
          const double z = (HighOrder::kZeta * kInv4Pi) * (s2 * s2) * (iR2 * iR2 * iR2 * iR);
          k0 += z * axy.x;
          k1 += z * axy.y;
          k2 += z * st.az[j];
        }
      } else {
        auto sum = [&](auto uniform, double is2, double zk) {
#pragma unroll 4
          for (int j = 0; j < cnt; ++j) {
            const double2 xy = st.xy[j], zh = st.zh[j], axy = st.axy[j];
            const double dx = xt - xy.x, dy = yt - xy.y, dz = zt - zh.x;
            const double r2 = dx * dx + dy * dy + dz * dz;
            const double s2 = hst + zh.y;
            double i2 = is2, c = zk;
            if constexpr (!decltype(uniform)::value) {
              const double is = fast_rsqrt(s2);
              i2 = is * is;
              c = kInv2Pi15 * i2 * is;
            }
            const double z = r2 >= 1500.0 * s2 ? 0.0 : c * exp(-0.5 * (r2 * i2));  // NaN stays NaN
            k0 += z * axy.x;
            k1 += z * axy.y;
            k2 += z * st.az[j];
          }
        };
        if (one) {
          const double is = fast_rsqrt(hst0 + hs0);
          sum(TrueType{}, is * is, kInv2Pi15 * (is * is) * is);
        } else {
          sum(FalseType{}, 0.0, 0.0);
        }
      }
    }
    __syncthreads();  // the previous tile's sums have been read
    red[(w * 3 + 0) * 32 + lane] = k0;
    red[(w * 3 + 1) * 32 + lane] = k1;
    red[(w * 3 + 2) * 32 + lane] = k2;
    __syncthreads();
    row_run_sums<3>(run, red, 1.0, a.partial, cap, a.nch);
    row += run.nrows;
  }
}

// field[m][i] = sum over chunks of partial[c][m][i], m = 0..2.
static __global__ void field_reduce_kernel(const double *partial, int nch, int64_t cap, double *field) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cap; i += (int64_t)gridDim.x * blockDim.x) {
    for (int m = 0; m < 3; ++m) {
      double v = 0.0;
      for (int c = 0; c < nch; ++c) v += partial[((int64_t)c * 6 + m) * cap + i];
      field[m * cap + i] = v;
    }
  }
}

// Per-wake O(N) diagnostics and the reduction of the quadratic row sums, FP64.
// Fields (per CTA partial, summed on the host in CTA order):
//   0-2 sum alpha, 3-5 sum x x alpha, 6-8 sum x x (x x alpha), 9 Zc numerator,
//   10 Zc denominator, 11-13 velocity at the origin (getVi), 14 helicity,
//   15 KE pair sum, 16 KEF pair sum, 17 KE self terms, 18 KEF self terms,
//   19 enstrophy pair sum, 20 enstrophyF pair sum, 21 enstrophy self terms
//   5 |a|^2 / (2 pi s^3), 22 enstrophyF self terms 15 |a|^2 / (8 pi s^3)
//   (ENST(sigma) / ENSTF(sigma), highorder.h:101-110; 19-22 stay zero for the
//   Gaussian kernel, whose ENST / ENSTF are zero).
__device__ __forceinline__ double block_sum(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r += red[i];
  return r;
}

static __global__ void diag_wake_kernel(const double *x0, const double *sig, const double *partial, int nch, int64_t cap,
                                 int64_t lo, int64_t hi, int quad, int ker, double *out) {
  __shared__ double red[32];
  double f[kDiagFields];
#pragma unroll
  for (int m = 0; m < kDiagFields; ++m) f[m] = 0.0;
  for (int64_t i = lo + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < hi; i += (int64_t)gridDim.x * blockDim.x) {
    const double x = x0[i], y = x0[cap + i], z = x0[2 * cap + i];
    const double ax = x0[3 * cap + i], ay = x0[4 * cap + i], az = x0[5 * cap + i];
    f[0] += ax; f[1] += ay; f[2] += az;
    const double cx = y * az - z * ay, cy = z * ax - x * az, cz = x * ay - y * ax;
    f[3] += cx; f[4] += cy; f[5] += cz;
    f[6] += y * cz - z * cy; f[7] += z * cx - x * cz; f[8] += x * cy - y * cx;
    const double om = sqrt(ax * ax + ay * ay + az * az);
    const double rr = x * x + y * y;
    f[9] += om * z * rr;
    f[10] += om * rr;
    // getVi at the origin with the particle's own radius: d = -x
    const double s = sig[i];
    const double r2 = rr + z * z;
    const double q = (ker == kHighOrder ? pair_terms_ho(r2, s * s).q : pair_terms(r2, s * s).q) * kInv4Pi;
    f[11] += q * (ay * (-z) - az * (-y));
    f[12] += q * (az * (-x) - ax * (-z));
    f[13] += q * (ax * (-y) - ay * (-x));
    if (quad) {
      double h = 0, ke = 0, kef = 0;
      for (int c = 0; c < nch; ++c) {
        h += partial[((int64_t)c * 6 + 0) * cap + i];
        ke += partial[((int64_t)c * 6 + 1) * cap + i];
        kef += partial[((int64_t)c * 6 + 2) * cap + i];
      }
      f[14] += h; f[15] += ke; f[16] += kef;
      if (ker == kHighOrder) {
        double en = 0, enf = 0;
        for (int c = 0; c < nch; ++c) {
          en += partial[((int64_t)c * 6 + 3) * cap + i];
          enf += partial[((int64_t)c * 6 + 4) * cap + i];
        }
        f[19] += en; f[20] += enf;
      }
    }
    const double a2 = ax * ax + ay * ay + az * az;
    f[17] += a2 / s * (kInv4Pi * 0.5);    // |a|^2 / (8 pi s)
    f[18] += a2 / s * (kInv4Pi * 0.75);   // 3 |a|^2 / (16 pi s)
    if (ker == kHighOrder) {
      const double is3 = 1.0 / (s * s * s);
      f[21] += a2 * is3 * (kInv4Pi * 10.0);  // 5 |a|^2 / (2 pi s^3)
      f[22] += a2 * is3 * (kInv4Pi * 7.5);   // 15 |a|^2 / (8 pi s^3)
    }
  }
  for (int m = 0; m < kDiagFields; ++m) {
    const double r = block_sum(f[m], red);
    if (threadIdx.x == 0) out[(int64_t)blockIdx.x * kDiagFields + m] = r;
  }
}

// Candidate pairs of PAWAN's particle merge (__wake::merge, wake.cpp:112-159).
// PAWAN merges j into i (i < j) when |x_i - x_j| < 0.125 (r_i + r_j), both
// strengths are non-zero and the strengths are not aligned; its loop is
// sequential (a merge moves x_i and zeroes alpha_j), so the host replays it
// (pgpu_merge).  These kernels find, from the state at entry, every pair with
// i < n_elig, i < j < n, non-zero strengths and
// |x_i - x_j| < reach (r_i + r_j), reach = 0.25, twice PAWAN's, so the host can
// keep using the list while a merged x_i stays within 0.125 (r_i + r_min) of
// where it started.
//
// Search: a uniform grid of cell size h = 2 reach r_max.  merge_keys_kernel
// gives every particle with a non-zero strength its cell key (zero strengths
// get a key above every cell's, so no search finds them); the keys are sorted
// with their indices and merge_gather_kernel copies (x, y, z, r) into key
// order.  merge_grid_kernel then scans, for each i, the cells covering
// [x_i - reach (r_i + r_max), x_i + reach (r_i + r_max)] in every axis (at
// most 3 per axis; floor(x / h) is monotonic in x, so no pair within reach is
// missed at a cell boundary), finding each cell's run of sorted keys by
// binary search.  Cell coordinates are wrapped to 21 bits per axis in the key;
// far cells that share a key only add pairs the distance test rejects.
//
// Pairs are packed (i << 32 | j << 1 | out), wake indices, so that sorting the
// keys orders them by i, then j; out = 1 marks a pair surely outside PAWAN's
// reach at entry (|x_i - x_j|^2 >= (0.125 (r_i + r_j))^2 (1 + 1e-12), a
// margin far above the rounding of either side's distance), which cannot
// merge before x_i has moved.  count may exceed max_pairs, and then only the
// first max_pairs are stored (the host retries with room for all of them).
constexpr unsigned long long kMergeNoCell = ~0ull;

__device__ __forceinline__ int64_t merge_cell(double x, double h) {
  return (int64_t)fmin(fmax(floor(x / h), -4.0e18), 4.0e18);
}
__device__ __forceinline__ unsigned long long merge_cell_key(int64_t cx, int64_t cy, int64_t cz) {
  const unsigned long long m = (1ull << 21) - 1;
  return (((unsigned long long)cx & m) << 42) | (((unsigned long long)cy & m) << 21) | ((unsigned long long)cz & m);
}
__device__ __forceinline__ bool merge_nonzero(const double *x0, int64_t cap, int64_t g) {
  return x0[3 * cap + g] != 0.0 || x0[4 * cap + g] != 0.0 || x0[5 * cap + g] != 0.0;
}

static __global__ void merge_keys_kernel(const double *x0, int64_t cap, int64_t off, int64_t n, double h,
                                         unsigned long long *keys, int *idx) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t g = off + j;
    keys[j] = merge_nonzero(x0, cap, g)
                  ? merge_cell_key(merge_cell(x0[g], h), merge_cell(x0[cap + g], h), merge_cell(x0[2 * cap + g], h))
                  : kMergeNoCell;
    idx[j] = (int)j;
  }
}

// (x, y, z, r) of the particles in sorted key order.
static __global__ void merge_gather_kernel(const double *x0, const double *sig, int64_t cap, int64_t off, int64_t n,
                                           const int *idx, double4 *rec) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t g = off + idx[e];
    rec[e] = make_double4(x0[g], x0[cap + g], x0[2 * cap + g], sig[g]);
  }
}

struct MergeArgs {
  const double *x0;  // [6][cap] state
  const double *sig;
  int64_t cap, off, n, n_elig;
  double reach, h, rmax;
  const unsigned long long *keys;  // sorted cell keys
  const int *idx;                  // particle of each sorted key
  const double4 *rec;              // (x, y, z, r) in sorted key order
  unsigned long long *pairs;
  unsigned long long *count;
  int64_t max_pairs;
};

static __global__ void merge_grid_kernel(MergeArgs a) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= a.n_elig) return;
  const int64_t g = a.off + i;
  if (!merge_nonzero(a.x0, a.cap, g)) return;
  const double x[3] = {a.x0[g], a.x0[a.cap + g], a.x0[2 * a.cap + g]};
  const double ri = a.sig[g];
  const double ext = a.reach * (ri + a.rmax);
  int64_t c0[3], c1[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    c0[m] = merge_cell(x[m] - ext, a.h);
    c1[m] = merge_cell(x[m] + ext, a.h);
  }
  for (int64_t cx = c0[0]; cx <= c1[0]; ++cx)
    for (int64_t cy = c0[1]; cy <= c1[1]; ++cy)
      for (int64_t cz = c0[2]; cz <= c1[2]; ++cz) {
        const unsigned long long key = merge_cell_key(cx, cy, cz);
        int64_t lo = 0, hi = a.n;  // first sorted key >= key
        while (lo < hi) {
          const int64_t mid = (lo + hi) >> 1;
          if (a.keys[mid] < key) lo = mid + 1;
          else hi = mid;
        }
        for (int64_t e = lo; e < a.n && a.keys[e] == key; ++e) {
          const int64_t j = a.idx[e];
          if (j <= i) continue;
          const double4 p = a.rec[e];
          const double dx = x[0] - p.x, dy = x[1] - p.y, dz = x[2] - p.z;
          const double d2 = dx * dx + dy * dy + dz * dz;
          const double lim = a.reach * (ri + p.w);
          if (d2 < lim * lim) {
            const double pawan = 0.125 * (ri + p.w);
            const unsigned long long out = d2 >= pawan * pawan * (1.0 + 1e-12) ? 1ull : 0ull;
            const unsigned long long k = atomicAdd(a.count, 1ull);
            if ((int64_t)k < a.max_pairs)
              a.pairs[k] = ((unsigned long long)i << 32) | ((unsigned long long)j << 1) | out;
          }
        }
      }
}

// Velocity induced at arbitrary points by particles [lo, hi) with each
// particle's own radius (PAWAN __interaction::getVi, interaction.cpp:453-477;
// the blade-airstation inflow of getInflow, :399-451), with the q of the
// selected kernel (KER), FP64.
//
// Bound by the FP64 pipe (about 24 operations per far pair), once the device
// is full: a rotor has a few hundred airstations and a wake 1e5-1e6 particles,
// so the lanes are particles, read once into registers for kProbePoints points,
// and blockIdx.y splits the particles into chunks of `per`.  Each CTA reduces its
// sums and writes part[chunk][3 npts]; probe_reduce_kernel adds the chunks in
// order.  Gaussian pairs at u >= kFarU64 take the far limit q = 1/rho^3, which
// equals the closed form to double rounding; the closed form runs under a
// warp vote.
// 400 points of 100,000 particles, whole call: 0.19 ms with 4 points per CTA (118
// registers, two CTAs per SM), 0.30 with 8 (158), 0.24 with 2; 51.6 ms for one thread per
// point over all particles (4 CTAs) with the closed form for every pair.
constexpr int kProbeBlock = 256;
constexpr int kProbePoints = 4;

template <int KER = kGaussian>
__global__ void __launch_bounds__(kProbeBlock) probe_kernel(const double *x0, const double *sig, int64_t cap, int64_t lo,
                                                            int64_t hi, int64_t per, const double *pts, int64_t npts,
                                                            double *part) {
  constexpr int NW = kProbeBlock / 32;
  __shared__ double red[NW][3 * kProbePoints];
  __shared__ double spt[3 * kProbePoints];
  const int64_t p0 = blockIdx.x * (int64_t)kProbePoints;
  const int np = (int)min((int64_t)kProbePoints, npts - p0);
  const int64_t s0 = lo + blockIdx.y * per, s1 = min(hi, s0 + per);
  if (threadIdx.x < 3 * np) spt[threadIdx.x] = pts[3 * p0 + threadIdx.x];
  __syncthreads();
  double u[kProbePoints][3];
#pragma unroll
  for (int k = 0; k < kProbePoints; ++k) u[k][0] = u[k][1] = u[k][2] = 0.0;
  // whole warps stay in the loop for the vote: lanes past the end repeat the
  // last particle with zero strength
  for (int64_t jb = s0 + (threadIdx.x & ~31); jb < s1; jb += kProbeBlock) {
    const int64_t j = jb + (threadIdx.x & 31);
    const bool valid = j < s1;
    const int64_t jj = valid ? j : s1 - 1;
    const double xs = x0[jj], ys = x0[cap + jj], zs = x0[2 * cap + jj];
    const double ax = valid ? x0[3 * cap + jj] : 0.0, ay = valid ? x0[4 * cap + jj] : 0.0,
                 az = valid ? x0[5 * cap + jj] : 0.0;
    const double s2 = sig[jj] * sig[jj], is = fast_rsqrt(s2);
#pragma unroll
    for (int k = 0; k < kProbePoints; ++k) {
      if (k >= np) break;
      const double dx = spt[3 * k] - xs, dy = spt[3 * k + 1] - ys, dz = spt[3 * k + 2] - zs;
      const double r2 = dx * dx + dy * dy + dz * dz;
      double q;
      if constexpr (KER == kHighOrder) {
        q = pair_terms_ho(r2, s2).q;
      } else {
        const bool near = !(r2 >= kFarU64 * s2);  // a NaN radius takes the closed form, which passes it on
        const double ir = fast_rsqrt(r2);
        q = ir * ir * ir;
        if (__any_sync(0xffffffffu, near)) {
          if (near) q = pair_terms(r2, s2, ir, is).q;
        }
      }
      if (valid) {
        u[k][0] += q * (ay * dz - az * dy);
        u[k][1] += q * (az * dx - ax * dz);
        u[k][2] += q * (ax * dy - ay * dx);
      }
    }
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < kProbePoints; ++k)
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      double v = u[k][m];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (l == 0) red[w][3 * k + m] = v;
    }
  __syncthreads();
  if (threadIdx.x < 3 * np) {
    double v = 0.0;
    for (int k = 0; k < NW; ++k) v += red[k][threadIdx.x];
    part[blockIdx.y * 3 * npts + 3 * p0 + threadIdx.x] = v * kInv4Pi;
  }
}

// The same with the lanes over the points, for calls whose points fill the
// device by themselves (probe_by_points): a thread sums all particles for its
// point, so there are no partial sums to store and reduce.
template <int KER = kGaussian>
__global__ void __launch_bounds__(kProbeBlock) probe_points_kernel(const double *x0, const double *sig, int64_t cap,
                                                                   int64_t lo, int64_t hi, const double *pts,
                                                                   int64_t npts, double *vel) {
  __shared__ double sx[kProbeBlock][8];  // position, sigma^2, strength, 1/sigma
  const int64_t pi = blockIdx.x * (int64_t)kProbeBlock + threadIdx.x;
  const bool valid = pi < npts;
  const int64_t pl = valid ? pi : npts - 1;
  const double x = pts[3 * pl], y = pts[3 * pl + 1], z = pts[3 * pl + 2];
  double u[3] = {0.0, 0.0, 0.0};
  for (int64_t sb = lo; sb < hi; sb += kProbeBlock) {
    __syncthreads();
    const int64_t j = sb + threadIdx.x;
    if (j < hi) {
      double *s = sx[threadIdx.x];
      for (int m = 0; m < 3; ++m) {
        s[m] = x0[m * cap + j];
        s[4 + m] = x0[(3 + m) * cap + j];
      }
      s[3] = sig[j] * sig[j];
      s[7] = fast_rsqrt(s[3]);
    }
    __syncthreads();
    const int cnt = (int)min((int64_t)kProbeBlock, hi - sb);
#pragma unroll 2
    for (int k = 0; k < cnt; ++k) {
      const double *s = sx[k];
      const double dx = x - s[0], dy = y - s[1], dz = z - s[2], s2 = s[3];
      const double r2 = dx * dx + dy * dy + dz * dz;
      double q;
      if constexpr (KER == kHighOrder) {
        q = pair_terms_ho(r2, s2).q;
      } else {
        const bool near = !(r2 >= kFarU64 * s2);
        const double ir = fast_rsqrt(r2);
        q = ir * ir * ir;
        if (__any_sync(0xffffffffu, near)) {
          if (near) q = pair_terms(r2, s2, ir, s[7]).q;
        }
      }
      u[0] += q * (s[5] * dz - s[6] * dy);
      u[1] += q * (s[6] * dx - s[4] * dz);
      u[2] += q * (s[4] * dy - s[5] * dx);
    }
  }
  if (valid)
    for (int m = 0; m < 3; ++m) vel[3 * pi + m] = u[m] * kInv4Pi;
}

static __global__ void probe_reduce_kernel(const double *part, int chunks, int64_t n3, double *vel) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n3; i += (int64_t)gridDim.x * blockDim.x) {
    double v = 0.0;
#pragma unroll 8
    for (int c = 0; c < chunks; ++c) v += part[c * n3 + i];
    vel[i] = v;
  }
}

// FP32 pipe throughput probe: kFfmaChains independent FMA chains per thread,
// all operands in registers.  The result is stored only if it equals a value
// it cannot take, so the loop is not eliminated.
constexpr int kFfmaChains = 8;
static __global__ void __launch_bounds__(256) ffma_peak_kernel(float *out, int iters, float a, float b) {
  float x[kFfmaChains];
#pragma unroll
  for (int k = 0; k < kFfmaChains; ++k) x[k] = threadIdx.x * 1e-3f + k;
  for (int i = 0; i < iters; i += 4) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int k = 0; k < kFfmaChains; ++k) x[k] = fmaf(x[k], a, b);
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < kFfmaChains; ++k) s += x[k];
  if (s == -1.2345e30f) *out = s;
}

// The same probe with the packed two-wide FMA of sm_100 (__ffma2_rn): each
// instruction does two FP32 FMAs.
static __global__ void __launch_bounds__(256) ffma2_peak_kernel(float *out, int iters, float a, float b) {
  float2 x[kFfmaChains / 2];
  const float2 a2 = make_float2(a, a), b2 = make_float2(b, b);
#pragma unroll
  for (int k = 0; k < kFfmaChains / 2; ++k) x[k] = make_float2(threadIdx.x * 1e-3f + 2 * k, threadIdx.x * 1e-3f + 2 * k + 1);
  for (int i = 0; i < iters; i += 4) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int k = 0; k < kFfmaChains / 2; ++k) x[k] = __ffma2_rn(x[k], a2, b2);
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < kFfmaChains / 2; ++k) s += x[k].x + x[k].y;
  if (s == -1.2345e30f) *out = s;
}

// The same probe for the FP64 pipe (DFMA), the bound of the FP64 mode's pair
// kernel.
static __global__ void __launch_bounds__(256) dfma_peak_kernel(float *out, int iters, double a, double b) {
  double x[kFfmaChains];
#pragma unroll
  for (int k = 0; k < kFfmaChains; ++k) x[k] = threadIdx.x * 1e-3 + k;
  for (int i = 0; i < iters; i += 4) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int k = 0; k < kFfmaChains; ++k) x[k] = fma(x[k], a, b);
  }
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < kFfmaChains; ++k) s += x[k];
  if (s == -1.2345e300) *out = (float)s;
}

}  // namespace pgpu
