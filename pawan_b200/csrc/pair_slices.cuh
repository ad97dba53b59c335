// FP32 (compensated) pair kernel for systems too small to fill the device with
// the CTA-wide target tiles of pair_f32.cuh, and for wakes of dense filaments,
// where its finer boxes find more far pairs.  Bound by the FP32 pipe from a few thousand
// particles on (64% busy on 20,000 particles, warps mostly waiting for it), by
// latency below.  The 5000-particle station ring: 62 us per evaluation (4.1e11
// pairs/s) against 167 us with 128 x 2 tiles (20 x 16 items, mostly idle SMs).
//
// The unit of work is a row: a tile of 32 targets and eight slices of 32 SL
// sources, one per warp of a CTA.  All rows of all systems form one list
// and every CTA takes an equal run of it, whatever tile it starts or ends in, so
// the device is evenly full at any size.  The warps of a CTA hold the same
// targets and stage their own slices (no CTA barrier between rows); at a tile's
// end the CTA adds its warps' sums in warp order into the tile's next partial.
// The arithmetic is that of pair_f32.cuh: packed far limit for slices whose box
// is far from the targets' box, closed form for the others, one compensation
// group per slice.  The order of every sum is fixed by the sizes.
//
// High-order kernel (KER): every pair takes its full terms, two sources per
// packed instruction, 42 FP32 operations in slices far from the targets and 58
// in the others (two less where one sigma serves the slice), against 68 scalar
// instructions in the generic body; no pair is cheap enough for wider tiles to
// pay, so it takes these slices at any size.
#pragma once

namespace pgpu {

constexpr int kSliceWarps = 8;

// Minimum and maximum over a warp (redux.sync on FP32: sm_100a).
__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ void reduce_box(WarpBox &b) {
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    b.lo[m] = warp_min(b.lo[m]);
    b.hi[m] = warp_max(b.hi[m]);
  }
  b.hs = warp_max(b.hs);
}

// The rows of one target tile that a CTA takes: from `row` up to its own end
// row1 or the tile's last row.
struct RowRun {
  PlanEntry pe;
  int64_t first;  // the tile's first row
  int64_t t0, tend, s1;  // first target of the tile, ends of the targets and of the sources
  // Row r holds the slices of group (r mult) mod rows-per-tile: any run of rows
  // samples the whole system evenly, so the slices around the tile, which
  // take the closed form, spread over the CTAs.
  int64_t g;
  int nrows;
  int c;  // this CTA's partial of the tile
  bool last;  // holds the tile's last row
};
__device__ __forceinline__ RowRun row_run(const PlanEntry *plan, int nsys, int64_t rpc, int64_t row, int64_t row1) {
  RowRun r;
  r.pe = plan[find_plan(plan, nsys, row)];
  const int64_t rps = r.pe.chunk;  // rows per target tile
  const int64_t tile = (row - r.pe.item_start) / rps;
  r.first = r.pe.item_start + tile * rps;
  r.t0 = r.pe.off + r.pe.toff + tile * 32;
  r.tend = r.pe.off + r.pe.toff + r.pe.tn;
  r.s1 = r.pe.off + r.pe.n;
  r.g = ((row - r.first) * r.pe.mult) % rps;
  r.nrows = (int)(min(r.first + rps, row1) - row);
  r.c = (int)(row / rpc - r.first / rpc);
  r.last = row + r.nrows == r.first + rps;
  return r;
}
// The CTA's sums of a tile, red[warp][component][target] (NC components), in
// warp order and times `scale` into its partial; the CTA of the tile's last row
// also clears the partials that no CTA has.
template <int NC>
__device__ __forceinline__ void row_run_sums(const RowRun &r, const double *red, double scale, double *partial,
                                             int64_t cap, int nch) {
  const int clear = r.last ? nch : r.c + 1;
  for (int e = threadIdx.x; e < NC * 32; e += 32 * kSliceWarps) {
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < kSliceWarps; ++k) v += red[k * NC * 32 + e];
    const int64_t i = r.t0 + e % 32;
    if (i >= r.tend) continue;
    double *o = partial + (e / 32) * cap + i;
    o[r.c * 6 * cap] = v * scale;
    for (int k = r.c + 1; k < clear; ++k) o[k * 6 * cap] = 0.0;
  }
}

// REF: with n_s, for far pairs formed from a reference point (far_slice).
template <int SL, bool SPLIT, bool REF = true> struct SliceStage {
  float4 P[32 * SL], Q[32 * SL];  // pair-interleaved as in pair_f32.cuh
  float4 N[REF ? 32 * SL : 1];
  float4 L[SPLIT ? 32 * SL : 1];
};

// Source k of a slice (position p, strength and volume q), its n_s taken
// about the slice's reference point.
template <int SL, bool SPLIT, bool REF>
__device__ __forceinline__ void stage_source(SliceStage<SL, SPLIT, REF> &st, int k, float4 p, float4 q, float rx,
                                             float ry, float rz) {
  const int e = (k >> 1) * 8 + (k & 1);
  float *dp = reinterpret_cast<float *>(st.P) + e, *dq = reinterpret_cast<float *>(st.Q) + e,
        *dn = reinterpret_cast<float *>(st.N) + e;
  dp[0] = p.x; dp[2] = p.y; dp[4] = p.z; dp[6] = p.w;
  dq[0] = q.x; dq[2] = q.y; dq[4] = q.z; dq[6] = q.w;
  if constexpr (!REF) return;
  const float px = p.x - rx, py = p.y - ry, pz = p.z - rz;
  dn[0] = py * q.z - pz * q.y;
  dn[2] = pz * q.x - px * q.z;
  dn[4] = px * q.y - py * q.x;
}

// The Gaussian sums of one target over source pairs r0, r0 + step, ... (n of
// them) of a staged slice: the far limit, or the closed form (its diffusion
// into sdv).
template <int SL, bool SPLIT>
__device__ __forceinline__ void far_slice(const SliceStage<SL, SPLIT> &st, int n, int r0, int step, const float2 *X,
                                          const float2 *AT, float xr0, float xr1, float xr2, float2 *sv, float2 *sd,
                                          float2 *sp) {
  float2 B3[3];
  far_b3(xr0, xr1, xr2, AT, B3);
#pragma unroll 2
  for (int k = 0; k < n; ++k) {
    const int r = r0 + k * step;
    const float4 pa = st.P[2 * r], pb = st.P[2 * r + 1], qa = st.Q[2 * r], qb = st.Q[2 * r + 1], na = st.N[2 * r],
                 nb = st.N[2 * r + 1];
    far_pair2(make_float2(pa.x, pa.y), make_float2(pa.z, pa.w), make_float2(pb.x, pb.y), make_float2(qa.x, qa.y),
              make_float2(qa.z, qa.w), make_float2(qb.x, qb.y), make_float2(na.x, na.y), make_float2(na.z, na.w),
              make_float2(nb.x, nb.y), X, AT, B3, sv, sd, sp);
  }
}
// The far limit without a reference point: w = alpha_s x d per pair (28 packed
// operations), for slices whose sources may lie far apart.  AT = -3 alpha_t;
// sv sums q w, sp q alpha_s.
template <int SL, bool SPLIT>
__device__ __forceinline__ void far_slice_direct(const SliceStage<SL, SPLIT, false> &st, int n, int r0, int step,
                                                 const float2 *X, const float2 *AT, float2 *sv, float2 *sd,
                                                 float2 *sp) {
  const float2 M1 = make_float2(-1.f, -1.f);
#pragma unroll 2
  for (int k = 0; k < n; ++k) {
    const int r = r0 + k * step;
    const float4 pa = st.P[2 * r], pb = st.P[2 * r + 1], qa = st.Q[2 * r], qb = st.Q[2 * r + 1];
    const float2 ax = make_float2(qa.x, qa.y), ay = make_float2(qa.z, qa.w), az = make_float2(qb.x, qb.y);
    const float2 dx = __ffma2_rn(make_float2(pa.x, pa.y), M1, X[0]);
    const float2 dy = __ffma2_rn(make_float2(pa.z, pa.w), M1, X[1]);
    const float2 dz = __ffma2_rn(make_float2(pb.x, pb.y), M1, X[2]);
    float2 r2 = __fmul2_rn(dx, dx);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dz, dz, r2);
    const float2 ir = make_float2(fast_rsqrt(r2.x), fast_rsqrt(r2.y));
    const float2 A = __fmul2_rn(ir, ir);
    const float2 q = __fmul2_rn(A, ir);
    const float2 F = __fmul2_rn(q, A);
    const float2 wx = make_float2(ay.x * dz.x - az.x * dy.x, ay.y * dz.y - az.y * dy.y);
    const float2 wy = make_float2(az.x * dx.x - ax.x * dz.x, az.y * dx.y - ax.y * dz.y);
    const float2 wz = make_float2(ax.x * dy.x - ay.x * dx.x, ax.y * dy.y - ay.y * dx.y);
    sv[0] = __ffma2_rn(q, wx, sv[0]);
    sv[1] = __ffma2_rn(q, wy, sv[1]);
    sv[2] = __ffma2_rn(q, wz, sv[2]);
    float2 dot = __fmul2_rn(AT[0], wx);
    dot = __ffma2_rn(AT[1], wy, dot);
    dot = __ffma2_rn(AT[2], wz, dot);
    const float2 fd = __fmul2_rn(F, dot);
    sd[0] = __ffma2_rn(fd, dx, sd[0]);
    sd[1] = __ffma2_rn(fd, dy, sd[1]);
    sd[2] = __ffma2_rn(fd, dz, sd[2]);
    sp[0] = __ffma2_rn(q, ax, sp[0]);
    sp[1] = __ffma2_rn(q, ay, sp[1]);
    sp[2] = __ffma2_rn(q, az, sp[2]);
  }
}
template <bool SPLIT, bool CROSS, int SL, bool REF>
__device__ __forceinline__ void mid_slice(const SliceStage<SL, SPLIT, REF> &st, int n, int r0, int step, const float2 *X,
                                          const float *xl, const float *at, float hst, float vt, const MidSigma2 *uni, float2 *sv,
                                          float2 *sd, float2 *sp, float *sdv, unsigned &nfull) {
  float2 sdv2[3] = {dup2(0.f), dup2(0.f), dup2(0.f)};
#pragma unroll 2
  for (int k = 0; k < n; ++k) {
    const int r = r0 + k * step;
    const float4 pa = st.P[2 * r], pb = st.P[2 * r + 1], qa = st.Q[2 * r], qb = st.Q[2 * r + 1];
    float2 lx = dup2(0.f), ly = lx, lz = lx;
    if constexpr (SPLIT) {
      const float4 la = st.L[2 * r], lb = st.L[2 * r + 1];
      lx = make_float2(la.x, la.y); ly = make_float2(la.z, la.w); lz = make_float2(lb.x, lb.y);
    }
    mid_pair2<SPLIT, CROSS>(make_float2(pa.x, pa.y), make_float2(pa.z, pa.w), make_float2(pb.x, pb.y),
                            make_float2(pb.z, pb.w), make_float2(qa.x, qa.y), make_float2(qa.z, qa.w),
                            make_float2(qb.x, qb.y), make_float2(qb.z, qb.w), lx, ly, lz, X, xl, at, hst, kFarU * hst,
                            vt, uni, sv, sd, sp, sdv2, nfull);
  }
#pragma unroll
  for (int m = 0; m < 3; ++m) sdv[m] = sdv2[m].x + sdv2[m].y;
}

template <int SL, bool SPLIT, int KER = kGaussian>
__global__ void __launch_bounds__(32 * kSliceWarps, 2) pair_slices_kernel(PairArgs<float> a) {
  constexpr int W = kSliceWarps, S = 32 * SL, TT = 32;
  using Stage = SliceStage<SL, SPLIT>;
  constexpr size_t kStageBytes = W * sizeof(Stage), kRedBytes = (size_t)W * 6 * TT * sizeof(double);
  __shared__ __align__(16) unsigned char smem[kStageBytes > kRedBytes ? kStageBytes : kRedBytes];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Stage &st = reinterpret_cast<Stage *>(smem)[w];
  double *red = reinterpret_cast<double *>(smem);  // [W][6][TT], after the slices
  // rows of this CTA: plan items are rows, eight slices of one target tile
  const int64_t rpc = a.plan[a.nsys].chunk;
  const int64_t row1 = min((blockIdx.x + 1) * rpc, a.plan[a.nsys].item_start);
  for (int64_t row = blockIdx.x * rpc; row < row1;) {
    const RowRun run = row_run(a.plan, a.nsys, rpc, row, row1);
    const int64_t s1 = run.s1;
    int64_t g = run.g;

    // this lane's share of a slice, fetched ahead of the slice in work
    float4 gp[SL], gq[SL], gl[SPLIT ? SL : 1];
    auto fetch = [&](int64_t sb) {
#pragma unroll
      for (int j = 0; j < SL; ++j) {
        const int64_t i = sb + lane + 32 * j;
        gp[j] = i < s1 ? a.P[i] : pad_P<float>();
        gq[j] = i < s1 ? a.Q[i] : pad_Q<float>();
        if constexpr (SPLIT) gl[j] = i < s1 ? a.L[i] : pad_Q<float>();
      }
    };
    int64_t sb = run.pe.off + (g * W + w) * S;
    if (sb < s1) fetch(sb);

    int64_t ti = min(run.t0 + lane, run.tend - 1);
    if (a.targets) ti = run.pe.off + a.targets[ti];
    const float4 pt = a.P[ti], qt = a.Q[ti];
    float4 lt = pad_Q<float>();
    if constexpr (SPLIT) lt = a.L[ti];
    const float at[3] = {qt.x, qt.y, qt.z}, xl[3] = {lt.x, lt.y, lt.z};
    const float2 X[3] = {dup2(pt.x), dup2(pt.y), dup2(pt.z)};
    // Gaussian: -3 alpha_t, the far limit's constant folded in.  High-order: the
    // -3 of F waits for the fold, since the rounding of -3 alpha_t would turn
    // alpha_t for every source alike (norm-wise error of dalpha on the
    // 5000-particle ring: 2.3e-6 with it, 1.1e-6 without).
    constexpr float kAt = KER == kHighOrder ? 1.f : -3.f;
    const float2 AT[3] = {dup2(kAt * qt.x), dup2(kAt * qt.y), dup2(kAt * qt.z)};
    float vh[3] = {0.f, 0.f, 0.f}, vl[3] = {0.f, 0.f, 0.f}, dh[3] = {0.f, 0.f, 0.f}, dl[3] = {0.f, 0.f, 0.f};
    unsigned nfull = 0;
    WarpBox tb;
    tb.init();
    tb.add(pt.x, pt.y, pt.z, pt.w);
    reduce_box(tb);
    // one radius among the targets (equality with the largest, which no NaN passes)
    const bool one_t = __all_sync(0xffffffffu, pt.w == tb.hs);

    for (int r = 0; r < run.nrows; ++r) {
      const int64_t cur = sb;
      g += run.pe.mult;
      if (g >= run.pe.chunk) g -= run.pe.chunk;
      sb = run.pe.off + (g * W + w) * S;
      if (cur >= s1) {  // past the last source: this warp has no slice in the row
        if (r + 1 < run.nrows && sb < s1) fetch(sb);
        continue;
      }
      __syncwarp();
      const float rx = __shfl_sync(0xffffffffu, gp[0].x, 0), ry = __shfl_sync(0xffffffffu, gp[0].y, 0),
                  rz = __shfl_sync(0xffffffffu, gp[0].z, 0);
      WarpBox sbox;
      sbox.init();
#pragma unroll
      for (int j = 0; j < SL; ++j) {
        const float4 p = gp[j], q = gq[j];
        stage_source(st, lane + 32 * j, p, q, rx, ry, rz);
        if constexpr (SPLIT) {
          float *dl_ = reinterpret_cast<float *>(st.L) + ((lane + 32 * j) >> 1) * 8 + (lane & 1);
          dl_[0] = gl[j].x; dl_[2] = gl[j].y; dl_[4] = gl[j].z;
        }
        if (cur + lane + 32 * j < s1) sbox.add(p.x, p.y, p.z, p.w);
      }
      reduce_box(sbox);
      const bool far = all_far(tb, sbox);
      bool one = one_t;  // one sigma for all of the slice's pairs
#pragma unroll
      for (int j = 0; j < SL; ++j) one = one && (gp[j].w == sbox.hs || cur + lane + 32 * j >= s1);
      __syncwarp();
      if (r + 1 < run.nrows && sb < s1) fetch(sb);
      const int npr = (int)(min((int64_t)S, s1 - cur) + 1) >> 1;  // an odd tail pairs with a padding source

      float2 sv[3], sd[3], sp[3];
      float sdv[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int m = 0; m < 3; ++m) sv[m] = sd[m] = sp[m] = dup2(0.f);
      if constexpr (KER == kHighOrder) {
        float2 zs[3] = {dup2(0.f), dup2(0.f), dup2(0.f)};
        auto sums = [&](const HoSigma2 *uni) {
          if (far) {
            float2 B[3], sw = dup2(0.f);
            far_b3(pt.x - rx, pt.y - ry, pt.z - rz, AT, B);
#pragma unroll 2
            for (int r = 0; r < npr; ++r) {
              const float4 pa = st.P[2 * r], pb = st.P[2 * r + 1], qa = st.Q[2 * r], qb = st.Q[2 * r + 1],
                           na = st.N[2 * r], nb = st.N[2 * r + 1];
              ho_far_pair2(make_float2(pa.x, pa.y), make_float2(pa.z, pa.w), make_float2(pb.x, pb.y),
                           make_float2(pb.z, pb.w), make_float2(qa.x, qa.y), make_float2(qa.z, qa.w),
                           make_float2(qb.x, qb.y), make_float2(qb.z, qb.w), make_float2(na.x, na.y),
                           make_float2(na.z, na.w), make_float2(nb.x, nb.y), X, pt.w, uni, AT, B, sv, sd, sp, zs, sw);
            }
#pragma unroll
            for (int m = 0; m < 3; ++m) sdv[m] = qt.w * (zs[m].x + zs[m].y) - (sw.x + sw.y) * at[m];
          } else {
#pragma unroll 2
            for (int r = 0; r < npr; ++r) {
              const float4 pa = st.P[2 * r], pb = st.P[2 * r + 1], qa = st.Q[2 * r], qb = st.Q[2 * r + 1];
              ho_near_pair2(make_float2(pa.x, pa.y), make_float2(pa.z, pa.w), make_float2(pb.x, pb.y),
                            make_float2(pb.z, pb.w), make_float2(qa.x, qa.y), make_float2(qa.z, qa.w),
                            make_float2(qb.x, qb.y), make_float2(qb.z, qb.w), X, at, pt.w, qt.w, uni, AT, sv, sd, sp,
                            zs);
            }
#pragma unroll
            for (int m = 0; m < 3; ++m) sdv[m] = zs[m].x + zs[m].y;
          }
        };
        // one sigma: its powers leave the loop (a padding source's terms
        // vanish with R^-2.5 at rho ~ 1e18)
        if (__all_sync(0xffffffffu, one)) {
          const HoSigma2 g = ho_sigma2(dup2(tb.hs + sbox.hs));
          sums(&g);
        } else {
          sums(nullptr);
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          sdv[m] *= (float)HighOrder::kZd;
          sd[m] = __fmul2_rn(sd[m], dup2(-3.f));
        }
      } else if (far) {
        far_slice(st, npr, 0, 1, X, AT, pt.x - rx, pt.y - ry, pt.z - rz, sv, sd, sp);
      } else if (__all_sync(0xffffffffu, one)) {
        // one sigma, as in every wake shed with one radius: its factors leave
        // the loop (an odd tail's padding source carries no strength, so its
        // sigma does not matter)
        const MidSigma2 g = mid_sigma2(dup2(tb.hs + sbox.hs));
        mid_slice<SPLIT, true>(st, npr, 0, 1, X, xl, at, pt.w, qt.w, &g, sv, sd, sp, sdv, nfull);
      } else {
        mid_slice<SPLIT, true>(st, npr, 0, 1, X, xl, at, pt.w, qt.w, nullptr, sv, sd, sp, sdv, nfull);
      }
      fold_group_f32(far, pt.x - rx, pt.y - ry, pt.z - rz, at, a.nu2, sv, sd, sp, sdv, vh, vl, dh, dl);
    }
    // lanes past the end repeat the last target
    const unsigned wsum = __reduce_add_sync(0xffffffffu, run.t0 + lane < run.tend ? nfull : 0u);
    if (lane == 0 && wsum) atomicAdd(a.nfull, (unsigned long long)wsum);

    __syncthreads();  // every warp is done with its slices
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      red[(w * 6 + m) * TT + lane] = (double)vh[m] + (double)vl[m];
      red[(w * 6 + 3 + m) * TT + lane] = (double)dh[m] + (double)dl[m];
    }
    __syncthreads();
    row_run_sums<6>(run, red, kInv4Pi, a.partial, a.cap, a.nch);
    __syncthreads();  // before the next tile's slices overwrite the sums
    row += run.nrows;
  }
}

// How many pairs of a system take the closed form in slices and in CTA-wide
// tiles (choose_slices): one CTA per sampled target position, against every
// `stride`-th block of 128 sources of its system.  out[sample] = (32-source slices not far
// from 32 targets, 128-source tiles not far from 160 targets, the span of a
// warp of 128 x 2 tiles, blocks).
struct NearSample {
  int64_t off, n, t;  // first particle and particles of the system, first target
};
static __global__ void __launch_bounds__(256) near_share_kernel(const float4 *P, const NearSample *samples,
                                                                int max_blocks, int4 *out) {
  __shared__ int n32, n128;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const NearSample s = samples[blockIdx.x];
  const int64_t end = s.off + s.n, blocks = (s.n + 127) / 128, stride = (blocks + max_blocks - 1) / max_blocks;
  if (threadIdx.x == 0) n32 = n128 = 0;
  __syncthreads();
  WarpBox t32, t160;
  t160.init();
  for (int j = 0; j < 5; ++j) {
    const float4 p = P[min(s.t + lane + 32 * j, end - 1)];
    t160.add(p.x, p.y, p.z, p.w);
    if (j == 0) {
      t32 = t160;
      reduce_box(t32);
    }
  }
  reduce_box(t160);
  for (int64_t b = w * stride; b < blocks; b += 8 * stride) {
    WarpBox tile;
    tile.init();
    int near = 0;
    for (int j = 0; j < 4; ++j) {
      const float4 p = P[min(s.off + 128 * b + 32 * j + lane, end - 1)];
      WarpBox slice;
      slice.init();
      slice.add(p.x, p.y, p.z, p.w);
      tile.add(p.x, p.y, p.z, p.w);
      reduce_box(slice);
      near += !all_far(t32, slice);
    }
    reduce_box(tile);
    if (lane == 0) {
      atomicAdd(&n32, near);
      atomicAdd(&n128, (int)!all_far(t160, tile));
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) out[blockIdx.x] = make_int4(n32, n128, (int)((blocks + stride - 1) / stride), 0);
}

}  // namespace pgpu
