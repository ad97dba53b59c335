// FP32 (compensated) pair kernel for systems too small to fill the device with
// the CTA-wide target tiles of pair_f32.cuh, and for dense filaments, where its
// finer boxes find more far pairs.  Bound by the FP32 pipe from a few thousand
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

template <int SL, bool SPLIT> struct SliceStage {
  float4 P[32 * SL], Q[32 * SL], N[32 * SL];  // pair-interleaved as in pair_f32.cuh
  float4 L[SPLIT ? 32 * SL : 1];
};

template <int SL, bool SPLIT>
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
    const PlanEntry pe = a.plan[find_plan(a.plan, a.nsys, row)];
    const int64_t rps = pe.chunk;  // rows per target tile
    const int64_t tile = (row - pe.item_start) / rps;
    const int64_t first = pe.item_start + tile * rps;  // the tile's first row
    const int nrows = (int)(min(first + rps, row1) - row);
    const int c = (int)(row / rpc - first / rpc);  // this CTA's partial of the tile
    const int64_t t0 = pe.off + pe.toff + tile * TT;
    const int64_t tend = pe.off + pe.toff + pe.tn;  // end of the targets
    const int64_t s1 = pe.off + pe.n;
    // Row r holds the slices of group (r mult) mod rps: any run of rows
    // samples the whole system evenly, so the slices around the tile, which
    // take the closed form, spread over the CTAs.
    int64_t g = ((row - first) * pe.mult) % rps;

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
    int64_t sb = pe.off + (g * W + w) * S;
    if (sb < s1) fetch(sb);

    const int64_t ti = min(t0 + lane, tend - 1);
    const float4 pt = a.P[ti], qt = a.Q[ti];
    float4 lt = pad_Q<float>();
    if constexpr (SPLIT) lt = a.L[ti];
    const float at[3] = {qt.x, qt.y, qt.z}, xl[3] = {lt.x, lt.y, lt.z};
    const float2 X[3] = {dup2(pt.x), dup2(pt.y), dup2(pt.z)};
    const float2 AT3[3] = {dup2(-3.f * qt.x), dup2(-3.f * qt.y), dup2(-3.f * qt.z)};
    float vh[3] = {0.f, 0.f, 0.f}, vl[3] = {0.f, 0.f, 0.f}, dh[3] = {0.f, 0.f, 0.f}, dl[3] = {0.f, 0.f, 0.f};
    unsigned nfull = 0;
    WarpBox tb;
    tb.init();
    tb.add(pt.x, pt.y, pt.z, pt.w);
    reduce_box(tb);
    const float thmin = warp_min(pt.w);

    for (int r = 0; r < nrows; ++r) {
      const int64_t cur = sb;
      g += pe.mult;
      if (g >= rps) g -= rps;
      sb = pe.off + (g * W + w) * S;
      if (cur >= s1) {  // past the last source: this warp has no slice in the row
        if (r + 1 < nrows && sb < s1) fetch(sb);
        continue;
      }
      __syncwarp();
      const float rx = __shfl_sync(0xffffffffu, gp[0].x, 0), ry = __shfl_sync(0xffffffffu, gp[0].y, 0),
                  rz = __shfl_sync(0xffffffffu, gp[0].z, 0);
      WarpBox sbox;
      sbox.init();
      float hmin = 3.0e38f;
#pragma unroll
      for (int j = 0; j < SL; ++j) {
        const int e = ((lane + 32 * j) >> 1) * 8 + (lane & 1);
        float *dp = reinterpret_cast<float *>(st.P) + e, *dq = reinterpret_cast<float *>(st.Q) + e,
              *dn = reinterpret_cast<float *>(st.N) + e;
        const float4 p = gp[j], q = gq[j];
        dp[0] = p.x; dp[2] = p.y; dp[4] = p.z; dp[6] = p.w;
        dq[0] = q.x; dq[2] = q.y; dq[4] = q.z; dq[6] = q.w;
        const float px = p.x - rx, py = p.y - ry, pz = p.z - rz;
        dn[0] = py * q.z - pz * q.y;
        dn[2] = pz * q.x - px * q.z;
        dn[4] = px * q.y - py * q.x;
        if constexpr (SPLIT) {
          float *dl_ = reinterpret_cast<float *>(st.L) + e;
          dl_[0] = gl[j].x; dl_[2] = gl[j].y; dl_[4] = gl[j].z;
        }
        if (cur + lane + 32 * j < s1) {
          sbox.add(p.x, p.y, p.z, p.w);
          hmin = fminf(hmin, p.w);
        }
      }
      reduce_box(sbox);
      const bool far = all_far(tb, sbox);
      __syncwarp();
      if (r + 1 < nrows && sb < s1) fetch(sb);
      const int npr = (int)(min((int64_t)S, s1 - cur) + 1) >> 1;  // an odd tail pairs with a padding source

      float2 sv[3], sd[3], sp[3];
      float sdv[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int m = 0; m < 3; ++m) sv[m] = sd[m] = sp[m] = dup2(0.f);
      if (far) {
        float2 B3[3];
        far_b3(pt.x - rx, pt.y - ry, pt.z - rz, AT3, B3);
#pragma unroll 2
        for (int r = 0; r < npr; ++r) {
          const float4 pa = st.P[2 * r], pb = st.P[2 * r + 1], qa = st.Q[2 * r], qb = st.Q[2 * r + 1],
                       na = st.N[2 * r], nb = st.N[2 * r + 1];
          far_pair2(make_float2(pa.x, pa.y), make_float2(pa.z, pa.w), make_float2(pb.x, pb.y),
                    make_float2(qa.x, qa.y), make_float2(qa.z, qa.w), make_float2(qb.x, qb.y),
                    make_float2(na.x, na.y), make_float2(na.z, na.w), make_float2(nb.x, nb.y), X, AT3, B3, sv, sd, sp);
        }
      } else {
        float2 sdv2[3] = {dup2(0.f), dup2(0.f), dup2(0.f)};
        auto mid = [&](const MidSigma2 *uni) {
#pragma unroll 2
          for (int r = 0; r < npr; ++r) {
            const float4 pa = st.P[2 * r], pb = st.P[2 * r + 1], qa = st.Q[2 * r], qb = st.Q[2 * r + 1];
            float2 lx = dup2(0.f), ly = lx, lz = lx;
            if constexpr (SPLIT) {
              const float4 la = st.L[2 * r], lb = st.L[2 * r + 1];
              lx = make_float2(la.x, la.y); ly = make_float2(la.z, la.w); lz = make_float2(lb.x, lb.y);
            }
            mid_pair2<SPLIT>(make_float2(pa.x, pa.y), make_float2(pa.z, pa.w), make_float2(pb.x, pb.y),
                             make_float2(pb.z, pb.w), make_float2(qa.x, qa.y), make_float2(qa.z, qa.w),
                             make_float2(qb.x, qb.y), make_float2(qb.z, qb.w), lx, ly, lz, X, xl, at, pt.w,
                             kFarU * pt.w, qt.w, uni, sv, sd, sp, sdv2, nfull);
          }
        };
        // one sigma for all of the slice's pairs, as in every wake shed with
        // one radius: its factors leave the loop (an odd tail's padding
        // source carries no strength, so its sigma does not matter)
        if (warp_min(hmin) == sbox.hs && thmin == tb.hs) {
          const MidSigma2 g = mid_sigma2(dup2(tb.hs + sbox.hs));
          mid(&g);
        } else {
          mid(nullptr);
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) sdv[m] = sdv2[m].x + sdv2[m].y;
      }
      fold_group_f32(far, pt.x - rx, pt.y - ry, pt.z - rz, at, a.nu2, sv, sd, sp, sdv, vh, vl, dh, dl);
    }
    const unsigned wsum = __reduce_add_sync(0xffffffffu, nfull);
    if (lane == 0 && wsum) atomicAdd(a.nfull, (unsigned long long)wsum);

    __syncthreads();  // every warp is done with its slices
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      red[(w * 6 + m) * TT + lane] = (double)vh[m] + (double)vl[m];
      red[(w * 6 + 3 + m) * TT + lane] = (double)dh[m] + (double)dl[m];
    }
    __syncthreads();
    // the CTA of the tile's last row also clears the partials no CTA has
    const int clear = row + nrows == first + rps ? a.nch : c + 1;
    for (int e = threadIdx.x; e < 6 * TT; e += 32 * W) {
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < W; ++k) v += red[k * 6 * TT + e];
      const int64_t i = t0 + e % TT;
      if (i >= tend) continue;
      double *o = a.partial + (e / TT) * a.cap + i;
      o[c * 6 * a.cap] = v * kInv4Pi;
      for (int k = c + 1; k < clear; ++k) o[k * 6 * a.cap] = 0.0;
    }
    __syncthreads();  // before the next tile's slices overwrite the sums
    row += nrows;
  }
}

}  // namespace pgpu
