// FP64 pair kernel over the row list of pair_slices.cuh: rows of 32 targets by
// eight slices of 32 SL sources, one slice per warp.
//
// Bound by the FP64 pipe (64 lanes per SM and clock): 30 operations per pair of
// a far slice (u >= 100, where the far limit equals the closed form to double
// rounding), the closed form under a warp vote in the others; high-order kernel
// 43 per pair.  The records are staged as double2 (x, y), (z, sigma^2/2),
// (ax, ay), (az, volume) and n_s, so that a far pair loads nine 8-byte words
// (an FP64 operation takes a warp two issue cycles of one scheduler, a 16-byte
// broadcast load about two of the SM).  The compensated (hi, lo) sums live in
// shared memory, touched once per slice: 24 registers less per thread, which
// go to loads and roots in flight at 16 warps per SM.
#pragma once

namespace pgpu {

template <int SL> struct SliceStage64 {
  double2 xy[32 * SL], zh[32 * SL], axy[32 * SL], azv[32 * SL], nxy[32 * SL];
  double nz[32 * SL];
};

__device__ __forceinline__ bool bounded(const WarpBox &b) {
  const float lo = fminf(fminf(b.lo[0], b.lo[1]), b.lo[2]), hi = fmaxf(fmaxf(b.hi[0], b.hi[1]), b.hi[2]);
  return lo > -1e18f && hi < 1e18f && b.hs < 1e36f;
}

template <int SL, int KER>
__global__ void __launch_bounds__(32 * kSliceWarps, 2) pair_slices64_kernel(PairArgs<double> a) {
  constexpr int W = kSliceWarps, S = 32 * SL;
  // dynamic shared memory: the warps' slices, then their (hi, lo) sums,
  // [warp][component][lane] (sums_hi is also the reduction buffer)
  extern __shared__ __align__(16) unsigned char dyn64[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  SliceStage64<SL> &st = reinterpret_cast<SliceStage64<SL> *>(dyn64)[w];
  double *sums_hi = reinterpret_cast<double *>(dyn64 + W * sizeof(SliceStage64<SL>));
  double *hi = sums_hi + w * 6 * 32 + lane, *lo = hi + W * 6 * 32;
  const int64_t rpc = a.plan[a.nsys].chunk;
  const int64_t row1 = min((blockIdx.x + 1) * rpc, a.plan[a.nsys].item_start);
  for (int64_t row = blockIdx.x * rpc; row < row1;) {
    const RowRun run = row_run(a.plan, a.nsys, rpc, row, row1);
    const int64_t s1 = run.s1;
    int64_t g = run.g;
    const int64_t ti = min(run.t0 + lane, run.tend - 1);
    const double4 pt = a.P[ti], qt = a.Q[ti];
    const double xt[3] = {pt.x, pt.y, pt.z}, at[3] = {qt.x, qt.y, qt.z}, hst = pt.w, vt = qt.w;
    const double at3[3] = {-3.0 * at[0], -3.0 * at[1], -3.0 * at[2]};
    WarpBox tb;
    tb.init();
    tb.add((float)pt.x, (float)pt.y, (float)pt.z, (float)pt.w);
    reduce_box(tb);
    tb.widen();
    const double hst0 = __shfl_sync(0xffffffffu, hst, 0);
    const bool one_t = __all_sync(0xffffffffu, hst == hst0);
#pragma unroll
    for (int m = 0; m < 6; ++m) hi[32 * m] = lo[32 * m] = 0.0;
    unsigned nfull = 0;

    for (int r = 0; r < run.nrows; ++r) {
      const int64_t cur = run.pe.off + (g * W + w) * S;
      g += run.pe.mult;
      if (g >= run.pe.chunk) g -= run.pe.chunk;
      if (cur >= s1) continue;  // past the last source: this warp has no slice in the row
      __syncwarp();
      WarpBox sbox;
      sbox.init();
      double rx = 0, ry = 0, rz = 0;  // reference point: the slice's first source
      double hs0 = 0;
      bool one = one_t;  // one sigma for all of the slice's pairs
#pragma unroll
      for (int j = 0; j < SL; ++j) {
        const int64_t i = cur + lane + 32 * j;
        const double4 p = i < s1 ? a.P[i] : pad_P<double>();
        const double4 q = i < s1 ? a.Q[i] : pad_Q<double>();
        if (j == 0) {
          rx = __shfl_sync(0xffffffffu, p.x, 0);
          ry = __shfl_sync(0xffffffffu, p.y, 0);
          rz = __shfl_sync(0xffffffffu, p.z, 0);
          hs0 = __shfl_sync(0xffffffffu, p.w, 0);
        }
        one = one && (p.w == hs0 || i >= s1);
        const int e = lane + 32 * j;
        const double px = p.x - rx, py = p.y - ry, pz = p.z - rz;
        st.xy[e] = make_double2(p.x, p.y);
        st.zh[e] = make_double2(p.z, p.w);
        st.axy[e] = make_double2(q.x, q.y);
        st.azv[e] = make_double2(q.z, q.w);
        st.nxy[e] = make_double2(py * q.z - pz * q.y, pz * q.x - px * q.z);
        st.nz[e] = px * q.y - py * q.x;
        if (i < s1) sbox.add((float)p.x, (float)p.y, (float)p.z, (float)p.w);
      }
      reduce_box(sbox);
      sbox.widen();
      one = __all_sync(0xffffffffu, one);
      const double is1 = one ? fast_rsqrt(hst0 + hs0) : 0.0;  // then 1/sigma leaves the loop
      // far by the boxes, as the tiles of pair_body_generic; positions below
      // 1e18 keep rho^2 of a far pair a positive normal number, so that its
      // root needs no test
      const bool far = all_far(tb, sbox, KER == kGaussian ? (float)kFarU64 : kFarU) && bounded(tb) && bounded(sbox);
      __syncwarp();
      const int cnt = (int)min((int64_t)S, s1 - cur);

      double sv[3] = {0, 0, 0}, sd[3] = {0, 0, 0}, sp[3] = {0, 0, 0}, sdv[3] = {0, 0, 0};
      if (far) {
        const double xr0 = xt[0] - rx, xr1 = xt[1] - ry, xr2 = xt[2] - rz;
        const double b3[3] = {xr1 * at3[2] - xr2 * at3[1], xr2 * at3[0] - xr0 * at3[2], xr0 * at3[1] - xr1 * at3[0]};
        double sw = 0.0;
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
          const double2 xy = st.xy[j], axy = st.axy[j], nxy = st.nxy[j];
          const double nz = st.nz[j];
          const double z = st.zh[j].x, az = st.azv[j].x;
          double q, F;
          const double dx = xt[0] - xy.x, dy = xt[1] - xy.y, dz = xt[2] - z;
          if constexpr (KER == kGaussian) {
            // far limit: q' = r^3, F' = -3 r^5 (the -3 is in at3 and b3), no diffusion
            const double ir = rsqrt_normal(dx * dx + dy * dy + dz * dz);
            const double A = ir * ir;
            q = A * ir;
            F = q * A;
          } else {
            const double s2 = hst + st.zh[j].y;
            const double R = fma(dz, dz, fma(dy, dy, fma(dx, dx, s2)));
            const double iR = rsqrt_normal(R);
            const double iR2 = iR * iR, iR5 = iR2 * iR2 * iR, iR7 = iR5 * iR2;
            q = fma(1.5, s2, R) * iR5;
            F = fma(2.5, s2, R) * iR7;
            const double zd = (s2 * s2) * (iR7 * iR2);
            sdv[0] = fma(zd, axy.x, sdv[0]);
            sdv[1] = fma(zd, axy.y, sdv[1]);
            sdv[2] = fma(zd, az, sdv[2]);
            sw = fma(zd, st.azv[j].y, sw);
          }
          sp[0] += q * axy.x; sp[1] += q * axy.y; sp[2] += q * az;
          sv[0] += q * nxy.x; sv[1] += q * nxy.y; sv[2] += q * nz;
          const double fd =
              F * (axy.x * b3[0] + axy.y * b3[1] + az * b3[2] + nxy.x * at3[0] + nxy.y * at3[1] + nz * at3[2]);
          sd[0] += fd * dx; sd[1] += fd * dy; sd[2] += fd * dz;
        }
        if constexpr (KER == kHighOrder) {
#pragma unroll
          for (int m = 0; m < 3; ++m) sdv[m] = HighOrder::kZd * (vt * sdv[m] - sw * at[m]);
        }
        // velocity = (sum q alpha_s) x X' + sum q n_s
        const double n0 = sv[0], n1 = sv[1], n2 = sv[2];
        sv[0] = sp[1] * xr2 - sp[2] * xr1 + n0;
        sv[1] = sp[2] * xr0 - sp[0] * xr2 + n1;
        sv[2] = sp[0] * xr1 - sp[1] * xr0 + n2;
      } else {
#pragma unroll 2
        for (int j = 0; j < cnt; ++j) {
          const double2 xy = st.xy[j], zh = st.zh[j], axy = st.axy[j], azv = st.azv[j];
          const double dx = xt[0] - xy.x, dy = xt[1] - xy.y, dz = xt[2] - zh.x;
          const double r2 = dx * dx + dy * dy + dz * dz, s2 = hst + zh.y;
          double q, F;
          if constexpr (KER == kGaussian) {
            const double ir = fast_rsqrt(r2);
            const double A = ir * ir;
            q = A * ir;
            F = -3.0 * q * A;
            const bool near = r2 < kFarU64 * s2;
            if (__any_sync(0xffffffffu, near)) {
              if (near) {
                const PairTerms<double> t = pair_terms(r2, s2, ir, one ? is1 : fast_rsqrt(s2));
                q = t.q; F = t.F;
                sdv[0] += t.zd * (vt * axy.x - azv.y * at[0]);
                sdv[1] += t.zd * (vt * axy.y - azv.y * at[1]);
                sdv[2] += t.zd * (vt * azv.x - azv.y * at[2]);
                ++nfull;
              }
            }
          } else {
            const PairTerms<double> t = pair_terms_ho(r2, s2);
            q = t.q; F = t.F;
            sdv[0] += t.zd * (vt * axy.x - azv.y * at[0]);
            sdv[1] += t.zd * (vt * axy.y - azv.y * at[1]);
            sdv[2] += t.zd * (vt * azv.x - azv.y * at[2]);
          }
          // w = alpha_s x d, d . (alpha_t x alpha_s) = alpha_t . w
          const double wx = axy.y * dz - azv.x * dy, wy = azv.x * dx - axy.x * dz, wz = axy.x * dy - axy.y * dx;
          sv[0] += q * wx; sv[1] += q * wy; sv[2] += q * wz;
          const double fd = F * (at[0] * wx + at[1] * wy + at[2] * wz);
          sd[0] += fd * dx; sd[1] += fd * dy; sd[2] += fd * dz;
          sp[0] += q * axy.x; sp[1] += q * axy.y; sp[2] += q * azv.x;
        }
      }
      // da = alpha_t x (sum q alpha_s) + sum F (d.c) d + 2 nu sum z (v_t a_s - v_s a_t)
      const double add[6] = {sv[0], sv[1], sv[2],
                             at[1] * sp[2] - at[2] * sp[1] + sd[0] + a.nu2 * sdv[0],
                             at[2] * sp[0] - at[0] * sp[2] + sd[1] + a.nu2 * sdv[1],
                             at[0] * sp[1] - at[1] * sp[0] + sd[2] + a.nu2 * sdv[2]};
#pragma unroll
      for (int m = 0; m < 6; ++m) two_sum_acc(hi[32 * m], lo[32 * m], add[m]);
    }
    if constexpr (KER == kGaussian) {
      const unsigned wsum = __reduce_add_sync(0xffffffffu, run.t0 + lane < run.tend ? nfull : 0u);
      if (lane == 0 && wsum) atomicAdd(a.nfull, (unsigned long long)wsum);
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) hi[32 * m] += lo[32 * m];
    __syncthreads();
    row_run_sums<6>(run, sums_hi, kInv4Pi, a.partial, a.cap, a.nch);
    __syncthreads();  // before the next tile's sums
    row += run.nrows;
  }
}

template <int SL> constexpr size_t slices64_smem() {
  return kSliceWarps * (sizeof(SliceStage64<SL>) + 2 * 6 * 32 * sizeof(double));
}

}  // namespace pgpu
