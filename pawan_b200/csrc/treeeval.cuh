// Surrogate evaluation on the octree of tree.cuh, FP32 with compensated sums.
//
// Far cells.  Beyond a few cell widths the Gaussian regularisation is below
// FP32 resolution (tests/test_math_fits.py), so a far cell acts through the
// singular kernel, written with phi(d) = 1/|d| (4 pi units, as the pair kernel):
//   velocity    alpha_s x d / rho^3                     = -alpha_s x grad phi(d)
//   stretching  b/rho^3 - 3 (d.b) d / rho^5, b = alpha_t x alpha_s  = -D2(d) b
// Expanding d = r - y about the cell centroid (r = x_t - c, y = x_s - c) in
// powers of y, with A = sum alpha, M_ab = sum alpha_a y_b,
// Q_abc = sum alpha_a y_b y_c, T_abcd = sum alpha_a y_b y_c y_d and Dn the
// n-th derivative tensors of phi at r:
//   u_i = -eps_iab [A_a D1_b - M_ac D2_bc + 1/2 Q_acd D3_bcd - 1/6 T_acde D4_bcde]
//   s_i = -[D2_ik B_k - D3_ikc N_kc + 1/2 D4_ikcd P_kcd - 1/6 D5_ikcde R_kcde],
//         B = alpha_t x A, N_.c = alpha_t x M_.c, P_.cd = alpha_t x Q_.cd,
//         R_.cde = alpha_t x T_.cde.
// `order` 0 keeps the monopole, 1 adds the dipole, 2 the quadrupole, 3 the
// octupole.  The contractions below never form the derivative tensors; the
// order-3 contractions were checked in a CPU restatement against the full
// tensor contraction, and tests/test_surrogate.py checks the result end to
// end (the error falls with the order against the direct sum).
//
// Near leaves.  Exact pair sums with the same three-regime FP32 terms as the
// direct kernel.
#pragma once
#include "kernels.cuh"
#include "mlp.cuh"
#include "tree.cuh"

namespace pgpu {

__device__ __forceinline__ void cross3f(const float *a, const float *b, float *c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}

// Velocity u and stretching s (4 pi units) induced at a target (position x,
// strength at) by a far cell (data v), to the given order.
__device__ __forceinline__ void far_expand(const float *v, const float *x, const float *at, int order, float *u,
                                           float *s) {
  const float r[3] = {x[0] - v[0], x[1] - v[1], x[2] - v[2]};
  const float r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
  const float ir = fast_rsqrt(r2);
  const float ir2 = ir * ir, ir3 = ir * ir2, ir5 = ir3 * ir2, ir7 = ir5 * ir2, ir9 = ir7 * ir2;
  const float A[3] = {v[3], v[4], v[5]};
  float t[3];
  cross3f(A, r, t);
  for (int i = 0; i < 3; ++i) u[i] = ir3 * t[i];
  float B[3];
  cross3f(at, A, B);
  const float rB = r[0] * B[0] + r[1] * B[1] + r[2] * B[2];
  for (int i = 0; i < 3; ++i) s[i] = ir3 * B[i] - 3.f * ir5 * rB * r[i];
  if (order < 1) return;
  // ---- dipole
  const float *M = v + 6;  // M[a*3+b]
  float Mr[3];
  for (int a = 0; a < 3; ++a) Mr[a] = M[3 * a] * r[0] + M[3 * a + 1] * r[1] + M[3 * a + 2] * r[2];
  const float mx[3] = {M[5] - M[7], M[6] - M[2], M[1] - M[3]};
  cross3f(Mr, r, t);
  for (int i = 0; i < 3; ++i) u[i] += 3.f * ir5 * t[i] - ir3 * mx[i];
  float N[3][3];  // N[k][c] = (at x M_.c)_k
  for (int c = 0; c < 3; ++c) {
    const float col[3] = {M[c], M[3 + c], M[6 + c]};
    float n[3];
    cross3f(at, col, n);
    N[0][c] = n[0]; N[1][c] = n[1]; N[2][c] = n[2];
  }
  float Nr[3], NTr[3];
  for (int i = 0; i < 3; ++i) {
    Nr[i] = N[i][0] * r[0] + N[i][1] * r[1] + N[i][2] * r[2];
    NTr[i] = N[0][i] * r[0] + N[1][i] * r[1] + N[2][i] * r[2];
  }
  const float rNr = r[0] * Nr[0] + r[1] * Nr[1] + r[2] * Nr[2];
  const float trN = N[0][0] + N[1][1] + N[2][2];
  for (int i = 0; i < 3; ++i) s[i] += -15.f * ir7 * rNr * r[i] + 3.f * ir5 * (Nr[i] + NTr[i] + r[i] * trN);
  if (order < 2) return;
  // ---- quadrupole; Q_a packed (00,01,02,11,12,22)
  const float *Qp = v + 15;
  float sv[3], tv[3], W[3][3];
  for (int a = 0; a < 3; ++a) {
    const float *q = Qp + 6 * a;
    W[a][0] = q[0] * r[0] + q[1] * r[1] + q[2] * r[2];
    W[a][1] = q[1] * r[0] + q[3] * r[1] + q[4] * r[2];
    W[a][2] = q[2] * r[0] + q[4] * r[1] + q[5] * r[2];
    sv[a] = r[0] * W[a][0] + r[1] * W[a][1] + r[2] * W[a][2];
    tv[a] = q[0] + q[3] + q[5];
  }
  const float wx[3] = {W[1][2] - W[2][1], W[2][0] - W[0][2], W[0][1] - W[1][0]};
  float sr[3], tr[3];
  cross3f(sv, r, sr);
  cross3f(tv, r, tr);
  for (int i = 0; i < 3; ++i) u[i] += 7.5f * ir7 * sr[i] - 1.5f * ir5 * (2.f * wx[i] + tr[i]);
  // P_k (symmetric over cd) = (at x Q_.cd)_k
  float P[3][6];
  for (int e = 0; e < 6; ++e) {
    const float col[3] = {Qp[e], Qp[6 + e], Qp[12 + e]};
    float p[3];
    cross3f(at, col, p);
    P[0][e] = p[0]; P[1][e] = p[1]; P[2][e] = p[2];
  }
  float Pr[3][3], rPr[3], trP[3];
  for (int k = 0; k < 3; ++k) {
    const float *q = P[k];
    Pr[k][0] = q[0] * r[0] + q[1] * r[1] + q[2] * r[2];
    Pr[k][1] = q[1] * r[0] + q[3] * r[1] + q[4] * r[2];
    Pr[k][2] = q[2] * r[0] + q[4] * r[1] + q[5] * r[2];
    rPr[k] = r[0] * Pr[k][0] + r[1] * Pr[k][1] + r[2] * Pr[k][2];
    trP[k] = q[0] + q[3] + q[5];
  }
  const float srPr = r[0] * rPr[0] + r[1] * rPr[1] + r[2] * rPr[2];
  const float sPrk = Pr[0][0] + Pr[1][1] + Pr[2][2];  // sum_k (P_k r)_k
  const float rtr = r[0] * trP[0] + r[1] * trP[1] + r[2] * trP[2];
  // sum_k P_k[i][k]: P_k packed; entry (i,k)
  auto pik = [&](int k, int i) {
    const int a = min(i, k), b = max(i, k);
    const int e = a == 0 ? b : (a == 1 ? 2 + b : 5);
    return P[k][e];
  };
  for (int i = 0; i < 3; ++i) {
    const float sumPk = r[0] * Pr[0][i] + r[1] * Pr[1][i] + r[2] * Pr[2][i];
    const float spik = pik(0, i) + pik(1, i) + pik(2, i);
    const float d4p = 105.f * ir9 * r[i] * srPr -
                      15.f * ir7 * (rPr[i] + 2.f * sumPk + 2.f * r[i] * sPrk + r[i] * rtr) +
                      3.f * ir5 * (trP[i] + 2.f * spik);
    s[i] -= 0.5f * d4p;
  }
  if (order < 3) return;
  // ---- octupole; T_a packed (000,001,002,011,012,022,111,112,122,222).
  // For a symmetric third-order tensor S: Sr[b][d] = S_bde r_e (symmetric),
  // S1 = Sr r, S0 = S1.r, tS_b = S_bdd, and S_ccd r_d = tS.r.
  //   u_i += 1/6 eps_iab [105 S0_a r_b / rho^9 - 45 (S1_ab + r_b (tS_a.r)) / rho^7 + 9 tS_ab / rho^5]
  //   s_i += 1/6 D5_ikcde R_kcde, R_k = (alpha_t x T_.)_k, by the pairings of
  //   D5 = -945 r r r r r / rho^11 + 105 sum_10 (delta r r r) / rho^9 - 15 sum_15 (delta delta r) / rho^7
  const float ir11 = ir9 * ir2;
  auto sym3 = [&](const float *S, float Sr[3][3], float *S1, float &S0, float *tS) {
    // S index of (b, c, d), b <= c <= d sorted
    Sr[0][0] = S[0] * r[0] + S[1] * r[1] + S[2] * r[2];
    Sr[0][1] = S[1] * r[0] + S[3] * r[1] + S[4] * r[2];
    Sr[0][2] = S[2] * r[0] + S[4] * r[1] + S[5] * r[2];
    Sr[1][1] = S[3] * r[0] + S[6] * r[1] + S[7] * r[2];
    Sr[1][2] = S[4] * r[0] + S[7] * r[1] + S[8] * r[2];
    Sr[2][2] = S[5] * r[0] + S[8] * r[1] + S[9] * r[2];
    Sr[1][0] = Sr[0][1]; Sr[2][0] = Sr[0][2]; Sr[2][1] = Sr[1][2];
    for (int b = 0; b < 3; ++b) S1[b] = Sr[b][0] * r[0] + Sr[b][1] * r[1] + Sr[b][2] * r[2];
    S0 = S1[0] * r[0] + S1[1] * r[1] + S1[2] * r[2];
    tS[0] = S[0] + S[3] + S[5];
    tS[1] = S[1] + S[6] + S[8];
    tS[2] = S[2] + S[7] + S[9];
  };
  const float *Tp = v + 40;
  {
    float S0[3], S1[3][3], tS[3][3], Sr[3][3];
    for (int a = 0; a < 3; ++a) sym3(Tp + 10 * a, Sr, S1[a], S0[a], tS[a]);
    for (int i = 0; i < 3; ++i) {
      const int a1 = (i + 1) % 3, b1 = (i + 2) % 3;  // eps_i a1 b1 = +1
      const float x1 = 105.f * ir9 * (S0[a1] * r[b1] - S0[b1] * r[a1]);
      const float sa1 = tS[a1][0] * r[0] + tS[a1][1] * r[1] + tS[a1][2] * r[2];
      const float sb1 = tS[b1][0] * r[0] + tS[b1][1] * r[1] + tS[b1][2] * r[2];
      const float x2 = -45.f * ir7 * ((S1[a1][b1] - S1[b1][a1]) + (sa1 * r[b1] - sb1 * r[a1]));
      const float x3 = 9.f * ir5 * (tS[a1][b1] - tS[b1][a1]);
      u[i] += (x1 + x2 + x3) * (1.f / 6.f);
    }
  }
  {
    // R_k = (alpha_t x T_.)_k, each a symmetric third-order tensor
    float R[3][10];
    for (int e = 0; e < 10; ++e) {
      const float col[3] = {Tp[e], Tp[10 + e], Tp[20 + e]};
      float p[3];
      cross3f(at, col, p);
      R[0][e] = p[0]; R[1][e] = p[1]; R[2][e] = p[2];
    }
    float M[3][3][3], r1[3][3], r0[3], tk[3][3];
    for (int k = 0; k < 3; ++k) sym3(R[k], M[k], r1[k], r0[k], tk[k]);
    float rr0 = 0.f, tr1 = 0.f, rsg = 0.f, trt = 0.f;
    for (int k = 0; k < 3; ++k) {
      rr0 += r[k] * r0[k];
      tr1 += r1[k][k];
      rsg += r[k] * (tk[k][0] * r[0] + tk[k][1] * r[1] + tk[k][2] * r[2]);
      trt += tk[k][k];
    }
    for (int i = 0; i < 3; ++i) {
      float rk1 = 0.f, rkt = 0.f, psi = 0.f;
      for (int k = 0; k < 3; ++k) {
        rk1 += r[k] * r1[k][i];
        rkt += r[k] * tk[k][i];
        psi += M[k][i][k];
      }
      const float ti_r = tk[i][0] * r[0] + tk[i][1] * r[1] + tk[i][2] * r[2];
      const float t1 = -945.f * ir11 * r[i] * rr0;
      const float t2 = 105.f * ir9 * (r0[i] + 3.f * rk1 + 3.f * r[i] * tr1 + 3.f * r[i] * rsg);
      const float t3 = -15.f * ir7 * (3.f * r[i] * trt + 3.f * rkt + 3.f * ti_r + 6.f * psi);
      s[i] += (t1 + t2 + t3) * (1.f / 6.f);
    }
  }
}

// The expansion to order ORD <= 2 of two far cells at once (lane .x the even
// cell, .y the odd one), added to u and s.  The terms are those of far_expand,
// arranged by strength component: with Phi_a = sum alpha_a phi,
//   u = -curl-like  -eps_kab d_b Phi_a,   s_i = d_i (alpha_t . u) = sum_a (H^a V_a)_i,
// H^a the Hessian of Phi_a and V_a the (negated) rows of alpha_t's cross matrix,
// two components each.  Per a, with m = M_a, Q = Q_a:
//   grad = c2 r + ir^3 m + 3 ir^5 Q r
//   H V  = r (c1 r.V + w.V) + w (r.V) + c2 V + 3 ir^5 Q V
//   c2 = -A ir^3 - 3 ir^5 m.r - 7.5 ir^7 r.Q r + 1.5 ir^5 tr Q
//   c1 = 3 A ir^5 + 15 ir^7 m.r + 52.5 ir^9 r.Q r - 7.5 ir^7 tr Q
//   w  = -3 ir^5 m - 15 ir^7 Q r
// About 190 packed operations at order 2; far_expand forms alpha_t x A, M and Q
// per target, about 310 (1M coaxial rings, 1250 far cells per target:
// evaluation 97 ms instead of 105 ms).
template <int ORD>
__device__ __forceinline__ void far_expand2(const float2 *v, const float2 *x, const float2 *at, const float2 *nat,
                                            float2 *u, float2 *s) {
  const float2 M1 = dup2(-1.f);
  const float2 r[3] = {__ffma2_rn(v[0], M1, x[0]), __ffma2_rn(v[1], M1, x[1]), __ffma2_rn(v[2], M1, x[2])};
  const float2 r2 = __ffma2_rn(r[2], r[2], __ffma2_rn(r[1], r[1], __fmul2_rn(r[0], r[0])));
  const float2 ir = make_float2(fast_rsqrt(r2.x), fast_rsqrt(r2.y));
  const float2 ir2 = __fmul2_rn(ir, ir), ir3 = __fmul2_rn(ir2, ir);
  const float2 nir3 = __fmul2_rn(ir3, M1);
  const float2 k3 = __fmul2_rn(__fmul2_rn(ir3, ir2), dup2(3.f));  // 3 ir^5
  const float2 nk3 = __fmul2_rn(k3, M1);
  const float2 k15 = __fmul2_rn(__fmul2_rn(k3, ir2), dup2(5.f));  // 15 ir^7
  const float2 nk15 = __fmul2_rn(k15, M1), nk75 = __fmul2_rn(k15, dup2(-0.5f));
  const float2 k525 = __fmul2_rn(__fmul2_rn(k15, ir2), dup2(3.5f));  // 52.5 ir^9
  const float2 hk3 = __fmul2_rn(k3, dup2(0.5f));
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int p = (a + 1) % 3, q = (a + 2) % 3;
    // -V_a: component p is -alpha_t[q], component q is +alpha_t[p]
    const float2 Vp = nat[q], Vq = at[p];
    float2 c2 = __fmul2_rn(v[3 + a], nir3), c1 = __fmul2_rn(v[3 + a], k3);
    float2 w[3], Qr[3];
    const float2 *m = v + 6 + 3 * a, *Q = v + 15 + 6 * a;  // Q packed (00,01,02,11,12,22)
    if constexpr (ORD >= 1) {
      const float2 mr = __ffma2_rn(m[2], r[2], __ffma2_rn(m[1], r[1], __fmul2_rn(m[0], r[0])));
      c2 = __ffma2_rn(nk3, mr, c2);
      c1 = __ffma2_rn(k15, mr, c1);
#pragma unroll
      for (int i = 0; i < 3; ++i) w[i] = __fmul2_rn(nk3, m[i]);
    }
    if constexpr (ORD >= 2) {
      Qr[0] = __ffma2_rn(Q[2], r[2], __ffma2_rn(Q[1], r[1], __fmul2_rn(Q[0], r[0])));
      Qr[1] = __ffma2_rn(Q[4], r[2], __ffma2_rn(Q[3], r[1], __fmul2_rn(Q[1], r[0])));
      Qr[2] = __ffma2_rn(Q[5], r[2], __ffma2_rn(Q[4], r[1], __fmul2_rn(Q[2], r[0])));
      const float2 rQr = __ffma2_rn(Qr[2], r[2], __ffma2_rn(Qr[1], r[1], __fmul2_rn(Qr[0], r[0])));
      const float2 tr = __fadd2_rn(__fadd2_rn(Q[0], Q[3]), Q[5]);
      c2 = __ffma2_rn(hk3, tr, __ffma2_rn(nk75, rQr, c2));
      c1 = __ffma2_rn(nk75, tr, __ffma2_rn(k525, rQr, c1));
#pragma unroll
      for (int i = 0; i < 3; ++i) w[i] = __ffma2_rn(nk15, Qr[i], w[i]);
    }
    // gradient components p and q: u[q] -= g_p, u[p] += g_q
    float2 gp = __fmul2_rn(c2, r[p]), gq = __fmul2_rn(c2, r[q]);
    if constexpr (ORD >= 1) {
      gp = __ffma2_rn(ir3, m[p], gp);
      gq = __ffma2_rn(ir3, m[q], gq);
    }
    if constexpr (ORD >= 2) {
      gp = __ffma2_rn(k3, Qr[p], gp);
      gq = __ffma2_rn(k3, Qr[q], gq);
    }
    u[q] = __ffma2_rn(gp, M1, u[q]);
    u[p] = __fadd2_rn(u[p], gq);
    const float2 rv = __ffma2_rn(r[q], Vq, __fmul2_rn(r[p], Vp));
    float2 t = __fmul2_rn(c1, rv);
    if constexpr (ORD >= 1) t = __ffma2_rn(w[q], Vq, __ffma2_rn(w[p], Vp, t));
    s[p] = __ffma2_rn(c2, Vp, s[p]);
    s[q] = __ffma2_rn(c2, Vq, s[q]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      s[i] = __ffma2_rn(r[i], t, s[i]);
      if constexpr (ORD >= 1) s[i] = __ffma2_rn(w[i], rv, s[i]);
      if constexpr (ORD >= 2) {
        constexpr int S[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
        const float2 qv = __ffma2_rn(Q[S[i][q]], Vq, __fmul2_rn(Q[S[i][p]], Vp));
        s[i] = __ffma2_rn(k3, qv, s[i]);
      }
    }
  }
}

// Input features of the far-field correction network for one (target, far
// cell) pair, and the scales of its outputs.  With r = x_t - c (c the cell's
// particle centroid, the expansion origin), rho = |r|, rh = r/rho, w the cube
// width, A = sum alpha, Q_j = sum alpha_j y y^T (y = x_s - c) the second
// moments and C = sum_j (A_j/|A|) Q_j:
//   0-2 rh, 3 4w/rho, 4 4 sigma_c/rho, 5-7 A/|A|,
//   8-10 4 eps_ijk (Q_j rh)_k / (|A| w^2), 11-13 4 rh.Q_j.rh / (|A| w^2),
//   14-16 4 tr Q_j / (|A| w^2), 17-19 16 C rh/(|A| rho^2),
//   20-22 alpha_t/|alpha_t|, 23 16 rh.C.rh/(|A| rho^2)
// The residual of the monopole+dipole expansion is led by the quadrupole
// term, whose velocity is exactly
//   (-3 eps_ijk (Q_j rh)_k + (7.5 rh.Q_j.rh - 1.5 tr Q_j) (e_j x rh)_i) / rho^4
// (4 pi units), a function of slots 0-2 and 8-16 alone; its stretching
// also involves alpha_t, and for strengths close to one direction (Q_j ~
// A_j C / |A|) it depends on C through C rh and rh.C.rh.  sigma_c (the cell's
// mean smoothing radius) carries what is left of the Gaussian regularisation
// for cells only a few radii away.  The network predicts the residual in
// units of the quadrupole scale: velocity / (|A| w^2 / rho^4), stretching /
// (|A| |alpha_t| w^2 / rho^5) (4 pi units).
__device__ __forceinline__ void far_features(const float *v, const float *x, const float *at, float *f, float &sv,
                                             float &ss) {
  const float r[3] = {x[0] - v[0], x[1] - v[1], x[2] - v[2]};
  const float r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
  const float ir = fast_rsqrt(r2);
  const float rh[3] = {r[0] * ir, r[1] * ir, r[2] * ir};
  for (int i = 0; i < 3; ++i) f[i] = rh[i];
  const float w = v[34];
  f[3] = 4.f * w * ir;
  f[4] = 4.f * sqrtf(2.f * v[38]) * ir;
  const float am = sqrtf(v[3] * v[3] + v[4] * v[4] + v[5] * v[5]);
  const float ia = am > 0.f ? 1.f / am : 0.f;
  const float ah[3] = {v[3] * ia, v[4] * ia, v[5] * ia};
  for (int i = 0; i < 3; ++i) f[5 + i] = ah[i];
  const float qs = w > 0.f ? 4.f * ia / (w * w) : 0.f;
  float P[3][3];  // P[j] = Q_j rh
  for (int j = 0; j < 3; ++j) {
    const float *Q = v + 15 + 6 * j;
    P[j][0] = Q[0] * rh[0] + Q[1] * rh[1] + Q[2] * rh[2];
    P[j][1] = Q[1] * rh[0] + Q[3] * rh[1] + Q[4] * rh[2];
    P[j][2] = Q[2] * rh[0] + Q[4] * rh[1] + Q[5] * rh[2];
    f[11 + j] = qs * (rh[0] * P[j][0] + rh[1] * P[j][1] + rh[2] * P[j][2]);
    f[14 + j] = qs * (Q[0] + Q[3] + Q[5]);
  }
  f[8] = qs * (P[1][2] - P[2][1]);
  f[9] = qs * (P[2][0] - P[0][2]);
  f[10] = qs * (P[0][1] - P[1][0]);
  // C = sum_a ah_a Q_a, packed (00,01,02,11,12,22)
  float Cp[6];
  for (int e = 0; e < 6; ++e) Cp[e] = ah[0] * v[15 + e] + ah[1] * v[21 + e] + ah[2] * v[27 + e];
  const float Cr[3] = {Cp[0] * rh[0] + Cp[1] * rh[1] + Cp[2] * rh[2], Cp[1] * rh[0] + Cp[3] * rh[1] + Cp[4] * rh[2],
                       Cp[2] * rh[0] + Cp[4] * rh[1] + Cp[5] * rh[2]};
  const float cs = 16.f * ia * ir * ir;
  for (int i = 0; i < 3; ++i) f[17 + i] = cs * Cr[i];
  const float tm = sqrtf(at[0] * at[0] + at[1] * at[1] + at[2] * at[2]);
  const float it = tm > 0.f ? 1.f / tm : 0.f;
  for (int i = 0; i < 3; ++i) f[20 + i] = at[i] * it;
  f[23] = cs * (rh[0] * Cr[0] + rh[1] * Cr[1] + rh[2] * Cr[2]);
  const float q2 = (w * ir) * (w * ir);
  sv = am * ir * ir * q2;
  ss = am * tm * ir * ir * ir * q2;
}

struct TreeEvalArgs {
  const CellData *cd;
  const TreeCell *cells;
  const int *leaves;
  int nleaves;
  const int *far_off, *far_cnt, *far_list;
  const int *near_off, *near_cnt;
  const int2 *near_runs;  // sorted-order particle ranges of the near field
  const float4 *Ps, *Qs;  // sorted records
  const int *idx;         // sorted position -> index within the system
  int64_t off;            // slot offset of the system
  double *partial;        // chunk 0 of [nch][6][cap]
  int64_t cap;
  float nu2;
  int order;
  // owned targets [own_lo, own_hi) (indices within the system); a context
  // with a target range evaluates and writes only these
  int own_lo, own_hi;
};

// Warp-independent form: every warp takes work items (target leaf, slice of
// 32 of its targets) from an atomic counter and stages its own source tiles,
// synchronising only within the warp.  Leaves average ~130 particles, so
// whole-leaf CTAs leave most warps idle; independent warps keep ~48 warps per
// SM busy.  items[k] = (leaf index, slice); counter[0] must be 0 at launch.
constexpr int kWarpTile = 64;
constexpr int kWarpCells = 16;
constexpr int kNearGroup = 16;  // pairs of a compensation group of the near field
constexpr int kWarpsPerCta = 4;

// Per-warp shared buffers (all carved from dynamic shared memory, after the
// packed network when the correction is on).
constexpr int kPairFloats = 33;  // centroid, A, M, Q: what the order-2 expansion reads
struct WarpSmem {
  union {
    float sc[kWarpCells][kCellFloats];
    float2 sc2[kWarpCells / 2][kPairFloats];  // cell pairs, interleaved
    SliceStage<kWarpTile / 32, false, false> near;
  };
};
struct WarpSmemMlp {
  __nv_bfloat16 sF[32][kInPad + 8];
  float sO[32][kOutPad];
};
constexpr int kWarpsPerCtaMlp = 12;  // warps sharing one copy of the network
template <bool MLP> constexpr int eval_warps() { return MLP ? kWarpsPerCtaMlp : kWarpsPerCta; }
template <bool MLP> constexpr size_t eval_smem() {
  return (MLP ? sizeof(MlpPacked) : 0) + eval_warps<MLP>() * (sizeof(WarpSmem) + (MLP ? sizeof(WarpSmemMlp) : 0));
}

template <bool MLP>
__global__ void __launch_bounds__(32 * eval_warps<MLP>()) tree_eval_warp_kernel(TreeEvalArgs a, const int2 *items,
                                                                             int nitems, unsigned *counter,
                                                                             const MlpPacked *mlp) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t off0 = MLP ? sizeof(MlpPacked) : 0;
  WarpSmem &ws = reinterpret_cast<WarpSmem *>(dyn_smem + off0)[w];
  WarpSmemMlp &wm = reinterpret_cast<WarpSmemMlp *>(dyn_smem + off0 + eval_warps<MLP>() * sizeof(WarpSmem))[w];
  if constexpr (MLP) {
    // the packed network, shared by the CTA's warps
    const uint4 *src = reinterpret_cast<const uint4 *>(mlp);
    uint4 *dst = reinterpret_cast<uint4 *>(dyn_smem);
    for (int i = threadIdx.x; i < (int)(sizeof(MlpPacked) / 16); i += blockDim.x) dst[i] = src[i];
    __syncthreads();
  }
  const MlpPacked &W = *reinterpret_cast<const MlpPacked *>(dyn_smem);
  for (;;) {
    int item = 0;
    if (lane == 0) item = (int)atomicAdd(counter, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= nitems) break;
    const int2 it = items[item];
    const int li = it.x;
    const TreeCell tc = a.cells[a.leaves[li]];
    // A slice of at most 16 targets (half of the leaves' last slices) gives
    // each of them two lanes, h = 0 and 1, which take every other pair of the
    // far cells and near sources and add their sums at the end (1M coaxial
    // rings: 90 ms instead of 97 ms).
    const int left = tc.end - (tc.start + it.y * 32);
    const bool half = !MLP && a.order <= 2 && left <= 16;
    const int h = half ? lane >> 4 : 0, step = half ? 2 : 1;
    const int t0 = tc.start + it.y * 32 + (half ? lane & 15 : lane);
    const int t = min(t0, tc.end - 1);
    const int ti = a.idx[t];
    const bool mine = t0 < tc.end && ti >= a.own_lo && ti < a.own_hi;
    if (!__any_sync(0xffffffffu, mine)) continue;  // a slice with no owned target
    const float4 pt = a.Ps[t], qt = a.Qs[t];
    const float xt[3] = {pt.x, pt.y, pt.z}, at[3] = {qt.x, qt.y, qt.z};
    const float hst = pt.w, vt = qt.w;
    float vh[3] = {0, 0, 0}, vl[3] = {0, 0, 0}, dh[3] = {0, 0, 0}, dl[3] = {0, 0, 0};
    const int fo = a.far_off[li], fn = a.far_cnt[li];
    // far cells, orders up to 2 without the network: two cells per packed
    // instruction, one compensated addition per kWarpCells cells
    auto far2 = [&](auto ord) {
      constexpr int ORD = decltype(ord)::value;
      const float2 x2[3] = {dup2(xt[0]), dup2(xt[1]), dup2(xt[2])};
      const float2 at2[3] = {dup2(at[0]), dup2(at[1]), dup2(at[2])};
      const float2 nat2[3] = {dup2(-at[0]), dup2(-at[1]), dup2(-at[2])};
      constexpr int nf = ORD == 0 ? 6 : ORD == 1 ? 15 : kPairFloats;
      for (int c0 = 0; c0 < fn; c0 += kWarpCells) {
        const int cn = min(kWarpCells, fn - c0), cp = (cn + 2 * step - 1) & ~(2 * step - 1);
        __syncwarp();
        for (int k = lane; k < cp * nf; k += 32) {
          const int cc = k / nf, e = k - cc * nf;
          // the last pairs are filled up with the last cell, without strength
          const float val = a.cd[a.far_list[fo + c0 + min(cc, cn - 1)]].v[e];
          reinterpret_cast<float *>(&ws.sc2[cc >> 1][e])[cc & 1] = cc < cn || e < 3 ? val : 0.f;
        }
        __syncwarp();
        float2 u2[3] = {dup2(0.f), dup2(0.f), dup2(0.f)}, s2[3] = {dup2(0.f), dup2(0.f), dup2(0.f)};
        for (int j = h; j < cp / 2; j += step) far_expand2<ORD>(ws.sc2[j], x2, at2, nat2, u2, s2);
        for (int m = 0; m < 3; ++m) {
          two_sum_acc(vh[m], vl[m], u2[m].x + u2[m].y);
          two_sum_acc(dh[m], dl[m], s2[m].x + s2[m].y);
        }
      }
    };
    const bool packed = !MLP && a.order <= 2;
    if constexpr (!MLP) {
      if (a.order == 2) far2(IntType<2>{});
      else if (a.order == 1) far2(IntType<1>{});
      else if (a.order == 0) far2(IntType<0>{});
    }
    for (int c0 = packed ? fn : 0; c0 < fn; c0 += kWarpCells) {
      const int cn = min(kWarpCells, fn - c0);
      __syncwarp();
      // the cell data the expansion reads: the third moments only at order 3
      const int nf = a.order >= 3 ? kCellFloats : 40;
      for (int e = lane; e < cn * nf; e += 32)
        ws.sc[e / nf][e % nf] = a.cd[a.far_list[fo + c0 + e / nf]].v[e % nf];
      __syncwarp();
      float su[3] = {0, 0, 0}, ss[3] = {0, 0, 0};
      for (int j = 0; j < cn; ++j) {
        float u[3], s[3];
        far_expand(ws.sc[j], xt, at, a.order, u, s);
        for (int m = 0; m < 3; ++m) { su[m] += u[m]; ss[m] += s[m]; }
        if constexpr (MLP) {
          float f[kIn], scv, scs;
          far_features(ws.sc[j], xt, at, f, scv, scs);
          for (int i = 0; i < kIn; i += 2) *reinterpret_cast<uint32_t *>(&wm.sF[lane][i]) = pack_bf16(f[i], f[i + 1]);
          for (int i = kIn; i < kInPad; i += 2) *reinterpret_cast<uint32_t *>(&wm.sF[lane][i]) = 0u;
          __syncwarp();
          mlp_tile16(W, wm.sF, wm.sO, lane);
          mlp_tile16(W, wm.sF + 16, wm.sO + 16, lane);
          __syncwarp();
          for (int m = 0; m < 3; ++m) {
            su[m] += scv * wm.sO[lane][m];
            ss[m] += scs * wm.sO[lane][3 + m];
          }
          __syncwarp();
        }
      }
      for (int m = 0; m < 3; ++m) {
        two_sum_acc(vh[m], vl[m], su[m]);
        two_sum_acc(dh[m], dl[m], ss[m]);
      }
    }
    // Near field: the slices of pair_slices.cuh over the leaf's runs.  Slices
    // far from the warp's targets (every pair at u >= 50) take the far limit,
    // the others the closed form, with sigma's factors out of the loop where
    // one radius serves the slice.  It is most of the evaluation (about 28,000
    // near particles per target on the 1M coaxial rings) and bound by the FP32
    // pipe.  A lane's sums are compensated every kNearGroup pairs: groups of 64
    // sources put dalpha of a 5000-particle Gaussian ring off by 4.1e-6, 32 by
    // 2.7e-6 (norm-wise).  The far limit takes w per pair: the sources of a run
    // may lie anywhere between two leaves, and w costs no more than staging n_s
    // (evaluation 91 ms; 97 ms with the direct kernel's reference points).
    const float2 X2[3] = {dup2(xt[0]), dup2(xt[1]), dup2(xt[2])};
    const float2 AT3[3] = {dup2(-3.f * at[0]), dup2(-3.f * at[1]), dup2(-3.f * at[2])};
    WarpBox tb;
    tb.init();
    tb.add(xt[0], xt[1], xt[2], hst);
    reduce_box(tb);
    const bool one_t = __all_sync(0xffffffffu, hst == tb.hs);  // one radius among the targets (no NaN passes)
    constexpr int SL = kWarpTile / 32;
    auto &st = ws.near;
    unsigned nfull = 0;
    const int no = a.near_off[li], nn = a.near_cnt[li];
    for (int ni = 0; ni < nn; ++ni) {
      const int2 run = a.near_runs[no + ni];
      for (int sb = run.x; sb < run.y; sb += kWarpTile) {
        __syncwarp();
        WarpBox sbx;
        sbx.init();
        float hs[SL];
#pragma unroll
        for (int j = 0; j < SL; ++j) {
          const int i = sb + lane + 32 * j;
          const float4 p = i < run.y ? a.Ps[i] : pad_P<float>();
          const float4 q = i < run.y ? a.Qs[i] : pad_Q<float>();
          stage_source(st, lane + 32 * j, p, q, 0.f, 0.f, 0.f);
          if (i < run.y) sbx.add(p.x, p.y, p.z, p.w);
          hs[j] = p.w;
        }
        reduce_box(sbx);
        bool one = one_t;  // one sigma for all of the slice's pairs
#pragma unroll
        for (int j = 0; j < SL; ++j) one = one && (hs[j] == sbx.hs || sb + lane + 32 * j >= run.y);
        const bool far_tile = all_far(tb, sbx);
        __syncwarp();
        // source pairs; an odd tail pairs with a padding source (zero strength, far away)
        const int npr = (min(kWarpTile, run.y - sb) + 1) >> 1;
        const int n = half ? (npr + 1) >> 1 : npr;  // an odd pair pairs with padding sources (every slot is staged)
        one = __all_sync(0xffffffffu, one);
        const MidSigma2 g = mid_sigma2(dup2(tb.hs + sbx.hs));
        // one compensation group per kNearGroup pairs of a lane
        for (int b = 0; b < n; b += kNearGroup) {
          const int r0 = h + b * step, nb = min(kNearGroup, n - b);
          float2 sv[3], sd[3], sp[3];
          float sdv[3] = {0.f, 0.f, 0.f};
#pragma unroll
          for (int m = 0; m < 3; ++m) sv[m] = sd[m] = sp[m] = dup2(0.f);
          if (far_tile) {
            far_slice_direct(st, nb, r0, step, X2, AT3, sv, sd, sp);
          } else if (one) {
            mid_slice<false, false>(st, nb, r0, step, X2, xt, at, hst, vt, &g, sv, sd, sp, sdv, nfull);
          } else {
            mid_slice<false, false>(st, nb, r0, step, X2, xt, at, hst, vt, nullptr, sv, sd, sp, sdv, nfull);
          }
          fold_group_f32<false>(false, 0.f, 0.f, 0.f, at, a.nu2, sv, sd, sp, sdv, vh, vl, dh, dl);
        }
      }
    }
    double out[6];
    for (int m = 0; m < 3; ++m) {
      out[m] = (double)vh[m] + (double)vl[m];
      out[3 + m] = (double)dh[m] + (double)dl[m];
    }
    if (half)
      for (int m = 0; m < 6; ++m) out[m] += __shfl_xor_sync(0xffffffffu, out[m], 16);
    if (mine && h == 0) {
      double *o = a.partial + a.off + ti;
      for (int m = 0; m < 6; ++m) o[m * a.cap] = out[m] * kInv4Pi;
    }
  }
}

// Training samples of the correction network from the current octree: each
// warp draws (leaf, target, far cell) with a hash of (seed, sample), computes
// the features, the exact FP64 contribution of the cell's particles (the
// direct kernel's formula) and the expansion to the surrogate's order
// (a.order), and stores the scaled residual.  Rows whose leaf has no far cell
// after 32 draws are all zero.
__global__ void mlp_sample_kernel(TreeEvalArgs a, const int *far_leaves, int nfar_leaves, int nsamples,
                                  unsigned long long seed, float *X, float *T) {
  const int lane = threadIdx.x & 31;
  const int wg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (int smp = wg; smp < nsamples; smp += nw) {
    int li = -1, t = 0, fj = 0;
    if (lane == 0) {
      unsigned long long h = seed ^ (0x9E3779B97F4A7C15ULL * (unsigned long long)(smp + 1));
      h ^= h >> 33; h *= 0xFF51AFD7ED558CCDULL; h ^= h >> 33; h *= 0xC4CEB9FE1A85EC53ULL; h ^= h >> 33;
      const int l = far_leaves[(int)(h % (unsigned long long)nfar_leaves)];
      const TreeCell tc = a.cells[a.leaves[l]];
      li = l;
      t = tc.start + (int)((h >> 20) % (unsigned long long)(tc.end - tc.start));
      fj = (int)((h >> 40) % (unsigned long long)a.far_cnt[l]);
    }
    li = __shfl_sync(0xffffffffu, li, 0);
    t = __shfl_sync(0xffffffffu, t, 0);
    fj = __shfl_sync(0xffffffffu, fj, 0);
    float *xo = X + (int64_t)smp * kIn;
    float *to = T + (int64_t)smp * kOut;
    if (li < 0) {
      if (lane < kIn) xo[lane] = 0.f;
      if (lane < kOut) to[lane] = 0.f;
      continue;
    }
    const int ci = a.far_list[a.far_off[li] + fj];
    const TreeCell cc = a.cells[ci];
    const float *v = a.cd[ci].v;
    const float4 pt = a.Ps[t], qt = a.Qs[t];
    const float xt[3] = {pt.x, pt.y, pt.z}, at[3] = {qt.x, qt.y, qt.z};
    double ex[6] = {0, 0, 0, 0, 0, 0};
    for (int j = cc.start + lane; j < cc.end; j += 32) {
      const float4 p = a.Ps[j], q = a.Qs[j];
      const double d[3] = {(double)pt.x - p.x, (double)pt.y - p.y, (double)pt.z - p.z};
      const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
      const PairTerms<double> k = pair_terms(r2, (double)pt.w + (double)p.w);
      const double as[3] = {q.x, q.y, q.z}, a_t[3] = {qt.x, qt.y, qt.z};
      const double w3[3] = {as[1] * d[2] - as[2] * d[1], as[2] * d[0] - as[0] * d[2], as[0] * d[1] - as[1] * d[0]};
      const double c3[3] = {a_t[1] * as[2] - a_t[2] * as[1], a_t[2] * as[0] - a_t[0] * as[2], a_t[0] * as[1] - a_t[1] * as[0]};
      const double dc = d[0] * c3[0] + d[1] * c3[1] + d[2] * c3[2];
      for (int m = 0; m < 3; ++m) {
        ex[m] += k.q * w3[m];
        ex[3 + m] += k.q * c3[m] + k.F * dc * d[m];
      }
    }
    for (int m = 0; m < 6; ++m)
      for (int o = 16; o > 0; o >>= 1) ex[m] += __shfl_down_sync(0xffffffffu, ex[m], o);
    if (lane == 0) {
      float f[kIn], scv, scs, u[3], s[3];
      far_features(v, xt, at, f, scv, scs);
      far_expand(v, xt, at, a.order, u, s);
      for (int i = 0; i < kIn; ++i) xo[i] = f[i];
      for (int m = 0; m < 3; ++m) {
        to[m] = scv > 0.f ? (float)((ex[m] - u[m]) / scv) : 0.f;
        to[3 + m] = scs > 0.f ? (float)((ex[3 + m] - s[m]) / scs) : 0.f;
      }
    }
  }
}

// (leaf, slice) work items: count[li] = ceil(size / 32), then written at the
// exclusive-scan offsets.
__global__ void slice_count_kernel(const TreeCell *cells, const int *leaves, int nleaves, int *cnt) {
  const int li = blockIdx.x * blockDim.x + threadIdx.x;
  if (li < nleaves) {
    const TreeCell c = cells[leaves[li]];
    cnt[li] = (c.end - c.start + 31) / 32;
  }
}
__global__ void slice_write_kernel(const int *cnt, const int *off, int nleaves, int2 *items) {
  const int li = blockIdx.x * blockDim.x + threadIdx.x;
  if (li < nleaves)
    for (int k = 0; k < cnt[li]; ++k) items[off[li] + k] = make_int2(li, k);
}

// Max-norm errors of the surrogate rates (chunk 0 of partial) at the sampled
// targets against the exact sums: res[0] = max |dv|^2, res[1] = max |v|^2,
// res[2] = max |d dalpha|^2, res[3] = max |dalpha|^2 (ordered-float atomics).
__global__ void sample_compare_kernel(const double *exact, int chunks, int nt, const int *targets, int64_t off,
                                      const double *partial, int64_t cap, unsigned *res) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  double ex[6];
  for (int m = 0; m < 6; ++m) {
    double v = 0;
    for (int c = 0; c < chunks; ++c) v += exact[((int64_t)c * 6 + m) * nt + t];
    ex[m] = v;
  }
  const int64_t i = off + targets[t];
  double dv = 0, v2 = 0, da = 0, a2 = 0;
  for (int m = 0; m < 3; ++m) {
    const double s = partial[m * cap + i], sa = partial[(3 + m) * cap + i];
    dv += (s - ex[m]) * (s - ex[m]);
    v2 += ex[m] * ex[m];
    da += (sa - ex[3 + m]) * (sa - ex[3 + m]);
    a2 += ex[3 + m] * ex[3 + m];
  }
  atomicMax(&res[0], f2ord((float)dv));
  atomicMax(&res[1], f2ord((float)v2));
  atomicMax(&res[2], f2ord((float)da));
  atomicMax(&res[3], f2ord((float)a2));
}

}  // namespace pgpu
