// Tangent (JVP) and adjoint (VJP) of the classic RK4 and Lawson-RK6 shooting
// modes (jax_scripts/lib/timestepping.py:17-44 and :83-125), from one
// description of an explicit (Lawson) Runge-Kutta step:
//
//   x_1 = f0,  k_s = h v(x_s),
//   x_s = e^{p_s} f0 + sum_{j<s} a_sj e^{p_s - p_j} k_j,
//   f'  = e^{P} f0 + sum_j b_j e^{P - p_j} k_j,
//
// where e = exp(tau h L) (masked) is the integrating factor and p_s counts the
// factors applied before stage s.  Lawson-RK6 applies e after stages 1, 3, 4,
// 5, 6 and 7 (p = 0 1 1 2 3 4 5 6, P = 6, tau = 1/6); classic RK4 has no
// factor (e = 1) and its v includes the dissipation L x (loss_functions.py:53).
// The reference repeats the multiplications by e; here powers of e are formed
// by repeated multiplication too, and the stage weights are products with the
// rational coefficients (rounding differences of order 1e-16, far inside the
// parity bound).
//
// With dh = dT / steps, d(e^m) = m tau L e^m dh:
//   dk_s  = (dh/h) k_s + h (N'(x_s) dx_s [+ L dx_s])
//   dx_s  = e^{p_s} (df0 + p_s c f0) + sum_{j<s} a_sj e^{p_s-p_j} (dk_j + (p_s-p_j) c k_j),  c = tau L dh
// and in reverse, from the cotangent fbar' of f':
//   kbar_j = b_j e^{P-p_j} fbar',  f0bar = e^P fbar'
//   for s = S..1:  xbar_s = N'(x_s)^T (h kbar_s) [+ h L kbar_s];
//                  f0bar += e^{p_s} xbar_s,  kbar_j += a_sj e^{p_s-p_j} xbar_s (j < s)
//   hbar = sum_s <kbar_s, k_s>/h + the e^m terms (<ybar, m tau L e^m y>).
#pragma once

#include "kernels_adj.cuh"
#include "kernels_fx.cuh"

namespace ecs {

// Stage count, factor exponent and dissipation-in-v of a scheme.
__host__ __device__ constexpr int fxl_stages(int scheme) { return scheme == FX_RK6 ? 8 : 4; }
__host__ __device__ constexpr double fxl_tau(int scheme) { return scheme == FX_RK6 ? 1.0 / 6.0 : 0.0; }
__host__ __device__ constexpr bool fxl_diss_in_v(int scheme) { return scheme == FX_RK4; }
// p_s (s = 1..S) and P (s = S + 1)
__host__ __device__ constexpr int fxl_p(int scheme, int s) {
  if (scheme != FX_RK6) return 0;
  return s == 1 ? 0 : s <= 3 ? 1 : s <= 8 ? s - 2 : 6;   // 0 1 1 2 3 4 5 6 ; P = 6
}
// a_sj (s = 2..S, j < s); s = S + 1 gives the final weights b_j
__host__ __device__ constexpr double fxl_a(int scheme, int s, int j) {
  if (scheme == FX_RK4) {
    if (s == 5) return j == 1 ? 1.0 / 6.0 : j == 2 ? 1.0 / 3.0 : j == 3 ? 1.0 / 3.0 : 1.0 / 6.0;   // :44
    return (s == 2 && j == 1) ? 0.5 : (s == 3 && j == 2) ? 0.5 : (s == 4 && j == 3) ? 1.0 : 0.0;  // :40-43
  }
  switch (s) {   // timestepping.py:112-124
    case 2: return j == 1 ? 1.0 / 6.0 : 0.0;
    case 3: return (j == 1 || j == 2) ? 1.0 / 12.0 : 0.0;
    case 4: return j == 2 ? -4.0 / 33.0 : j == 3 ? 5.0 / 11.0 : 0.0;
    case 5: return j == 1 ? -1.0 / 4.0 : j == 2 ? -29.0 / 44.0 : j == 3 ? 31.0 / 22.0 : 0.0;
    case 6: return j == 1 ? 3.0 / 11.0 : j == 2 ? 8.0 / 33.0 : j == 3 ? -4.0 / 11.0 : j == 4 ? 1.0 / 11.0
                 : j == 5 ? 14.0 / 33.0 : 0.0;
    case 7: return j == 1 ? -17.0 / 48.0 : j == 2 ? -5.0 / 12.0 : j == 3 ? 1.0 : j == 4 ? 1.0
                 : j == 5 ? -13.0 / 12.0 : j == 6 ? 11.0 / 16.0 : 0.0;
    case 8: return j == 1 ? 20.0 / 39.0 : j == 2 ? 12.0 / 39.0 : j == 3 ? -31.0 / 39.0 : j == 4 ? -1.0 / 39.0
                 : j == 5 ? 34.0 / 39.0 : j == 6 ? -11.0 / 39.0 : j == 7 ? 16.0 / 39.0 : 0.0;
    default:   // 9: final weights
      return (j == 1 || j == 8) ? 13.0 / 200.0 : (j == 3 || j == 7) ? 4.0 / 25.0
           : (j == 4 || j == 6) ? 11.0 / 40.0 : 0.0;
  }
}

// Trajectory record of one step: f0, k_1..k_S (as computed, before any
// factor), the stage inputs x_2..x_S.  2 S box vectors.
__host__ __device__ constexpr int fxr_f() { return 0; }
__host__ __device__ constexpr int fxr_k(int s) { return s; }
__host__ __device__ constexpr int fxr_x(int scheme, int s) { return fxl_stages(scheme) + s - 1; }
__host__ __device__ constexpr int fxr_n(int scheme) { return 2 * fxl_stages(scheme); }

// e^m for a small non-negative m by repeated multiplication (e^0 = 1, also
// where the masked factor is 0).
template <typename R> __device__ __forceinline__ R fxl_pow(R e, int m) {
  R r = R(1);
  for (int i = 0; i < m; ++i) r *= e;
  return r;
}

// ---------------------------------------------------------------------------
// Tangent column pass.  Slots per tangent: df0, dx (the current stage input),
// dk_1..dk_S.  STAGE 0: inverse transforms of df0 (the first stage input).
// STAGE s = 1..S: the forward transform of the tangent row pass at x_s gives
// N'(x_s) dx_s, hence dk_s; then the next stage input dx_{s+1} (or, at s = S,
// the step's result df') and its inverse transforms.
// ---------------------------------------------------------------------------
enum FxtSlot { FT_F = 0, FT_X = 1, FT_K1 = 2 };
__host__ __device__ constexpr int fxt_nslot(int scheme) { return fxl_stages(scheme) + 2; }

template <typename R>
struct ColFxtParams {
  const cplx<R>* H;     // [B][NH][K][N]
  cplx<R>* G;           // [B][NG][K][N]
  cplx<R>* D;           // tangent slots [B][nslot][2][K][M]
  int nslot;
  const cplx<R>* rec;   // this step's record [2S][2][K][M]
  const double* dT;     // [B]
  double h, dscale;     // dh = dT * dscale
  const cplx<R>* tw;
  R nu, eta;
  int B, produce;
};

// Slots that stage s reads before its stores: df0, the stage input (with the
// dissipation in v), and the dk_j of the next stage input's weights.
__host__ __device__ constexpr unsigned fxt_dmask(int scheme, int s) {
  unsigned m = 1u << FT_F;
  if (s == 0) return m;
  if (fxl_diss_in_v(scheme) && s > 1) m |= 1u << FT_X;
  for (int j = 1; j < s; ++j)
    if (fxl_a(scheme, s + 1, j) != 0.0) m |= 1u << (FT_K1 + j - 1);
  return m;
}

template <typename R, int N, int SCHEME, int STAGE>
__global__ void __launch_bounds__(COLWARPS * 32, 1) k_col_fxt(ColFxtParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  constexpr int S = fxl_stages(SCHEME);
  ECS_COL_PROLOGUE(popc_c(fxt_dmask(SCHEME, STAGE)), 1);   // the multipliers
  const int c = id.ch, b = id.b, ky = id.ky;
  const size_t row = ((size_t)c * K + ky) * M;
  cplx<R>* D = p.D + (size_t)b * p.nslot * VEC + row;
  const cplx<R>* Q = p.rec + row;
  const R h = (R)p.h;
  const R dh = (R)(p.dT[b] * p.dscale);
  const R dh_h = dh / h;
  const R coeff = c == 0 ? p.nu : p.eta;
  constexpr unsigned DM = fxt_dmask(SCHEME, STAGE);
  Operands<X, DM> op(rows);
  op.begin(D, VEC);
  const TableRow<X, rows_fit(popc_c(DM), 1)> mu(rows + popc_c(DM) * M, mu_row<X>(p.tw, ky));
  cplx<R> r[E];
  if (STAGE > 0) col_load_rhs(p.H, b, c, ky, xf, r);
  op.load(D, VEC, true, xf);
  cplx<R> x[E];
#pragma unroll
  for (int i = 0; i < E; ++i) {
      x[i] = mk<R>(0, 0);
      const int slot = xf.slot(i);
      if (slot < 0) continue;
      auto DV = [&](int d) -> cplx<R> { return op.get(d, i, slot); };
      auto DW = [&](int d, cplx<R> v) { D[d * VEC + slot] = v; };
      auto Qv = [&](int q) -> cplx<R> { return __ldg(Q + q * VEC + slot); };
      if (STAGE == 0) {
        x[i] = DV(FT_F);
        continue;
      }
      const R L = diss_L<R>(xf.kx(i), (R)ky, coeff);   // zero at (0,0)
      const bool msk = !(slot == 0 && ky == 0);
      // the integrating factor of the linearisation's step (as k_fx_setup forms it)
      const R e = SCHEME == FX_RK6 ? (msk ? exp(h / R(6) * L) : R(0)) : R(1);
      const R cf = R(fxl_tau(SCHEME)) * L * dh;   // d(e^m) = m cf e^m
      cplx<R> rv = r[i];                          // N'(x_s) dx_s (no forcing)
      if constexpr (fxl_diss_in_v(SCHEME)) rv = cadd(rv, cscale(STAGE == 1 ? DV(FT_F) : DV(FT_X), L));
      const cplx<R> dk = cadd(cscale(Qv(fxr_k(STAGE)), dh_h), cscale(rv, h));
      DW(FT_K1 + STAGE - 1, dk);
      constexpr int sn = STAGE + 1;               // S + 1: the step's result
      constexpr int pn = fxl_p(SCHEME, sn);
      cplx<R> acc = cscale(cadd(DV(FT_F), cscale(Qv(fxr_f()), R(pn) * cf)), fxl_pow(e, pn));
#pragma unroll
      for (int q = 1; q <= STAGE; ++q) {
        const double a = fxl_a(SCHEME, sn, q);
        if (a == 0.0) continue;
        const int m = pn - fxl_p(SCHEME, q);
        const cplx<R> dkj = q == STAGE ? dk : DV(FT_K1 + q - 1);
        acc = cadd(acc, cscale(cadd(dkj, cscale(Qv(fxr_k(q)), R(m) * cf)), R(a) * fxl_pow(e, m)));
      }
      if (STAGE < S) DW(FT_X, acc);
      else DW(FT_F, acc);
      x[i] = acc;
  }
  if (!p.produce) return;
  col_inverse_uv(x, p.G, b, c, ky, id.act, xf, mu);
}

// ---------------------------------------------------------------------------
// Adjoint column pass.  Slots per cotangent: f0bar (FA_F; on entry to a step's
// reverse sweep the cotangent of the step's result f'), kbar_1..kbar_S.
// STAGE S + 1 (seed): kbar_j = b_j e^{P-p_j} f'bar, f0bar = e^P f'bar, and the
// emission of lambda_S = h kbar_S.  STAGE s = S..1: the forward transforms of
// the adjoint row pass at x_s give N'(x_s)^T (h kbar_s), hence xbar_s, which is
// distributed to f0bar and kbar_j (j < s); then lambda_{s-1} is emitted
// (nothing after s = 1).  hbar is accumulated per (b, ky, channel) in hacc.
// ---------------------------------------------------------------------------
enum FxaSlot { FA_F = 0, FA_K1 = 1 };
__host__ __device__ constexpr int fxa_nslot(int scheme) { return fxl_stages(scheme) + 1; }

template <typename R>
struct ColFxaParams {
  const cplx<R>* H;     // [B][NHA][K][N]
  cplx<R>* G;           // [B][NG][K][N] (fields 0..2 written)
  cplx<R>* J;           // adjoint slots [B][nslot][2][K][M]
  int nslot;
  const cplx<R>* rec;   // this step's record [2S][2][K][M]
  double* hacc;         // [B][K][2]
  double h;
  const cplx<R>* tw;
  R nu, eta;
  int B;
};

// Slots that a stage reads before its stores: f0bar, kbar_s and the kbar_j that
// xbar_s is distributed to (and kbar_{s-1}, the next emission).
__host__ __device__ constexpr unsigned fxa_jmask(int scheme, int s) {
  unsigned m = 1u << FA_F;
  if (s > fxl_stages(scheme)) return m;
  m |= 1u << (FA_K1 + s - 1);
  for (int j = 1; j < s; ++j)
    if (fxl_a(scheme, s, j) != 0.0 || j == s - 1) m |= 1u << (FA_K1 + j - 1);
  return m;
}

template <typename R, int N, int SCHEME, int STAGE>
__global__ void __launch_bounds__(COLWARPS * 32, 1) k_col_fxa(ColFxaParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  constexpr int S = fxl_stages(SCHEME);
  constexpr bool SEED = STAGE == S + 1;
  ECS_COL_PROLOGUE(popc_c(fxa_jmask(SCHEME, STAGE)), 1);   // the multipliers
  const int c = id.ch, b = id.b, ky = id.ky;
  const size_t row = ((size_t)c * K + ky) * M;
  cplx<R>* J = p.J + (size_t)b * p.nslot * VEC + row;
  const cplx<R>* Q = p.rec + row;
  const R h = (R)p.h;
  const R coeff = c == 0 ? p.nu : p.eta;
  constexpr unsigned JM = fxa_jmask(SCHEME, STAGE);
  Operands<X, JM> op(rows);
  op.begin(J, VEC);
  const TableRow<X, !SEED && rows_fit(popc_c(JM), 1)> mu(rows + popc_c(JM) * M, mu_row<X>(p.tw, ky));
  cplx<R> xa[E];
  if (!SEED) col_adj_xb(p.H, b, c, ky, xf, mu, xa);
  op.load(J, VEC, true, xf);
  double hpart = 0.0, hdiv = 0.0;   // hdiv: the terms over h
  cplx<R> lam[E];
#pragma unroll
  for (int i = 0; i < E; ++i) {
      lam[i] = mk<R>(0, 0);
      const int slot = xf.slot(i);
      if (slot < 0) continue;
      const R L = diss_L<R>(xf.kx(i), (R)ky, coeff);
      const bool msk = !(slot == 0 && ky == 0);
      const R e = SCHEME == FX_RK6 ? (msk ? exp(h / R(6) * L) : R(0)) : R(1);
      const R tl = R(fxl_tau(SCHEME)) * L;        // d(e^m)/dh = m tl e^m
      auto JV = [&](int q) -> cplx<R> { return op.get(q, i, slot); };
      auto JW = [&](int q, cplx<R> v) { J[q * VEC + slot] = v; };
      auto Qv = [&](int q) -> cplx<R> { return __ldg(Q + q * VEC + slot); };
      auto ip = [&](cplx<R> a, cplx<R> bb) { return (double)a.x * (double)bb.x + (double)a.y * (double)bb.y; };
      cplx<R> kb = mk<R>(0, 0);   // the kbar whose h-multiple feeds the next adjoint row pass
      if constexpr (SEED) {
        constexpr int P = fxl_p(SCHEME, S + 1);
        const cplx<R> fb = JV(FA_F);
        const R eP = fxl_pow(e, P);
        JW(FA_F, cscale(fb, eP));
        if (P > 0) hpart += ip(fb, cscale(Qv(fxr_f()), R(P) * tl * eP));
#pragma unroll
        for (int q = 1; q <= S; ++q) {
          const double bw = fxl_a(SCHEME, S + 1, q);
          const int m = P - fxl_p(SCHEME, q);
          const R em = fxl_pow(e, m);
          const cplx<R> kq = cscale(fb, R(bw) * em);
          JW(FA_K1 + q - 1, kq);
          if (bw != 0.0 && m > 0) hpart += ip(fb, cscale(Qv(fxr_k(q)), R(bw) * R(m) * tl * em));
          if (q == S) kb = kq;
        }
      } else {
        constexpr int ps = fxl_p(SCHEME, STAGE);
        const cplx<R> ks = JV(FA_K1 + STAGE - 1);   // kbar_s, complete
        hdiv += ip(ks, Qv(fxr_k(STAGE)));
        cplx<R> xb = xa[i];
        if (fxl_diss_in_v(SCHEME)) xb = cadd(xb, cscale(ks, h * L));
        const R eps = fxl_pow(e, ps);
        JW(FA_F, cadd(JV(FA_F), cscale(xb, eps)));
        if (ps > 0) hpart += ip(xb, cscale(Qv(fxr_f()), R(ps) * tl * eps));
#pragma unroll
        for (int q = 1; q < STAGE; ++q) {
          const double a = fxl_a(SCHEME, STAGE, q);
          if (a == 0.0 && q < STAGE - 1) continue;
          cplx<R> kq = JV(FA_K1 + q - 1);
          if (a != 0.0) {
            const int m = ps - fxl_p(SCHEME, q);
            const R em = fxl_pow(e, m);
            kq = cadd(kq, cscale(xb, R(a) * em));
            JW(FA_K1 + q - 1, kq);
            if (m > 0) hpart += ip(xb, cscale(Qv(fxr_k(q)), R(a) * R(m) * tl * em));
          }
          if (q == STAGE - 1) kb = kq;
        }
      }
      lam[i] = cscale(cscale(kb, h), ky == 0 ? R(1) : R(0.5));   // h kb / c_ky
  }
  col_hacc(p.hacc, id, id.act, xf, hpart + hdiv / (double)h);
  if (STAGE == 1) return;
  col_adj_emit(lam, p.G, b, c, ky, id.act, xf);
}

}  // namespace ecs
