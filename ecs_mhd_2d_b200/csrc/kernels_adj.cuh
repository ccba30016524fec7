// Adjoint (reverse-mode) kernels of the shooting map: the VJP used by
// adjoint descent (reference: jax.value_and_grad of loss_RPO,
// jax_scripts/adjoint_descent.py:90-91) and as the transpose preconditioner
// of Newton-GMRES (jax.vjp of objective_RPO, jax_scripts/newton.py:168-170).
//
// Inner products: box vectors use <X, Y> = Re sum conj(X) Y, real fields the
// Euclidean dot.  With these, the transposes of the box transforms are
//   to_box^T(Y)   = n^2 irfft2(Y / c_ky)        (c_ky = 1 for ky = 0, else 2)
//   from_box^T(w) = (c_ky / n^2) rfft2(w)
// so one adjoint right-hand side is again a column pass and a row pass
// (Basdevant form of the products, see kernels.cuh):
//   lambda -> P1bar = Re sum (-kx ky) lambda_w e^{ik.x},  P2bar = Re sum (ky^2 - kx^2) lambda_w e^{ik.x},
//             P3bar = Re sum k^2 lambda_j e^{ik.x}
//   -> product adjoints with the primal fields
//        ubar  =  2u P1bar - v P2bar + B_y P3bar,   vbar  = -2v P1bar - u P2bar - B_x P3bar,
//        Bxbar = -2B_x P1bar + B_y P2bar - v P3bar, Bybar =  2B_y P1bar + B_x P2bar + u P3bar
//   -> 4 forward transforms
//   -> Xbar_c = (c_ky/n^2) sum_m (-i mu_m) rfft2(fbar_mc), mu_m in {ky/k^2, -kx/k^2}.
#pragma once

#include "kernels.cuh"
#include "kernels_rk43.cuh"
#include "kernels_tan.cuh"

namespace ecs {

// ---------------------------------------------------------------------------
// Adjoint row pass
// ---------------------------------------------------------------------------
template <typename R>
struct RowAdjParams {
  const cplx<R>* G;     // [B][NG][K][N]: fields 0..2 hold the inverse columns of the P1, P2, P3 cotangents (/c_ky)
  cplx<R>* H;           // [B][NHA][K][N]: rfft2 rows of the 4 adjoint fields
  const R* phys;        // primal physical fields of this stage: phys + b * phys_bstride is [N][NPH][N]
  long phys_bstride;    // 0: one primal shared by the batch
  const StepCtl* ctl;   // optional per-candidate control: batch elements whose ctl.done is set are skipped
  const cplx<R>* tw;
  int B;
};

// Product adjoints of one point: (P1bar, P2bar) and P3bar -> (ubar, vbar) and (Bxbar, Bybar).
template <typename R>
__device__ __forceinline__ void row_adj_product(cplx<R> p12, R p3, cplx<R> uv, cplx<R> bb, cplx<R>& a, cplx<R>& q) {
  const R p1 = p12.x, p2 = p12.y, u = uv.x, v = uv.y, bx = bb.x, by = bb.y;
  a = mk<R>(R(2) * u * p1 - v * p2 + by * p3, -R(2) * v * p1 - u * p2 - bx * p3);
  q = mk<R>(-R(2) * bx * p1 + by * p2 - v * p3, R(2) * by * p1 + bx * p2 + u * p3);
}

// Rows x0 .. x0 + XT - 1 of cotangent b; s_G holds the three product rows and then the
// four adjoint rows (each warp reads and writes its own column of the tile).  CX
// (cluster-resident passes): the tile is there already unless load_g, and the adjoint rows
// go to the column warps' rows at `hcols` (scatter_h_tile) unless that is null.
template <int XT, bool CX = false, class X>
__device__ __forceinline__ void row_adj_body(const RowAdjParams<typename X::R>& p, int b, int x0, const X& xf,
                                             cplx<typename X::R>* s_G, bool load_g = true,
                                             cplx<typename X::R>* hcols = nullptr) {
  using R = typename X::R;
  constexpr int E = X::E, L = X::L, K = X::K, N = X::N;
  const int w = threadIdx.x / L;
  constexpr bool EARLY = E <= 4;        // see row_tan_body
  const cplx<R>* ph = phys_row<R, N>(p.phys + (size_t)b * p.phys_bstride, x0 + w) + xf.l;
  cplx<R> puv[E], pbb[E];
  auto load_phys = [&]() {
#pragma unroll
    for (int j = 0; j < E; ++j) { puv[j] = ph[L * j]; pbb[j] = ph[N + L * j]; }
  };
  if constexpr (EARLY) load_phys();
  if (!CX || load_g) load_tile<R, N, XT>(s_G, p.G + (size_t)b * NG * K * N, 3 * K, x0);
  __syncthreads();
  cplx<R> P12[E], P3[E];   // (P1bar, P2bar) and (P3bar, 0)
  row_inverse<XT, true>(s_G, w, xf, P12, P3);
  if constexpr (!EARLY) load_phys();
#pragma unroll
  for (int j = 0; j < E; ++j) {
    cplx<R> a, q;
    row_adj_product<R>(P12[j], P3[j].x, puv[j], pbb[j], a, q);
    P12[j] = a; P3[j] = q;
  }
  row_forward<XT, true>(P12, P3, s_G, w, xf);
  __syncthreads();
  if constexpr (CX) {
    if (hcols) { scatter_h_tile<XT, true>(s_G, hcols, x0, xf); return; }
  }
  store_tile<R, N, XT>(p.H + (size_t)b * NHA * K * N, s_G, NHA * K, x0);
}

template <typename R, int N, int XT>
__global__ void __launch_bounds__(XT * Xf<R, N>::L) k_row_adj(RowAdjParams<R> p) {
  using X = Xf<R, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_x = reinterpret_cast<cplx<R>*>(smem_raw);
  const int tiles = N / XT;
  const int b = blockIdx.x / tiles, x0 = (blockIdx.x - b * tiles) * XT;
  load_tables<X>(s_x, p.tw);
  pdl_wait();
  pdl_trigger();
  if (p.ctl && p.ctl[b].done) return;   // the whole CTA belongs to batch element b
  row_adj_body<XT>(p, b, x0, X(s_x, threadIdx.x >> 5), s_x + X::smem(XT / X::G));
}

// ---------------------------------------------------------------------------
// Adjoint column pass
// ---------------------------------------------------------------------------
enum AdjStage : int {
  AJ_PRE = 0,                        // Lawson-RK4: seed the step adjoint from obar
  AJ_S4 = 4, AJ_S3 = 3, AJ_S2 = 2, AJ_S1 = 1,
  AJ43_INIT = 10,                    // Lawson-RK4(3): adjoint of the initial k1 = t v(x0)
  AJ43_PRE = 11,                     // seed an accepted attempt from (xbar_f, k5bar)
  AJ43_S5 = 15, AJ43_S4 = 14, AJ43_S3 = 13, AJ43_S2 = 12,
  AJ43_IPRE = 16,                    // seed the adjoint RHS of the initial k1
};
// Adjoint slots. Lawson-RK4: OB (obar / fbar), F2, A1, K2, B3.
enum AdjSlot4 { J_OB = 0, J_F2, J_A1, J_K2, J_B3, J_NS4 };
// Lawson-RK4(3): X0 (x0bar carried), K1 (k1bar carried), XF, X2, XB, K1P (k1'bar), K2, K3P (k3'bar), K2P (k2'bar), K1PP
enum AdjSlot43 { JJ_X0 = 0, JJ_K1, JJ_X2, JJ_XB, JJ_K1P, JJ_K1PP, JJ_K2, JJ_K2P, JJ_K3P, JJ_NS43 };

template <typename R>
struct ColAdjParams {
  const cplx<R>* H;     // [B][NHA][K][N]
  cplx<R>* G;           // [B][NG][K][N] (fields 0..2 written)
  cplx<R>* J;           // adjoint slots [B][nslot][2][K][M]
  int nslot;
  const cplx<R>* rec;   // primal record of this step / attempt
  const cplx<R>* rec_prev;   // Lawson-RK4 AJ_S1: record of the previous step (null at the first step)
  double* hacc;         // [B][K][2] accumulators of dL/dh (RK4) or dL/dt (RK4(3))
  double t, h;
  const cplx<R>* tw;
  R nu, eta;
  int B, stage;
  // Several candidates (Lawson-RK4 stages): ctl[b] gives candidate b's step h
  // and done flag (skipped once done); rec / rec_prev + b * rec_bstride its record.
  const StepCtl* ctl;
  long rec_bstride;
};

__device__ __forceinline__ double rdot2(double ax, double ay, double bx, double by) { return ax * bx + ay * by; }

// Record rows (bits of Rk4Rec) that a Lawson-RK4 stage reads (AJ_S1: of the step before).
__host__ __device__ constexpr unsigned adj4_qmask(int stage) {
  return stage == AJ_S4 ? (1u << Q_F) | (1u << Q_K1) | (1u << Q_K2) | (1u << Q_K3)
       : stage == AJ_S3 ? (1u << Q_K2)
       : stage == AJ_S2 ? (1u << Q_F) | (1u << Q_K1) : (1u << Q_K4);
}
// Slots (bits of AdjSlot4 / AdjSlot43) that the algebra of a stage reads; they are
// loaded together before the stage's stores.
__host__ __device__ constexpr unsigned adj_jmask(int stage) {
  return stage == AJ_PRE || stage == AJ_S1 ? (1u << J_OB)
       : stage == AJ_S4 ? (1u << J_F2) | (1u << J_A1) | (1u << J_K2) | (1u << J_B3)
       : stage == AJ_S3 ? (1u << J_F2) | (1u << J_K2)
       : stage == AJ_S2 ? (1u << J_F2) | (1u << J_A1)
       : stage == AJ43_PRE || stage == AJ43_IPRE ? (1u << JJ_K1)
       : stage == AJ43_S5 || stage == AJ43_INIT ? (1u << JJ_X0)
       : stage == AJ43_S4 ? (1u << JJ_X2) | (1u << JJ_K3P) | (1u << JJ_K2P) | (1u << JJ_K1PP)
       : stage == AJ43_S3 ? (1u << JJ_XB) | (1u << JJ_K2)
       : stage == AJ43_S2 ? (1u << JJ_XB) | (1u << JJ_K1P) : 0u;
}

// (c_ky/n^2) sum_m (-i mu_m) rfft2 of the adjoint rows of channel c in H: the box
// cotangent N'(P)^T lambda at the lane's algebra elements.
template <class X, class Mu>
__device__ __forceinline__ void col_adj_rows(const cplx<typename X::R>* h0, const cplx<typename X::R>* h1, int ky, const X& xf,
                                           const Mu& mu, cplx<typename X::R> (&xb)[X::E]) {
  using R = typename X::R;
  constexpr int E = X::E, L = X::L;
  const R cky = ky == 0 ? R(1) : R(2);
  cplx<R> v1[E];
#pragma unroll
  for (int j = 0; j < E; ++j) { xb[j] = h0[xf.l + L * j]; v1[j] = h1[xf.l + L * j]; }
  xf.template to_spec2<false>(xb, v1);
  mu.wait();
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int s = xf.slot(j);
    if (s < 0) { xb[j] = mk<R>(0, 0); continue; }
    const cplx<R> m = mu(s);
    xb[j] = cscale(cadd(cimul(xb[j], -m.x), cimul(v1[j], -m.y)), cky);
  }
}
template <class X, class Mu>
__device__ __forceinline__ void col_adj_xb(const cplx<typename X::R>* H, int b, int c, int ky, const X& xf, const Mu& mu,
                                           cplx<typename X::R> (&xb)[X::E]) {
  const cplx<typename X::R>* h0 = H + ((size_t)(b * NHA + 2 * c) * X::K + ky) * X::N;
  col_adj_rows(h0, h0 + (size_t)X::K * X::N, ky, xf, mu, xb);
}

// Inverse column transforms of lambda/c_ky times the product multipliers: the
// product cotangents P1bar, P2bar (channel w) or P3bar (channel j) in G,
// unscaled: Re sum mult_f lam e^{ik.x} (the row pass doubles ky > 0).
template <int CX = 0, class X>
__device__ __forceinline__ void col_adj_emit(const cplx<typename X::R> (&lam)[X::E], cplx<typename X::R>* G, int b, int c,
                                             int ky, bool act, const X& xf,
                                             cplx<typename X::R>* gtile = nullptr) {
  using R = typename X::R;
  constexpr int E = X::E;
  auto mult = [&](cplx<R> (&z)[E], int f) {
#pragma unroll
    for (int j = 0; j < E; ++j)
      z[j] = X::none(j) ? mk<R>(0, 0) : cscale_rn(lam[j], prod_mult<R>(f, xf.kx(j), (R)ky));
  };
  cplx<R> z[E];
  if (c == 0) {
    cplx<R> z1[E];
    mult(z, 0); mult(z1, 1);
    xf.template from_spec2<true>(z, z1);
    col_put<CX>(z, G, NG, b, 0, ky, act, xf, gtile);
    col_put<CX>(z1, G, NG, b, 1, ky, act, xf, gtile);
  } else {
    mult(z, 2);
    xf.template from_spec<true>(z);
    col_put<CX>(z, G, NG, b, 2, ky, act, xf, gtile);
  }
}

// Sum over the lanes of a column's group, added to hacc by its first lane.
template <class X>
__device__ __forceinline__ void col_hacc(double* hacc, const ColId<X>& id, bool act, const X& xf, double part) {
#pragma unroll
  for (int o = X::L / 2; o >= 1; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (act && xf.l == 0) hacc[((size_t)id.b * X::K + id.ky) * 2 + id.ch] += part;
}

// The algebra of an adjoint stage at one mode from the cotangent Xb of its adjoint
// right-hand side: returns the cotangent fed to the next one (times h or t) and adds the
// terms of the step-size accumulator to hpart, those over h (or t) to hdiv.  JV(q) reads
// and JW(q, v) writes slot q, QV(q) reads the record, E() gives exp(h/2 L) mask
// (Lawson-RK4); prev: a step precedes (AJ_S1), whose recorded k4 QP() gives.
template <int STAGE, typename R, class JVf, class JWf, class QVf, class Ef, class QPf>
__device__ __forceinline__ cplx<R> adj_algebra(R h, R t, R L, cplx<R> Xb, bool prev, double& hpart, double& hdiv, JVf&& JV,
                                               JWf&& JW, QVf&& QV, Ef&& E, QPf&& QP) {
  constexpr bool rk43 = STAGE >= AJ43_INIT;
  auto ip = [&](cplx<R> a, cplx<R> bb) { return rdot2(a.x, a.y, bb.x, bb.y); };
  cplx<R> kb = mk<R>(0, 0);
  if (!rk43) {
    const R e = E();
    const R dedh = e * L / R(2);
    switch (STAGE) {
      case AJ_PRE: {
        const cplx<R> ob = JV(J_OB);
        JW(J_F2, ob); JW(J_A1, cdiv_k<6>(ob));
        JW(J_K2, cdiv_k<3>(ob)); JW(J_B3, cdiv_k<3>(ob));
        kb = cdiv_k<6>(ob);                                   // k4bar
        hdiv += ip(kb, QV(Q_K4));
      } break;
      case AJ_S4: {
        const cplx<R> f2b = cadd(JV(J_F2), Xb), b3b = cadd(JV(J_B3), Xb);
        const cplx<R> b2b = JV(J_K2), b1b = JV(J_A1);
        const cplx<R> f = QV(Q_F), k1 = QV(Q_K1);
        const double eb = ip(b3b, QV(Q_K3)) + ip(b2b, QV(Q_K2)) + ip(b1b, cscale(k1, e)) +
                          ip(f2b, cscale(f, e));
        hpart += eb * (double)dedh;
        kb = cscale(b3b, e);                                     // k3bar
        hdiv += ip(kb, QV(Q_K3));
        JW(J_F2, cscale(f2b, e));                      // f1bar
        JW(J_A1, cscale(b1b, e));                      // a1bar
        JW(J_K2, cscale(b2b, e));                      // k2bar
      } break;
      case AJ_S3: {
        JW(J_F2, cadd(JV(J_F2), Xb));
        kb = cadd(JV(J_K2), cscale(Xb, R(0.5)));        // k2bar final
        hdiv += ip(kb, QV(Q_K2));
      } break;
      case AJ_S2: {
        const cplx<R> f1b = cadd(JV(J_F2), Xb);
        const cplx<R> a1b = cadd(JV(J_A1), cscale(Xb, R(0.5)));
        const double eb = ip(a1b, QV(Q_K1)) + ip(f1b, QV(Q_F));
        hpart += eb * (double)dedh;
        kb = cscale(a1b, e);                                     // k1bar
        hdiv += ip(kb, QV(Q_K1));
        JW(J_OB, cscale(f1b, e));                      // fbar (without the RHS1 term)
      } break;
      default: {   // AJ_S1: fbar += X1bar; then seed the previous step (if any)
        const cplx<R> fb = cadd(JV(J_OB), Xb);
        JW(J_OB, fb);
        if (prev) {
          JW(J_F2, fb); JW(J_A1, cdiv_k<6>(fb));
          JW(J_K2, cdiv_k<3>(fb)); JW(J_B3, cdiv_k<3>(fb));
          kb = cdiv_k<6>(fb);
          hdiv += ip(kb, QP());
        }
      } break;
    }
    kb = cscale(kb, h);
  } else {
    const cplx<R> eg = QV(RR_E);   // (e, e L h/2) of the attempt, e = exp(t L h/2)
    const R e = eg.x;
    const R dedt = eg.y;
    switch (STAGE) {
      case AJ43_PRE:      // from (xbar_f, k5bar) in (X0, K1) slots: RHS5 input = k5bar
      case AJ43_IPRE: {   // initial k1 = t v(x0): input = k1bar
        kb = JV(JJ_K1);
        hdiv += ip(kb, QV(STAGE == AJ43_PRE ? RR_K5 : RR_K1));
      } break;
      case AJ43_S5: {     // xbar_f += Xbar5; distribute to x2, k1'', k2', k3', k4
        const cplx<R> xfb = cadd(JV(JJ_X0), Xb);
        JW(JJ_X2, xfb);
        JW(JJ_K1PP, cdiv_k<6>(cscale(xfb, h)));
        JW(JJ_K2P, cdiv_k<3>(cscale(xfb, h)));
        JW(JJ_K3P, cdiv_k<3>(cscale(xfb, h)));
        kb = cdiv_k<6>(cscale(xfb, h));                       // k4bar
        hdiv += ip(kb, QV(RR_K4));
      } break;
      case AJ43_S4: {     // Y4 = x2 + h k3'
        const cplx<R> x2b = cadd(JV(JJ_X2), Xb);
        const cplx<R> k3pb = cadd(JV(JJ_K3P), cscale(Xb, h));
        const cplx<R> k2pb = JV(JJ_K2P), k1ppb = JV(JJ_K1PP);
        const cplx<R> x0 = QV(RR_X0), k1 = QV(RR_K1);
        const double eb = ip(k3pb, QV(RR_K3)) + ip(k2pb, QV(RR_K2)) +
                          ip(k1ppb, cscale(k1, e)) + ip(x2b, cscale(x0, e));
        hpart += eb * (double)dedt;
        kb = cscale(k3pb, e);                                    // k3bar
        hdiv += ip(kb, QV(RR_K3));
        JW(JJ_K2, cscale(k2pb, e));                    // k2bar (partial)
        JW(JJ_K1P, cscale(k1ppb, e));                  // k1'bar (partial)
        JW(JJ_XB, cscale(x2b, e));                     // xbar (partial)
      } break;
      case AJ43_S3: {     // Y3 = x + h k2/2
        JW(JJ_XB, cadd(JV(JJ_XB), Xb));
        kb = cadd(JV(JJ_K2), cscale(cscale(Xb, h), R(0.5)));   // k2bar final
        hdiv += ip(kb, QV(RR_K2));
      } break;
      case AJ43_S2: {     // Y2 = x + h k1'/2; then x0bar, k1bar of this attempt
        const cplx<R> xbb = cadd(JV(JJ_XB), Xb);
        const cplx<R> k1pb = cadd(JV(JJ_K1P), cscale(cscale(Xb, h), R(0.5)));
        const double eb = ip(k1pb, QV(RR_K1)) + ip(xbb, QV(RR_X0));
        hpart += eb * (double)dedt;
        JW(JJ_X0, cscale(xbb, e));
        JW(JJ_K1, cscale(k1pb, e));
      } break;
      default: {          // AJ43_INIT: initial k1 = t v(x0): x0bar += Xbar
        JW(JJ_X0, cadd(JV(JJ_X0), Xb));
      } break;
    }
    kb = cscale(kb, t);
  }
  return kb;
}

template <typename R, int N, int STAGE>
__global__ void __launch_bounds__(COLWARPS * 32, 1) k_col_adj(ColAdjParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  ECS_COL_PROLOGUE(popc_c(adj_jmask(STAGE)), 1);   // the multipliers
  const int ch = id.ch, b = id.b, ky = id.ky;
  if (p.ctl && p.ctl[b].done) return;
  const size_t row = ((size_t)ch * K + ky) * M;
  cplx<R>* J = p.J + (size_t)b * p.nslot * VEC + row;
  const cplx<R>* Q = p.rec + (size_t)b * p.rec_bstride + row;
  const cplx<R>* Qp = p.rec_prev ? p.rec_prev + (size_t)b * p.rec_bstride + row : nullptr;
  const R h = p.ctl ? (R)p.ctl[b].h : (R)p.h, t = (R)p.t;
  constexpr bool rk43 = STAGE >= AJ43_INIT;
  constexpr bool has_rhs = !(STAGE == AJ_PRE || STAGE == AJ43_PRE || STAGE == AJ43_IPRE);
  const R coeff = ch == 0 ? p.nu : p.eta;
  double hpart = 0.0, hdiv = 0.0;   // hdiv: the terms over h (RK4) or t (RK4(3))
  constexpr unsigned JM = adj_jmask(STAGE);
  Operands<X, JM> op(rows);
  op.begin(J, VEC);
  const TableRow<X, has_rhs && rows_fit(popc_c(JM), 1)> mu(rows + popc_c(JM) * M, mu_row<X>(p.tw, ky));
  cplx<R> xb[E];
  if (has_rhs) col_adj_xb(p.H, b, ch, ky, xf, mu, xb);
  op.load(J, VEC, true, xf);
  cplx<R> lam[E];   // next adjoint-RHS input lambda / c_ky (multipliers applied per product below)
#pragma unroll
  for (int i = 0; i < E; ++i) {
      lam[i] = mk<R>(0, 0);
      const int slot = xf.slot(i);
      if (slot < 0) continue;
      const cplx<R> kb = adj_algebra<STAGE, R>(
          h, t, diss_L<R>(xf.kx(i), (R)ky, coeff), has_rhs ? xb[i] : mk<R>(0, 0), Qp != nullptr, hpart, hdiv,
          [&](int q) -> cplx<R> { return op.get(q, i, slot); }, [&](int q, cplx<R> v) { J[q * VEC + slot] = v; },
          [&](int q) -> cplx<R> { return __ldg(Q + q * VEC + slot); },
          [&]() { return slot == 0 && ky == 0 ? R(0) : exp(h / R(2) * diss_L<R>(xf.kx(i), (R)ky, coeff)); },
          [&]() -> cplx<R> { return __ldg(Qp + Q_K4 * VEC + slot); });
      // lambda = kb; the product multipliers vanish at (0,0), which the mask removes
      lam[i] = cscale(kb, ky == 0 ? R(1) : R(0.5));   // kb / c_ky, exactly
  }
  col_hacc(p.hacc, id, true, xf, hpart + hdiv / (double)(rk43 ? t : h));
  if (STAGE == AJ43_S2 || STAGE == AJ43_INIT || (STAGE == AJ_S1 && !Qp)) return;   // nothing follows
  col_adj_emit(lam, p.G, b, ch, ky, true, xf);
}

// Rejected Lawson-RK4(3) attempt in reverse: k1_next = e (e k1) ((e, e L h/2) from the attempt's record).
template <typename R>
__global__ void k_adj_reject(cplx<R>* J, int nslot, const cplx<R>* rec, double* hacc, int n, int B) {
  const Geom g = make_geom(n);
  const size_t VEC = (size_t)2 * g.K * g.M;
  // one warp per (b, ky) column so that hacc[b][ky] has a single writer
  const int lane = threadIdx.x & 31;
  const int colid = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (colid >= B * g.K) return;
  const int b = colid / g.K, ky = colid - b * g.K;
  cplx<R>* Jb = J + (size_t)b * nslot * VEC;
  double part = 0.0;
  for (int ch = 0; ch < 2; ++ch)
    for (int slot = lane; slot < g.M; slot += 32) {
      const size_t o = ((size_t)ch * g.K + ky) * g.M + slot;
      const cplx<R> eg = rec[RR_E * VEC + o];   // (e, e L h/2) of the attempt
      const R e = eg.x;
      const R dedt = eg.y;
      const cplx<R> k1 = rec[RR_K1 * VEC + o], k1e = cscale(k1, e);
      const cplx<R> kppb = Jb[JJ_K1 * VEC + o];
      const cplx<R> kpb = cscale(kppb, e);
      part += (rdot2(kppb.x, kppb.y, k1e.x, k1e.y) + rdot2(kpb.x, kpb.y, k1.x, k1.y)) * (double)dedt;
      Jb[JJ_K1 * VEC + o] = cscale(kpb, e);
    }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (lane == 0) hacc[((size_t)b * g.K + ky) * 2] += part;
}

// Head of the adjoint: from Ybar = cotangent of sym(Phi) (box, already
// -(c/n^2) rfft2(c_out)), Phibar = sym^T(Ybar) and sxbar = <Phibar, i kx Phi>
// (symmetry.py:4-25; shift_x uses masked kx).  One cluster of SUM_CL CTAs per batch
// element (at n = 128 one CTA took 42 us, a cluster takes 9.5).
template <typename R>
__global__ void __cluster_dims__(SUM_CL, 1, 1) k_adj_head(const cplx<R>* Ybar, const cplx<R>* phi, const double* sx, int sx_shared, double sy,
                           int odd, int rot, cplx<R>* Phibar, long pb_stride, double* sxbar, int n) {
  const Geom g = make_geom(n);
  const size_t VEC = (size_t)2 * g.K * g.M;
  const int b = blockIdx.x / SUM_CL, r = blockIdx.x % SUM_CL;
  const double s = sx[sx_shared ? 0 : b];
  const cplx<R>* Y = Ybar + (size_t)b * VEC;
  cplx<R>* P = Phibar + (size_t)b * pb_stride;
  double part = 0.0, none = 0.0;
  for (size_t i = (size_t)r * blockDim.x + threadIdx.x; i < VEC; i += (size_t)SUM_CL * blockDim.x) {
    // i indexes the SOURCE mode kappa (the mode of Phi); its image is kx_out
    const int slot = i % g.M; const int ky = (i / g.M) % g.K; const int c = (int)(i / ((size_t)g.K * g.M));
    const int kap = slot_to_kx(slot, g.kmax, g.M);
    const int kout = odd ? -kap : kap;
    const int sout = kout >= 0 ? kout : kout + g.M;
    cplx<R> y = Y[((size_t)c * g.K + ky) * g.M + sout];
    if (rot) { y.y = -y.y; if (c == 1) { y.x = -y.x; y.y = -y.y; } }   // R^T = sign_c conj
    if (odd) { y.x = -y.x; y.y = -y.y; }
    const bool m = !(kap == 0 && ky == 0);
    double sn, cs;
    sincos(m ? (double)ky * sy : 0.0, &sn, &cs);
    y = cmul(mk<R>((R)cs, (R)-sn), y);
    sincos(m ? (double)kap * s : 0.0, &sn, &cs);
    y = cmul(mk<R>((R)cs, (R)-sn), y);
    P[i] = y;
    const cplx<R> ph = phi[i];
    const R km = m ? (R)kap : R(0);
    // <y, i kap phi> = Re(conj(y) * i kap phi)
    part += (double)y.x * (double)(-km * ph.y) + (double)y.y * (double)(km * ph.x);
  }
  cluster_sum2(part, none);
  if (r == 0 && threadIdx.x == 0) sxbar[b] = part;
}

// Ybar = -(c_ky/n^2) * box  (transpose of out = base - irfft2(.))
template <typename R>
__global__ void k_box_scale_c(cplx<R>* v, long stride, int n, int B, R sign_over_n2) {
  const Geom g = make_geom(n);
  const size_t VEC = (size_t)2 * g.K * g.M;
  const long total = (long)B * VEC;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int b = (int)(i / VEC); const size_t o = i - (size_t)b * VEC;
    const int ky = (o / g.M) % g.K;
    cplx<R>* q = v + (size_t)b * stride + o;
    *q = cscale(*q, (ky == 0 ? R(1) : R(2)) * sign_over_n2);
  }
}

// Z = fbar0 * n^2 / c_ky (so that from_box(Z) = to_box^T(fbar0)).
template <typename R>
__global__ void k_box_to_fields_adj(const cplx<R>* fb, long stride, cplx<R>* Z, int n, int B) {
  const Geom g = make_geom(n);
  const size_t VEC = (size_t)2 * g.K * g.M;
  const long total = (long)B * VEC;
  const R n2 = R(n) * R(n);
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int b = (int)(i / VEC); const size_t o = i - (size_t)b * VEC;
    const int ky = (o / g.M) % g.K;
    Z[i] = cscale(fb[(size_t)b * stride + o], n2 / (ky == 0 ? R(1) : R(2)));
  }
}

// g += cT vt / (2n^2) + csx vx / (2n^2)  (phase-condition transposes, loss_functions.py:124-129)
template <typename R>
__global__ void k_adj_phase(R* gfields, const R* vt, const R* vx, const double* cT, const double* csx, int n, int B) {
  const long per = 2L * n * n;
  const long total = (long)B * per;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int b = (int)(i / per); const long o = i - (long)b * per;
    gfields[i] += (R)((cT[b] * (double)vt[o] + csx[b] * (double)vx[o]) / (double)per);
  }
}

// Deterministic reduction of the [B][K][2] accumulators: out[b] = scale * sum hacc[b].
static __global__ void k_reduce_hacc(const double* hacc, int K, double scale, double* out, int B) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  double s = 0.0;
  for (int k = 0; k < 2 * K; ++k) s += hacc[(size_t)b * 2 * K + k];
  out[b] = s * scale;
}

// Reverse segment r of several candidates' gradient sweeps, aligned at each
// candidate's end: candidate b (nseg[b] segments) works on its segment
// g = nseg[b] - 1 - r, whose start state is ckpt[g][b]; a candidate with g < 0
// is done (skipped by every launch of the segment).
template <typename R>
__global__ void k_grad_segment(cplx<R>* F, const cplx<R>* ckpt, const int* nseg, int r, StepCtl* ctl, long vec,
                               int B) {
  const long total = (long)B * vec;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int b = (int)(i / vec);
    const int g = nseg[b] - 1 - r;
    if (i % vec == 0) ctl[b].done = g < 0 ? 1 : 0;
    if (g >= 0) F[i] = ckpt[((size_t)g * B + b) * vec + (i % vec)];
  }
}

}  // namespace ecs
