// Column passes of the other fixed-step shooting modes of mismatch_RPO
// (jax_scripts/lib/loss_functions.py:48-85), sharing the row passes and the
// adaptive stepper's slot array S [B][S_NSLOT][2][K][M]:
//   FX_RK4  classic RK4 with dissipation in the right-hand side (timestepping.py:17-44)
//   FX_RK6  Lawson sixth-order RK, e = exp(h/6 L) mask (timestepping.py:83-125)
//   FX_TD4  two-derivative RK4 (timestepping.py:127-149): each step evaluates the
//           right-hand side at f and f_temp and its Jacobian-vector product there
//           (the tangent row pass on the recorded physical fields of that point)
// One launch per stage; STAGE 0 starts a run (inverse transforms of F).  Modes
// outside the box: RK4 and TDRK4 leave them unchanged (their right-hand side
// is masked), Lawson-RK6 zeroes them (masked integrating factor), as the
// reference does.
#pragma once

#include "kernels.cuh"
#include "kernels_rk43.cuh"
#include "kernels_adj.cuh"

namespace ecs {

enum FxScheme : int { FX_RK4 = 0, FX_RK6 = 1, FX_TD4 = 2 };
// slots: F, then K1..K7 (RK4 uses K1..K3, RK6 K1..K7); TDRK4: K1, A1, FT, K2
enum FxSlot { X_F = 0, X_K1 = 1, X_A1 = 2, X_FT = 3, X_K2T = 4 };
// TDRK4 trajectory record per step (for the tangent and adjoint): the step's
// start state, k1, a1, f_temp, k2, a2.
enum TdRec { TR_F = 0, TR_K1, TR_A1, TR_FT, TR_K2, TR_A2, TR_NREC };

template <typename R>
struct ColFxParams {
  const cplx<R>* H;     // [B][NH][K][N]
  cplx<R>* G;           // [B][NG][K][N]
  cplx<R>* S;           // [B][S_NSLOT][2][K][M]
  const R* Etab;        // [B][2][K][M] e = exp(h/6 L) mask (RK6)
  const StepCtl* ctl;   // [B] (h)
  const cplx<R>* fhat;  // [K][M]
  const cplx<R>* tw;
  R nu, eta;
  int B, produce;
  cplx<R>* rec;         // linearisation (batch 1): record of this step, or null: TDRK4 [TR_NREC][2][K][M];
                        // RK4 / Lawson-RK6 [f0, k_1..k_S, x_2..x_S] (see kernels_fxl.cuh)
};

// The right-hand side entering a stage: 0 none, 1 full (forcing), 2 Jacobian-vector product (no forcing).
__host__ __device__ constexpr int fx_rhs(int scheme, int stage) {
  return stage == 0 ? 0 : (scheme == FX_TD4 && (stage == 2 || stage == 4)) ? 2 : 1;
}
__host__ __device__ constexpr int fx_stages(int scheme) { return scheme == FX_RK6 ? 8 : 4; }

// Slots that a stage reads before it writes any (bits of FxSlot); they are loaded
// together before the stage's stores.
__host__ __device__ constexpr unsigned fx_smask(int scheme, int stage) {
  const unsigned F = 1u << X_F;
  if (stage == 0) return F;
  if (scheme == FX_RK4)
    return F | (stage == 2 || stage == 4 ? 1u << X_K1 : 0u) | (stage >= 3 ? 1u << (X_K1 + 1) : 0u) |
           (stage == 4 ? 1u << (X_K1 + 2) : 0u);
  if (scheme == FX_RK6) return stage == 8 ? F | (1u << X_K1) | (1u << (X_K1 + 2)) | (1u << (X_K1 + 3)) |
                                                (1u << (X_K1 + 5)) | (1u << (X_K1 + 6))
                                          : F | (((1u << (stage - 1)) - 1u) << X_K1);
  return stage == 1 ? F : stage == 2 ? F | (1u << X_K1) : stage == 3 ? 1u << X_FT
       : F | (1u << X_K1) | (1u << X_A1) | (1u << X_K2T);
}

// The algebra of a stage at one mode: the stage input from the derivative v (forcing
// included).  Q(q) reads and W(q, a) writes slot q, E() gives the factor e (Lawson-RK6)
// and put(q, a) records.
template <int SCHEME, int STAGE, typename R, class Qf, class Wf, class Ef, class Pf>
__device__ __forceinline__ cplx<R> fx_algebra(R h, R L, cplx<R> v, Qf&& Q, Wf&& W, Ef&& E, Pf&& put) {
  constexpr unsigned SM = fx_smask(SCHEME, STAGE);
  cplx<R> xin = mk<R>(0, 0);
  if (STAGE == 0) {
    xin = Q(X_F);
  } else if (SCHEME == FX_RK4) {
    // v_fn includes dissipation L x at the stage input x (loss_functions.py:53, mhd_jax.py:171-173)
    const cplx<R> f = Q(X_F);
    cplx<R> xs = f;
    if (STAGE == 2) xs = cadd(f, cdiv_k<2>(Q(X_K1)));
    if (STAGE == 3) xs = cadd(f, cdiv_k<2>(Q(X_K1 + 1)));
    if (STAGE == 4) xs = cadd(f, Q(X_K1 + 2));
    const cplx<R> k = cscale(cadd(v, cscale(xs, L)), h);            // timestepping.py:40-43
    // record: f0, k_s, x_{s+1}
    if (STAGE == 1) put(0, f);
    put(STAGE, k);
    if (STAGE < 4) {
      W(X_K1 + STAGE - 1, k);
      xin = STAGE < 3 ? cadd(f, cdiv_k<2>(k)) : cadd(f, k);
      put(4 + STAGE, xin);
    } else {
      const cplx<R> fn = cadd(cadd(cadd(cadd(f, cdiv_k<6>(Q(X_K1))), cdiv_k<3>(Q(X_K1 + 1))),
                                   cdiv_k<3>(Q(X_K1 + 2))), cdiv_k<6>(k));   // :44
      W(X_F, fn);
      xin = fn;
    }
  } else if (SCHEME == FX_RK6) {
    const R e = E();
    const cplx<R> k = cscale(v, h);
    // record: f0, k_s (before any factor)
    if (STAGE == 1) put(0, Q(X_F));
    put(STAGE, k);
    // f, k1..k_{STAGE-1} and the new k, times e after stages 1, 3..7 and stored
    constexpr bool SC = STAGE != 2 && STAGE != 8;
    cplx<R> f = Q(X_F), K_[9];
#pragma unroll
    for (int q = 1; q < 9; ++q) K_[q] = mk<R>(0, 0);
#pragma unroll
    for (int q = 1; q < STAGE; ++q)
      if ((SM >> (X_K1 + q - 1)) & 1u) K_[q] = Q(X_K1 + q - 1);
    K_[STAGE] = k;
    if (SC) {
      f = cscale_rn(f, e);
      W(X_F, f);
#pragma unroll
      for (int q = 1; q <= STAGE; ++q) { K_[q] = cscale_rn(K_[q], e); W(X_K1 + q - 1, K_[q]); }
    } else if (STAGE == 2) {
      W(X_K1 + 1, k);
    }
    switch (STAGE) {
      case 1:   // :110-112
        xin = cadd(f, cdiv_k<6>(K_[1]));
        break;
      case 2:   // :113
        xin = cadd(cadd(f, cdiv_k<12>(K_[1])), cdiv_k<12>(K_[2]));
        break;
      case 3:   // :114-115
        xin = cadd(csub(f, cdiv_k<33>(cscale(K_[2], R(4)))), cdiv_k<11>(cscale(K_[3], R(5))));
        break;
      case 4:   // :116-117
        xin = cadd(csub(csub(f, cdiv_k<4>(K_[1])), cdiv_k<44>(cscale(K_[2], R(29)))),
                   cdiv_k<22>(cscale(K_[3], R(31))));
        break;
      case 5:   // :118-119
        xin = cadd(cadd(csub(cadd(cadd(f, cdiv_k<11>(cscale(K_[1], R(3)))), cdiv_k<33>(cscale(K_[2], R(8)))),
                             cdiv_k<11>(cscale(K_[3], R(4)))), cdiv_k<11>(K_[4])),
                   cdiv_k<33>(cscale(K_[5], R(14))));
        break;
      case 6:   // :120-121
        xin = cadd(csub(cadd(cadd(csub(csub(f, cdiv_k<48>(cscale(K_[1], R(17)))), cdiv_k<12>(cscale(K_[2], R(5)))),
                                  K_[3]), K_[4]), cdiv_k<12>(cscale(K_[5], R(13)))),
                   cdiv_k<16>(cscale(K_[6], R(11))));
        break;
      case 7:   // :122-123
        xin = cadd(csub(cadd(csub(csub(cadd(cadd(f, cdiv_k<39>(cscale(K_[1], R(20)))),
                                                cdiv_k<39>(cscale(K_[2], R(12)))),
                                           cdiv_k<39>(cscale(K_[3], R(31)))), cdiv_k<39>(K_[4])),
                                 cdiv_k<39>(cscale(K_[5], R(34)))), cdiv_k<39>(cscale(K_[6], R(11)))),
                   cdiv_k<39>(cscale(K_[7], R(16))));
        break;
      default: {   // 8: :124
        const R c1 = R(13) / R(200), c3 = R(4) / R(25), c4 = R(11) / R(40);
        const cplx<R> fn = cadd(cadd(cadd(f, cscale(cadd(K_[1], k), c1)), cscale(cadd(K_[3], K_[7]), c3)),
                                cscale(cadd(K_[4], K_[6]), c4));
        W(X_F, fn);
        xin = fn;
      } break;
    }
    if (STAGE < 8) put(8 + STAGE, xin);   // the stage input x_{s+1}
  } else {   // FX_TD4, timestepping.py:137-144; v_fn and its derivative include dissipation
    switch (STAGE) {
      case 1: {   // k1 = h v(f); next: the transforms of k1 (tangent input of jac(f, k1))
        const cplx<R> k1 = cscale(cadd(v, cscale(Q(X_F), L)), h);
        W(X_K1, k1);
        put(TR_F, Q(X_F)); put(TR_K1, k1);
        xin = k1;
      } break;
      case 2: {   // a1 = h jac(f, k1); f_temp = f + k1/2 + a1/8
        const cplx<R> k1 = Q(X_K1);
        const cplx<R> a1 = cscale(cadd(v, cscale(k1, L)), h);
        W(X_A1, a1);
        const cplx<R> ft = cadd(cadd(Q(X_F), cdiv_k<2>(k1)), cdiv_k<8>(a1));
        W(X_FT, ft);
        put(TR_A1, a1); put(TR_FT, ft);
        xin = ft;
      } break;
      case 3: {   // k2 = h v(f_temp)
        const cplx<R> k2 = cscale(cadd(v, cscale(Q(X_FT), L)), h);
        W(X_K2T, k2);
        put(TR_K2, k2);
        xin = k2;
      } break;
      default: {  // a2 = h jac(f_temp, k2); f = f + k1 + a1/6 + a2/3
        const cplx<R> a2 = cscale(cadd(v, cscale(Q(X_K2T), L)), h);
        put(TR_A2, a2);
        const cplx<R> fn = cadd(cadd(cadd(Q(X_F), Q(X_K1)), cdiv_k<6>(Q(X_A1))), cdiv_k<3>(a2));
        W(X_F, fn);
        xin = fn;
      } break;
    }
  }
  return xin;
}

template <typename R, int N, int SCHEME, int STAGE>
__global__ void __launch_bounds__(COLWARPS * 32, 1) k_col_fx(ColFxParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  constexpr int rhs = fx_rhs(SCHEME, STAGE);
  ECS_COL_PROLOGUE(popc_c(fx_smask(SCHEME, STAGE)), 2);   // the forcing, the multipliers
  const int c = id.ch, b = id.b, ky = id.ky;
  const R h = (R)p.ctl[b].h;
  const R coeff = c == 0 ? p.nu : p.eta;
  const size_t row = ((size_t)c * K + ky) * M;
  cplx<R>* S = p.S + (size_t)b * S_NSLOT * VEC + row;
  const R* Et = p.Etab + (size_t)b * VEC + row;
  cplx<R>* rec = p.rec ? p.rec + row : nullptr;
  constexpr unsigned SM = fx_smask(SCHEME, STAGE);
  Operands<X, SM> op(rows);
  op.begin(S, VEC);
  constexpr int n = popc_c(SM);
  const TableRow<X, rhs == 1 && rows_fit(n, 2)> forcing(rows + n * M, p.fhat + ky * M);
  const TableRow<X, rows_fit(n, 2)> mu(rows + (n + 1) * M, mu_row<X>(p.tw, ky));
  cplx<R> r[E];
  if (rhs) col_load_rhs(p.H, b, c, ky, xf, r);
  op.load(S, VEC, true, xf);
  cplx<R> x[E];
#pragma unroll
  for (int i = 0; i < E; ++i) {
    x[i] = mk<R>(0, 0);
    const int slot = xf.slot(i);
    if (slot < 0) continue;
    cplx<R> v = mk<R>(0, 0);
    if (rhs) {
      v = r[i];
      if (rhs == 1 && c == 0 && !(slot == 0 && ky == 0)) v = cadd(v, forcing(slot));
    }
    x[i] = fx_algebra<SCHEME, STAGE, R>(h, diss_L<R>(xf.kx(i), (R)ky, coeff), v,
                                        [&](int q) -> cplx<R> { return op.get(q, i, slot); },
                                        [&](int q, cplx<R> a) { S[q * VEC + slot] = a; }, [&]() { return __ldg(Et + slot); },
                                        [&](int q, cplx<R> a) { if (rec) rec[q * VEC + slot] = a; });
  }
  if (!p.produce) return;
  col_inverse_uv(x, p.G, b, c, ky, id.act, xf, mu);
}

// ---------------------------------------------------------------------------
// TDRK4 tangent.  With the quadratic right-hand side, N'(f) x = N'(x) f, so the
// tangent of a1 = h J(f) k1 is (dh/h) a1 + h [N'(f) dk1 + N'(k1) df + L dk1]:
// one "dual" tangent row pass of two tangent field sets against two primal
// field sets.  Per step, along (df, dT):
//   dk1 = (dh/h) k1 + h J(f) df
//   da1 = (dh/h) a1 + h [N'(f) dk1 + N'(k1) df + L dk1]
//   dft = df + dk1/2 + da1/8
//   dk2 = (dh/h) k2 + h J(f_temp) dft
//   da2 = (dh/h) a2 + h [N'(f_temp) dk2 + N'(k2) dft + L dk2]
//   df' = df + dk1 + da1/6 + da2/3
// Ga holds the transforms of df / dft, Gb those of dk1 / dk2.
// ---------------------------------------------------------------------------
template <typename R>
struct RowTan2Params {
  const cplx<R>* Ga;    // [B][NG][K][N] tangent paired with phys_b
  const cplx<R>* Gb;    // [B][NG][K][N] tangent paired with phys_a
  cplx<R>* H;           // [B][NH][K][N]
  const R* phys_a;      // primal point (f or f_temp), B_x/B_y with the mean field: [N][NPH][N]
  const R* phys_b;      // stage derivative (k1 or k2), no mean field: [N][NPH][N]
  const cplx<R>* tw;
  int B;
};

// Linearised products dP of one tangent (du, dv, dbx, dby) about one field set (u, v, bx, by), accumulated.
template <typename R>
__device__ __forceinline__ void acc_tan_products(R u, R v, R bx, R by, R du, R dv, R dbx, R dby, cplx<R>& W, R& p3) {
  // (sums of two products with a fixed order of rounding, whatever code surrounds them)
  W.x += R(2) * (fpm(u, du, v, dv) - fpm(bx, dbx, by, dby));   // dP1
  W.y += fpp(bx, dby, by, dbx) - fpp(u, dv, v, du);            // dP2
  p3 += fpp(u, dby, by, du) - fpp(v, dbx, bx, dv);             // dP3
}

// Rows x0 .. x0 + XT - 1 of tangent b; the tile of Ga holds the H tile at the end (each
// warp reads and writes its own column of the tiles).  CX: as in row_tan_body.
template <int XT, bool CX = false, class X>
__device__ __forceinline__ void row_tan2_body(const RowTan2Params<typename X::R>& p, int b, int x0, const X& xf,
                                              cplx<typename X::R>* s_Ga, cplx<typename X::R>* s_Gb, bool load_g = true,
                                              cplx<typename X::R>* hcols = nullptr) {
  using R = typename X::R;
  constexpr int E = X::E, L = X::L, K = X::K, N = X::N;
  const int w = threadIdx.x / L;
  if (!CX || load_g) {
    load_tile<R, N, XT>(s_Ga, p.Ga + (size_t)b * NG * K * N, NG * K, x0);
    load_tile<R, N, XT>(s_Gb, p.Gb + (size_t)b * NG * K * N, NG * K, x0);
  }
  __syncthreads();
  cplx<R> W[E];
  R p3[E];
#pragma unroll
  for (int j = 0; j < E; ++j) { W[j] = mk<R>(0, 0); p3[j] = R(0); }
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {   // pass 0: Gb about phys_a; pass 1: Ga about phys_b
    const cplx<R>* ph = phys_row<R, N>(pass == 0 ? p.phys_a : p.phys_b, x0 + w) + xf.l;
    cplx<R> duv[E], dbb[E];
    row_inverse<XT>(pass == 0 ? s_Gb : s_Ga, w, xf, duv, dbb);
#pragma unroll
    for (int j = 0; j < E; ++j) {
      const cplx<R> uv = ph[L * j], bb = ph[N + L * j];
      acc_tan_products<R>(uv.x, uv.y, bb.x, bb.y, duv[j].x, duv[j].y, dbb[j].x, dbb[j].y, W[j], p3[j]);
    }
  }
  cplx<R> Z[E];
#pragma unroll
  for (int j = 0; j < E; ++j) Z[j] = mk<R>(p3[j], R(0));
  row_forward<XT>(W, Z, s_Ga, w, xf);
  __syncthreads();
  if constexpr (CX) {
    if (hcols) { scatter_h_tile<XT>(s_Ga, hcols, x0, xf); return; }
  }
  store_tile<R, N, XT>(p.H + (size_t)b * NH * K * N, s_Ga, NH * K, x0);
}

template <typename R, int N, int XT>
__global__ void __launch_bounds__(XT * Xf<R, N>::L) k_row_tan2(RowTan2Params<R> p) {
  using X = Xf<R, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_x = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_Ga = s_x + X::smem(XT / X::G);
  const int tiles = N / XT;
  const int b = blockIdx.x / tiles, x0 = (blockIdx.x - b * tiles) * XT;
  load_tables<X>(s_x, p.tw);
  pdl_wait();
  pdl_trigger();
  row_tan2_body<XT>(p, b, x0, X(s_x, threadIdx.x >> 5), s_Ga, s_Ga + NG * X::K * (XT + 1));
}

enum TdTanSlot { DT_F = 0, DT_K1, DT_A1, DT_FT, DT_K2, DT_NSLOT };

template <typename R>
struct ColTdjParams {
  const cplx<R>* H;     // [B][NH][K][N]
  cplx<R>* Ga;          // [B][NG][K][N]
  cplx<R>* Gb;          // [B][NG][K][N]
  cplx<R>* D;           // tangent slots [B][nslot][2][K][M]
  int nslot;
  const cplx<R>* rec;   // primal record of this step [TR_NREC][2][K][M]
  const double* dT;     // [B]
  double h, dscale;     // dh = dT * dscale
  const cplx<R>* tw;
  R nu, eta;
  int B, produce;
};

__host__ __device__ constexpr unsigned tdj_dmask(int stage) {   // slots read (bits of TdTanSlot)
  return stage <= 1 ? 1u << DT_F : stage == 2 ? (1u << DT_F) | (1u << DT_K1) : stage == 3 ? 1u << DT_FT
       : (1u << DT_F) | (1u << DT_K1) | (1u << DT_A1) | (1u << DT_K2);
}

// The record row that a stage reads.
__host__ __device__ constexpr int tdj_qrow(int stage) {
  return stage == 1 ? (int)TR_K1 : stage == 2 ? (int)TR_A1 : stage == 3 ? (int)TR_K2 : (int)TR_A2;
}
// The algebra of a stage at one mode: its output from the derivative r and the record's q.
template <int STAGE, typename R, class DVf, class DWf>
__device__ __forceinline__ cplx<R> tdj_algebra(R h, R dpar_h, R L, cplx<R> r, cplx<R> q, DVf&& DV, DWf&& DW) {
  // d(h X) = (dh/h) (h X) + h dX, with the recorded h X and dX = r + L dx (no forcing)
  auto dk = [&](cplx<R> dxin) { return lin2_rn(q, dpar_h, cadd(r, cscale(dxin, L)), h); };
  cplx<R> xin = mk<R>(0, 0);
  switch (STAGE) {
    case 0: xin = DV(DT_F); break;
    case 1: { const cplx<R> dk1 = dk(DV(DT_F)); DW(DT_K1, dk1); xin = dk1; } break;
    case 2: {
      const cplx<R> dk1 = DV(DT_K1);
      const cplx<R> da1 = dk(dk1);
      DW(DT_A1, da1);
      const cplx<R> dft = cadd(cadd(DV(DT_F), cdiv_k<2>(dk1)), cdiv_k<8>(da1));
      DW(DT_FT, dft);
      xin = dft;
    } break;
    case 3: { const cplx<R> dk2 = dk(DV(DT_FT)); DW(DT_K2, dk2); xin = dk2; } break;
    default: {
      const cplx<R> da2 = dk(DV(DT_K2));
      const cplx<R> dfn = cadd(cadd(cadd(DV(DT_F), DV(DT_K1)), cdiv_k<6>(DV(DT_A1))), cdiv_k<3>(da2));
      DW(DT_F, dfn);
      xin = dfn;
    } break;
  }
  return xin;
}

template <typename R, int N, int STAGE>
__global__ void __launch_bounds__(COLWARPS * 32, 1) k_col_tdj(ColTdjParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  ECS_COL_PROLOGUE(popc_c(tdj_dmask(STAGE)), 2);   // the record row, the multipliers
  const int c = id.ch, b = id.b, ky = id.ky;
  const size_t row = ((size_t)c * K + ky) * M;
  cplx<R>* D = p.D + (size_t)b * p.nslot * VEC + row;
  const cplx<R>* Q = p.rec + row;
  const R h = (R)p.h;
  const R dpar = (R)(p.dT[b] * p.dscale);   // dh
  const R dpar_h = dpar / h;
  const R coeff = c == 0 ? p.nu : p.eta;
  constexpr unsigned DM = tdj_dmask(STAGE);
  Operands<X, DM> op(rows);
  op.begin(D, VEC);
  const TableRow<X, STAGE != 0> rq(rows + popc_c(DM) * M, Q + tdj_qrow(STAGE) * VEC);
  const TableRow<X, true> mu(rows + (popc_c(DM) + 1) * M, mu_row<X>(p.tw, ky));
  cplx<R> r[E];
  if (STAGE != 0) col_load_rhs(p.H, b, c, ky, xf, r);
  op.load(D, VEC, true, xf);
  cplx<R> x[E];
#pragma unroll
  for (int i = 0; i < E; ++i) {
      x[i] = mk<R>(0, 0);
      const int slot = xf.slot(i);
      if (slot < 0) continue;
      x[i] = tdj_algebra<STAGE, R>(h, dpar_h, diss_L<R>(xf.kx(i), (R)ky, coeff), STAGE != 0 ? r[i] : mk<R>(0, 0),
                                   STAGE != 0 ? rq(slot) : mk<R>(0, 0), [&](int d) -> cplx<R> { return op.get(d, i, slot); },
                                   [&](int d, cplx<R> v) { D[d * VEC + slot] = v; });
  }
  if (!p.produce) return;
  // dk1, dk2 go to Gb (paired with the point f / f_temp); df, dft, df' to Ga
  col_inverse_uv(x, (STAGE == 1 || STAGE == 3) ? p.Gb : p.Ga, b, c, ky, id.act, xf, mu);
}

// ---------------------------------------------------------------------------
// TDRK4 adjoint.  Reverse of one step (lambda = h xbar is the input of each
// adjoint row pass; N'(x)^T from the transposed product chain of kernels_adj.cuh):
//   seed: a2bar = fbar'/3, k1bar = fbar', a1bar = fbar'/6, fbar = fbar'
//   dual pass, lambda = h a2bar at (f_temp, k2):  k2bar = N'(ft)^T lambda + h L a2bar,  ftbar = N'(k2)^T lambda
//   pass, lambda = h k2bar at f_temp:             ftbar += N'(ft)^T lambda + h L k2bar
//   fbar += ftbar, k1bar += ftbar/2, a1bar += ftbar/8
//   dual pass, lambda = h a1bar at (f, k1):       k1bar += N'(f)^T lambda + h L a1bar,  fbar += N'(k1)^T lambda
//   pass, lambda = h k1bar at f:                  fbar += N'(f)^T lambda + h L k1bar
// and hbar += <a2bar, a2>/h + <k2bar, k2>/h + <a1bar, a1>/h + <k1bar, k1>/h.
// ---------------------------------------------------------------------------
template <typename R>
struct RowAdj2Params {
  const cplx<R>* G;     // [B][NG][K][N]: fields 0..2 the product cotangents of lambda (/c_ky)
  cplx<R>* Ha;          // [B][NHA][K][N]: rfft2 rows of N'(phys_a)^T
  cplx<R>* Hb;          // [B][NHA][K][N]: rfft2 rows of N'(phys_b)^T
  const R* phys_a;      // [N][NPH][N]
  const R* phys_b;      // [N][NPH][N]
  const cplx<R>* tw;
  int B;
};

template <typename R, int N, int XT>
__global__ void __launch_bounds__(XT * Xf<R, N>::L) k_row_adj2(RowAdj2Params<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, L = X::L, K = X::K;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_x = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_G = s_x + X::smem(XT / X::G);
  const int tiles = N / XT;
  const int b = blockIdx.x / tiles, x0 = (blockIdx.x - b * tiles) * XT;
  const int w = threadIdx.x / L;
  const X xf(s_x, threadIdx.x >> 5);
  load_tables<X>(s_x, p.tw);
  pdl_wait();
  pdl_trigger();
  load_tile<R, N, XT>(s_G, p.G + (size_t)b * NG * K * N, 3 * K, x0);
  __syncthreads();
  cplx<R> P12[E], P3[E];
  row_inverse<XT, true>(s_G, w, xf, P12, P3);
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const cplx<R>* ph = phys_row<R, N>(pass == 0 ? p.phys_a : p.phys_b, x0 + w) + xf.l;
    cplx<R> A[E], Bv[E];
#pragma unroll
    for (int j = 0; j < E; ++j) row_adj_product<R>(P12[j], P3[j].x, ph[L * j], ph[N + L * j], A[j], Bv[j]);
    row_forward<XT, true>(A, Bv, s_G, w, xf);
    __syncthreads();
    store_tile<R, N, XT>((pass == 0 ? p.Ha : p.Hb) + (size_t)b * NHA * K * N, s_G, NHA * K, x0);
    __syncthreads();
  }
}

enum TdAdjSlot { JT_F = 0, JT_K1, JT_A1, JT_FT, JT_K2, JT_A2, JT_NSLOT };
enum TdAdjStage { TA_SEED = 0, TA_B = 1, TA_C = 2, TA_D = 3, TA_E = 4 };

template <typename R>
struct ColTdaParams {
  const cplx<R>* Ha;    // [B][NHA][K][N]
  const cplx<R>* Hb;    // [B][NHA][K][N] (dual passes)
  cplx<R>* G;           // [B][NG][K][N] (fields 0..2 written)
  cplx<R>* J;           // adjoint slots [B][nslot][2][K][M]
  int nslot;
  const cplx<R>* rec;   // primal record of this step [TR_NREC][2][K][M]
  double* hacc;         // [B][K][2]
  double h;
  const cplx<R>* tw;
  R nu, eta;
  int B;
};

__host__ __device__ constexpr unsigned tda_jmask(int stage) {   // slots read (bits of TdAdjSlot)
  return stage == TA_SEED ? 1u << JT_F
       : stage == TA_B ? 1u << JT_A2
       : stage == TA_C ? (1u << JT_F) | (1u << JT_K1) | (1u << JT_A1) | (1u << JT_FT) | (1u << JT_K2)
       : stage == TA_D ? (1u << JT_F) | (1u << JT_K1) | (1u << JT_A1) : (1u << JT_F) | (1u << JT_K1);
}

template <typename R, int N, int STAGE>
__global__ void __launch_bounds__(COLWARPS * 32, 1) k_col_tda(ColTdaParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  ECS_COL_PROLOGUE(popc_c(tda_jmask(STAGE)), 2);   // the record row, the multipliers
  const int c = id.ch, b = id.b, ky = id.ky;
  const size_t row = ((size_t)c * K + ky) * M;
  cplx<R>* J = p.J + (size_t)b * p.nslot * VEC + row;
  const cplx<R>* Q = p.rec + row;
  const R h = (R)p.h;
  const R coeff = c == 0 ? p.nu : p.eta;
  constexpr unsigned JM = tda_jmask(STAGE);
  Operands<X, JM> op(rows);
  op.begin(J, VEC);
  constexpr int QV = STAGE == TA_SEED ? (int)TR_A2 : STAGE == TA_B ? (int)TR_K2 : STAGE == TA_C ? (int)TR_A1 : (int)TR_K1;
  const TableRow<X, STAGE != TA_E> rq(rows + popc_c(JM) * M, Q + QV * VEC);
  const TableRow<X, STAGE != TA_SEED> mu(rows + (popc_c(JM) + 1) * M, mu_row<X>(p.tw, ky));
  cplx<R> xa[E], xbb[E];
  if (STAGE != TA_SEED) col_adj_xb(p.Ha, b, c, ky, xf, mu, xa);
  if (STAGE == TA_B || STAGE == TA_D) col_adj_xb(p.Hb, b, c, ky, xf, mu, xbb);
  op.load(J, VEC, true, xf);
  double hdiv = 0.0;   // the terms over h
  cplx<R> lam[E];
#pragma unroll
  for (int i = 0; i < E; ++i) {
      lam[i] = mk<R>(0, 0);
      const int slot = xf.slot(i);
      if (slot < 0) continue;
      const R L = diss_L<R>(xf.kx(i), (R)ky, coeff);
      auto JV = [&](int q) -> cplx<R> { return op.get(q, i, slot); };
      auto JW = [&](int q, cplx<R> v) { J[q * VEC + slot] = v; };
      auto ip = [&](cplx<R> a) {
        const cplx<R> v = rq(slot);
        return (double)a.x * (double)v.x + (double)a.y * (double)v.y;
      };
      cplx<R> kb = mk<R>(0, 0);   // cotangent whose h-multiple feeds the next adjoint pass
      switch (STAGE) {
        case TA_SEED: {
          const cplx<R> fb = JV(JT_F);
          const cplx<R> a2b = cdiv_k<3>(fb);
          JW(JT_A2, a2b); JW(JT_K1, fb); JW(JT_A1, cdiv_k<6>(fb));
          hdiv += ip(a2b);
          kb = a2b;
        } break;
        case TA_B: {
          const cplx<R> k2b = cadd(xa[i], cscale(JV(JT_A2), h * L));
          JW(JT_K2, k2b); JW(JT_FT, xbb[i]);
          hdiv += ip(k2b);
          kb = k2b;
        } break;
        case TA_C: {
          const cplx<R> ftb = cadd(cadd(JV(JT_FT), xa[i]), cscale(JV(JT_K2), h * L));
          JW(JT_F, cadd(JV(JT_F), ftb));
          JW(JT_K1, cadd(JV(JT_K1), cdiv_k<2>(ftb)));
          const cplx<R> a1b = cadd(JV(JT_A1), cdiv_k<8>(ftb));
          JW(JT_A1, a1b);
          hdiv += ip(a1b);
          kb = a1b;
        } break;
        case TA_D: {
          const cplx<R> k1b = cadd(cadd(JV(JT_K1), xa[i]), cscale(JV(JT_A1), h * L));
          JW(JT_K1, k1b);
          JW(JT_F, cadd(JV(JT_F), xbb[i]));
          hdiv += ip(k1b);
          kb = k1b;
        } break;
        default: {   // TA_E: the cotangent of the step's start state
          JW(JT_F, cadd(cadd(JV(JT_F), xa[i]), cscale(JV(JT_K1), h * L)));
        } break;
      }
      lam[i] = cscale(cscale(kb, h), ky == 0 ? R(1) : R(0.5));   // h kb / c_ky
  }
  col_hacc(p.hacc, id, id.act, xf, hdiv / (double)h);
  if (STAGE == TA_E) return;
  col_adj_emit(lam, p.G, b, c, ky, id.act, xf);
}

// Box entries back into the full half spectrum, leaving every other entry as it is
// (RK4 / TDRK4 carry the modes outside the box unchanged).
template <typename R>
__global__ void k_scatter_box_keep(const cplx<R>* box, cplx<R>* full, int n, int B) {
  const Geom g = make_geom(n);
  const int nh = n / 2 + 1;
  const long total = (long)B * 2 * n * nh;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int ky = i % nh; const long r = i / nh; const int pos = r % n; const long bc = r / n;
    const int slot = (ky < g.K) ? pos_to_slot(pos, n, g.kmax, g.M) : -1;
    if (slot >= 0) full[i] = box[(bc * g.K + ky) * g.M + slot];
  }
}

// Recurrence matrix of snapshots (jax_scripts/generate_turbulence.py:136-146):
// dist[j][i] = || |fs_j| - |fs_i| ||_2 over the len complex entries of a
// snapshot (spectral magnitudes: blind to translations).  One block per pair
// j >= i (the matrix is symmetric), FP64 accumulation, a fixed-order tree.
template <typename R>
__global__ void k_recurrence(const cplx<R>* fs, int S, long len, double* dist) {
  const int i = blockIdx.x, j = blockIdx.y;
  if (j < i) return;
  const cplx<R>* a = fs + (size_t)j * len;
  const cplx<R>* b = fs + (size_t)i * len;
  double acc = 0.0;
  for (long k = threadIdx.x; k < len; k += blockDim.x) {
    const double d = hypot((double)a[k].x, (double)a[k].y) - hypot((double)b[k].x, (double)b[k].y);
    acc += d * d;
  }
  __shared__ double red[32];
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    const double r = sqrt(t);
    dist[(size_t)j * S + i] = r;
    dist[(size_t)i * S + j] = r;
  }
}

// e = exp(h/div L) mask and h = (T/nc)/ms per batch element (timestepping.py:69-72, :105-108).
template <typename R>
__global__ void k_fx_setup(const double* T, int nc, int ms, int div, StepCtl* ctl, R* Etab, int n, double nu,
                           double eta, int B) {
  const Geom g = make_geom(n);
  const long per = 2L * g.K * g.M;
  const long total = (long)B * per;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int b = (int)(i / per);
    const double tseg = T[b] / (double)nc;
    const R h = (R)(tseg / (double)ms);
    if (i % per == 0) { ctl[b].t = tseg; ctl[b].h = (double)h; }
    const int slot = i % g.M; const long r = i / g.M; const int ky = r % g.K; const int c = (r / g.K) & 1;
    const int kx = slot_to_kx(slot, g.kmax, g.M);
    const R L = diss_L<R>((R)kx, (R)ky, (R)(c == 0 ? nu : eta));
    const bool msk = !(kx == 0 && ky == 0);
    Etab[i] = msk ? exp(h / R(div) * L) : R(0);
  }
}

}  // namespace ecs
