// Tangent (forward-mode) kernels of the shooting map: the JVP used as the
// Newton-GMRES matvec (reference: jax.jvp of objective_RPO, jax_scripts/lib/utils.py:108).
//
// A batch of B tangents shares one primal trajectory.  The primal solve records,
// per step (Lawson-RK4) or attempt (Lawson-RK4(3)), the compact stage inputs and
// stage derivatives; the tangent pass regenerates the primal's 4 physical
// fields (u, v, B_x, B_y) for a chunk of stages in one batched launch pair
// (shared by all tangents) and then advances the tangents with the linearised
// products of the Basdevant form (see kernels.cuh)
//   dP1 = 2 (u du - v dv) - 2 (B_x dB_x - B_y dB_y)
//   dP2 = B_x dB_y + B_y dB_x - u dv - v du
//   dP3 = u dB_y + B_y du - v dB_x - B_x dv
// and the product rule through the integrating factor, e' = e L h'/2.
#pragma once

#include "kernels.cuh"
#include "kernels_rk43.cuh"

namespace ecs {


// ---------------------------------------------------------------------------
// Regeneration of primal physical fields for a list of recorded stage inputs.
// ---------------------------------------------------------------------------
template <typename R>
struct ColRegenParams {
  const cplx<R>* rec;     // record base
  const long* items;      // [nitems] offsets (in box vectors) of the stage inputs in rec
  cplx<R>* G;             // [nitems][NG][K][N]
  const cplx<R>* tw;
  int nitems;
};

template <typename R, int N>
__global__ void __launch_bounds__(COLWARPS * 32) k_col_regen(ColRegenParams<R> p) {
  using X = Xf<R, N>;
  constexpr int K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  __shared__ __align__(16) cplx<R> s_x[X::smem(COLWARPS)];
  load_tables<X>(s_x, p.tw);
  __syncthreads();
  const X xf(s_x, threadIdx.x >> 5);
  const ColId<X> id(p.nitems);   // the items in the place of batch elements
  if (id.none) return;
  const cplx<R>* y = p.rec + (size_t)p.items[id.b] * VEC + (size_t)(id.ch * K + id.ky) * M;
  cplx<R> x[X::E];
#pragma unroll
  for (int i = 0; i < X::E; ++i) {
    x[i] = mk<R>(0, 0);
    if (X::none(i)) continue;
    const int slot = xf.slot(i);
    if (slot >= 0) x[i] = y[slot];
  }
  col_inverse_uv(x, p.G, id.b, id.ch, id.ky, id.act, xf, TableRow<X, false>(nullptr, mu_row<X>(p.tw, id.ky)));
}

// Physical fields of each item: Phys[it][x][2][N] (see phys_row; B_x, B_y include b0).
template <typename R>
struct RowPhysParams {
  const cplx<R>* G;   // [nitems][NG][K][N]
  R* phys;            // [nitems][N][NPH][N]
  const cplx<R>* tw;
  R b0x, b0y;
  int nitems;
};

template <typename R, int N, int XT>
__global__ void __launch_bounds__(XT * Xf<R, N>::L) k_row_phys(RowPhysParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, L = X::L, K = X::K;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_x = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_G = s_x + X::smem(XT / X::G);
  const int tiles = N / XT;
  const int it = blockIdx.x / tiles, x0 = (blockIdx.x - it * tiles) * XT;
  load_tables<X>(s_x, p.tw);
  load_tile<R, N, XT>(s_G, p.G + (size_t)it * NG * K * N, NG * K, x0);
  __syncthreads();
  const X xf(s_x, threadIdx.x >> 5);
  const int w = threadIdx.x / L;
  cplx<R>* ph = const_cast<cplx<R>*>(phys_row<R, N>(p.phys + (size_t)it * N * NPH * N, x0 + w)) + xf.l;
  cplx<R> uv[E], bb[E];
  row_inverse<XT>(s_G, w, xf, uv, bb);
#pragma unroll
  for (int j = 0; j < E; ++j) {
    ph[L * j] = uv[j];
    ph[N + L * j] = mk<R>(bb[j].x + p.b0x, bb[j].y + p.b0y);   // B carries the mean field (mhd_jax.py:145-149)
  }
}

// ---------------------------------------------------------------------------
// Tangent row pass: linearised products around the primal physical fields.
// ---------------------------------------------------------------------------
template <typename R>
struct RowTanParams {
  const cplx<R>* G;     // tangent [B][NG][K][N]
  cplx<R>* H;           // tangent [B][NH][K][N]
  const R* phys;        // primal physical fields of this stage: phys + b * phys_bstride is [N][NPH][N]
  long phys_bstride;    // 0: one primal shared by the batch
  const cplx<R>* tw;
  const StepCtl* ctl;   // optional per-candidate control: batch elements whose ctl.done is set are skipped
  int B;
};

// The linearised products of one row in physical space: (dP1, dP2) and dP3.
template <typename R>
__device__ __forceinline__ cplx<R> tan_p12(cplx<R> d, cplx<R> db, cplx<R> uv, cplx<R> bb) {
  return mk<R>(R(2) * (fpm(uv.x, d.x, uv.y, d.y) - fpm(bb.x, db.x, bb.y, db.y)),
               fpp(bb.x, db.y, bb.y, db.x) - fpp(uv.x, d.y, uv.y, d.x));
}
template <typename R>
__device__ __forceinline__ R tan_p3(cplx<R> d, cplx<R> db, cplx<R> uv, cplx<R> bb) {
  return fpp(uv.x, db.y, bb.y, d.x) - fpp(uv.y, db.x, bb.x, d.y);
}

// Rows x0 .. x0 + XT - 1 of tangent b, one group per row; s_G and s_H are the tile
// buffers (NG and NH rows of K x (XT + 1), the same memory allowed: see row_rhs_body).
// CX (cluster-resident passes): s_G already holds the tile (written
// by the column pass) unless load_g, and the H tile goes to the column groups'
// rows at `hcols` (scatter_h_tile) unless that is null (global H).
template <int XT, bool CX = false, class X>
__device__ __forceinline__ void row_tan_body(const RowTanParams<typename X::R>& p, int b, int x0, const X& xf,
                                             cplx<typename X::R>* s_G, cplx<typename X::R>* s_H, bool load_g = true,
                                             cplx<typename X::R>* hcols = nullptr) {
  using R = typename X::R;
  constexpr int E = X::E, L = X::L, K = X::K, N = X::N;
  const int w = threadIdx.x / L;
  // primal (u, v), (B_x, B_y) of this row, loaded first so that the loads overlap
  // the tile load and the inverse transforms where a lane holds four values or fewer;
  // else they would hold 4 E registers across the transform, and are loaded after it
  constexpr bool EARLY = E <= 4;
  const cplx<R>* ph = phys_row<R, N>(p.phys + (size_t)b * p.phys_bstride, x0 + w) + xf.l;
  cplx<R> puv[E], pbb[E];
  auto load_phys = [&]() {
#pragma unroll
    for (int j = 0; j < E; ++j) { puv[j] = ph[L * j]; pbb[j] = ph[N + L * j]; }
  };
  if constexpr (EARLY) load_phys();
  if (!CX || load_g) load_tile<R, N, XT>(s_G, p.G + (size_t)b * NG * K * N, NG * K, x0);
  __syncthreads();
  cplx<R> duv[E], dbb[E];
  row_inverse<XT>(s_G, w, xf, duv, dbb);
  if constexpr (!EARLY) load_phys();
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const cplx<R> d = duv[j], db = dbb[j];
    duv[j] = tan_p12<R>(d, db, puv[j], pbb[j]);
    dbb[j] = mk<R>(tan_p3<R>(d, db, puv[j], pbb[j]), R(0));
  }
  row_forward<XT>(duv, dbb, s_H, w, xf);
  __syncthreads();
  if constexpr (CX) {
    if (hcols) { scatter_h_tile<XT>(s_H, hcols, x0, xf); return; }
  }
  store_tile<R, N, XT>(p.H + (size_t)b * NH * K * N, s_H, NH * K, x0);
}

template <typename R, int N, int XT>
__global__ void __launch_bounds__(XT * Xf<R, N>::L) k_row_tan(RowTanParams<R> p) {
  using X = Xf<R, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_x = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_G = s_x + X::smem(XT / X::G);
  const int tiles = N / XT;
  const int b = blockIdx.x / tiles, x0 = (blockIdx.x - b * tiles) * XT;
  load_tables<X>(s_x, p.tw);
  pdl_wait();
  pdl_trigger();
  if (p.ctl && p.ctl[b].done) return;   // the whole CTA belongs to batch element b
  row_tan_body<XT>(p, b, x0, X(s_x, threadIdx.x >> 5), s_G, s_G);
}

// ---------------------------------------------------------------------------
// Tangent column pass: forward transform of the linearised products and the
// tangent of the stepper algebra.
// ---------------------------------------------------------------------------
enum TanStage : int {
  TS_START = 0,                  // inverse transforms of the tangent state (dF / dX0)
  T4_S1 = 1, T4_S2, T4_S3, T4_S4,   // Lawson-RK4 stages
  T43_INIT = 10, T43_A, T43_B, T43_C, T43_D, T43_E,   // Lawson-RK4(3) stages
  T43_START = 16,                // inverse transforms of dX0 (before T43_INIT)
  T43_EA = 17,                   // T43_E of an attempt, then T43_A of the next (accepted) attempt, one launch
};
// Tangent slots (Lawson-RK4 uses the first three).
enum TanSlot { D_F = 0, D_A1, D_K2, D_NS4 = 3 };

template <typename R>
struct ColTanParams {
  const cplx<R>* H;     // [B][NH][K][N]
  cplx<R>* G;           // [B][NG][K][N]
  cplx<R>* D;           // tangent slots [B][nslot][2][K][M]
  int nslot;
  const cplx<R>* rec;   // primal record of this step/attempt
  const double* dT;     // [B]
  double t, h;          // Lawson-RK4: t unused; Lawson-RK4(3): t = T, h = attempt step
  double dscale;        // Lawson-RK4: dh = dT * dscale; Lawson-RK4(3): dt = dT * dscale
  const cplx<R>* tw;
  R nu, eta;
  int B, stage, produce;
  // Several candidates, one tangent each (ecs_jvp_multi; Lawson-RK4 stages):
  // ctl[b] gives candidate b's step size h and done flag (skipped once done),
  // rec + b * rec_bstride its record, dscale_b[b] its dT scale, and
  // etab + b * 2 K M its factor exp(h/2 L) mask.  All null/0 for one candidate.
  const StepCtl* ctl;
  long rec_bstride;
  const double* dscale_b;
  const R* etab;
  const cplx<R>* rec2;  // T43_EA: the next attempt's record (h is the next attempt's step)
};

// Record vectors (bits of Rk4Rec / Rk43Rec; tan_qmask2: of the next attempt, from
// rec2) and tangent slots (bits of TanSlot / Rk43Slot) that the algebra of a stage
// reads; they are loaded together before the stage's stores.
__host__ __device__ constexpr unsigned tan_qmask(int stage) {
  return stage == T4_S1 ? (1u << Q_F) | (1u << Q_K1)
       : stage == T4_S2 ? (1u << Q_K2)
       : stage == T4_S3 ? (1u << Q_F) | (1u << Q_K1) | (1u << Q_K2) | (1u << Q_K3)
       : stage == T4_S4 ? (1u << Q_K4)
       : stage == T43_INIT ? (1u << RR_K1)
       : stage == T43_A ? (1u << RR_X0) | (1u << RR_K1) | (1u << RR_E)
       : stage == T43_B ? (1u << RR_K2)
       : stage == T43_C ? (1u << RR_X0) | (1u << RR_K1) | (1u << RR_K2) | (1u << RR_K3) | (1u << RR_E)
       : stage == T43_D ? (1u << RR_K4)
       : stage == T43_E || stage == T43_EA ? (1u << RR_K5) : 0u;
}
__host__ __device__ constexpr unsigned tan_qmask2(int stage) {
  return stage == T43_EA ? (1u << RR_X0) | (1u << RR_K1) | (1u << RR_E) : 0u;
}
__host__ __device__ constexpr unsigned tan_dmask(int stage) {
  return stage == TS_START || stage == T4_S1 || stage == T4_S2 || stage == T4_S4 ? (1u << D_F)
       : stage == T4_S3 ? (1u << D_F) | (1u << D_A1) | (1u << D_K2)
       : stage == T43_START ? (1u << S_X0)
       : stage == T43_A ? (1u << S_X0) | (1u << S_K1)
       : stage == T43_B ? (1u << S_XE)
       : stage == T43_C ? (1u << S_XE) | (1u << S_K1E) | (1u << S_K2)
       : stage == T43_D ? (1u << S_K1) | (1u << S_K2) | (1u << S_K3) | (1u << S_X2)
       : stage == T43_E || stage == T43_EA ? (1u << S_XF) : 0u;
}

__host__ __device__ constexpr int tan_rows(int stage) {
  return popc_c(tan_dmask(stage)) + popc_c(tan_qmask(stage)) + popc_c(tan_qmask2(stage));
}

// What the algebra of a tangent stage needs beside its operands.
template <typename R>
struct TanCol {
  R h, t, dpar, dpar_h, dpar_t;   // dpar: dh (Lawson-RK4) or dt (Lawson-RK4(3))
  const R* etab;                  // the column's factors exp(h/2 L) mask, or null
  __device__ __forceinline__ TanCol(const ColTanParams<R>& p, int b, size_t at) {
    h = p.ctl ? (R)p.ctl[b].h : (R)p.h; t = (R)p.t;
    dpar = (R)(p.dT[b] * (p.dscale_b ? p.dscale_b[b] : p.dscale));
    dpar_h = dpar / h; dpar_t = dpar / t;
    etab = p.etab ? p.etab + at : nullptr;
  }
};
__host__ __device__ constexpr bool tan_has_rhs(int stage) { return !(stage == TS_START || stage == T43_A || stage == T43_START); }
__host__ __device__ constexpr bool tan_has_input(int stage) { return !(stage == T43_INIT || stage == T43_E); }

// The algebra of a tangent stage at one mode: the stage input from the derivative dv
// (the tangent has no forcing).  QV(q), Q2V(q) read rows of the primal record (and of
// the next attempt's), DV(d) reads and DW(d, v) writes tangent slot d.
template <int STAGE, typename R, class QVf, class Q2Vf, class DVf, class DWf>
__device__ __forceinline__ cplx<R> tan_algebra(const TanCol<R>& c, R L, bool in_mask, cplx<R> dv, int slot, QVf&& QV,
                                               Q2Vf&& Q2V, DVf&& DV, DWf&& DW) {
  const R h = c.h, t = c.t, dpar = c.dpar, dpar_h = c.dpar_h, dpar_t = c.dpar_t;
  const R* etab = c.etab;
  constexpr bool rk43 = STAGE >= T43_INIT;
  cplx<R> xin = mk<R>(0, 0);
  if (!rk43) {
    // Lawson-RK4: e = exp(h/2 L) mask, de = e L dh/2; dk = dh v + h dv with v = k/h
    const R ex = etab ? __ldg(etab + slot) : in_mask ? exp(h / R(2) * L) : R(0);
    const R de = ex * L * (dpar / R(2));
    auto dk_of = [&](int q) { return lin2_rn(QV(q), dpar_h, dv, h); };
    switch (STAGE) {
      case TS_START: xin = DV(D_F); break;
      case T4_S1: {
        const cplx<R> dk1 = dk_of(Q_K1);
        const cplx<R> df1 = lin2_rn(QV(Q_F), de, DV(D_F), ex);
        const cplx<R> da1 = lin2_rn(QV(Q_K1), de, dk1, ex);
        DW(D_F, df1); DW(D_A1, da1);
        xin = cadd(df1, cscale(da1, R(0.5)));
      } break;
      case T4_S2: {
        const cplx<R> dk2 = dk_of(Q_K2);
        DW(D_K2, dk2);
        xin = cadd(DV(D_F), cscale(dk2, R(0.5)));
      } break;
      case T4_S3: {
        const cplx<R> dk3 = dk_of(Q_K3);
        const cplx<R> f1 = cscale_rn(QV(Q_F), ex), a1 = cscale_rn(QV(Q_K1), ex);
        const cplx<R> df2 = lin2_rn(f1, de, DV(D_F), ex);
        const cplx<R> db1 = lin2_rn(a1, de, DV(D_A1), ex);
        const cplx<R> db2 = lin2_rn(QV(Q_K2), de, DV(D_K2), ex);
        const cplx<R> db3 = lin2_rn(QV(Q_K3), de, dk3, ex);
        xin = cadd(df2, db3);
        DW(D_F, cadd(cadd(cadd(df2, cdiv_k<6>(db1)), cdiv_k<3>(db2)), cdiv_k<3>(db3)));
      } break;
      default: {   // T4_S4
        const cplx<R> dk4 = dk_of(Q_K4);
        xin = cadd(DV(D_F), cdiv_k<6>(dk4));
        DW(D_F, xin);
      } break;
    }
  } else {
    // Lawson-RK4(3): e = exp(t L h/2), de = e L h/2 dt; dk = dt v + t dv with v = k/t;
    // (e, e L h/2) of this attempt from the primal record (stages A and C use them)
    const cplx<R> eg = (STAGE == T43_A || STAGE == T43_C) ? QV(RR_E) : mk<R>(0, 0);
    [[maybe_unused]] const R ex = eg.x;
    [[maybe_unused]] const R de = eg.y * dpar;
    auto dk_of = [&](int q) { return lin2_rn(QV(q), dpar_t, dv, t); };
    // the A and E algebra, written with explicitly rounded operations: the
    // merged pass T43_EA computes exactly what T43_E followed by T43_A does
    auto stage_e = [&]() { return lin2_rn(QV(RR_K5), dpar_t, dv, t); };   // dk5
    auto stage_a = [&](cplx<R> x0, cplx<R> k1, cplx<R> eg_, cplx<R> dx0, cplx<R> dk1, R h_) {
      const R e_ = eg_.x, de_ = mul_rn(eg_.y, dpar);
      const cplx<R> dxe = lin2_rn(x0, de_, dx0, e_), dk1e = lin2_rn(k1, de_, dk1, e_);
      DW(S_XE, dxe); DW(S_K1E, dk1e);
      cplx<R> half = cscale(dk1e, h_);
      half.x = mul_rn(half.x, R(0.5)); half.y = mul_rn(half.y, R(0.5));
      return mk<R>(add_rn(dxe.x, half.x), add_rn(dxe.y, half.y));
    };
    switch (STAGE) {
      case T43_START: xin = DV(S_X0); break;
      case T43_INIT: DW(S_K1, dk_of(RR_K1)); break;
      case T43_A: xin = stage_a(QV(RR_X0), QV(RR_K1), eg, DV(S_X0), DV(S_K1), h); break;
      case T43_B: {
        const cplx<R> dk2 = dk_of(RR_K2);
        DW(S_K2, dk2);
        xin = cadd(DV(S_XE), cscale(cscale(dk2, h), R(0.5)));
      } break;
      case T43_C: {
        const cplx<R> dk3 = dk_of(RR_K3);
        const cplx<R> xe = cscale_rn(QV(RR_X0), ex), k1e = cscale_rn(QV(RR_K1), ex);
        const cplx<R> dx2 = lin2_rn(xe, de, DV(S_XE), ex);
        const cplx<R> dk1ee = lin2_rn(k1e, de, DV(S_K1E), ex);
        const cplx<R> dk2e = lin2_rn(QV(RR_K2), de, DV(S_K2), ex);
        const cplx<R> dk3e = lin2_rn(QV(RR_K3), de, dk3, ex);
        DW(S_X2, dx2); DW(S_K1, dk1ee); DW(S_K2, dk2e); DW(S_K3, dk3e);
        xin = cadd_scaled_rn(dx2, dk3e, h);
      } break;
      case T43_D: {
        const cplx<R> dk4 = dk_of(RR_K4);
        const cplx<R> acc = cadd(cadd(cadd(cdiv_k<6>(DV(S_K1)), cdiv_k<3>(DV(S_K2))),
                                      cdiv_k<3>(DV(S_K3))), cdiv_k<6>(dk4));
        xin = cadd_scaled_rn(DV(S_X2), acc, h);
        DW(S_XF, xin);
      } break;
      case T43_E: {   // accepted attempt, promote (dxf, dk5) -> (dx0, dk1)
        DW(S_K1, stage_e());
        DW(S_X0, DV(S_XF));
      } break;
      default: {      // T43_EA: T43_E, then T43_A of the next attempt on the promoted values
        const cplx<R> dk1 = stage_e(), dx0 = DV(S_XF);
        DW(S_K1, dk1);
        DW(S_X0, dx0);
        xin = stage_a(Q2V(RR_X0), Q2V(RR_K1), Q2V(RR_E), dx0, dk1, h);
      } break;
    }
  }
  return xin;
}

// A tangent column stage of one column; `rows`: shared room for its operands.
template <int STAGE, class X>
__device__ __forceinline__ void col_tan_body(const ColTanParams<typename X::R>& p, const ColId<X>& id, const X& xf,
                                             cplx<typename X::R>* rows) {
  using R = typename X::R;
  constexpr int E = X::E, K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  const int ch = id.ch, b = id.b, ky = id.ky;
  const bool act = id.act && !(p.ctl && p.ctl[b].done);
  if (!__any_sync(0xffffffffu, act)) return;
  const size_t row = ((size_t)ch * K + ky) * M;
  cplx<R>* D = p.D + (size_t)b * p.nslot * VEC + row;
  const cplx<R>* Q = p.rec + (size_t)b * p.rec_bstride + row;
  const cplx<R>* Q2 = p.rec2 + row;
  const TanCol<R> c(p, b, (size_t)b * VEC + row);
  constexpr unsigned DM = tan_dmask(STAGE), QM = tan_qmask(STAGE), QM2 = tan_qmask2(STAGE);
  // Group layout: the operands of half of the lane's elements at a time; up to two slots
  // whole and before the transform (more would not fit into the registers beside it).
  constexpr int EH = X::STAGED ? E : (E + 1) / 2;
  constexpr bool EARLY = X::GROUP && popc_c(DM) <= 2;
  Operands<X, DM, EARLY ? E : EH> d(rows);
  Operands<X, QM, EH> q(rows + popc_c(DM) * M);
  Operands<X, QM2, EH> q2(rows + (popc_c(DM) + popc_c(QM)) * M);
  d.begin(D, VEC); q.begin(Q, VEC); q2.begin(Q2, VEC);
  constexpr int n = tan_rows(STAGE);
  const TableRow<X, rows_fit(n, 1)> mu(rows + n * M, mu_row<X>(p.tw, ky));
  if constexpr (EARLY) d.load(D, VEC, act, xf);
  cplx<R> r[E], x[E];
  if (tan_has_rhs(STAGE)) col_load_rhs(p.H, b, ch, ky, xf, r);
  const R coeff = ch == 0 ? p.nu : p.eta;
#pragma unroll
  for (int i0 = 0; i0 < E; i0 += EH) {
    if constexpr (!EARLY) d.load(D, VEC, act, xf, i0);
    q.load(Q, VEC, act, xf, i0);
    q2.load(Q2, VEC, act, xf, i0);
#pragma unroll
    for (int i = i0; i < i0 + EH && i < E; ++i) {
      x[i] = mk<R>(0, 0);
      if (X::none(i)) continue;
      const int slot = act ? xf.slot(i) : -1;
      if (slot < 0) continue;
      x[i] = tan_algebra<STAGE>(c, diss_L<R>(xf.kx(i), (R)ky, coeff), !(slot == 0 && ky == 0),
                                tan_has_rhs(STAGE) ? r[i] : mk<R>(0, 0), slot,
                                [&](int a) { return q.get(a, i, slot); }, [&](int a) { return q2.get(a, i, slot); },
                                [&](int a) { return d.get(a, i, slot); },
                                [&](int a, cplx<R> v) { D[a * VEC + slot] = v; });
    }
  }
  if (p.produce && tan_has_input(STAGE)) col_inverse_uv(x, p.G, b, ch, ky, act, xf, mu);
}

template <typename R, int N, int STAGE, bool GRP = false>
__global__ void __launch_bounds__(COLWARPS * 32, GRP ? 3 : 1) k_col_tan(ColTanParams<R> p) {
  using X = Xf<R, N, GRP>;
  ECS_COL_PROLOGUE(tan_rows(STAGE), 1);   // the multipliers
  col_tan_body<STAGE>(p, id, xf, rows);
}

// Rejected Lawson-RK4(3) attempt: the carried k1 becomes e^2 k1 (timestepping.py:267,275,297);
// its tangent is d(e (e k1)) with e' = e L h/2 dt ((e, e L h/2) from the attempt's record).
// The carried dk1 at entry o after a rejected attempt (record rec), dpar = dT * dscale.
template <typename R>
__device__ __forceinline__ cplx<R> tan_reject_k1(const cplx<R>* rec, size_t VEC, size_t o, R dpar, cplx<R> dk1) {
  const cplx<R> eg = rec[RR_E * VEC + o];   // (e, e L h/2) of the attempt
  const R e = eg.x;
  const R de = eg.y * dpar;
  const cplx<R> k1 = rec[RR_K1 * VEC + o];
  const cplx<R> k1e = cscale_rn(k1, e);
  const cplx<R> dk1e = lin2_rn(k1, de, dk1, e);
  return lin2_rn(k1e, de, dk1e, e);
}
// Entry o of tangent Db (slots of one tangent).
template <typename R>
__device__ __forceinline__ void tan_reject_at(cplx<R>* Db, const cplx<R>* rec, size_t VEC, size_t o, R dpar) {
  Db[S_K1 * VEC + o] = tan_reject_k1<R>(rec, VEC, o, dpar, Db[S_K1 * VEC + o]);
}

template <typename R>
__global__ void k_tan_reject(cplx<R>* D, int nslot, const cplx<R>* rec, const double* dT, double dscale, int n,
                             int B) {
  const Geom g = make_geom(n);
  const size_t VEC = (size_t)2 * g.K * g.M;
  const long total = (long)B * VEC;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int b = (int)(i / VEC);
    const size_t o = i - (size_t)b * VEC;
    tan_reject_at<R>(D + (size_t)b * nslot * VEC, rec, VEC, o, (R)(dT[b] * dscale));
  }
}

// W[b] = dPhi[b] + i kx dsx[b] Phi (the tangent of shift_x before the symmetry
// action, symmetry.py:4-5; kx masked).
template <typename R>
__global__ void k_tan_shift(const cplx<R>* dphi, long dstride, const cplx<R>* phi, const double* dsx, cplx<R>* W,
                            int n, int B) {
  const Geom g = make_geom(n);
  const size_t VEC = (size_t)2 * g.K * g.M;
  const long total = (long)B * VEC;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int b = (int)(i / VEC);
    const size_t o = i - (size_t)b * VEC;
    const int slot = o % g.M; const int ky = (o / g.M) % g.K;
    const int kx = slot_to_kx(slot, g.kmax, g.M);
    const R kxm = (kx == 0 && ky == 0) ? R(0) : (R)kx;
    W[i] = cadd(dphi[(size_t)b * dstride + o], cimul(cscale(phi[o], (R)dsx[b]), kxm));
  }
}

// Sums over the CTAs of a cluster of two partial sums per thread, in a fixed order: valid
// in thread 0 of its first CTA.
constexpr int SUM_CL = 8;
__device__ __forceinline__ void cluster_sum2(double& a, double& b) {
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  __shared__ double s1[32], s2[32], all[2][SUM_CL];
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) { a += __shfl_xor_sync(0xffffffffu, a, o); b += __shfl_xor_sync(0xffffffffu, b, o); }
  if ((threadIdx.x & 31) == 0) { s1[threadIdx.x >> 5] = a; s2[threadIdx.x >> 5] = b; }
  cl.sync();   // (also: every CTA has started before a peer writes its shared memory)
  if (threadIdx.x == 0) {
    a = b = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { a += s1[w]; b += s2[w]; }
    const unsigned r = cl.block_rank();
    *cl.map_shared_rank(&all[0][r], 0) = a;
    *cl.map_shared_rank(&all[1][r], 0) = b;
  }
  cl.sync();
  if (cl.block_rank() == 0 && threadIdx.x == 0) {
    a = b = 0.0;
    for (int r = 0; r < SUM_CL; ++r) { a += all[0][r]; b += all[1][r]; }
  }
}

// Tangents of the phase conditions: dpt = mean(vt * du0), dpx = mean(vx * du0)
// over 2 n^2 entries (loss_functions.py:124-125); one cluster of SUM_CL CTAs per tangent
// (at n = 128 one CTA took 55 us, a cluster takes 9.6).
template <typename R>
__global__ void __cluster_dims__(SUM_CL, 1, 1) k_phase_dot(const R* vt, const R* vx, const R* du, double* dpt, double* dpx,
                                                          int n) {
  const int b = blockIdx.x / SUM_CL, r = blockIdx.x % SUM_CL;
  const long cnt = 2L * n * n;
  const R* d = du + (size_t)b * cnt;
  double st = 0.0, sx = 0.0;
  for (long i = r * (long)blockDim.x + threadIdx.x; i < cnt; i += (long)SUM_CL * blockDim.x) {
    st += (double)vt[i] * d[i];
    sx += (double)vx[i] * d[i];
  }
  cluster_sum2(st, sx);
  if (r == 0 && threadIdx.x == 0) { dpt[b] = st / (double)cnt; dpx[b] = sx / (double)cnt; }
}

}  // namespace ecs
