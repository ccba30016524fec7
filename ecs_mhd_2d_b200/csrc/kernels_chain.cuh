// Cluster-resident tangent sweep of the adaptive Lawson-RK4(3) linearisation:
// one launch runs a whole list of tangent passes (the column stages, the row
// passes between them and the elementwise updates of rejected attempts) that
// the launch-per-pass sweep (k_col_tan / k_row_tan / k_tan_reject) issues one
// kernel each, for the same batch of tangents at a fixed linearisation
// (reference: jax.jvp of objective_RPO, jax_scripts/lib/utils.py:108, through
// the adaptive stepper of jax_scripts/lib/timestepping.py:151-335).
//
// One thread-block cluster of CL = N / W CTAs of W warps serves one tangent
// (W = 16: 8 CTAs at n = 128, a portable cluster; W = 8: 16 CTAs, half the
// warps per SM and no register cap below 255):
//   * a column pass gives each warp a fixed column (ky, channel) of the box --
//     column c of tangent b on warp c / CL of CTA c % CL -- and runs the same
//     transforms and the same algebra per mode as k_col_tan (tan_algebra), so the
//     arithmetic and the rounding are those of the launch-per-pass sweep;
//   * a row pass gives CTA r the W physical rows W r .. W r + W - 1, one warp
//     per row, and runs k_row_tan's body (row_tan_body) with W-row tiles;
//   * a rejected attempt updates the tangent's carried k1 column by column on
//     the same warps as the column passes (tan_reject_k1).
// Consecutive passes of the same kind (column stages and rejects) touch only
// the warp's own box rows, so they follow each other without a barrier (a
// __syncwarp orders the lanes' writes before the next pass's reads).
// Between a column pass and a row pass the cluster synchronises with the
// hardware cluster barrier (arrive.release / wait.acquire), whose
// release/acquire makes one pass's writes visible to the next pass's readers on
// the other SMs of the cluster.  The barrier is a hardware barrier over CTAs
// that are co-scheduled by construction (a cluster), so no wait in this kernel
// spins on memory.
//
// What bounds a chain is the length of one warp's path through a pass, and on that
// path the instruction fetch: a pass is a straight line that every warp runs once, so
// code that does not stay in the instruction caches comes from L2.  A column pass
// therefore has ONE copy of its transforms for all stages, and only the algebra of the
// stage is selected at run time; the operands of the algebra are in shared memory, or
// on their way there before the forward transform starts.  Measured (one copy of the
// column body per stage and operands staged per pass -> this): 256 Lawson-RK4 steps of one
// state at n = 128 7.88 -> 6.84 ms, 1024 steps of 8 states at n = 64 16.1 -> 14.7 ms, an
// adaptive solve of T = 0.5 at n = 128 5.1 -> 4.3 ms.
//
// The intermediate arrays between the passes travel one of two ways (template
// flag DSM):
//   * DSM = false: through global memory (G, H; L2-resident at these sizes);
//   * DSM = true: through distributed shared memory -- a column pass writes its
//     inverse transforms straight into the G tiles of the CTAs that own those
//     physical rows (col_to_tiles), and a row pass sends its H tile to the
//     shared rows of the warps that transform those columns (scatter_h_tile),
//     so neither array leaves the cluster.  The first pass of a launch reads and
//     the last one writes global G / H, which carries the state from one launch
//     to the next (a launch ends before a row pass, at a regeneration chunk).
// With DSH (8-warp CTAs only, for shared-memory room) each column warp keeps its
// column's state slots in shared memory for the whole launch: loaded at the start,
// written back at the end.
//
// The same layout runs the primal: k_rk4_chain (fixed-step Lawson-RK4 steps)
// and k_rk43_chain (adaptive attempts with the error norm and the accept/reject
// decision in the kernel), below.
#pragma once

#include <utility>

#include "kernels_fx.cuh"
#include "kernels_tan.cuh"

namespace ecs {

enum ChainKind : int { CH_COL = 0, CH_ROW = 1, CH_REJECT = 2 };

// One pass of the sweep.  Record offsets are in box vectors from the record
// base; `item` indexes the physical fields of the launch's regeneration chunk.
struct ChainOp {
  int kind, stage, produce, pad;
  long rec, rec2;
  long item;
  double h;
};

// W warps per CTA = physical rows per CTA in a row pass; CL = N / W CTAs per cluster.
template <int N, int W> __host__ __device__ constexpr int chain_cl() { return N / W; }
// Warps per CTA that own columns in the column passes (2 K columns over CL CTAs).
template <int N, int W> __host__ __device__ constexpr int chain_colwarps() {
  return (2 * ((N - 1) / 3 + 1) + chain_cl<N, W>() - 1) / chain_cl<N, W>();
}
// Shared-memory regions of a chain kernel (offsets in complex entries): tables; with DSM
// the G tile and the column warps' H rows; a work area that the row tile (without DSM)
// and the column warps' staged operand rows (STG rows of M each) take in turn; SLOTS
// resident rows of M per column warp.
template <typename R, int N, int W, bool DSM, int STG, int SLOTS> struct ChainSmem {
  using X = Xf<R, N>;
  static constexpr int K = X::K, M = X::M, CW = chain_colwarps<N, W>();
  static constexpr int gt = X::smem(W);
  static constexpr int hc = gt + (DSM ? NG * K * (W + 1) : 0);
  static constexpr int work = hc + (DSM ? CW * 2 * N : 0);
  static constexpr int row = DSM ? 0 : NG * K * (W + 1);
  static constexpr int ds = work + (CW * STG * M > row ? CW * STG * M : row);
  static constexpr size_t bytes = (size_t)(ds + CW * SLOTS * M) * sizeof(cplx<R>);
};
// Staged rows: of the tangent sweep the record rows a stage reads (5, stage C) and,
// unless the slots are resident, its slots (8 together); of an attempt of the primal
// its slots (4), unless resident.  Lawson-RK4 steps keep F, A1, K2 and the real e.
// Resident beside them: the column's multipliers, and of the primal its forcing.
template <typename R, int N, int W, bool DSM, bool DSH>
using TanChainSmem = ChainSmem<R, N, W, DSM, DSH ? 5 : 8, (DSH ? S_NSLOT : 0) + 1>;
template <typename R, int N, int W, bool DSM> using Rk4ChainSmem = ChainSmem<R, N, W, DSM, 0, 6>;
template <typename R, int N, int W>
using Rk43ChainSmem = ChainSmem<R, N, W, true, W == 8 ? 0 : 4, (W == 8 ? S_NSLOT : 0) + 2>;

template <typename R>
struct ChainParams {
  ColTanParams<R> col;   // H, G, D, nslot, dT, t, dscale, tw, nu, eta, B of every column pass
  RowTanParams<R> row;   // G, H, tw of every row pass
  const cplx<R>* rec;    // record base
  const R* phys;         // [item - item0][N][NPH][N]: the regeneration chunk
  long item0;            // first item of the chunk
  const ChainOp* ops;
  int op0, op1;
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;\n" ::: "memory");
}

// The column that the calling warp owns in its state's column passes, or -1: warp w of
// CTA `rank` owns column w CL + rank (channel its lowest bit).
template <int N, int W> __device__ __forceinline__ int chain_column(int rank) {
  const int w = (int)(threadIdx.x >> 5), c = w * chain_cl<N, W>() + rank;
  return w < chain_colwarps<N, W>() && c < 2 * ((N - 1) / 3 + 1) ? c : -1;
}

// Rows `mask` of a column (row q at from + q pitch, M entries) on their way to
// consecutive shared rows at `to`; returns the place after them.
template <typename R, int M>
__device__ __forceinline__ cplx<R>* stage_rows(cplx<R>* to, const cplx<R>* from, size_t pitch, unsigned mask) {
  for (; mask; mask &= mask - 1) {
    const cplx<R>* q = from + (__ffs((int)mask) - 1) * pitch;
    for (int s = threadIdx.x & 31; s < M; s += 32) cp_async_c<R>(to + s, q + s);
    to += M;
  }
  return to;
}
// A resident row of a column's table, as TableRow reads one.
template <typename R> struct SharedRow {
  const cplx<R>* s;
  __device__ __forceinline__ void wait() const {}
  __device__ __forceinline__ cplx<R> operator()(int slot) const { return s[slot]; }
};
__device__ __forceinline__ void staged_wait() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncwarp();
}

// The derivative of a column from its product rows: the warp's shared rows `hrows`, or
// (null) global H; one copy of the transforms.
template <class X>
__device__ __forceinline__ void chain_rhs(const cplx<typename X::R>* H, const ColId<X>& id, const X& xf,
                                          const cplx<typename X::R>* hrows, cplx<typename X::R> (&r)[X::E]) {
  const cplx<typename X::R>* h0 =
      hrows ? hrows : H + ((size_t)(id.b * NH + (id.ch == 0 ? 0 : 2)) * X::K + id.ky) * X::N;
  col_rhs_rows(h0, h0 + (hrows ? (size_t)X::N : (size_t)X::K * X::N), id.ch, id.ky, xf, r);
}

// The stage's algebra on the lane's modes; ops(std::integral_constant of the stage).
template <int STAGE, bool DSH, class X>
__device__ __forceinline__ void chain_tan_algebra(const TanCol<typename X::R>& c, typename X::R coeff, const ColId<X>& id,
                                                  const X& xf, const cplx<typename X::R>* rows, cplx<typename X::R>* D,
                                                  size_t DS, const cplx<typename X::R> (&r)[X::E],
                                                  cplx<typename X::R> (&x)[X::E]) {
  using R = typename X::R;
  constexpr int M = X::M;
  constexpr unsigned DM = tan_dmask(STAGE), QM = tan_qmask(STAGE), QM2 = tan_qmask2(STAGE);
  constexpr int NQ = popc_c(QM), NQ2 = popc_c(QM2);
#pragma unroll
  for (int i = 0; i < X::E; ++i) {
    const int slot = xf.slot(i);
    if (slot < 0) continue;
    x[i] = tan_algebra<STAGE>(c, diss_L<R>(xf.kx(i), (R)id.ky, coeff), !(slot == 0 && id.ky == 0),
                              tan_has_rhs(STAGE) ? r[i] : mk<R>(0, 0), slot,
                              [&](int q) { return rows[bit_rank(QM, q) * M + slot]; },
                              [&](int q) { return rows[(NQ + bit_rank(QM2, q)) * M + slot]; },
                              [&](int d) { return DSH ? D[d * M + slot] : rows[(NQ + NQ2 + bit_rank(DM, d)) * M + slot]; },
                              [&](int d, cplx<R> v) { D[d * DS + slot] = v; });
  }
}

template <int W, bool DSM, bool DSH, class X>
__device__ __forceinline__ void chain_col(const ChainParams<typename X::R>& P, const ChainOp& op, TanCol<typename X::R> c,
                                          const ColId<X>& id, const X& xf, const cplx<typename X::R>* hrows,
                                          cplx<typename X::R>* gtile, cplx<typename X::R>* dsh, cplx<typename X::R>* rows,
                                          const SharedRow<typename X::R>& mu) {
  using R = typename X::R;
  constexpr int K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  const ColTanParams<R>& p = P.col;
  c.h = (R)op.h;   // (the adaptive stages use dpar / t, not dpar / h)
  const size_t at = ((size_t)id.ch * K + id.ky) * M;
  cplx<R>* D = DSH ? dsh : p.D + (size_t)id.b * p.nslot * VEC + at;
  constexpr size_t DS = DSH ? (size_t)M : VEC;
  const cplx<R>* rec = P.rec + (size_t)op.rec * VEC;
  if (op.kind == CH_REJECT) {
    for (int s = xf.l; s < M; s += 32) D[S_K1 * DS + s] = tan_reject_k1<R>(rec, VEC, at + s, c.dpar, D[S_K1 * DS + s]);
    return;
  }
  cplx<R>* to = stage_rows<R, M>(rows, rec + at, VEC, tan_qmask(op.stage));
  to = stage_rows<R, M>(to, P.rec + (size_t)op.rec2 * VEC + at, VEC, tan_qmask2(op.stage));
  if constexpr (!DSH) stage_rows<R, M>(to, D, VEC, tan_dmask(op.stage));
  cplx<R> r[X::E], x[X::E];
#pragma unroll
  for (int i = 0; i < X::E; ++i) r[i] = x[i] = mk<R>(0, 0);
  if (tan_has_rhs(op.stage)) chain_rhs(p.H, id, xf, hrows, r);
  staged_wait();
  const R coeff = id.ch == 0 ? p.nu : p.eta;
  switch (op.stage) {
    case T43_START: chain_tan_algebra<T43_START, DSH>(c, coeff, id, xf, rows, D, DS, r, x); break;
    case T43_INIT: chain_tan_algebra<T43_INIT, DSH>(c, coeff, id, xf, rows, D, DS, r, x); break;
    case T43_A: chain_tan_algebra<T43_A, DSH>(c, coeff, id, xf, rows, D, DS, r, x); break;
    case T43_B: chain_tan_algebra<T43_B, DSH>(c, coeff, id, xf, rows, D, DS, r, x); break;
    case T43_C: chain_tan_algebra<T43_C, DSH>(c, coeff, id, xf, rows, D, DS, r, x); break;
    case T43_D: chain_tan_algebra<T43_D, DSH>(c, coeff, id, xf, rows, D, DS, r, x); break;
    case T43_EA: chain_tan_algebra<T43_EA, DSH>(c, coeff, id, xf, rows, D, DS, r, x); break;
    default: chain_tan_algebra<T43_E, DSH>(c, coeff, id, xf, rows, D, DS, r, x); break;
  }
  if (op.produce && tan_has_input(op.stage))
    col_inverse_uv<DSM ? W : 0>(x, p.G, id.b, id.ch, id.ky, true, xf, mu, gtile);
}

// Grid: B clusters of CL CTAs (cluster b = tangent b; the cluster shape is a
// launch attribute), W * 32 threads each.
template <typename R, int N, int W, bool DSM, bool DSH>
__global__ void __launch_bounds__(W * 32, 1) k_tan_chain(ChainParams<R> P) {
  using X = Xf<R, N>;
  constexpr int K = X::K, M = X::M, CL = chain_cl<N, W>();
  constexpr size_t VEC = (size_t)2 * K * M;
  using SM = TanChainSmem<R, N, W, DSM, DSH>;
  static_assert(DSH || popc_c(tan_qmask(T43_C)) + popc_c(tan_dmask(T43_C)) <= 8, "staged rows");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_base = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_gt = s_base + SM::gt;
  const X xf(s_base, threadIdx.x >> 5);
  const int b = blockIdx.x / CL, rank = blockIdx.x - b * CL;
  const int cw = chain_column<N, W>(rank), wc = cw < 0 ? 0 : (int)(threadIdx.x >> 5);
  const ColId<X> id(cw < 0 ? 0 : cw, b, b + 1);
  cplx<R>* my_h = s_base + SM::hc + (size_t)wc * 2 * N;
  cplx<R>* my_rows = s_base + SM::work + (size_t)wc * (DSH ? 5 : 8) * M;
  cplx<R>* my_mu = s_base + SM::ds + (size_t)wc * ((DSH ? S_NSLOT : 0) + 1) * M;
  cplx<R>* dsh = my_mu + M;
  cplx<R>* dglob = P.col.D + (size_t)b * P.col.nslot * VEC + ((size_t)id.ch * K + id.ky) * M;
  load_tables<X>(s_base, P.col.tw);
  pdl_wait();   // launched with programmatic serialization: the predecessor's writes are visible past here
  if (cw >= 0) {
    for (int e = xf.l; e < M; e += 32) my_mu[e] = mu_row<X>(P.col.tw, id.ky)[e];
    if constexpr (DSH)
      for (int d = 0; d < S_NSLOT; ++d)
        for (int e = xf.l; e < M; e += 32) dsh[d * M + e] = dglob[d * VEC + e];
  }
  const TanCol<R> tc(P.col, b, 0);
  if constexpr (DSM) cluster_barrier();   // every CTA has started before a peer writes its shared memory
  else __syncthreads();
  int prev = -1;   // kind class of the previous pass: 0 column-like, 1 row
  ChainOp next = P.ops[P.op0];
  for (int i = P.op0; i < P.op1; ++i) {
    const ChainOp op = next;
    if (i + 1 < P.op1) next = P.ops[i + 1];   // on its way during this pass
    const int cls = op.kind == CH_ROW ? 1 : 0;
    if (prev >= 0 && (cls != prev || cls == 1)) cluster_barrier();
    else if (prev >= 0) __syncwarp();
    prev = cls;
    const bool first = i == P.op0, last = i == P.op1 - 1;   // global G / H at the launch's ends
    if (cls) {
      RowTanParams<R> rp = P.row;
      rp.phys = P.phys + (size_t)(op.item - P.item0) * N * NPH * N;
      cplx<R>* tile = DSM ? s_gt : s_base + SM::work;
      row_tan_body<W, DSM>(rp, b, rank * W, xf, tile, tile, first, last ? nullptr : s_base + SM::hc);
    } else if (cw >= 0) {
      chain_col<W, DSM, DSH>(P, op, tc, id, xf, (DSM && !first) ? my_h : nullptr, (DSM && !last) ? s_gt : nullptr, dsh, my_rows,
                             SharedRow<R>{my_mu});
    }
  }
  if constexpr (DSH) {   // the slots back to global memory for the next launch and the JVP output
    __syncwarp();
    if (cw >= 0)
      for (int d = 0; d < S_NSLOT; ++d)
        for (int e = xf.l; e < M; e += 32) dglob[d * VEC + e] = dsh[d * M + e];
  }
  if constexpr (DSM) cluster_barrier();   // no CTA leaves while a peer may still write its shared memory
}

// ---------------------------------------------------------------------------
// Lawson-RK4 steps of the primal (timestepping.lawson_rk4,
// jax_scripts/lib/timestepping.py:69-80) in one launch: cluster b advances
// state b through `steps` steps, each stage a row pass (k_row_rhs's body,
// W-row tiles) and a column pass (k_col_rk4's transforms and algebra), with the same
// layout and barriers as k_tan_chain.  The stage input of the first stage is in G (from
// a COL_START column pass before the launch).  Each column warp keeps its column's
// state, A1, K2, e, forcing and multipliers in shared memory; the state goes back to global F at the end.
// ---------------------------------------------------------------------------
template <typename R>
struct Rk4ChainParams {
  ColParams<R> col;   // stage and produce are set per stage
  RowParams<R> row;
  long steps;
  int last_produce;   // inverse transforms after the last stage (the next stage input)
  long rec_step;      // col.rec: entries from a step's record to the next step's
  long phys_step;     // row.phys: values from a stage's record to the next stage's
};

template <int STAGE, class X>
__device__ __forceinline__ void chain_rk4_algebra(const ColParams<typename X::R>& p, const ColId<X>& id, const X& xf,
                                                  const Rk4Rows<typename X::R>& w, typename X::R h,
                                                  const SharedRow<typename X::R>& forcing,
                                                  const cplx<typename X::R> (&r)[X::E], cplx<typename X::R> (&x)[X::E]) {
  using C = cplx<typename X::R>;
  // loaded together: a load of a row cannot move over a store to another
  C f[X::E], a1[X::E], k2[X::E];
  typename X::R e[X::E];
#pragma unroll
  for (int i = 0; i < X::E; ++i) {
    const int slot = xf.slot(i);
    if (slot < 0) continue;
    f[i] = w.F[slot];
    if (STAGE == COL_RK4_S3) { a1[i] = w.A1[slot]; k2[i] = w.K2[slot]; }
    if (rk4_reads_e(STAGE)) e[i] = w.e[slot];
  }
  col_rk4_algebra<STAGE>(p, id, xf, w, h, [&](int q, int i, int) { return q == 0 ? f[i] : q == 1 ? a1[i] : k2[i]; },
                         [&](int i, int) { return e[i]; }, forcing, r, x);
}

template <typename R, int N, int W, bool DSM>
__global__ void __launch_bounds__(W * 32, 1) k_rk4_chain(Rk4ChainParams<R> P) {
  using X = Xf<R, N>;
  constexpr int M = X::M, CL = chain_cl<N, W>();
  using SM = Rk4ChainSmem<R, N, W, DSM>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_base = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_gt = s_base + SM::gt;
  cplx<R>* s_hc = s_base + SM::hc;
  const X xf(s_base, threadIdx.x >> 5);
  const int b = blockIdx.x / CL, rank = blockIdx.x - b * CL;
  const int cw = chain_column<N, W>(rank), wc = cw < 0 ? 0 : (int)(threadIdx.x >> 5);
  const ColId<X> id(cw < 0 ? 0 : cw, b, b + 1);
  const size_t at = ((size_t)(b * 2 + id.ch) * X::K + id.ky) * M;
  cplx<R>* my_s = s_base + SM::ds + (size_t)wc * 6 * M;
  R* my_e = reinterpret_cast<R*>(my_s + 3 * M);
  const SharedRow<R> forcing{my_s + 4 * M}, mu{my_s + 5 * M};
  const Rk4Rows<R> w{my_s, my_s + M, my_s + 2 * M, my_e};
  const cplx<R>* my_h = DSM ? s_hc + (size_t)wc * 2 * N : nullptr;
  load_tables<X>(s_base, P.col.tw);
  pdl_wait();   // launched with programmatic serialization: the predecessor's writes are visible past here
  if (P.col.use_done && P.col.ctl[b].done) return;   // the whole cluster
  if (cw >= 0)
    for (int s = xf.l; s < M; s += 32) {
      my_s[s] = P.col.F[at + s]; my_e[s] = P.col.Etab[at + s];
      my_s[4 * M + s] = P.col.fhat[id.ky * M + s]; my_s[5 * M + s] = mu_row<X>(P.col.tw, id.ky)[s];
    }
  const R h = (R)P.col.ctl[b].h;
  if constexpr (DSM) cluster_barrier();   // every CTA has started before a peer writes its shared memory
  else __syncthreads();
  for (long step = 0; step < P.steps; ++step) {
    ColParams<R> col = P.col;
    if (col.rec) col.rec += step * P.rec_step;
#pragma unroll 1
    for (int st = COL_RK4_S1; st <= COL_RK4_S4; ++st) {
      if (step > 0 || st > COL_RK4_S1) cluster_barrier();   // column pass -> row pass
      const bool first = step == 0 && st == COL_RK4_S1, last = step == P.steps - 1 && st == COL_RK4_S4;
      cplx<R>* tile = DSM ? s_gt : s_base + SM::work;
      RowParams<R> row = P.row;
      if (row.phys) row.phys += (step * 4 + st - COL_RK4_S1) * P.phys_step;
      row_rhs_body<W, DSM>(row, b, rank * W, xf, tile, tile, first, s_hc);
      cluster_barrier();                                     // row pass -> column pass
      if (cw < 0) continue;
      cplx<R> r[X::E], x[X::E];
      chain_rhs(P.col.H, id, xf, my_h, r);
      switch (st) {
        case COL_RK4_S1: chain_rk4_algebra<COL_RK4_S1>(col, id, xf, w, h, forcing, r, x); break;
        case COL_RK4_S2: chain_rk4_algebra<COL_RK4_S2>(col, id, xf, w, h, forcing, r, x); break;
        case COL_RK4_S3: chain_rk4_algebra<COL_RK4_S3>(col, id, xf, w, h, forcing, r, x); break;
        default: chain_rk4_algebra<COL_RK4_S4>(col, id, xf, w, h, forcing, r, x); break;
      }
      if (!last || P.last_produce)
        col_inverse_uv<DSM ? W : 0>(x, P.col.G, b, id.ch, id.ky, true, xf, mu, (DSM && !last) ? s_gt : nullptr);
    }
  }
  __syncwarp();
  if (cw >= 0)
    for (int s = xf.l; s < M; s += 32) P.col.F[at + s] = my_s[s];
  if constexpr (DSM) cluster_barrier();   // no CTA leaves while a peer may still write its shared memory
}

// ---------------------------------------------------------------------------
// Steps of the other fixed-step modes (RK4, Lawson-RK6, TDRK4; kernels_fx.cuh) in one
// launch, with the layout of k_rk4_chain; the slots, e, forcing and multipliers of a
// column stay in shared memory.  The passes are k_row_rhs's (k_row_tan's for TDRK4's
// Jacobian-vector products, on the physical fields that the row's own warp left in
// row.phys the pass before) and k_col_fx's.  The stage input of the first stage is in G.
// Measured, 32 steps, launch per pass -> this: n = 128, batch 1 Lawson-RK6 2.85 -> 1.98 ms,
// RK4 1.38 -> 0.95, TDRK4 1.38 -> 1.00; batch 7 Lawson-RK6 3.36 -> 1.99; n = 64, batch 8
// 1.78 -> 1.11, 0.87 -> 0.56, 0.86 -> 0.58, batch 24 2.69 -> 1.67, 1.26 -> 0.80, 1.20 -> 0.84.
// ---------------------------------------------------------------------------
template <typename R>
struct FxChainParams {
  ColFxParams<R> col;
  RowParams<R> row;   // phys, phys_bstride: TDRK4
  long steps;
  long rec_step;      // col.rec: entries from a step's record to the next step's
};

__host__ __device__ constexpr int fx_nslot(int scheme) { return scheme == FX_RK6 ? 8 : scheme == FX_TD4 ? 5 : 4; }
template <typename R, int N, int W, int SCHEME> using FxChainSmem = ChainSmem<R, N, W, true, 0, fx_nslot(SCHEME) + 3>;

template <int SCHEME, int STAGE, class X>
__device__ __forceinline__ void chain_fx_algebra(typename X::R h, typename X::R coeff, const ColId<X>& id, const X& xf,
                                                 cplx<typename X::R>* S, const typename X::R* e,
                                                 const SharedRow<typename X::R>& forcing, cplx<typename X::R>* rec,
                                                 const cplx<typename X::R> (&r)[X::E], cplx<typename X::R> (&x)[X::E]) {
  using R = typename X::R;
  constexpr int M = X::M;
  constexpr size_t VEC = (size_t)2 * X::K * M;
#pragma unroll
  for (int i = 0; i < X::E; ++i) {
    x[i] = mk<R>(0, 0);
    const int slot = xf.slot(i);
    if (slot < 0) continue;
    cplx<R> v = r[i];
    if (fx_rhs(SCHEME, STAGE) == 1 && id.ch == 0 && !(slot == 0 && id.ky == 0)) v = cadd(v, forcing(slot));
    x[i] = fx_algebra<SCHEME, STAGE, R>(h, diss_L<R>(xf.kx(i), (R)id.ky, coeff), v,
                                        [&](int q) -> cplx<R> { return S[q * M + slot]; },
                                        [&](int q, cplx<R> a) { S[q * M + slot] = a; }, [&]() { return e[slot]; },
                                        [&](int q, cplx<R> a) { if (rec) rec[q * VEC + slot] = a; });
  }
}
template <int SCHEME, class X, int... ST, typename... A>
__device__ __forceinline__ void chain_fx_stage(int st, std::integer_sequence<int, ST...>, A&&... a) {
  ((st == ST + 1 ? chain_fx_algebra<SCHEME, ST + 1, X>(a...) : (void)0), ...);
}

template <typename R, int N, int W, int SCHEME>
__global__ void __launch_bounds__(W * 32, 1) k_fx_chain(FxChainParams<R> P) {
  using X = Xf<R, N>;
  constexpr int M = X::M, CL = chain_cl<N, W>(), NS = fx_nslot(SCHEME);
  constexpr size_t VEC = (size_t)2 * X::K * M;
  using SM = FxChainSmem<R, N, W, SCHEME>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_base = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_gt = s_base + SM::gt;
  cplx<R>* s_hc = s_base + SM::hc;
  const X xf(s_base, threadIdx.x >> 5);
  const int b = blockIdx.x / CL, rank = blockIdx.x - b * CL;
  const int cw = chain_column<N, W>(rank), wc = cw < 0 ? 0 : (int)(threadIdx.x >> 5);
  const ColId<X> id(cw < 0 ? 0 : cw, b, b + 1);
  const size_t at = ((size_t)id.ch * X::K + id.ky) * M;
  cplx<R>* F = P.col.S + (size_t)b * S_NSLOT * VEC + X_F * VEC + at;
  cplx<R>* S = s_base + SM::ds + (size_t)wc * (NS + 3) * M;
  R* e = reinterpret_cast<R*>(S + NS * M);
  const SharedRow<R> forcing{S + (NS + 1) * M}, mu{S + (NS + 2) * M};
  const cplx<R>* my_h = s_hc + (size_t)wc * 2 * N;
  load_tables<X>(s_base, P.col.tw);
  pdl_wait();   // launched with programmatic serialization: the predecessor's writes are visible past here
  if (cw >= 0)
    for (int s = xf.l; s < M; s += 32) {
      S[X_F * M + s] = F[s];
      if (SCHEME == FX_RK6) e[s] = P.col.Etab[(size_t)b * VEC + at + s];
      S[(NS + 1) * M + s] = P.col.fhat[id.ky * M + s];
      S[(NS + 2) * M + s] = mu_row<X>(P.col.tw, id.ky)[s];
    }
  const R h = (R)P.col.ctl[b].h, coeff = id.ch == 0 ? P.col.nu : P.col.eta;
  cluster_barrier();   // every CTA has started before a peer writes its shared memory
  RowTanParams<R> tan{};
  tan.G = P.row.G; tan.H = P.row.H; tan.phys = P.row.phys; tan.phys_bstride = P.row.phys_bstride; tan.tw = P.row.tw;
  for (long step = 0; step < P.steps; ++step) {
    cplx<R>* rec = P.col.rec ? P.col.rec + step * P.rec_step + at : nullptr;
#pragma unroll 1
    for (int st = 1; st <= fx_stages(SCHEME); ++st) {
      if (step > 0 || st > 1) cluster_barrier();   // column pass -> row pass
      const bool first = step == 0 && st == 1, last = step == P.steps - 1 && st == fx_stages(SCHEME);
      if (SCHEME == FX_TD4 && fx_rhs(SCHEME, 2) == 2 && (st & 1) == 0)
        row_tan_body<W, true>(tan, b, rank * W, xf, s_gt, s_gt, false, s_hc);
      else
        row_rhs_body<W, true>(P.row, b, rank * W, xf, s_gt, s_gt, first, s_hc);
      cluster_barrier();                            // row pass -> column pass
      if (cw < 0) continue;
      cplx<R> r[X::E], x[X::E];
      chain_rhs(P.col.H, id, xf, my_h, r);
      chain_fx_stage<SCHEME, X>(st, std::make_integer_sequence<int, fx_stages(SCHEME)>{}, h, coeff, id, xf, S,
                                (const R*)e, forcing, rec, r, x);
      if (!last) col_inverse_uv<W>(x, P.col.G, b, id.ch, id.ky, true, xf, mu, s_gt);
    }
  }
  __syncwarp();
  if (cw >= 0)
    for (int s = xf.l; s < M; s += 32) F[s] = S[X_F * M + s];
  cluster_barrier();   // no CTA leaves while a peer may still write its shared memory
}

// ---------------------------------------------------------------------------
// The adjoint of a run of Lawson-RK4 steps (k_row_adj's and k_col_adj's passes, stages
// AJ_S4 .. AJ_S1 of each step, last step first) in one launch, with the layout of
// k_rk4_chain: cluster b runs cotangent b.  The slots, e and the multipliers of a column
// stay in shared memory, its dL/dh accumulator in a register; the record rows of a stage
// are on their way to shared memory before its transforms.  The first row pass reads
// global G (an AJ_PRE pass, or the launch before), and the last column pass writes it if
// a step precedes.
// Measured, transpose products of 64 steps, launch per pass -> this: n = 64, batch 1
// 1.75 -> 1.37 ms, batch 8 1.94 -> 1.37; n = 128, batch 1 2.40 -> 2.33, batch 7 3.47 -> 2.35.
// ---------------------------------------------------------------------------
template <typename R>
struct AdjChainParams {
  ColAdjParams<R> col;   // rec: of step 0 of the run; h (or ctl), J, nslot, hacc, ...
  RowAdjParams<R> row;   // phys: of stage 1 of step `lo`
  long rec_step;         // entries from a step's record to the next step's
  long phys_step;        // values from a stage's physical fields to the next stage's
  int hi, lo;            // steps hi .. lo, downwards
};
template <typename R, int N, int W> using AdjChainSmem = ChainSmem<R, N, W, true, 4, (int)J_NS4 + 2>;

template <int STAGE, class X>
__device__ __forceinline__ void chain_adj_algebra(typename X::R h, typename X::R coeff, const ColId<X>& id, const X& xf,
                                                  bool prev, double& hpart, double& hdiv, cplx<typename X::R>* J,
                                                  const typename X::R* e, const cplx<typename X::R>* rows,
                                                  const cplx<typename X::R> (&xb)[X::E], cplx<typename X::R> (&lam)[X::E]) {
  using R = typename X::R;
  constexpr int M = X::M;
  constexpr unsigned QM = adj4_qmask(STAGE);
#pragma unroll
  for (int i = 0; i < X::E; ++i) {
    lam[i] = mk<R>(0, 0);
    const int slot = xf.slot(i);
    if (slot < 0) continue;
    const cplx<R> kb = adj_algebra<STAGE, R>(
        h, R(0), diss_L<R>(xf.kx(i), (R)id.ky, coeff), xb[i], prev, hpart, hdiv,
        [&](int q) -> cplx<R> { return J[q * M + slot]; }, [&](int q, cplx<R> v) { J[q * M + slot] = v; },
        [&](int q) -> cplx<R> { return rows[bit_rank(QM, q) * M + slot]; }, [&]() { return e[slot]; },
        [&]() -> cplx<R> { return rows[slot]; });
    lam[i] = cscale(kb, id.ky == 0 ? R(1) : R(0.5));   // kb / c_ky, exactly
  }
}

template <typename R, int N, int W>
__global__ void __launch_bounds__(W * 32, 1) k_adj_chain(AdjChainParams<R> P) {
  using X = Xf<R, N>;
  constexpr int K = X::K, M = X::M, CL = chain_cl<N, W>(), NS = (int)J_NS4;
  constexpr size_t VEC = (size_t)2 * K * M;
  using SM = AdjChainSmem<R, N, W>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_base = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_gt = s_base + SM::gt;
  cplx<R>* s_hc = s_base + SM::hc;
  const X xf(s_base, threadIdx.x >> 5);
  const int b = blockIdx.x / CL, rank = blockIdx.x - b * CL;
  const int cw = chain_column<N, W>(rank), wc = cw < 0 ? 0 : (int)(threadIdx.x >> 5);
  const ColId<X> id(cw < 0 ? 0 : cw, b, b + 1);
  const size_t at = ((size_t)id.ch * K + id.ky) * M;
  cplx<R>* Jg = P.col.J + (size_t)b * P.col.nslot * VEC + at;
  cplx<R>* rows = s_base + SM::work + (size_t)wc * 4 * M;
  cplx<R>* J = s_base + SM::ds + (size_t)wc * (NS + 2) * M;
  R* e = reinterpret_cast<R*>(J + NS * M);
  const SharedRow<R> mu{J + (NS + 1) * M};
  const cplx<R>* my_h = s_hc + (size_t)wc * 2 * N;
  const cplx<R>* rec = P.col.rec + (size_t)b * P.col.rec_bstride + at;
  double* hacc = P.col.hacc + ((size_t)b * K + id.ky) * 2 + id.ch;
  load_tables<X>(s_base, P.col.tw);
  pdl_wait();   // launched with programmatic serialization: the predecessor's writes are visible past here
  if (P.col.ctl && P.col.ctl[b].done) return;   // the whole cluster
  const R h = P.col.ctl ? (R)P.col.ctl[b].h : (R)P.col.h, coeff = id.ch == 0 ? P.col.nu : P.col.eta;
  double acc = 0.0;
  if (cw >= 0) {
    acc = *hacc;
    for (int s = xf.l; s < M; s += 32) {
      for (int q = 0; q < NS; ++q) J[q * M + s] = Jg[q * VEC + s];
      e[s] = s == 0 && id.ky == 0 ? R(0) : exp(h / R(2) * diss_L<R>((R)slot_to_kx(s, X::KMAX, M), (R)id.ky, coeff));
      J[(NS + 1) * M + s] = mu_row<X>(P.col.tw, id.ky)[s];
    }
  }
  cluster_barrier();   // every CTA has started before a peer writes its shared memory
  for (int it = P.hi; it >= P.lo; --it) {
    const cplx<R>* Q = rec + it * P.rec_step;
#pragma unroll 1
    for (int k = AJ_S4; k >= AJ_S1; --k) {
      const bool first = it == P.hi && k == AJ_S4, last = it == P.lo && k == AJ_S1, prev = it > 0;
      if (!first) cluster_barrier();   // column pass -> row pass
      RowAdjParams<R> row = P.row;
      row.phys += ((long)(it - P.lo) * 4 + k - AJ_S1) * P.phys_step;
      row_adj_body<W, true>(row, b, rank * W, xf, s_gt, first, s_hc);
      cluster_barrier();               // row pass -> column pass
      if (cw < 0) continue;
      if (k > AJ_S1) stage_rows<R, M>(rows, Q, VEC, adj4_qmask(k));
      else if (prev) stage_rows<R, M>(rows, Q - P.rec_step, VEC, adj4_qmask(AJ_S1));
      cplx<R> xb[X::E], lam[X::E];
      col_adj_rows(my_h, my_h + N, id.ky, xf, mu, xb);
      staged_wait();
      double hpart = 0.0, hdiv = 0.0;
      switch (k) {
        case AJ_S4: chain_adj_algebra<AJ_S4>(h, coeff, id, xf, prev, hpart, hdiv, J, e, rows, xb, lam); break;
        case AJ_S3: chain_adj_algebra<AJ_S3>(h, coeff, id, xf, prev, hpart, hdiv, J, e, rows, xb, lam); break;
        case AJ_S2: chain_adj_algebra<AJ_S2>(h, coeff, id, xf, prev, hpart, hdiv, J, e, rows, xb, lam); break;
        default: chain_adj_algebra<AJ_S1>(h, coeff, id, xf, prev, hpart, hdiv, J, e, rows, xb, lam); break;
      }
      double part = hpart + hdiv / (double)h;   // col_hacc
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      acc += part;
      if (k > AJ_S1 || prev) col_adj_emit<W>(lam, P.col.G, b, id.ch, id.ky, true, xf, last ? nullptr : s_gt);
    }
  }
  if (cw >= 0) {
    __syncwarp();
    for (int s = xf.l; s < M; s += 32)
      for (int q = 0; q < NS; ++q) Jg[q * VEC + s] = J[q * M + s];
    if (xf.l == 0) *hacc = acc;
  }
  cluster_barrier();   // no CTA leaves while a peer may still write its shared memory
}

// ---------------------------------------------------------------------------
// Tangents of a run of TDRK4 steps (k_row_tan's, k_row_tan2's and k_col_tdj's passes) in one
// launch, with the layout of k_rk4_chain.  The tiles of df and of dk1 / dk2 lie beside each
// other; the H tile of a single row pass takes the second's place, that of a dual one the
// first's.  The first row pass reads global Ga and the last column pass writes it.
// Measured, tangents of 64 steps, launch per pass -> this: n = 64, batch 1 1.96 -> 1.40 ms,
// batch 12 2.22 -> 1.39; n = 128, batch 1 2.74 -> 2.36, batch 7 3.77 -> 2.33.
// ---------------------------------------------------------------------------
template <typename R>
struct TdChainParams {
  ColTdjParams<R> col;   // rec: of step 0 of the run
  const R* phys;         // [2 cnt][N][NPH][N] states f, f_temp of the run's steps, then k1, k2
  int cnt, produce;
};
template <typename R, int N, int W> struct TdChainSmem {   // the second tile after the first's regions
  using S = ChainSmem<R, N, W, true, 1, (int)DT_NSLOT + 1>;
  static constexpr int gtb = (int)(S::bytes / sizeof(cplx<R>));
  static constexpr size_t bytes = S::bytes + (size_t)NG * S::K * (W + 1) * sizeof(cplx<R>);
};
template <int STAGE, class X>
__device__ __forceinline__ void chain_tdj_algebra(typename X::R h, typename X::R dpar_h, typename X::R coeff,
                                                  const ColId<X>& id, const X& xf, cplx<typename X::R>* S,
                                                  const cplx<typename X::R>* q, const cplx<typename X::R> (&r)[X::E],
                                                  cplx<typename X::R> (&x)[X::E]) {
  using R = typename X::R;
#pragma unroll
  for (int i = 0; i < X::E; ++i) {
    x[i] = mk<R>(0, 0);
    const int slot = xf.slot(i);
    if (slot < 0) continue;
    x[i] = tdj_algebra<STAGE, R>(h, dpar_h, diss_L<R>(xf.kx(i), (R)id.ky, coeff), r[i], q[slot],
                                 [&](int d) -> cplx<R> { return S[d * X::M + slot]; },
                                 [&](int d, cplx<R> v) { S[d * X::M + slot] = v; });
  }
}

template <typename R, int N, int W>
__global__ void __launch_bounds__(W * 32, 1) k_tdj_chain(TdChainParams<R> P) {
  using X = Xf<R, N>;
  constexpr int K = X::K, M = X::M, CL = chain_cl<N, W>(), NS = (int)DT_NSLOT;
  constexpr size_t VEC = (size_t)2 * K * M, PST = (size_t)N * NPH * N;
  using SM = typename TdChainSmem<R, N, W>::S;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_base = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_ga = s_base + SM::gt;
  cplx<R>* s_gb = s_base + TdChainSmem<R, N, W>::gtb;
  cplx<R>* s_hc = s_base + SM::hc;
  const X xf(s_base, threadIdx.x >> 5);
  const int b = blockIdx.x / CL, rank = blockIdx.x - b * CL;
  const int cw = chain_column<N, W>(rank), wc = cw < 0 ? 0 : (int)(threadIdx.x >> 5);
  const ColId<X> id(cw < 0 ? 0 : cw, b, b + 1);
  const size_t at = ((size_t)id.ch * K + id.ky) * M;
  cplx<R>* D = P.col.D + (size_t)b * P.col.nslot * VEC + at;
  cplx<R>* row = s_base + SM::work + (size_t)wc * M;
  cplx<R>* S = s_base + SM::ds + (size_t)wc * (NS + 1) * M;
  const SharedRow<R> mu{S + NS * M};
  const cplx<R>* my_h = s_hc + (size_t)wc * 2 * N;
  load_tables<X>(s_base, P.col.tw);
  pdl_wait();   // launched with programmatic serialization: the predecessor's writes are visible past here
  if (cw >= 0)
    for (int s = xf.l; s < M; s += 32) {
      S[DT_F * M + s] = D[DT_F * VEC + s];
      S[NS * M + s] = mu_row<X>(P.col.tw, id.ky)[s];
    }
  const R h = (R)P.col.h, dpar_h = (R)(P.col.dT[b] * P.col.dscale) / h, coeff = id.ch == 0 ? P.col.nu : P.col.eta;
  cluster_barrier();   // every CTA has started before a peer writes its shared memory
  for (int it = 0; it < P.cnt; ++it) {
#pragma unroll 1
    for (int st = 1; st <= 4; ++st) {
      if (it > 0 || st > 1) cluster_barrier();   // column pass -> row pass
      const bool first = it == 0 && st == 1, last = it == P.cnt - 1 && st == 4;
      const R* pa = P.phys + (size_t)(2 * it + (st > 2)) * PST;   // f, or f_temp
      if (st & 1) {
        RowTanParams<R> q{};
        q.G = P.col.Ga; q.phys = pa;
        row_tan_body<W, true>(q, b, rank * W, xf, s_ga, s_gb, first, s_hc);
      } else {
        RowTan2Params<R> q{};
        q.phys_a = pa; q.phys_b = pa + (size_t)2 * P.cnt * PST;   // and k1, or k2
        row_tan2_body<W, true>(q, b, rank * W, xf, s_ga, s_gb, false, s_hc);
      }
      cluster_barrier();                          // row pass -> column pass
      if (cw < 0) continue;
      stage_rows<R, M>(row, P.col.rec + (size_t)it * TR_NREC * VEC + at, VEC, 1u << tdj_qrow(st));
      cplx<R> r[X::E], x[X::E];
      chain_rhs(P.col.H, id, xf, my_h, r);
      staged_wait();
      switch (st) {
        case 1: chain_tdj_algebra<1>(h, dpar_h, coeff, id, xf, S, row, r, x); break;
        case 2: chain_tdj_algebra<2>(h, dpar_h, coeff, id, xf, S, row, r, x); break;
        case 3: chain_tdj_algebra<3>(h, dpar_h, coeff, id, xf, S, row, r, x); break;
        default: chain_tdj_algebra<4>(h, dpar_h, coeff, id, xf, S, row, r, x); break;
      }
      if (!last || P.produce)
        col_inverse_uv<W>(x, P.col.Ga, b, id.ch, id.ky, true, xf, mu, last ? nullptr : (st & 1) ? s_gb : s_ga);
    }
  }
  __syncwarp();
  if (cw >= 0)
    for (int s = xf.l; s < M; s += 32) D[DT_F * VEC + s] = S[DT_F * M + s];
  cluster_barrier();   // no CTA leaves while a peer may still write its shared memory
}

// ---------------------------------------------------------------------------
// Adaptive Lawson-RK4(3) attempts of the primal (timestepping.lawson_rk43,
// jax_scripts/lib/timestepping.py:151-335) in one launch: cluster b runs state
// b's attempts until it completes or `amax` attempts were made -- the column
// stages A..E (k_col_rk43's transforms and algebra), the four RHS row passes
// (k_row_rhs's body) and the error norm (k_row_err's body).  G and H never leave the
// cluster (an attempt starts from the slots alone).  Each CTA sends its error maximum to
// every CTA of the cluster, and after one cluster barrier every CTA makes the same
// accept/reject decision and step-size update (rk43_control, as the last block of
// k_row_err does) on its own copy of the control block, which CTA 0 writes back at the
// end.  Set-up, START and INIT passes run before the launch.
// Measured at n = 128 FP64, T = 0.2, atol 1e-8 (G and H through global memory, CTA 0
// deciding behind a second barrier -> this): batch 1 1.55 -> 1.45 ms, batch 8 4.28 -> 3.99;
// at n = 64 1.26 -> 1.03 and 2.08 -> 1.67.
// ---------------------------------------------------------------------------
template <typename R>
struct Rk43ChainParams {
  Col43Params<R> col;
  RowParams<R> row;
  double atol;
  double* rec_h;   // optional [B][cap] attempted step sizes
  int* rec_acc;    // optional [B][cap] accept flags
  long amax;       // attempts at most
};

template <int STAGE, bool DSH, class X>
__device__ __forceinline__ void chain_rk43_algebra(const Col43Params<typename X::R>& p, const R43Col<typename X::R>& c,
                                                   const ColId<X>& id, const X& xf, const cplx<typename X::R>* rows,
                                                   cplx<typename X::R>* S, size_t SS, const SharedRow<typename X::R>& forcing,
                                                   const cplx<typename X::R> (&r)[X::E], cplx<typename X::R> (&x)[X::E]) {
  using R = typename X::R;
  constexpr size_t VEC = (size_t)2 * X::K * X::M;
  constexpr int M = X::M;
  constexpr unsigned SMASK = r43_smask(STAGE);
  const R coeff = id.ch == 0 ? p.nu : p.eta;
  const int ix = DSH ? (c.pend ? S_XF : S_X0) : 0, ik = DSH ? (c.pend ? S_K5 : S_K1) : 1;   // stage A
#pragma unroll
  for (int i = 0; i < X::E; ++i) {
    const int slot = xf.slot(i);
    if (slot < 0) continue;
    const cplx<R> v = STAGE == R43_A ? mk<R>(0, 0) : with_forcing<R>(r[i], forcing, id.ch, id.ky, slot);
    cplx<R> xs = mk<R>(0, 0), ks = xs;
    if constexpr (STAGE == R43_A) { xs = (DSH ? S : rows)[ix * M + slot]; ks = (DSH ? S : rows)[ik * M + slot]; }
    x[i] = r43_algebra<STAGE>(c, diss_L<R>(xf.kx(i), (R)id.ky, coeff), v, xs, ks, VEC, slot,
                              [&](int q) { return DSH ? S[q * M + slot] : rows[bit_rank(SMASK, q) * M + slot]; },
                              [&](int q, cplx<R> a) { S[q * SS + slot] = a; });
  }
}

template <typename R, int N, int W>
__global__ void __launch_bounds__(W * 32, 1) k_rk43_chain(Rk43ChainParams<R> P) {
  using X = Xf<R, N>;
  constexpr int M = X::M, CL = chain_cl<N, W>();
  constexpr size_t VEC = (size_t)2 * X::K * M;
  constexpr bool DSH = W == 8;   // slots in shared memory
  constexpr size_t SS = DSH ? (size_t)M : VEC;
  using SM = Rk43ChainSmem<R, N, W>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_base = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_gt = s_base + SM::gt;
  cplx<R>* s_hc = s_base + SM::hc;
  __shared__ double s_max[W];
  __shared__ double s_errs[CL];   // the error maxima of the cluster's CTAs
  __shared__ StepCtl s_ctl;       // state b's control block, the same in every CTA
  const X xf(s_base, threadIdx.x >> 5);
  const int b = blockIdx.x / CL, rank = blockIdx.x - b * CL;
  const int cw = chain_column<N, W>(rank), wc = cw < 0 ? 0 : (int)(threadIdx.x >> 5);
  const ColId<X> id(cw < 0 ? 0 : cw, b, b + 1);
  cplx<R>* sglob = P.col.S + (size_t)b * S_NSLOT * VEC + ((size_t)id.ch * X::K + id.ky) * M;
  cplx<R>* my_s = s_base + SM::ds + (size_t)wc * ((DSH ? S_NSLOT : 0) + 2) * M;
  const SharedRow<R> forcing{my_s}, mu{my_s + M};
  cplx<R>* S = DSH ? my_s + 2 * M : sglob;
  cplx<R>* rows = s_base + SM::work + (size_t)wc * (DSH ? 0 : 4) * M;
  const cplx<R>* my_h = s_hc + (size_t)wc * 2 * N;
  load_tables<X>(s_base, P.col.tw);
  pdl_wait();   // launched with programmatic serialization: the predecessor's writes are visible past here
  if (threadIdx.x == 0) s_ctl = P.col.ctl[b];
  if (cw >= 0) {
    for (int e = xf.l; e < M; e += 32) {
      my_s[e] = P.col.fhat[id.ky * M + e];
      my_s[M + e] = mu_row<X>(P.col.tw, id.ky)[e];
    }
    if constexpr (DSH)
      for (int d = 0; d < S_NSLOT; ++d)
        for (int e = xf.l; e < M; e += 32) S[d * M + e] = sglob[d * VEC + e];
  }
  cluster_barrier();   // every CTA has started before a peer writes its shared memory
  for (long a = 0; a < P.amax && !s_ctl.done; ++a) {
    const R43Col<R> c(P.col, s_ctl, b, id.ch, id.ky, VEC, X::K, M);
#pragma unroll 1
    for (int st = R43_A; st <= R43_E; ++st) {
      if (st != R43_A) {
        row_rhs_body<W, true>(P.row, b, rank * W, xf, s_gt, s_gt, false, s_hc);
        cluster_barrier();
      }
      if (cw >= 0) {
        if constexpr (!DSH) stage_rows<R, M>(rows, sglob, VEC, st == R43_A ? r43_amask(c.pend) : r43_smask(st));
        cplx<R> r[X::E], x[X::E];
#pragma unroll
        for (int i = 0; i < X::E; ++i) r[i] = x[i] = mk<R>(0, 0);
        if (st != R43_A) chain_rhs(P.col.H, id, xf, my_h, r);
        if constexpr (!DSH) staged_wait();
        switch (st) {
          case R43_A: chain_rk43_algebra<R43_A, DSH>(P.col, c, id, xf, rows, S, SS, forcing, r, x); break;
          case R43_B: chain_rk43_algebra<R43_B, DSH>(P.col, c, id, xf, rows, S, SS, forcing, r, x); break;
          case R43_C: chain_rk43_algebra<R43_C, DSH>(P.col, c, id, xf, rows, S, SS, forcing, r, x); break;
          case R43_D: chain_rk43_algebra<R43_D, DSH>(P.col, c, id, xf, rows, S, SS, forcing, r, x); break;
          default: chain_rk43_algebra<R43_E, DSH>(P.col, c, id, xf, rows, S, SS, forcing, r, x); break;
        }
        if (st == R43_E) col_inverse1<W>(x, P.col.G, NG, b, id.ch, id.ky, true, xf, R(1) / (R(N) * R(N)), s_gt);
        else col_inverse_uv<W>(x, P.col.G, b, id.ch, id.ky, true, xf, mu, s_gt);
      }
      cluster_barrier();
    }
    const double bm = row_err_max<W>(P.col.G, b, rank * W, xf, s_gt, s_max, false);
    if (threadIdx.x < CL)
      *cooperative_groups::this_cluster().map_shared_rank(&s_errs[rank], (unsigned)threadIdx.x) = bm;
    cluster_barrier();
    if (threadIdx.x == 0) {
      double err = 0.0;
      for (int r = 0; r < CL; ++r) err = (s_errs[r] > err || isnan(s_errs[r])) ? s_errs[r] : err;
      const int at = s_ctl.attempts, cap = P.col.cap;
      const bool rec = rank == 0 && at < cap;
      rk43_control(s_ctl, P.atol, err, rec && P.rec_h ? P.rec_h + (size_t)b * cap : nullptr,
                   rec && P.rec_acc ? P.rec_acc + (size_t)b * cap : nullptr);
    }
    __syncthreads();
  }
  if (rank == 0 && threadIdx.x == 0) P.col.ctl[b] = s_ctl;
  if constexpr (DSH) {
    __syncwarp();
    if (cw >= 0)
      for (int d = 0; d < S_NSLOT; ++d)
        for (int e = xf.l; e < M; e += 32) sglob[d * VEC + e] = S[d * M + e];
  }
}   // (no CTA writes a peer's shared memory after the last cluster barrier)

}  // namespace ecs
