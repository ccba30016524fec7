// Hot-path kernels of the pseudo-spectral MHD right-hand side and the Lawson
// steppers.  One right-hand-side evaluation (reference: state_vel,
// jax_scripts/lib/mhd_jax.py:105-175) is split into two passes around the two
// transposes of a 2D FFT.
//
// Nonlinear terms.  The reference forms
//   dw/dt = -(u.grad w) + (B.grad j) + f,   dj/dt = k^2 rfft2(u B_y - v B_x)
// from 8 physical fields (the x and y derivatives of w and j and the uncurled
// velocities u, v, B_x, B_y, B with the mean field b0).  For divergence-free u
// and B with w = dv/dx - du/dy (and j likewise from B) the advection terms
// equal Basdevant's form
//   u.grad w = d_xy(v^2 - u^2) + (d_xx - d_yy)(u v)
// so that, with
//   P1 = (u^2 - v^2) - (B_x^2 - B_y^2),  P2 = B_x B_y - u v,  P3 = u B_y - v B_x,
//   dw/dt = mask (-kx ky P1^ + (ky^2 - kx^2) P2^ + f^),   dj/dt = k^2 mask P3^.
// Products of two fields on the 2/3-dealiased box alias only onto modes outside
// the box, so the retained modes of both forms are equal in exact arithmetic;
// this form needs 4 physical fields instead of 8 and 7 column transforms
// instead of 10.
//
//   column pass (one transform group per (batch, ky, channel), x contiguous; a
//   group is a warp, or 16 lanes in the group layout, see fft.cuh):
//     [forward FFTs along x of the product rows of the previous RHS: P1, P2
//      (channel w) or P3 (channel j)]
//     -> spectral epilogue (multipliers, dealias mask, forcing, stepper stage algebra)
//     -> stage input -> the two uncurling multipliers i ky/k^2, -i kx/k^2
//        -> 2 inverse FFTs along x -> G (u, v or B_x, B_y)
//   row pass (one warp per physical row x, CTA = XT rows staged in shared memory):
//     4 half-spectra rows of G -> 2 complex inverse FFTs (two real fields
//     packed per transform) -> P1, P2, P3 -> 2 forward FFTs -> split -> H
//
// The box layout and intermediate layouts are documented in common.cuh.
#pragma once

#include "common.cuh"
#include "fft.cuh"

#include <cooperative_groups.h>

namespace ecs {

// Field counts of the intermediate arrays (per batch element).
constexpr int NG = 4;    // G[b][NG][K][N]: inverse column transforms of u, v, B_x, B_y (no mean field)
constexpr int NH = 3;    // H[b][NH][K][N]: row transforms of P1, P2, P3
constexpr int NPH = 4;   // physical record rows: u, v, B_x + b0x, B_y + b0y
constexpr int NHA = 4;   // adjoint H[b][NHA][K][N]: row transforms of the cotangents of u, v, B_x, B_y

// ---------------------------------------------------------------------------
// spectral helpers
// ---------------------------------------------------------------------------

// (kx^2 + ky^2) (mhd_jax.py:154); zero at (0,0), as the mask makes it.  Exact in
// both precisions, as all these integer products.
template <typename R>
__device__ __forceinline__ R ksq_of(R kx, R ky) { return kx * kx + ky * ky; }

// Dissipation L = -(kx^2+ky^2) * coeff (mhd_jax.py:97-102), zero at (0,0).
template <typename R>
__device__ __forceinline__ R diss_L(R kx, R ky, R coeff) {
  return (-ksq_of<R>(kx, ky)) * coeff;
}

// Multiplier of the transformed product row f in {0: P1, 1: P2, 2: P3} in the
// nonlinear time derivative: -kx ky, ky^2 - kx^2 (channel w), k^2 (channel j).
// Zero at (0,0), which the mask removes.
template <typename R>
__device__ __forceinline__ R prod_mult(int f, R kx, R ky) {
  return f == 0 ? -kx * ky : f == 1 ? ky * ky - kx * kx : kx * kx + ky * ky;
}

// ---------------------------------------------------------------------------
// column-pass building blocks (one transform group per (batch, ky, channel))
// ---------------------------------------------------------------------------

// The column a lane's group works on.  Unit u of a state is channel u & 1 of the G
// columns ky from (u / 2) G on, for one warp (one channel per unit, so that its groups
// run the same transforms).  A group past the last column
// is not active: it computes on the last one and stores nothing; `none`: the warp
// has no unit at all.
template <class X> __host__ __device__ constexpr int col_units() { return 2 * ((X::K + X::G - 1) / X::G); }
template <class X>
struct ColId {
  bool act, none;
  int b, ch, ky;
  // A pass over B states: unit w % col_units of state w / col_units on warp w of the grid.
  __device__ __forceinline__ explicit ColId(int B) {
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    set(w % col_units<X>(), w / col_units<X>(), B);
  }
  __device__ __forceinline__ ColId(int u, int b_, int B) { set(u, b_, B); }
  __device__ __forceinline__ void set(int u, int b_, int B) {
    const int k = (u >> 1) * X::G + (int)(threadIdx.x & 31) / X::L;
    none = b_ >= B;
    act = !none && k < X::K;
    ch = u & 1;
    ky = k < X::K ? k : X::K - 1;
    b = none ? B - 1 : b_;
  }
};

__host__ __device__ constexpr int popc_c(unsigned m) { return m ? (int)(m & 1u) + popc_c(m >> 1) : 0; }
// Place of bit q among the bits of a mask: an intrinsic, which folds in unrolled code
// (a recursive call as an array index puts the array into local memory).
__device__ __forceinline__ int bit_rank(unsigned mask, int q) { return __popc(mask & ((1u << q) - 1u)); }

// The rows of MASK that a column pass's algebra reads, one complex value per mode each.
// Their latency overlaps the forward transform: where STAGED, they are on their way to
// shared memory (cp.async, no registers) from begin() on.  Elsewhere load() brings EH of
// the lane's elements together into registers, because a load of one row cannot move
// over a store to another.  Measured per launch at n = 128 FP64 (cold caches): loads after
// the transform -> staged, the table rows below included, 19.1 -> 16.6 us for Lawson-RK4
// stage 2 at batch 64 and 7.4 -> 5.7 us at batch 1.
constexpr int MAX_STAGED = 8;   // rows of a warp that fit beside the tables in 48 KB (FP64, n = 128)
template <class X, unsigned MASK, int EH = X::E> struct Operands {
  using R = typename X::R;
  using C = cplx<R>;
  static constexpr int n = popc_c(MASK);
  static constexpr bool STAGED = X::STAGED && n <= MAX_STAGED;
  C* s;
  C op[STAGED || n == 0 ? 1 : n][EH];
  __device__ __forceinline__ explicit Operands(C* rows) : s(rows) {}
  // Row q starts at from(q), or at from + q pitch.
  template <class F> __device__ __forceinline__ void begin(F&& from) {
    if constexpr (STAGED) {
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        if (!((MASK >> q) & 1u)) continue;
        const C* g = from(q);
        for (int e = threadIdx.x & 31; e < X::M; e += 32) cp_async_c<R>(s + bit_rank(MASK, q) * X::M + e, g + e);
      }
    }
  }
  __device__ __forceinline__ void begin(const C* from, size_t pitch) { begin([&](int q) { return from + q * pitch; }); }
  // After the transform: elements i0 .. i0 + EH - 1.
  template <class F> __device__ __forceinline__ void load(F&& from, bool act, const X& xf, int i0 = 0) {
    if constexpr (STAGED) {
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      __syncwarp();
    } else if constexpr (n > 0) {
#pragma unroll
      for (int e = 0; e < EH; ++e) {
        if (i0 + e >= X::E || X::none(i0 + e)) continue;
        const int slot = act ? xf.slot(i0 + e) : -1;
        if (slot < 0) continue;
#pragma unroll
        for (int q = 0; q < 16; ++q)
          if ((MASK >> q) & 1u) op[bit_rank(MASK, q)][e] = from(q)[slot];
      }
    }
  }
  __device__ __forceinline__ void load(const C* from, size_t pitch, bool act, const X& xf, int i0 = 0) {
    load([&](int q) { return from + q * pitch; }, act, xf, i0);
  }
  // Row q at element i, whose slot is `slot`.
  __device__ __forceinline__ C get(int q, int i, int slot) const {
    if constexpr (STAGED) return s[bit_rank(MASK, q) * X::M + slot];
    else return op[bit_rank(MASK, q)][i % EH];
  }
};

// A table row of a column (its multipliers, the forcing): staged with the operands if ON
// (wait for it with Operands::load), else read where it is used.
template <class X, bool ON> struct TableRow {
  using C = cplx<typename X::R>;
  static constexpr bool STAGED = ON && X::STAGED;
  const C* g;
  __device__ __forceinline__ TableRow(C* rows, const C* from) : g(STAGED ? rows : from) {
    if constexpr (STAGED)
      for (int e = threadIdx.x & 31; e < X::M; e += 32) cp_async_c<typename X::R>(rows + e, from + e);
  }
  // Before the first read, where no Operands::load came before it.
  __device__ __forceinline__ void wait() const {
    if constexpr (STAGED) {
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      __syncwarp();
    }
  }
  __device__ __forceinline__ C operator()(int slot) const { return STAGED ? g[slot] : __ldg(g + slot); }
};
// The multipliers' row of column ky in the device table.
template <class X> __device__ __forceinline__ const cplx<typename X::R>* mu_row(const cplx<typename X::R>* tab, int ky) {
  return tab + XfTable<typename X::R, X::N>::mu + ky * X::M;
}

// Warps per CTA of the column passes.
constexpr int COLWARPS = 4;
// Whether `extra` table rows are staged beside n operand rows, and the rows of room of a
// warp then.
__host__ __device__ constexpr bool rows_fit(int n, int extra) { return n + extra <= MAX_STAGED; }
template <class X> __host__ __device__ constexpr int col_rows(int n, int extra) {
  return !X::STAGED || n > MAX_STAGED ? 0 : rows_fit(n, extra) ? n + extra : n;
}
// Start of a column kernel with n operand rows and `extra` table rows: tables, the
// predecessor's results (programmatic launch), the warp's column `id`, its room `rows`.
#define ECS_COL_PROLOGUE(n, extra)                                                                          \
  __shared__ __align__(16) cplx<typename X::R> s_x[X::smem(COLWARPS) + COLWARPS * col_rows<X>(n, extra) * X::M];\
  load_tables<X>(s_x, p.tw);                                                                                \
  pdl_wait();                                                                                               \
  pdl_trigger();                                                                                            \
  __syncthreads();                                                                                          \
  const X xf(s_x, threadIdx.x >> 5);                                                                        \
  const ColId<X> id(p.B);                                                                                   \
  if (id.none) return;                                                                                      \
  [[maybe_unused]] cplx<typename X::R>* rows = s_x + X::smem(COLWARPS) + (int)(threadIdx.x >> 5) * col_rows<X>(n, extra) * X::M

// Nonlinear time derivative of channel ch (without forcing) at the lane's algebra
// elements of column ky from the product rows h0, h1 = the P1, P2 rows of
// column ky (ch 0), or h0 = its P3 row (ch 1), in global or shared memory:
//   ch 0: -kx ky rfft2(P1) + (ky^2 - kx^2) rfft2(P2),  ch 1: k^2 rfft2(P3).
template <class X>
__device__ __forceinline__ void col_rhs_rows(const cplx<typename X::R>* h0, const cplx<typename X::R>* h1, int ch, int ky,
                                             const X& xf, cplx<typename X::R> (&v)[X::E]) {
  using R = typename X::R;
  constexpr int E = X::E, L = X::L;
  const R rky = (R)ky;
  if constexpr (X::GROUP) {
    // one copy of the transform for both channels: P2 then P1 (channel w), or P3;
    // fma(m0, P1, RN(m1 P2)) as in the other layouts
    cplx<R> t[E];
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = mk<R>(0, 0);
#pragma unroll 1
    for (int f = ch == 0 ? 1 : 2; f >= 0; f = f == 1 ? 0 : -1) {
      const cplx<R>* h = f == 1 ? h1 : h0;
#pragma unroll
      for (int j = 0; j < E; ++j) t[j] = h[xf.l + L * j];
      xf.template to_spec<false>(t);
#pragma unroll
      for (int j = 0; j < E; ++j) {
        if (X::none(j)) continue;
        const R m = prod_mult<R>(f, xf.kx(j), rky);
        v[j] = mk<R>(fma(m, t[j].x, v[j].x), fma(m, t[j].y, v[j].y));
      }
    }
  } else if (ch == 0) {
    cplx<R> r[E];
#pragma unroll
    for (int j = 0; j < E; ++j) { v[j] = h0[xf.l + L * j]; r[j] = h1[xf.l + L * j]; }
    xf.template to_spec2<false>(v, r);
#pragma unroll
    for (int j = 0; j < E; ++j) {
      const R kx = xf.kx(j), m0 = prod_mult<R>(0, kx, rky), m1 = prod_mult<R>(1, kx, rky);
      v[j] = mk<R>(fpp(m0, v[j].x, m1, r[j].x), fpp(m0, v[j].y, m1, r[j].y));
    }
  } else {
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = h0[xf.l + L * j];
    xf.template to_spec<false>(v);
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = cscale(v[j], prod_mult<R>(2, xf.kx(j), rky));
  }
}

template <class X>
__device__ __forceinline__ void col_load_rhs(const cplx<typename X::R>* H, int b, int ch, int ky, const X& xf,
                                             cplx<typename X::R> (&v)[X::E]) {
  const cplx<typename X::R>* h0 = H + ((size_t)(b * NH + (ch == 0 ? 0 : 2)) * X::K + ky) * X::N;
  col_rhs_rows(h0, h0 + (size_t)X::K * X::N, ch, ky, xf, v);
}

// Cluster-resident passes (kernels_chain.cuh): a cluster of N / XT CTAs holds
// one state; CTA r keeps the G tile of physical rows x in [XT r, XT r + XT)
// (NG K rows of pitch XT + 1, at the same shared-memory offset in every CTA).

// A G row of a column pass written into the cluster's G tiles instead of
// global memory: position x goes to CTA x / XT, tile row `row`, column x % XT.
// `tile` is this CTA's tile.
template <int XT, class X>
__device__ __forceinline__ void col_to_tiles(const cplx<typename X::R> (&w)[X::E], cplx<typename X::R>* tile, int row,
                                             const X& xf) {
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
#pragma unroll
  for (int j = 0; j < X::E; ++j) {
    const int x = xf.l + X::L * j;
    cl.map_shared_rank(tile, (unsigned)(x / XT))[row * (XT + 1) + x % XT] = w[j];
  }
}

// A transformed row to field f of column ky of G[b] (nf fields per state; or, CX > 0
// and `gtile` given, to the cluster's G tiles).
template <int CX = 0, class X>
__device__ __forceinline__ void col_put(const cplx<typename X::R> (&w)[X::E], cplx<typename X::R>* G, int nf, int b, int f,
                                        int ky, bool act, const X& xf, cplx<typename X::R>* gtile = nullptr) {
  if (!act) return;
  if constexpr (CX > 0) {
    if (gtile) { col_to_tiles<CX>(w, gtile, f * X::K + ky, xf); return; }
  }
  cplx<typename X::R>* g = G + ((size_t)(b * nf + f) * X::K + ky) * X::N;
#pragma unroll
  for (int j = 0; j < X::E; ++j) g[xf.l + X::L * j] = w[j];
}

// The two uncurled fields i ky/k^2 x and -i kx/k^2 x (mhd_jax.py:140-141) over n^2
// of a stage input x (the lane's algebra elements, zero outside the box),
// transformed along x, to G fields 2c, 2c+1.
// `mu` gives the column's multipliers (TableRow of mu_row).
template <int CX = 0, class X, class Mu>
__device__ __forceinline__ void col_inverse_uv(const cplx<typename X::R> (&x)[X::E], cplx<typename X::R>* G, int b, int c,
                                               int ky, bool act, const X& xf, const Mu& mu,
                                               cplx<typename X::R>* gtile = nullptr) {
  using R = typename X::R;
  constexpr int E = X::E;
  // product rounded on its own: not contracted with the transform's sums
  auto mul = [&](cplx<R> z, R f) { return mk<R>(mul_rn(-f, z.y), mul_rn(f, z.x)); };
  if constexpr (X::GROUP) {   // one after the other, one copy of the transform
    cplx<R> f[E];
#pragma unroll
    for (int j = 0; j < E; ++j)
      if (!X::none(j)) f[j] = mu(xf.slot(j) < 0 ? 0 : xf.slot(j));
#pragma unroll 1
    for (int v = 0; v < 2; ++v) {
      cplx<R> z[E];
#pragma unroll
      for (int j = 0; j < E; ++j) z[j] = X::none(j) ? mk<R>(0, 0) : mul(x[j], v == 0 ? f[j].x : f[j].y);
      xf.template from_spec<true, true>(z);
      col_put<CX>(z, G, NG, b, 2 * c + v, ky, act, xf, gtile);
    }
  } else {
    cplx<R> wu[E], wv[E];
#pragma unroll
    for (int j = 0; j < E; ++j) {
      const int s = xf.slot(j);
      wu[j] = wv[j] = mk<R>(0, 0);
      if (s < 0) continue;
      const cplx<R> f = mu(s);
      wu[j] = mul(x[j], f.x);
      wv[j] = mul(x[j], f.y);
    }
    xf.template from_spec2<true>(wu, wv);
    col_put<CX>(wu, G, NG, b, 2 * c, ky, act, xf, gtile);
    col_put<CX>(wv, G, NG, b, 2 * c + 1, ky, act, xf, gtile);
  }
}

// One plain inverse transform along x of a box column, scaled, to field f of
// G[b] (nf fields per batch element; or to the cluster's G tiles, see col_put).
template <int CX = 0, class X>
__device__ __forceinline__ void col_inverse1(const cplx<typename X::R> (&x)[X::E], cplx<typename X::R>* G, int nf, int b,
                                             int f, int ky, bool act, const X& xf, typename X::R scale,
                                             cplx<typename X::R>* gtile = nullptr) {
  using R = typename X::R;
  cplx<R> w[X::E];
#pragma unroll
  for (int j = 0; j < X::E; ++j) w[j] = X::none(j) ? mk<R>(0, 0) : cscale_rn(x[j], scale);
  xf.template from_spec<true, true>(w);
  col_put<CX>(w, G, nf, b, f, ky, act, xf, gtile);
}

// ---------------------------------------------------------------------------
// Column pass of the forward RHS fused with the Lawson-RK4 stage algebra
// (reference: timestepping.lawson_rk4, jax_scripts/lib/timestepping.py:69-80).
// ---------------------------------------------------------------------------

// Lawson-RK4 record per step (box vectors): stage input X1 = F, stage
// derivatives k1..k4 (before twiddles) and stage inputs X2..X4.
enum Rk4Rec { Q_F = 0, Q_K1, Q_K2, Q_K3, Q_K4, Q_X2, Q_X3, Q_X4, Q_NREC };

enum ColStage : int {
  COL_START = 0,     // no RHS input; stage input = F (start of a step)
  COL_RK4_S1 = 1,    // finish k1, stage input X2
  COL_RK4_S2 = 2,    // finish k2, stage input X3
  COL_RK4_S3 = 3,    // finish k3, stage input X4
  COL_RK4_S4 = 4,    // finish k4 (state update), stage input X1 of next step
  COL_PLAIN = 5,     // finish RHS: OUT = v (+ L f0 if diss)   [state_vel]
};

template <typename R>
struct ColParams {
  const cplx<R>* H;      // [B][NH][K][N]
  cplx<R>* G;            // [B][NG][K][N]
  cplx<R>* F;            // [B][2][K][M]   state / accumulator
  cplx<R>* A1;           // [B][2][K][M]   e*k1
  cplx<R>* K2;           // [B][2][K][M]   k2
  cplx<R>* OUT;          // [B][2][K][M]   COL_PLAIN output
  const R* Etab;         // [B][2][K][M]   exp(h/2 L) * mask
  const StepCtl* ctl;    // [B]
  const cplx<R>* fhat;   // [K][M] box spectrum of the forcing (omega only)
  const cplx<R>* tw;     // tables (xf_table)
  R nu, eta;
  int B;
  int stage;
  int produce;           // write G for the stage input
  int diss;              // COL_PLAIN: add L f (f = F)
  cplx<R>* rec;          // optional record of this step: [Q_NREC][2][K][M] per batch element
  long rec_bstride;      // elements between batch elements in rec
  int use_done;          // skip batch elements whose ctl.done is set (slot pool)
};

// A column's rows of the state slots and of the factor e.
template <typename R> struct Rk4Rows { cplx<R>* F; cplx<R>* A1; cplx<R>* K2; const R* e; };

// Rows that a stage's algebra reads (0: F, 1: A1, 2: K2), and whether it reads e.
__host__ __device__ constexpr unsigned rk4_mask(int stage) { return stage == COL_RK4_S3 ? 7u : stage == COL_PLAIN ? 0u : 1u; }
__host__ __device__ constexpr bool rk4_reads_e(int stage) { return stage == COL_RK4_S1 || stage == COL_RK4_S3; }

// The algebra of a Lawson-RK4 stage: the stage input x (zero outside the box) from the
// derivative r without forcing.  get(q, i, slot) reads row q, get_e(i, slot) e,
// forcing(slot) the forcing of channel w; h is the step.
template <int STAGE, class X, class Get, class GetE, class Forcing>
__device__ __forceinline__ void col_rk4_algebra(const ColParams<typename X::R>& p, const ColId<X>& id, const X& xf,
                                                const Rk4Rows<typename X::R>& w, typename X::R h, Get&& get, GetE&& get_e,
                                                const Forcing& forcing,
                                                const cplx<typename X::R> (&r)[X::E], cplx<typename X::R> (&x)[X::E]) {
  using R = typename X::R;
  constexpr int E = X::E, K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  const int c = id.ch, b = id.b, ky = id.ky;
  cplx<R>* rb = p.rec ? p.rec + (size_t)b * p.rec_bstride + ((size_t)c * K + ky) * M : nullptr;
#pragma unroll
  for (int i = 0; i < E; ++i) {
    x[i] = mk<R>(0, 0);
    if (X::none(i)) continue;
    const int slot = xf.slot(i);
    if (slot < 0) continue;
    cplx<R> v = mk<R>(0, 0);
    if (STAGE != COL_START) {
      v = r[i];                                                             // zero at (0,0)
      if (c == 0 && !(slot == 0 && ky == 0)) v = cadd(v, forcing(slot));    // mask * rfft2(forcing)
    }
    auto put = [&](int q, cplx<R> a) { if (rb) rb[q * VEC + slot] = a; };
    [[maybe_unused]] const cplx<R> f0 = STAGE != COL_PLAIN ? get(0, i, slot) : mk<R>(0, 0);
    [[maybe_unused]] const R e = rk4_reads_e(STAGE) ? get_e(i, slot) : R(0);
    switch (STAGE) {
      case COL_START: x[i] = f0; break;
      case COL_RK4_S1: {   // k1 = h v(f); f = e f; k1 = e k1; X2 = f + k1/2   (timestepping.py:74-76)
        cplx<R> k1 = cscale(v, h);
        put(Q_F, f0); put(Q_K1, k1);
        const cplx<R> f = cscale_rn(f0, e);
        k1 = cscale_rn(k1, e);
        w.F[slot] = f; w.A1[slot] = k1;
        x[i] = cadd(f, cscale(k1, R(0.5)));
        put(Q_X2, x[i]);
      } break;
      case COL_RK4_S2: {   // k2 = h v(X2); X3 = f + k2/2   (:76-77)
        const cplx<R> k2 = cscale(v, h);
        w.K2[slot] = k2;
        x[i] = cadd(f0, cscale(k2, R(0.5)));
        put(Q_K2, k2); put(Q_X3, x[i]);
      } break;
      case COL_RK4_S3: {   // k3; f,k1,k2,k3 *= e; X4 = f + k3; acc = f + k1/6 + k2/3 + k3/3   (:77-80)
        cplx<R> k3 = cscale(v, h);
        put(Q_K3, k3);
        const cplx<R> f = cscale_rn(f0, e), a = cscale_rn(get(1, i, slot), e), q2 = cscale_rn(get(2, i, slot), e);
        k3 = cscale_rn(k3, e);
        x[i] = cadd(f, k3);
        put(Q_X4, x[i]);
        w.F[slot] = cadd(cadd(cadd(f, cdiv_k<6>(a)), cdiv_k<3>(q2)), cdiv_k<3>(k3));
      } break;
      case COL_RK4_S4: {   // k4; f = acc + k4/6   (:79-80)
        const cplx<R> k4 = cscale(v, h);
        put(Q_K4, k4);
        const cplx<R> f = cadd(f0, cdiv_k<6>(k4));
        w.F[slot] = f;
        x[i] = f;
      } break;
      default: {           // COL_PLAIN: state_vel output (mhd_jax.py:171-173)
        if (p.diss) v = cadd(v, cscale(w.F[slot], diss_L<R>(xf.kx(i), (R)ky, c == 0 ? p.nu : p.eta)));
        p.OUT[((size_t)(b * 2 + c) * K + ky) * M + slot] = v;
      } break;
    }
  }
}

// A Lawson-RK4 column stage of one column; `rows`: shared room for its operands.
template <int STAGE, class X>
__device__ __forceinline__ void col_rk4_body(const ColParams<typename X::R>& p, const ColId<X>& id, const X& xf,
                                             cplx<typename X::R>* rows) {
  using R = typename X::R;
  if (p.use_done && p.ctl[id.b].done) return;
  const size_t base = ((size_t)(id.b * 2 + id.ch) * X::K + id.ky) * X::M;
  const Rk4Rows<R> w{p.F + base, p.A1 + base, p.K2 + base, p.Etab + base};
  auto from = [&](int q) { return q == 0 ? w.F : q == 1 ? w.A1 : w.K2; };
  constexpr int n = popc_c(rk4_mask(STAGE));
  Operands<X, rk4_mask(STAGE)> op(rows);
  op.begin(from);
  R* my_e = reinterpret_cast<R*>(rows + n * X::M);
  const TableRow<X, STAGE != COL_START> forcing(rows + (n + 1) * X::M, p.fhat + id.ky * X::M);
  const TableRow<X, STAGE != COL_PLAIN> mu(rows + (n + 2) * X::M, mu_row<X>(p.tw, id.ky));
  const R h = (R)p.ctl[id.b].h;
  if constexpr (X::STAGED && rk4_reads_e(STAGE))
    for (int s = xf.l; s < X::M; s += 32) cp_async_v(my_e + s, w.e + s);
  cplx<R> r[X::E], x[X::E];
  if (STAGE != COL_START) col_load_rhs(p.H, id.b, id.ch, id.ky, xf, r);
  op.load(from, true, xf);
  col_rk4_algebra<STAGE>(p, id, xf, w, h, [&](int q, int i, int slot) { return op.get(q, i, slot); },
                         [&](int, int slot) { return X::STAGED ? my_e[slot] : __ldg(w.e + slot); }, forcing, r, x);
  if (p.produce) col_inverse_uv(x, p.G, id.b, id.ch, id.ky, true, xf, mu);
}

template <typename R, int N, int STAGE>
__global__ void __launch_bounds__(COLWARPS * 32, 1) k_col_rk4(ColParams<R> p) {
  using X = Xf<R, N>;
  ECS_COL_PROLOGUE(popc_c(rk4_mask(STAGE)), 3);   // e, the forcing, the multipliers
  col_rk4_body<STAGE>(p, id, xf, rows);
}

// state_vel (mhd_jax.py:105-175) reads and writes full rfft2 arrays [B][2][N][N/2+1]
// directly: the first column pass takes its stage input from the full state and the last
// one writes the full derivative, zero outside the box (the columns past it by warps of
// their own): 3 launches per call instead of 5, without the copies between the full array
// and the box.  With the host's shorter comparison of the forcing a call on one state at
// n = 64, which is all launches and host work, takes 58.8 us instead of 71.9.
template <typename R, int N>
__global__ void __launch_bounds__(COLWARPS * 32, 1) k_col_full_start(ColParams<R> p, const cplx<R>* full) {
  using X = Xf<R, N>;
  ECS_COL_PROLOGUE(0, 1);   // the multipliers
  const TableRow<X, true> mu(rows, mu_row<X>(p.tw, id.ky));
  const cplx<R>* f = full + (size_t)(id.b * 2 + id.ch) * N * (N / 2 + 1) + id.ky;
  cplx<R> x[X::E];
#pragma unroll
  for (int j = 0; j < X::E; ++j) x[j] = xf.slot(j) >= 0 ? f[(size_t)X::pos(xf.l, j) * (N / 2 + 1)] : mk<R>(0, 0);
  mu.wait();
  col_inverse_uv(x, p.G, id.b, id.ch, id.ky, true, xf, mu);
}

// Warps for the N/2 + 1 columns of either channel.  `full` may be `out`: every entry is
// read by the thread that writes it.
template <typename R, int N>
__global__ void __launch_bounds__(COLWARPS * 32, 1) k_col_full_vel(ColParams<R> p, const cplx<R>* full, cplx<R>* out) {
  using X = Xf<R, N>;
  constexpr int E = X::E, NK = N / 2 + 1;
  __shared__ __align__(16) cplx<R> s_x[X::smem(COLWARPS)];
  load_tables<X>(s_x, p.tw);
  pdl_wait();
  pdl_trigger();
  __syncthreads();
  const X xf(s_x, threadIdx.x >> 5);
  const int u = blockIdx.x * COLWARPS + (int)(threadIdx.x >> 5), b = u / (2 * NK), ch = u & 1, ky = (u >> 1) % NK;
  if (b >= p.B) return;
  const size_t at = (size_t)(b * 2 + ch) * N * NK + ky;
  cplx<R> r[E];
#pragma unroll
  for (int j = 0; j < E; ++j) r[j] = mk<R>(0, 0);
  if (ky < X::K) col_load_rhs(p.H, b, ch, ky, xf, r);
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int slot = ky < X::K ? xf.slot(j) : -1;
    const size_t o = at + (size_t)X::pos(xf.l, j) * NK;
    cplx<R> v = mk<R>(0, 0);
    if (slot >= 0) {
      v = r[j];                                                                                      // zero at (0,0)
      if (ch == 0 && !(slot == 0 && ky == 0)) v = cadd(v, __ldg(p.fhat + ky * X::M + slot));         // mask * rfft2(forcing)
      if (p.diss) v = cadd(v, cscale(full[o], diss_L<R>(xf.kx(j), (R)ky, ch == 0 ? p.nu : p.eta)));   // mhd_jax.py:171-173
    }
    out[o] = v;
  }
}

// ---------------------------------------------------------------------------
// Row pass of the forward RHS: products in physical space.
// ---------------------------------------------------------------------------

template <typename R>
struct RowParams {
  const cplx<R>* G;   // [B][NG][K][N]
  cplx<R>* H;         // [B][NH][K][N]
  R* phys;            // optional record of u, v, B_x, B_y: phys + b * phys_bstride is [N][NPH][N]
  long phys_bstride;
  const StepCtl* ctl; // per-batch control (done flags) or null
  const cplx<R>* tw;
  R b0x, b0y;
  int B;
};

// Physical-field record of one stage: phys[x][2][N] pairs (u, v) and (B_x, B_y) of
// row x, in the order e = l + L j of the row transforms' registers, so that a lane loads
// the pairs that its products need whole and a warp's loads are contiguous.
template <typename R, int N>
__device__ __forceinline__ const cplx<R>* phys_row(const R* base, int x) {
  return reinterpret_cast<const cplx<R>*>(base) + (size_t)x * 2 * N;
}

// Load a [nf][K][XT] tile of a [B][nf][K][N] array into shared memory with row
// pitch XT+1.  Asynchronous copies (cp.async: global -> shared without a
// register round trip; 16 bytes per complex double, 8 per complex float);
// each thread waits for its own copies before returning, and the caller's
// __syncthreads then makes the whole tile visible.
template <typename R, int N, int XT>
__device__ __forceinline__ void load_tile(cplx<R>* s, const cplx<R>* __restrict__ g, int nfK, int x0) {
  for (int i = threadIdx.x; i < nfK * XT; i += blockDim.x) {
    const int xt = i % XT, r = i / XT;
    cp_async_c<R>(s + r * (XT + 1) + xt, g + (size_t)r * N + x0 + xt);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}
template <typename R, int N, int XT>
__device__ __forceinline__ void store_tile(cplx<R>* __restrict__ g, const cplx<R>* s, int nfK, int x0) {
  for (int i = threadIdx.x; i < nfK * XT; i += blockDim.x) {
    const int xt = i % XT, r = i / XT;
    g[(size_t)r * N + x0 + xt] = s[r * (XT + 1) + xt];
  }
}

// Full Hermitian spectrum value at position q (natural order) of the packed
// pair A + iB, from half-spectrum rows sA, sB (pitch XT+1, column w).  The ky=0
// entries contribute only their real parts, as irfft does.
template <typename R, int N, int XT>
__device__ __forceinline__ cplx<R> packed_pair(const cplx<R>* sA, const cplx<R>* sB, int q, int w) {
  constexpr int K = (N - 1) / 3 + 1;
  if (q < K) {
    cplx<R> a = sA[q * (XT + 1) + w], bb = sB[q * (XT + 1) + w];
    if (q == 0) { a.y = 0; bb.y = 0; }
    return mk<R>(a.x - bb.y, a.y + bb.x);
  }
  if (q > N - K) {
    const int qq = N - q;
    cplx<R> a = sA[qq * (XT + 1) + w], bb = sB[qq * (XT + 1) + w];
    return mk<R>(a.x + bb.y, bb.x - a.y);
  }
  return mk<R>(0, 0);
}

// Full Hermitian spectrum value at position q of one real field (imaginary
// part of the transform left zero) from its half-spectrum row sA.
template <typename R, int N, int XT>
__device__ __forceinline__ cplx<R> packed_one(const cplx<R>* sA, int q, int w) {
  constexpr int K = (N - 1) / 3 + 1;
  if (q < K) {
    cplx<R> a = sA[q * (XT + 1) + w];
    if (q == 0) a.y = 0;
    return a;
  }
  if (q > N - K) return cconj(sA[(N - q) * (XT + 1) + w]);
  return mk<R>(0, 0);
}

// The packed pair's (packed_one: a single field's) spectrum in the registers of the
// row's group, natural order.
template <int XT, class X>
__device__ __forceinline__ void load_pair(const cplx<typename X::R>* sA, const cplx<typename X::R>* sB, int w, const X& xf,
                                          cplx<typename X::R> (&v)[X::E]) {
  using R = typename X::R;
#pragma unroll
  for (int j = 0; j < X::E; ++j)
    v[j] = X::none(j) ? mk<R>(0, 0) : packed_pair<R, X::N, XT>(sA, sB, xf.l + X::L * j, w);
}
template <int XT, class X>
__device__ __forceinline__ void load_one(const cplx<typename X::R>* sA, int w, const X& xf, cplx<typename X::R> (&v)[X::E]) {
  using R = typename X::R;
#pragma unroll
  for (int j = 0; j < X::E; ++j)
    v[j] = X::none(j) ? mk<R>(0, 0) : packed_one<R, X::N, XT>(sA, xf.l + X::L * j, w);
}

// Split a natural-order forward transform W of (P1 + i P2) into the half
// spectra of P1 and P2: put(q, p1, p2) for ky = q < K.
template <class X, typename Put>
__device__ __forceinline__ void split_rows(const cplx<typename X::R> (&W)[X::E], const X& xf, Put&& put) {
  using R = typename X::R;
  constexpr int E = X::E, L = X::L;
  const int lane = threadIdx.x & 31, l = xf.l, src = (lane & ~(L - 1)) | ((L - l) & (L - 1));
#pragma unroll
  for (int j = 0; j < E; ++j) {
    if (L * j >= X::K) continue;
    cplx<R> t = shfl_c<R>(W[E - 1 - j], src);
    const cplx<R> P = (l == 0) ? W[(E - j) % E] : t;
    const int q = l + L * j;
    if (q < X::K) {
      const cplx<R> Wq = W[j];
      put(q, mk<R>((Wq.x + P.x) * R(0.5), (Wq.y - P.y) * R(0.5)), mk<R>((Wq.y + P.y) * R(0.5), (P.x - Wq.x) * R(0.5)));
    }
  }
}
// The same into shared rows s1, s2 of a tile; store_one: the half spectrum of one
// real field's transform.
template <int XT, class X>
__device__ __forceinline__ void split_store(const cplx<typename X::R> (&W)[X::E], cplx<typename X::R>* s1,
                                            cplx<typename X::R>* s2, int w, const X& xf) {
  using C = cplx<typename X::R>;
  split_rows(W, xf, [&](int q, C a, C b) { s1[q * (XT + 1) + w] = a; s2[q * (XT + 1) + w] = b; });
}
template <int XT, class X>
__device__ __forceinline__ void store_one(const cplx<typename X::R> (&W)[X::E], cplx<typename X::R>* s1, int w, const X& xf) {
#pragma unroll
  for (int j = 0; j < X::E; ++j) {
    if (X::L * j >= X::K) continue;
    const int q = xf.l + X::L * j;
    if (q < X::K) s1[q * (XT + 1) + w] = W[j];
  }
}

// The inverse transforms of a row's packed spectra in tile column w: fields (0, 1) to
// a, (2, 3) to b (SINGLE: field 2 alone).
template <int XT, bool SINGLE = false, class X>
__device__ __forceinline__ void row_inverse(const cplx<typename X::R>* s_G, int w, const X& xf,
                                            cplx<typename X::R> (&a)[X::E], cplx<typename X::R> (&b)[X::E]) {
  constexpr int F = X::K * (XT + 1);
  load_pair<XT>(s_G, s_G + F, w, xf, a);
  if (SINGLE) load_one<XT>(s_G + 2 * F, w, xf, b);
  else load_pair<XT>(s_G + 2 * F, s_G + 3 * F, w, xf, b);
  xf.template to_spec2<true>(a, b);
  __syncwarp();
}

// The forward transforms of a row: the packed pair a to fields 0, 1 of tile column w, and
// b to field 2 (one real field) or, PAIRS, to fields 2, 3.
template <int XT, bool PAIRS = false, class X>
__device__ __forceinline__ void row_forward(cplx<typename X::R> (&a)[X::E], cplx<typename X::R> (&b)[X::E],
                                            cplx<typename X::R>* s_H, int w, const X& xf) {
  constexpr int F = X::K * (XT + 1);
  xf.template from_spec2<false>(a, b);
  split_store<XT>(a, s_H, s_H + F, w, xf);
  if (PAIRS) split_store<XT>(b, s_H + 2 * F, s_H + 3 * F, w, xf);
  else store_one<XT>(b, s_H + 2 * F, w, xf);
}

// The NH K rows of a row pass's H tile (pitch XT + 1, physical rows x0 ..
// x0 + XT - 1) sent to the groups of the cluster that transform them: row
// (f, ky) feeds channel f == 2 of column ky, which is unit c = 2 (ky / G) + (f == 2) of
// the state: place c / CL of CTA c % CL (CL = N / XT CTAs), group ky % G, with its two
// rows of N at hcols + ((c / CL) G + ky % G) 2 N: P1, P2 (channel 0), or P3 in the
// first (channel 1).
// ADJ: the 2 x 2 adjoint rows instead, (f, ky) to row f % 2 of channel f / 2.
template <int XT, bool ADJ = false, class X>
__device__ __forceinline__ void scatter_h_tile(const cplx<typename X::R>* s_H, cplx<typename X::R>* hcols, int x0,
                                               const X&) {
  constexpr int K = X::K, G = X::G, N = X::N, CL = X::N / XT;
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  for (int i = threadIdx.x; i < (ADJ ? NHA : NH) * K * XT; i += blockDim.x) {
    const int rr = i / XT, xt = i - rr * XT;
    const int f = rr / K, ky = rr - f * K;
    const int c = 2 * (ky / G) + (ADJ ? f >> 1 : f == 2 ? 1 : 0);
    cplx<typename X::R>* dst = cl.map_shared_rank(hcols, (unsigned)(c % CL));
    dst[(((c / CL) * G + ky % G) * 2 + (ADJ ? f & 1 : f == 2 ? 0 : f)) * N + x0 + xt] = s_H[rr * (XT + 1) + xt];
  }
}

// The products of one row in physical space.
template <typename R>
__device__ __forceinline__ cplx<R> rhs_p12(R u, R v, R bx, R by) {
  return mk<R>(fpm(u - v, u + v, bx - by, bx + by), fpm(bx, by, u, v));
}
template <typename R>
__device__ __forceinline__ R rhs_p3(R u, R v, R bx, R by) { return fpm(u, by, v, bx); }   // mhd_jax.py:163

// Rows x0 .. x0 + XT - 1 of state b, one group per row; s_G and s_H are the tile
// buffers (NG and NH rows of K x (XT + 1)).  They may be the same memory: a
// group reads and writes its own column of the tiles only, all reads first.
// CX (cluster-resident passes): s_G holds the tile unless load_g; the H tile
// goes to the column groups' rows at `hcols` unless that is null.
template <int XT, bool CX = false, class X>
__device__ __forceinline__ void row_rhs_body(const RowParams<typename X::R>& p, int b, int x0, const X& xf,
                                             cplx<typename X::R>* s_G, cplx<typename X::R>* s_H, bool load_g = true,
                                             cplx<typename X::R>* hcols = nullptr) {
  using R = typename X::R;
  constexpr int E = X::E, L = X::L, K = X::K, N = X::N;
  if (!CX || load_g) load_tile<R, N, XT>(s_G, p.G + (size_t)b * NG * K * N, NG * K, x0);
  __syncthreads();
  const int w = threadIdx.x / L;
  cplx<R> uv[E], bb[E];
  // pairs (u, v) and (B_x, B_y) without the mean field (mhd_jax.py:140-149)
  row_inverse<XT>(s_G, w, xf, uv, bb);
  cplx<R>* ph = p.phys ? const_cast<cplx<R>*>(phys_row<R, N>(p.phys + (size_t)b * p.phys_bstride, x0 + w)) : nullptr;
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const R u = uv[j].x, v = uv[j].y;
    const R bx = bb[j].x + p.b0x, by = bb[j].y + p.b0y;
    if (ph) { ph[xf.l + L * j] = uv[j]; ph[N + xf.l + L * j] = mk<R>(bx, by); }
    uv[j] = rhs_p12<R>(u, v, bx, by);
    bb[j] = mk<R>(rhs_p3<R>(u, v, bx, by), R(0));
  }
  row_forward<XT>(uv, bb, s_H, w, xf);
  __syncthreads();
  if constexpr (CX) {
    if (hcols) { scatter_h_tile<XT>(s_H, hcols, x0, xf); return; }
  }
  store_tile<R, N, XT>(p.H + (size_t)b * NH * K * N, s_H, NH * K, x0);
}

template <typename R, int N, int XT>
__global__ void __launch_bounds__(XT * Xf<R, N>::L) k_row_rhs(RowParams<R> p) {
  using X = Xf<R, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_x = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_G = s_x + X::smem(XT / X::G);
  const int tiles = N / XT;
  const int b = blockIdx.x / tiles, x0 = (blockIdx.x - b * tiles) * XT;
  load_tables<X>(s_x, p.tw);
  pdl_wait();
  pdl_trigger();
  if (p.ctl && p.ctl[b].done) return;   // whole block belongs to one batch element
  row_rhs_body<XT>(p, b, x0, X(s_x, threadIdx.x >> 5), s_G, s_G);
}

// ---------------------------------------------------------------------------
// Boundary transforms between real fields [B][2][N][N] and the box spectrum.
// ---------------------------------------------------------------------------

// Row pass of rfft2 restricted to ky < K: real rows of both channels -> H[B][2][K][N].
template <typename R>
struct RowFwdParams {
  const R* fields;    // [B][2][N][N]
  cplx<R>* H;         // [B][2][K][N]
  const cplx<R>* tw;
  int B;
};

template <typename R, int N, int XT>
__global__ void __launch_bounds__(XT * Xf<R, N>::L) k_row_to_box(RowFwdParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, K = X::K;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_x = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_H = s_x + X::smem(XT / X::G);
  const int tiles = N / XT;
  const int b = blockIdx.x / tiles, x0 = (blockIdx.x - b * tiles) * XT;
  load_tables<X>(s_x, p.tw);
  __syncthreads();
  const X xf(s_x, threadIdx.x >> 5);
  const int w = threadIdx.x / X::L, x = x0 + w;
  const R* u0 = p.fields + ((size_t)(b * 2 + 0) * N + x) * N;
  const R* u1 = p.fields + ((size_t)(b * 2 + 1) * N + x) * N;
  cplx<R> W[E];
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int y = X::pos(xf.l, j);
    W[j] = mk<R>(u0[y], u1[y]);
  }
  xf.template from_spec<false>(W);
  split_store<XT>(W, s_H, s_H + K * (XT + 1), w, xf);
  __syncthreads();
  store_tile<R, N, XT>(p.H + (size_t)b * 2 * K * N, s_H, 2 * K, x0);
}

// Column pass of rfft2: H columns -> box spectrum V (raw rfft2 values, no mask).
template <typename R>
struct ColBoxParams {
  const cplx<R>* H;   // [B][nf][K][N]
  cplx<R>* V;         // [B][nf][K][M] with batch stride vstride (elements)
  const cplx<R>* tw;
  long vstride;
  int B, nf;
};

// The boundary column passes number their columns (b f) K + ky consecutively:
// column `warp` G + group of warp `warp`.
template <typename R, int N>
__global__ void __launch_bounds__(128) k_col_to_box(ColBoxParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, K = X::K, M = X::M;
  __shared__ __align__(16) cplx<R> s_x[X::smem(COLWARPS)];
  load_tables<X>(s_x, p.tw);
  __syncthreads();
  const X xf(s_x, threadIdx.x >> 5);
  const int warp = blockIdx.x * COLWARPS + (threadIdx.x >> 5), cols = p.B * p.nf * K;
  if (warp * X::G >= cols) return;
  const int ci = warp * X::G + (int)(threadIdx.x & 31) / X::L;
  const bool act = ci < cols;
  const int col = act ? ci : cols - 1;   // col = (b*nf + f)*K + ky
  const cplx<R>* hin = p.H + (size_t)col * N;
  cplx<R> v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) v[j] = hin[xf.l + X::L * j];
  xf.template to_spec<false>(v);
  if (!act) return;
  const int b = col / (p.nf * K), fk = col - b * p.nf * K;
  cplx<R>* vout = p.V + (size_t)b * p.vstride + (size_t)fk * M;
#pragma unroll
  for (int j = 0; j < E; ++j) {
    if (X::none(j)) continue;
    const int slot = xf.slot(j);
    if (slot >= 0) vout[slot] = v[j];
  }
}

// Symmetry group action applied to a box spectrum value at (kx, ky) of channel c
// (reference: symmetry.shift_x / shift_reflect / rot180, jax_scripts/lib/symmetry.py:4-25).
// The source value must be read at kx_src = odd_ny ? -kx : kx.
struct SymOp {
  double sx;   // x shift
  double sy;   // y shift = ny * 2 pi / 8
  int odd;     // ny odd: reflect x and negate
  int rot;     // rot180: conj, channel signs [1, -1]
};

template <typename R>
__device__ __forceinline__ cplx<R> apply_sym(cplx<R> g, int kx_src, int ky, int c, const SymOp& s) {
  // masked wavenumbers: (0,0) is masked out, so both phases are 1 there
  const bool m = !(kx_src == 0 && ky == 0);
  double sn, cs;
  sincos(m ? (double)kx_src * s.sx : 0.0, &sn, &cs);
  cplx<R> a = cmul(mk<R>((R)cs, (R)sn), g);
  sincos(m ? (double)ky * s.sy : 0.0, &sn, &cs);   // ky is unchanged by the x reflection
  a = cmul(mk<R>((R)cs, (R)sn), a);
  if (s.odd) { a.x = -a.x; a.y = -a.y; }
  if (s.rot) { a.y = -a.y; if (c == 1) { a.x = -a.x; a.y = -a.y; } }
  return a;
}

// Column inverse from a box spectrum (2 channels) -> G2[B][2][K][N], with an
// optional symmetry action, optional scaling and optional multiplier (i kx).
template <typename R>
struct ColFromBoxParams {
  const cplx<R>* V;   // [B][2][K][M]
  cplx<R>* G;         // [B][2][K][N]
  const cplx<R>* tw;
  const double* sx;   // [B] or null
  int sx_shared;      // sx[0] applies to every batch element
  double sy;
  int odd, rot, use_sym;
  int mult_ikx;       // multiply by i kx (masked) before the inverse
  int B;
};

template <typename R, int N>
__global__ void __launch_bounds__(128) k_col_from_box(ColFromBoxParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, K = X::K, M = X::M;
  __shared__ __align__(16) cplx<R> s_x[X::smem(COLWARPS)];
  load_tables<X>(s_x, p.tw);
  __syncthreads();
  const X xf(s_x, threadIdx.x >> 5);
  const int warp = blockIdx.x * COLWARPS + (threadIdx.x >> 5), cols = p.B * 2 * K;
  if (warp * X::G >= cols) return;
  const int ci = warp * X::G + (int)(threadIdx.x & 31) / X::L;
  const bool act = ci < cols;
  const int col = act ? ci : cols - 1;   // col = (b*2 + c)*K + ky
  const int ky = col % K, bc = col / K, c = bc & 1, b = bc >> 1;
  const cplx<R>* vin = p.V + (size_t)col * M;
  SymOp so; so.sx = p.sx ? p.sx[p.sx_shared ? 0 : b] : 0.0; so.sy = p.sy; so.odd = p.odd; so.rot = p.rot;
  const R inv_n2 = R(1) / (R(N) * R(N));
  cplx<R> v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) {
    v[j] = mk<R>(0, 0);
    if (X::none(j)) continue;
    const int slot = xf.slot(j);
    if (slot < 0) continue;
    const int kx = slot_to_kx(slot, X::KMAX, M);
    cplx<R> val;
    if (p.use_sym) {
      const int ksrc = so.odd ? -kx : kx;
      const int ssrc = ksrc >= 0 ? ksrc : ksrc + M;
      val = apply_sym<R>(vin[ssrc], ksrc, ky, c, so);
    } else {
      val = vin[slot];
    }
    if (p.mult_ikx) val = cimul(val, (kx == 0 && ky == 0) ? R(0) : (R)kx);
    v[j] = cscale(val, inv_n2);
  }
  xf.template from_spec<true, true>(v);
  if (!act) return;
  cplx<R>* gout = p.G + (size_t)col * N;
#pragma unroll
  for (int j = 0; j < E; ++j) gout[xf.l + X::L * j] = v[j];
}

// Row c2r of the two channels G2[B][2][K][N] -> real fields.
//   mode 0: out = u
//   mode 1: out = base - u   (objective residual irfft2(f0 - f) with irfft2(f0) = base)
//   mode 2: out = base + u
// Optionally accumulates per-row sums of out^2 (loss) into rowsq[B][N].
template <typename R>
struct RowFromBoxParams {
  const cplx<R>* G;   // [B][2][K][N]
  R* out;             // [B][2][N][N]
  const R* base;      // [B][2][N][N] or null
  double* rowsq;      // [B][N] or null
  const cplx<R>* tw;
  int B, mode;
};

template <typename R, int N, int XT>
__global__ void __launch_bounds__(XT * Xf<R, N>::L) k_row_from_box(RowFromBoxParams<R> p) {
  using X = Xf<R, N>;
  constexpr int E = X::E, K = X::K;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_x = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_G = s_x + X::smem(XT / X::G);
  const int tiles = N / XT;
  const int b = blockIdx.x / tiles, x0 = (blockIdx.x - b * tiles) * XT;
  load_tables<X>(s_x, p.tw);
  load_tile<R, N, XT>(s_G, p.G + (size_t)b * 2 * K * N, 2 * K, x0);
  __syncthreads();
  const X xf(s_x, threadIdx.x >> 5);
  const int w = threadIdx.x / X::L, x = x0 + w;
  cplx<R> z[E];
#pragma unroll
  for (int j = 0; j < E; ++j) z[j] = packed_pair<R, N, XT>(s_G, s_G + K * (XT + 1), X::pos(xf.l, j), w);
  xf.template from_spec<true>(z);
  R* o0 = p.out + ((size_t)(b * 2 + 0) * N + x) * N;
  R* o1 = p.out + ((size_t)(b * 2 + 1) * N + x) * N;
  const R* b0 = p.base ? p.base + ((size_t)(b * 2 + 0) * N + x) * N : nullptr;
  const R* b1 = p.base ? p.base + ((size_t)(b * 2 + 1) * N + x) * N : nullptr;
  double sq = 0.0;
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int y = xf.l + X::L * j;
    R a = z[j].x, c = z[j].y;
    if (p.mode == 1) { a = b0[y] - a; c = b1[y] - c; }
    else if (p.mode == 2) { a = b0[y] + a; c = b1[y] + c; }
    o0[y] = a; o1[y] = c;
    sq += (double)a * (double)a + (double)c * (double)c;
  }
  if (p.rowsq) {
#pragma unroll
    for (int o = X::L / 2; o >= 1; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (xf.l == 0) p.rowsq[(size_t)b * N + x] = sq;
  }
}

// ---------------------------------------------------------------------------
// Small elementwise kernels
// ---------------------------------------------------------------------------

// Full rfft2 layout [B][2][N][N/2+1] <-> box [B][2][K][M].
template <typename R>
__global__ void k_gather_box(const cplx<R>* full, cplx<R>* box, int n, int B) {
  const Geom g = make_geom(n);
  const int nh = n / 2 + 1;
  const long total = (long)B * 2 * g.K * g.M;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int slot = i % g.M; const long r = i / g.M; const int ky = r % g.K; const long bc = r / g.K;
    const int kx = slot_to_kx(slot, g.kmax, g.M);
    const int pos = kx >= 0 ? kx : kx + n;
    box[i] = full[(bc * n + pos) * nh + ky];
  }
}

template <typename R>
__global__ void k_scatter_box(const cplx<R>* box, cplx<R>* full, int n, int B) {
  const Geom g = make_geom(n);
  const int nh = n / 2 + 1;
  const long total = (long)B * 2 * n * nh;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int ky = i % nh; const long r = i / nh; const int pos = r % n; const long bc = r / n;
    const int slot = (ky < g.K) ? pos_to_slot(pos, n, g.kmax, g.M) : -1;
    full[i] = slot >= 0 ? box[(bc * g.K + ky) * g.M + slot] : mk<R>(0, 0);
  }
}

// Lawson-RK4 setup: h = (T/nc)/ms and e = exp(h/2 L) * mask per batch element.
template <typename R>
__global__ void k_rk4_setup(const double* T, int nc, int ms, StepCtl* ctl, R* Etab, int n, double nu, double eta, int B) {
  const Geom g = make_geom(n);
  const long per = 2L * g.K * g.M;
  const long total = (long)B * per;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int b = (int)(i / per);
    const double tseg = T[b] / (double)nc;          // loss_functions.py:63 T/num_checkpoints
    const R h = (R)(tseg / (double)ms);              // timestepping.py:69 h = t/steps
    if (i % per == 0) { ctl[b].t = tseg; ctl[b].h = (double)h; }
    const int slot = i % g.M; const long r = i / g.M; const int ky = r % g.K; const int c = (r / g.K) & 1;
    const int kx = slot_to_kx(slot, g.kmax, g.M);
    const R L = diss_L<R>((R)kx, (R)ky, (R)(c == 0 ? nu : eta));
    const bool msk = !(kx == 0 && ky == 0);
    Etab[i] = msk ? exp(h / R(2) * L) : R(0);        // timestepping.py:70-72
  }
}

// out -= P_sym(rest): the symmetry action on modes outside the box, which in
// real space is x -> -x with negation (odd ny) and a 180 degree rotation with
// channel signs [1, -1] (rot); shift_x and the y-phase of shift_reflect use
// masked wavenumbers and leave these modes unchanged (symmetry.py:4-25).
template <typename R>
__global__ void k_sub_sym_phys(R* out, const R* rest, int odd, int rot, int n, int B) {
  const long total = (long)B * 2 * n * n;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int y = i % n; const long r = i / n; const int x = r % n; const long bc = r / n; const int c = bc & 1;
    const int sx = (odd ? -1 : 1) * (rot ? -1 : 1), sy = rot ? -1 : 1;
    const int xs = ((sx * x) % n + n) % n, ys = ((sy * y) % n + n) % n;
    R f = rest[(bc * n + xs) * n + ys];
    if (odd) f = -f;
    if (rot && c == 1) f = -f;
    out[i] -= f;
  }
}

// Per-row sums of squares of real fields [B][2][N][N]: rowsq[b][x] (one warp per (b, x)).
template <typename R>
__global__ void k_rowsq(const R* f, double* rowsq, int n) {
  const int bx = blockIdx.x, b = bx / n, x = bx % n;
  double s = 0.0;
  for (int c = 0; c < 2; ++c) {
    const R* row = f + ((size_t)(b * 2 + c) * n + x) * n;
    for (int y = threadIdx.x; y < n; y += 32) s += (double)row[y] * (double)row[y];
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x == 0) rowsq[bx] = s;
}

template <typename R>
__global__ void k_axpy(R* y, const R* x, R a, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) y[i] += a * x[i];
}

// Slot pool: initialise one slot's control (steps_total = 0 marks it inactive).
static __global__ void k_pool_init(StepCtl* ctl, int first, int count, int steps_total) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  StepCtl& c = ctl[first + i];
  c.steps_total = steps_total; c.steps_done = 0; c.done = steps_total > 0 ? 0 : 1;
  c.attempts = 0; c.accepted = 0; c.rejected = 0; c.pending_accept = 0;
}

// Slot pool: count `steps` finished steps per active slot; a slot whose budget is
// spent is marked done and skipped by every later launch.
static __global__ void k_pool_count(StepCtl* ctl, int B, int steps = 1) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  StepCtl& c = ctl[b];
  if (c.done || c.steps_total <= 0) return;
  c.steps_done += steps;
  if (c.steps_done >= c.steps_total) c.done = 1;
}

// Deterministic per-batch reduction of row partials: out[b] = scale * sum_x rowsq[b][x].
static __global__ void k_reduce_rows(const double* rowsq, double* out, int n, int B, double scale) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  double s = 0.0;
  for (int x = 0; x < n; ++x) s += rowsq[(size_t)b * n + x];
  out[b] = s * scale;
}

}  // namespace ecs
