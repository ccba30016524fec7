// Adaptive Lawson-RK4(3) ("EARK43") stepper, device resident.
//
// Reference: lawson_rk43 (jax_scripts/lib/timestepping.py:151-335).  One
// attempted step is five column launches (A..E) interleaved with four RHS row
// launches and one error row launch; the error reduction's last block performs
// the accept/reject decision and the step-size update on the device, so no host
// round trip happens per attempt.  Candidates that completed (|s-1| < 1e-10)
// skip all work, as the reference's lax.cond(complete, identity, do_step) does.
#pragma once

#include "kernels.cuh"

namespace ecs {

// Per-candidate state slots of the stepper, each a box vector [2][K][M].
// S_E holds (e, e L h/2) of the current attempt, e = exp(t L h/2) (written at
// stage A, read at stage C).
enum Rk43Slot { S_X0 = 0, S_K1, S_XE, S_K1E, S_K2, S_K3, S_X2, S_K4, S_XF, S_K5, S_E, S_NSLOT };
// Trajectory record per attempt (primal values needed by tangent/adjoint):
// start state, carried k1 (before twiddles), k2..k5, the stage inputs, and the
// attempt's integrating factor as (e, e L h/2) with e = exp(t L h/2), computed
// once here so that the tangent and adjoint passes do not recompute it per
// tangent (the same expression, so the same values).
enum Rk43Rec { RR_X0 = 0, RR_K1, RR_K2, RR_K3, RR_K4, RR_K5, RR_Y2, RR_Y3, RR_Y4, RR_XF, RR_E, RR_NREC };

enum Rk43Stage : int {
  R43_START = 6,  // no RHS input; inverse transforms of x0
  R43_INIT = 0,   // RHS of x0 finished: k1 = t v(x0)
  R43_A = 1,      // start of an attempt: promote accepted state, twiddle, input Y2
  R43_B = 2,      // k2 finished, input Y3
  R43_C = 3,      // k3 finished, twiddles, input Y4
  R43_D = 4,      // k4 finished, xf, input xf
  R43_E = 5,      // k5 finished, error field d = h (k5 - k4)/6 -> 2 inverse columns
};

template <typename R>
struct Col43Params {
  const cplx<R>* H;     // [B][NH][K][N]
  cplx<R>* G;           // [B][NG][K][N]
  cplx<R>* S;           // [B][S_NSLOT][2][K][M]
  StepCtl* ctl;         // [B]
  const cplx<R>* fhat;  // [K][M]
  const cplx<R>* tw;
  cplx<R>* rec;         // optional [B][cap][RR_NREC][2][K][M]
  int cap;
  R nu, eta;
  int B, stage;
};

// Slots (bits of Rk43Slot) that the algebra of an attempt stage reads; they are
// loaded together before the stage's stores.
__host__ __device__ constexpr unsigned r43_smask(int stage) {
  return stage == R43_START ? (1u << S_X0)
       : stage == R43_B ? (1u << S_XE)
       : stage == R43_C ? (1u << S_XE) | (1u << S_K1E) | (1u << S_K2) | (1u << S_E)
       : stage == R43_D ? (1u << S_K1) | (1u << S_K2) | (1u << S_K3) | (1u << S_X2)
       : stage == R43_E ? (1u << S_K4) : 0u;
}
// What an attempt stage needs beside its operands: the candidate's step and the column's
// record rows of the attempt (or null).
template <typename R>
struct R43Col {
  R t, h;
  int pend;
  cplx<R>* rec;
  __device__ __forceinline__ R43Col(const Col43Params<R>& p, const StepCtl& c, int b, int ch, int ky, size_t VEC, int K, int M) {
    t = (R)c.t; h = (R)c.h; pend = c.pending_accept;
    rec = p.rec ? p.rec + ((size_t)b * p.cap + (c.attempts < p.cap ? c.attempts : p.cap - 1)) * RR_NREC * VEC +
                      ((size_t)ch * K + ky) * M
                : nullptr;
  }
};
// Slots that stage A reads: the carried state and k1.
__host__ __device__ constexpr unsigned r43_amask(int pend) {
  return pend ? (1u << S_XF) | (1u << S_K5) : (1u << S_X0) | (1u << S_K1);
}

__host__ __device__ constexpr unsigned r43_omask(int stage) { return stage == R43_A ? r43_amask(0) : r43_smask(stage); }

// The algebra of an attempt stage at one mode: the stage input from the derivative v.
// SV(q) reads and SW(q, a) writes slot q (stage A reads its two operands as xs and ks).
template <int STAGE, typename R, class SVf, class SWf>
__device__ __forceinline__ cplx<R> r43_algebra(const R43Col<R>& c, R L, cplx<R> v, cplx<R> xs, cplx<R> ks, size_t VEC,
                                               int slot, SVf&& SV, SWf&& SW) {
  const R t = c.t, h = c.h;
  auto put = [&](int q, cplx<R> a) { if (c.rec) c.rec[q * VEC + slot] = a; };
  const cplx<R> kv = cscale_rn(v, t);              // mod_vel_fn = t * vel_fn (timestepping.py:243)
  cplx<R> xin = mk<R>(0, 0);
  switch (STAGE) {
    case R43_START: xin = SV(S_X0); break;
    case R43_INIT: SW(S_K1, kv); break;
    case R43_A: {                                  // :266-270
      if (c.pend) { SW(S_X0, xs); SW(S_K1, ks); }
      put(RR_X0, xs); put(RR_K1, ks);
      const R e = exp((t * L) * h / R(2));         // e = exp(mod_L * h/2), not masked (:263)
      const cplx<R> eg = mk<R>(e, e * (L * h * R(0.5)));
      SW(S_E, eg);
      put(RR_E, eg);
      const cplx<R> xe = cscale_rn(xs, e), k1e = cscale_rn(ks, e);
      SW(S_XE, xe); SW(S_K1E, k1e);
      xin = cadd(xe, cscale(cscale_rn(k1e, h), R(0.5)));
      put(RR_Y2, xin);
    } break;
    case R43_B: {                                  // :270-271
      SW(S_K2, kv);
      put(RR_K2, kv);
      xin = cadd(SV(S_XE), cscale(cscale_rn(kv, h), R(0.5)));
      put(RR_Y3, xin);
    } break;
    case R43_C: {                                  // :271-280
      put(RR_K3, kv);
      const R e = SV(S_E).x;
      const cplx<R> x2 = cscale_rn(SV(S_XE), e);
      const cplx<R> k1ee = cscale_rn(SV(S_K1E), e);
      const cplx<R> k2e = cscale_rn(SV(S_K2), e);
      const cplx<R> k3e = cscale_rn(kv, e);
      SW(S_X2, x2); SW(S_K1, k1ee);                // k1 carried on rejection is e^2 k1 (:297)
      SW(S_K2, k2e); SW(S_K3, k3e);
      xin = cadd_scaled_rn(x2, k3e, h);
      put(RR_Y4, xin);
    } break;
    case R43_D: {                                  // :280-281
      SW(S_K4, kv);
      put(RR_K4, kv);
      const cplx<R> acc = cadd(cadd(cadd(cdiv_k<6>(SV(S_K1)), cdiv_k<3>(SV(S_K2))), cdiv_k<3>(SV(S_K3))), cdiv_k<6>(kv));
      xin = cadd_scaled_rn(SV(S_X2), acc, h);
      SW(S_XF, xin);
      put(RR_XF, xin);
    } break;
    default: {                                     // R43_E: :282, :288
      SW(S_K5, kv);
      put(RR_K5, kv);
      xin = cdiv_k<6>(cscale_rn(csub(kv, SV(S_K4)), h));
    } break;
  }
  return xin;
}

// The derivative of channel ch at mode (slot, ky): r plus the forcing.
template <typename R, class Forcing>
__device__ __forceinline__ cplx<R> with_forcing(cplx<R> r, const Forcing& forcing, int ch, int ky, int slot) {
  return ch == 0 && !(slot == 0 && ky == 0) ? cadd(r, forcing(slot)) : r;   // r is zero at (0,0)
}

// An attempt stage of one column; `rows`: shared room for its operands.
template <int STAGE, class X>
__device__ __forceinline__ void col_rk43_body(const Col43Params<typename X::R>& p, const ColId<X>& id, const X& xf,
                                              cplx<typename X::R>* rows) {
  using R = typename X::R;
  constexpr int N = X::N, E = X::E, K = X::K, M = X::M;
  constexpr size_t VEC = (size_t)2 * K * M;
  const int ch = id.ch, b = id.b, ky = id.ky;
  if (p.ctl[b].done) return;
  const R43Col<R> c(p, p.ctl[b], b, ch, ky, VEC, K, M);
  cplx<R>* S = p.S + (size_t)b * S_NSLOT * VEC + ((size_t)ch * K + ky) * M;
  constexpr bool has_rhs = STAGE != R43_A && STAGE != R43_START;
  constexpr int n = popc_c(r43_omask(STAGE));
  Operands<X, r43_omask(STAGE)> op(rows);
  const TableRow<X, has_rhs> forcing(rows + n * M, p.fhat + ky * M);
  const TableRow<X, STAGE != R43_INIT && STAGE != R43_E> mu(rows + (n + 1) * M, mu_row<X>(p.tw, ky));
  // stage A: the carried state and k1, which an accepted attempt left in S_XF and S_K5
  const size_t at_x = STAGE == R43_A && c.pend ? (S_XF - S_X0) * VEC : 0, at_k = STAGE == R43_A && c.pend ? (S_K5 - S_K1) * VEC : 0;
  auto from = [&](int q) { return S + q * VEC + (q == S_X0 ? at_x : at_k); };
  if constexpr (STAGE == R43_A) op.begin(from); else op.begin(S, VEC);
  cplx<R> r[E], x[E];
  if (has_rhs) col_load_rhs(p.H, b, ch, ky, xf, r);
  if constexpr (STAGE == R43_A) op.load(from, true, xf); else op.load(S, VEC, true, xf);
  const R coeff = ch == 0 ? p.nu : p.eta;
#pragma unroll
  for (int i = 0; i < E; ++i) {
    x[i] = mk<R>(0, 0);
    const int slot = xf.slot(i);
    if (slot < 0) continue;
    const cplx<R> v = has_rhs ? with_forcing<R>(r[i], forcing, ch, ky, slot) : mk<R>(0, 0);
    x[i] = r43_algebra<STAGE>(c, diss_L<R>(xf.kx(i), (R)ky, coeff), v, STAGE == R43_A ? op.get(S_X0, i, slot) : mk<R>(0, 0),
                              STAGE == R43_A ? op.get(S_K1, i, slot) : mk<R>(0, 0), VEC, slot,
                              [&](int q) { return op.get(q, i, slot); },
                              [&](int q, cplx<R> a) { S[q * VEC + slot] = a; });
  }
  if (STAGE == R43_INIT) return;
  if (STAGE == R43_E) col_inverse1(x, p.G, NG, b, ch, ky, true, xf, R(1) / (R(N) * R(N)));
  else col_inverse_uv(x, p.G, b, ch, ky, true, xf, mu);
}

template <typename R, int N, int STAGE>
__global__ void __launch_bounds__(COLWARPS * 32, 1) k_col_rk43(Col43Params<R> p) {
  using X = Xf<R, N>;
  ECS_COL_PROLOGUE(popc_c(r43_omask(STAGE)), 2);   // the forcing, the multipliers
  col_rk43_body<STAGE>(p, id, xf, rows);
}

// Error norm max|irfft2(d)| of the two channels (timestepping.py:288-291) with
// the accept/reject decision and h update done by the last block of each
// candidate (timestepping.py:294-310).
template <typename R>
struct RowErrParams {
  const cplx<R>* G;     // [B][NG][K][N], fields 0,1 hold the inverse columns of d
  StepCtl* ctl;
  const cplx<R>* tw;
  double atol;
  double* rec_h;        // optional [B][cap] attempted step sizes ("hs", :239,:294)
  int* rec_acc;         // optional [B][cap] accept flags
  int cap;
  int B;
};

__device__ __forceinline__ void rk43_control(StepCtl& c, double atol, double err, double* rec_h, int* rec_acc) {
  const int a = c.attempts;
  const bool accept = err < atol;                          // :297 (false for NaN)
  if (rec_h) rec_h[a] = c.h;                               // :294
  if (rec_acc) rec_acc[a] = accept ? 1 : 0;
  if (accept) { c.s = c.s + c.h; c.accepted += 1; c.pending_accept = 1; }
  else { c.rejected += 1; c.pending_accept = 0; }
  c.fevals += 4;                                           // :285
  double hn = isnan(err) ? c.h / 2 : c.h * 0.9 * pow(atol / err, 0.25);   // :300-302
  const double ov = c.s + hn - 1.0;                        // :304-307 h - relu(s + h - 1)
  hn = hn - (isnan(ov) ? ov : (ov > 0.0 ? ov : 0.0));
  c.h = hn;
  c.err = err;
  c.attempts = a + 1;
  c.done = fabs(c.s - 1.0) < 1e-10 ? 1 : 0;                // :313
}

// max |irfft2(d)| over rows x0 .. x0 + XT - 1 of state b (the inverse column
// transforms of d in G fields 0 and 1, or in the tile s_G already unless load_g), one
// warp per row; s_max holds one value per warp; valid in every thread.
template <int XT, class X>
__device__ __forceinline__ double row_err_max(const cplx<typename X::R>* G, int b, int x0, const X& xf,
                                              cplx<typename X::R>* s_G, double* s_max, bool load_g = true) {
  using R = typename X::R;
  constexpr int N = X::N;
  if (load_g) load_tile<R, N, XT>(s_G, G + (size_t)b * NG * X::K * N, 2 * X::K, x0);
  __syncthreads();
  cplx<R> z[X::E];
  load_pair<XT>(s_G, s_G + X::K * (XT + 1), threadIdx.x / X::L, xf, z);
  xf.template to_spec<true, true>(z);
  double m = 0.0;
#pragma unroll
  for (int j = 0; j < X::E; ++j) {
    const double a = fabs((double)z[j].x), bb = fabs((double)z[j].y);
    m = (a > m || isnan(a)) ? a : m;
    m = (bb > m || isnan(bb)) ? bb : m;
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const double q = __shfl_xor_sync(0xffffffffu, m, o);
    m = (q > m || isnan(q)) ? q : m;
  }
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = m;
  __syncthreads();
  double bm = s_max[0];
  for (int i = 1; i < XT / X::G; ++i) bm = (s_max[i] > bm || isnan(s_max[i])) ? s_max[i] : bm;
  return bm;
}

template <typename R, int N, int XT>
__global__ void __launch_bounds__(XT * Xf<R, N>::L) k_row_err(RowErrParams<R> p) {
  using X = Xf<R, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<R>* s_x = reinterpret_cast<cplx<R>*>(smem_raw);
  cplx<R>* s_G = s_x + X::smem(XT / X::G);
  __shared__ double s_max[XT];
  __shared__ int s_last;
  const int tiles = N / XT;
  const int b = blockIdx.x / tiles, x0 = (blockIdx.x - b * tiles) * XT;
  load_tables<X>(s_x, p.tw);
  pdl_wait();
  pdl_trigger();
  StepCtl& c = p.ctl[b];
  if (c.done) return;
  const double bm = row_err_max<XT>(p.G, b, x0, X(s_x, threadIdx.x >> 5), s_G, s_max);
  if (threadIdx.x == 0) {
    // non-negative doubles (and NaN with the sign bit clear) order like their bit patterns
    atomicMax(&c.err_bits, (unsigned long long)__double_as_longlong(fabs(bm)));
    __threadfence();
    const unsigned prev = atomicAdd(&c.err_blocks, 1u);
    s_last = (prev == (unsigned)(tiles - 1));
  }
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    __threadfence();
    const double err = __longlong_as_double((long long)atomicAdd(&c.err_bits, 0ull));
    const int a = c.attempts;
    rk43_control(c, p.atol, err, p.rec_h && a < p.cap ? p.rec_h + (size_t)b * p.cap : nullptr,
                 p.rec_acc && a < p.cap ? p.rec_acc + (size_t)b * p.cap : nullptr);
    c.err_bits = 0ull;
    c.err_blocks = 0u;
  }
}

// Initial control state: t = T, h = h0, s = 0 (timestepping.py:255).
static __global__ void k_rk43_setup(const double* T, double h0, StepCtl* ctl, int B) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  StepCtl c;
  c.t = T[b]; c.h = h0; c.s = 0.0; c.err = 0.0;
  c.accepted = 0; c.rejected = 0; c.fevals = 1; c.done = 0;
  c.pending_accept = 0; c.attempts = 0; c.err_bits = 0ull; c.err_blocks = 0u; c.pad = 0;
  ctl[b] = c;
}

// Final state = x carried by the loop: xf if the last attempt was accepted.
template <typename R>
__global__ void k_rk43_resolve(cplx<R>* S, const StepCtl* ctl, cplx<R>* out, int n, int B) {
  const Geom g = make_geom(n);
  const size_t VEC = (size_t)2 * g.K * g.M;
  const long total = (long)B * VEC;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int b = (int)(i / VEC);
    const size_t o = i - (size_t)b * VEC;
    const cplx<R>* Sb = S + (size_t)b * S_NSLOT * VEC;
    out[i] = ctl[b].pending_accept ? Sb[S_XF * VEC + o] : Sb[S_X0 * VEC + o];
  }
}

static __global__ void k_count_done(const StepCtl* ctl, int* count, int B) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    int s = 0;
    for (int b = 0; b < B; ++b) s += ctl[b].done;
    *count = s;
  }
}

}  // namespace ecs
