// Transforms of length N in {64, 128, 256}, in two layouts (struct Xf below).
//
// The warp layout, which every pass uses but the column passes of batched FP64 tangents
// at N = 128: one transform per warp.  Lane l holds E = N/32 complex values v[j] at
// "positions" e = l + 32*j.
//
//  * fft_dif : natural-order input  -> permuted output (lane l, register j holds X[spec_pos<N>(l, j)])
//  * fft_dit : permuted input       -> natural-order output
//
// Both are unnormalised.  FWD uses exp(-2 pi i k/N), INV uses exp(+2 pi i k/N).
//
// One radix-E pass over the register digits (the length-E DFT over
// j, then the twiddles W_N^{l k1}), after which every register digit is a
// finished frequency digit and the remaining 32-point DFTs run over the lane
// digits.  Those are five "half-swap" radix-2 stages: stage t (lane bit t, span
// S = 2^t) swaps lane bit t with a finished register bit rb -- the lane whose
// bit t is c keeps the values whose register bit rb is c and sends the other
// half to lane ^ S -- so that the butterfly over bit t becomes register-local,
// with its sign taken from c:
//   lower = keep + recv,  upper = (1 - 2c) (keep - recv) W_{2S}^{l mod S}.
// Each lane sends E/2 values per stage (a plain shuffle butterfly sends all E),
// and no shared memory is used beyond the tables.  The DIT is the transposed
// sequence (each stage's butterfly transposed and swapped back, then the
// twiddles and the radix-E DFT).  The stage order (t, rb) and the resulting
// output permutation spec_pos are listed below for each N.
//
// Twiddles come from a table tw[k] = exp(-2 pi i k / N), k in [0, N/2),
// computed on the host in long double, and expanded on the host (twiddle_image)
// into the shared-memory layout: one contiguous sub-table per index stride
// r = 1, 2, 4, ...:
//   s_tw[tw_off(N, r) + i] = tw[i r],  i < N / (2 r),  tw_off(N, r) = N - N / r,
// so that the lanes of a stage read consecutive entries, followed by the
// radix-E pass's table s_tw[N + (k1-1)*32 + l] = W_N^{l k1}, k1 = 1..E-1.
//
// The group layout (FP64 at N = 128): two transforms per warp, each on 16 lanes of 8
// values (x[l + 16 j] in register j), natural order in and out: radix 16 (its last
// butterflies across lanes l, l + 8 after a half swap), twiddles, the transposition of the
// values through the group's N-entry shared buffer, radix 8.  The half-swap form above
// spends most of its issue slots on selects and shuffles (a 128-point transform: 245
// instructions per warp, 100 of them FP64); this form has few of either and 8 to 16
// shared-memory accesses per lane and transform.  The buffer is swizzled (entry (k, l) of
// output digit k at k 8 + (l ^ (k mod 8))): eight lanes' 16-byte accesses fall on different
// banks in both directions.  What it gives per launch stands at with_layout.
#pragma once

#include "common.cuh"

#include <math.h>

namespace ecs {

__host__ __device__ constexpr int tw_first(int N) { return (N / 32 - 1) * 32; }
// Shared-memory twiddle entries and the offset of the stride-r sub-table.
__host__ __device__ constexpr int tw_smem(int N) { return N + tw_first(N); }
__host__ __device__ constexpr int tw_off(int N, int r) { return N - N / r; }
template <typename R, bool INV>
__device__ __forceinline__ cplx<R> twid(const cplx<R>* __restrict__ tw, int idx) {
  cplx<R> w = tw[idx];
  if (INV) w.y = -w.y;
  return w;
}

// Multiply by -i (forward) or +i (inverse): W_4^1.
template <typename R, bool INV>
__device__ __forceinline__ cplx<R> mul_mi(cplx<R> a) {
  return INV ? mk<R>(-a.y, a.x) : mk<R>(a.y, -a.x);
}

// Multiply by W_8^1 = (1 -+ i) / sqrt(2).
template <typename R, bool INV>
__device__ __forceinline__ cplx<R> mul_w8(cplx<R> a) {
  const R c = R(0.70710678118654752440084436210484904);
  // products rounded on their own (no contraction with the following sums)
  return INV ? mk<R>(mul_rn(a.x - a.y, c), mul_rn(a.x + a.y, c)) : mk<R>(mul_rn(a.x + a.y, c), mul_rn(a.y - a.x, c));
}

// ---------------------------------------------------------------------------
// Output permutation: lane L, register t holds X[spec_pos<N>(L, t)] (Li, ti
// are the bits of L and t).
//   N =  64: stages (t, rb) = (4,0) (3,0) (2,0) (1,0) (0,0);
//            k = L4 + 2 L3 + 4 L2 + 8 L1 + 16 L0 + 32 t0
//   N = 128: stages (4,0) (3,1) (2,0) (1,1) (0,0);
//            k = k1 + 4 k2, k1 = L4 + 2 L3, k2 = L2 + 2 L1 + 4 L0 + 8 t1 + 16 t0
//   N = 256: stages (4,0) (3,1) (2,2) (1,0) (0,1);
//            k = k1 + 8 k2, k1 = L4 + 2 L3 + 4 L2, k2 = L1 + 2 L0 + 4 t2 + 8 t0 + 16 t1
// ---------------------------------------------------------------------------
template <int N> __host__ __device__ __forceinline__ int spec_pos(int L, int t) {
  auto b = [](int x, int i) { return (x >> i) & 1; };
  if constexpr (N == 64) {
    return b(L, 4) + 2 * b(L, 3) + 4 * b(L, 2) + 8 * b(L, 1) + 16 * b(L, 0) + 32 * b(t, 0);
  } else if constexpr (N == 128) {
    return b(L, 4) + 2 * b(L, 3) + 4 * (b(L, 2) + 2 * b(L, 1) + 4 * b(L, 0) + 8 * b(t, 1) + 16 * b(t, 0));
  } else {
    return b(L, 4) + 2 * b(L, 3) + 4 * b(L, 2) + 8 * (b(L, 1) + 2 * b(L, 0) + 4 * b(t, 2) + 8 * b(t, 0) + 16 * b(t, 1));
  }
}

// Stage list: register bit swapped out at lane bit t.
template <int N, int T> struct StageRB {
  static constexpr int v = N == 64 ? 0 : N == 128 ? ((T == 3 || T == 1) ? 1 : 0)
                                                   : (T == 4 ? 0 : T == 3 ? 1 : T == 2 ? 2 : T == 1 ? 0 : 1);
};

// Length-E DFT over the register index, natural order in and out.
template <typename R, bool INV>
__device__ __forceinline__ void dft4(cplx<R>& a0, cplx<R>& a1, cplx<R>& a2, cplx<R>& a3) {
  const cplx<R> s02 = cadd(a0, a2), d02 = csub(a0, a2), s13 = cadd(a1, a3), d13 = mul_mi<R, INV>(csub(a1, a3));
  a0 = cadd(s02, s13); a1 = cadd(d02, d13); a2 = csub(s02, s13); a3 = csub(d02, d13);
}

template <typename R, bool INV, int E>
__device__ __forceinline__ void dft_reg(cplx<R> (&x)[E]) {
  if constexpr (E == 2) {
    const cplx<R> a = x[0], b = x[1];
    x[0] = cadd(a, b); x[1] = csub(a, b);
  } else if constexpr (E == 4) {
    dft4<R, INV>(x[0], x[1], x[2], x[3]);
  } else {
    // radix-2 split: a_j = x_j + x_{j+4} (even outputs), b_j = (x_j - x_{j+4}) W_8^j (odd outputs)
    cplx<R> a0 = cadd(x[0], x[4]), a1 = cadd(x[1], x[5]), a2 = cadd(x[2], x[6]), a3 = cadd(x[3], x[7]);
    cplx<R> b0 = csub(x[0], x[4]);
    cplx<R> b1 = mul_w8<R, INV>(csub(x[1], x[5]));
    cplx<R> b2 = mul_mi<R, INV>(csub(x[2], x[6]));
    cplx<R> b3 = mul_mi<R, INV>(mul_w8<R, INV>(csub(x[3], x[7])));
    dft4<R, INV>(a0, a1, a2, a3);
    dft4<R, INV>(b0, b1, b2, b3);
    x[0] = a0; x[2] = a1; x[4] = a2; x[6] = a3;
    x[1] = b0; x[3] = b1; x[5] = b2; x[7] = b3;
  }
}

// The radix-E pass (DIF order: DFT, then W_N^{l k1}) and its transpose.
template <typename R, bool INV, int NT, int N, bool TRANSPOSED>
__device__ __forceinline__ void first_pass(cplx<R> (*const (&v)[NT])[N / 32], const cplx<R>* tw, int lane) {
  constexpr int E = N / 32;
  const cplx<R>* t1 = tw + N;
  if constexpr (!TRANSPOSED) {
#pragma unroll
    for (int a = 0; a < NT; ++a) dft_reg<R, INV, E>(*v[a]);
  }
#pragma unroll
  for (int k = 1; k < E; ++k) {
    const cplx<R> w = twid<R, INV>(t1, (k - 1) * 32 + lane);
#pragma unroll
    for (int a = 0; a < NT; ++a) (*v[a])[k] = cmul((*v[a])[k], w);
  }
  if constexpr (TRANSPOSED) {
#pragma unroll
    for (int a = 0; a < NT; ++a) dft_reg<R, INV, E>(*v[a]);
  }
}

// (1 - 2c) W_{2S}^{lane mod S} of a half-swap stage (W = 1 for S = 1; for
// S = 2 only the sign, the W_4 factor is applied as a swap).
template <typename R, bool INV, int N, int S>
__device__ __forceinline__ cplx<R> hs_factor(const cplx<R>* tw, int lane, R sg) {
  if constexpr (S > 2) {
    const cplx<R> w = twid<R, INV>(tw + tw_off(N, N / (2 * S)), lane & (S - 1));
    return mk<R>(sg * w.x, sg * w.y);
  } else {
    return mk<R>(sg, R(0));
  }
}

template <typename R, bool INV, int NT, int N, int T>
__device__ __forceinline__ void hs_dif(cplx<R> (*const (&v)[NT])[N / 32], const cplx<R>* tw, int lane) {
  constexpr int E = N / 32, S = 1 << T, RB = StageRB<N, T>::v;
  const bool c = (lane >> T) & 1;
  const cplx<R> f = hs_factor<R, INV, N, S>(tw, lane, c ? R(-1) : R(1));
#pragma unroll
  for (int a = 0; a < NT; ++a)
#pragma unroll
    for (int og = 0; og < E / 2; ++og) {
      const int r0 = (og & ((1 << RB) - 1)) | ((og >> RB) << (RB + 1)), r1 = r0 | (1 << RB);
      const cplx<R> keep = c ? (*v[a])[r1] : (*v[a])[r0];
      const cplx<R> send = c ? (*v[a])[r0] : (*v[a])[r1];
      const cplx<R> recv = shfl_xor_c<R>(send, S);
      (*v[a])[r0] = cadd(keep, recv);
      cplx<R> d = csub(keep, recv);
      if constexpr (S > 2) d = cmul(d, f);
      else {
        d = cscale(d, f.x);
        if constexpr (S == 2) { if (lane & 1) d = mul_mi<R, INV>(d); }
      }
      (*v[a])[r1] = d;
    }
}

template <typename R, bool INV, int NT, int N, int T>
__device__ __forceinline__ void hs_dit(cplx<R> (*const (&v)[NT])[N / 32], const cplx<R>* tw, int lane) {
  constexpr int E = N / 32, S = 1 << T, RB = StageRB<N, T>::v;
  const bool c = (lane >> T) & 1;
  const cplx<R> f = hs_factor<R, INV, N, S>(tw, lane, c ? R(-1) : R(1));
#pragma unroll
  for (int a = 0; a < NT; ++a)
#pragma unroll
    for (int og = 0; og < E / 2; ++og) {
      const int r0 = (og & ((1 << RB) - 1)) | ((og >> RB) << (RB + 1)), r1 = r0 | (1 << RB);
      cplx<R> y = (*v[a])[r1];
      if constexpr (S > 2) y = cmul(y, f);
      else {
        if constexpr (S == 2) { if (lane & 1) y = mul_mi<R, INV>(y); }
        y = cscale(y, f.x);
      }
      const cplx<R> x = (*v[a])[r0];
      const cplx<R> keep = cadd(x, y), send = csub(x, y);
      const cplx<R> recv = shfl_xor_c<R>(send, S);
      (*v[a])[r0] = c ? recv : keep;
      (*v[a])[r1] = c ? keep : recv;
    }
}

template <typename R, bool INV, int NT, int N>
__device__ __forceinline__ void fft_dif_n(cplx<R> (*const (&v)[NT])[N / 32], const cplx<R>* tw, int lane) {
  first_pass<R, INV, NT, N, false>(v, tw, lane);
  hs_dif<R, INV, NT, N, 4>(v, tw, lane);
  hs_dif<R, INV, NT, N, 3>(v, tw, lane);
  hs_dif<R, INV, NT, N, 2>(v, tw, lane);
  hs_dif<R, INV, NT, N, 1>(v, tw, lane);
  hs_dif<R, INV, NT, N, 0>(v, tw, lane);
}

template <typename R, bool INV, int NT, int N>
__device__ __forceinline__ void fft_dit_n(cplx<R> (*const (&v)[NT])[N / 32], const cplx<R>* tw, int lane) {
  hs_dit<R, INV, NT, N, 0>(v, tw, lane);
  hs_dit<R, INV, NT, N, 1>(v, tw, lane);
  hs_dit<R, INV, NT, N, 2>(v, tw, lane);
  hs_dit<R, INV, NT, N, 3>(v, tw, lane);
  hs_dit<R, INV, NT, N, 4>(v, tw, lane);
  first_pass<R, INV, NT, N, true>(v, tw, lane);
}

template <typename R, int N, bool INV>
__device__ __forceinline__ void fft_dif(cplx<R> (&v)[N / 32], const cplx<R>* __restrict__ tw, int lane) {
  cplx<R>(*const ptrs[1])[N / 32] = {&v};
  fft_dif_n<R, INV, 1, N>(ptrs, tw, lane);
}

template <typename R, int N, bool INV>
__device__ __forceinline__ void fft_dit(cplx<R> (&v)[N / 32], const cplx<R>* __restrict__ tw, int lane) {
  cplx<R>(*const ptrs[1])[N / 32] = {&v};
  fft_dit_n<R, INV, 1, N>(ptrs, tw, lane);
}

// Two independent transforms in lockstep (same direction and order): every
// stage issues both arrays' shuffles before their arithmetic, so one warp
// keeps twice the independent work in flight.
template <typename R, int N, bool INV>
__device__ __forceinline__ void fft_dif2(cplx<R> (&a)[N / 32], cplx<R> (&b)[N / 32], const cplx<R>* __restrict__ tw,
                                         int lane) {
  cplx<R>(*const ptrs[2])[N / 32] = {&a, &b};
  fft_dif_n<R, INV, 2, N>(ptrs, tw, lane);
}

template <typename R, int N, bool INV>
__device__ __forceinline__ void fft_dit2(cplx<R> (&a)[N / 32], cplx<R> (&b)[N / 32], const cplx<R>* __restrict__ tw,
                                         int lane) {
  cplx<R>(*const ptrs[2])[N / 32] = {&a, &b};
  fft_dit_n<R, INV, 2, N>(ptrs, tw, lane);
}

// The shared-memory twiddle image (tw_smem(N) entries) built from the half
// table half[k] = exp(-2 pi i k / N), k < N/2: the strided sub-tables, then the
// radix-E pass's table W_N^{l k1} (k >= N/2 taken as -W_N^{k - N/2}).  Built
// once on the host when a context is created.
template <typename C, int N>
__host__ __device__ inline void twiddle_image(const C* half, C* img) {
  for (int i = 0; i < N; ++i) {
    int r = 1, off = 0;
    while (r < N / 2 && i >= off + N / (2 * r)) { off += N / (2 * r); r *= 2; }
    const int src = (i - off) * r;
    img[i] = half[src < N / 2 ? src : 0];
  }
  for (int i = 0; i < tw_first(N); ++i) {
    const int k = ((i >> 5) + 1) * (i & 31);
    C w = half[k & (N / 2 - 1)];
    if (k & (N / 2)) { w.x = -w.x; w.y = -w.y; }
    img[N + i] = w;
  }
}

// ---------------------------------------------------------------------------
// Group transforms (FP64)
// ---------------------------------------------------------------------------

// a W with W = c - i s (forward) or its conjugate (inverse).
template <typename R, bool INV>
__device__ __forceinline__ cplx<R> mul_cs(cplx<R> a, R c, R s) { return cmul(a, mk<R>(c, INV ? s : -s)); }

// The radix-16 pass of N = 128 on 16 lanes, as 4 x 4: lane l holds x[l + 16 j'], that is
// x[a + 8 j] with a = l mod 8 and j = h + 2 j', h = l / 8.  First the radix-4 butterflies
// over (j, j + 4, j + 8, j + 12), which lie within a lane (j = h and h + 2), then the
// factors W_16^{j k}, then radix-4 butterflies over j mod 4: their first sums lie within a
// lane too (j = 0, 2 on lanes h = 0; 1, 3 on lanes h = 1), and the last ones pair lanes l
// and l ^ 8, which swap half their values for them.  Then the transposition hands lane k1
// the eight values of its output digit.
template <typename R, bool INV, bool ZMID>
__device__ __forceinline__ void dft16_lanes(cplx<R> (&x)[8], int l) {
  const R c1 = R(0.92387953251128675612818318939678829), s1 = R(0.38268343236508977172845998403039887);
  const bool h = (l >> 3) & 1;
  // x[0], x[2], x[4], x[6]: j = h + 0, 4, 8, 12;  x[1], x[3], x[5], x[7]: j = h + 2, 6, 10, 14.
  // ZMID (inputs 48..79 of 128 are zero, j = 6..9): x[3] and x[4].
  if constexpr (ZMID) {
    {
      const cplx<R> s13 = cadd(x[2], x[6]), d13 = mul_mi<R, INV>(csub(x[2], x[6])), a = x[0];
      x[0] = cadd(a, s13); x[2] = cadd(a, d13); x[4] = csub(a, s13); x[6] = csub(a, d13);
    }
    {
      const cplx<R> s02 = cadd(x[1], x[5]), d02 = csub(x[1], x[5]), b = x[7], ib = mul_mi<R, INV>(b);
      x[1] = cadd(s02, b); x[3] = csub(d02, ib); x[5] = csub(s02, b); x[7] = cadd(d02, ib);
    }
  } else {
    dft4<R, INV>(x[0], x[2], x[4], x[6]);
    dft4<R, INV>(x[1], x[3], x[5], x[7]);
  }
  // x[2 k] = A_h[k], x[2 k + 1] = A_{h+2}[k]; times W_16^{j k}
  if (h) {
    x[2] = mul_cs<R, INV>(x[2], c1, s1);
    x[4] = mul_w8<R, INV>(x[4]);
    x[6] = mul_cs<R, INV>(x[6], s1, c1);
    x[3] = mul_cs<R, INV>(x[3], s1, c1);
    x[5] = mul_mi<R, INV>(mul_w8<R, INV>(x[5]));
    x[7] = mul_cs<R, INV>(x[7], -c1, -s1);
  } else {
    x[3] = mul_w8<R, INV>(x[3]);
    x[5] = mul_mi<R, INV>(x[5]);
    x[7] = mul_mi<R, INV>(mul_w8<R, INV>(x[7]));
  }
  // s = x[2k] + x[2k+1], d = x[2k] - x[2k+1] (lanes h = 1: times W_4): s02, d02 / s13, d13 of output k
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const cplx<R> s = cadd(x[2 * k], x[2 * k + 1]), d = csub(x[2 * k], x[2 * k + 1]), e = mul_mi<R, INV>(d);
    x[2 * k] = s;
    x[2 * k + 1] = h ? e : d;
  }
  // lanes h = 0 take k = 0, 1 of both, lanes h = 1 k = 2, 3
  cplx<R> y[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {   // i = 2 (k mod 2) + (s or d)
    const cplx<R> keep = h ? x[4 + i] : x[i], send = h ? x[i] : x[4 + i];
    const cplx<R> recv = shfl_xor_c<R>(send, 8);
    y[i] = cadd(keep, recv);
    const cplx<R> t = csub(keep, recv);                       // s02 - s13 on lanes h = 0, its negative on h = 1
    y[4 + i] = h ? mk<R>(-t.x, -t.y) : t;
  }
  // X[k + 4 m]: m = 0: s02 + s13, 1: d02 + d13, 2: s02 - s13, 3: d02 - d13; k = 2 h + (i / 2)
  // register order: x[m + 4 kk], kk = k - 2 h
#pragma unroll
  for (int kk = 0; kk < 2; ++kk) {
    x[4 * kk] = y[2 * kk]; x[4 * kk + 1] = y[2 * kk + 1]; x[4 * kk + 2] = y[4 + 2 * kk]; x[4 * kk + 3] = y[4 + 2 * kk + 1];
  }
}

template <typename R, bool INV, bool ZBOX>
__device__ __forceinline__ void fft_group16(cplx<R> (&x)[8], const cplx<R>* tw, cplx<R>* xb, int l) {
  dft16_lanes<R, INV, ZBOX>(x, l);
  const int a = l & 7, h2 = (l >> 3) * 2;
#pragma unroll
  for (int kk = 0; kk < 2; ++kk)
#pragma unroll
    for (int m = 0; m < 4; ++m) {   // output digit k1 = 2 h + kk + 4 m; k1 = 0 has no twiddle
      const int k1 = h2 + kk + 4 * m;
      if (kk == 0 && m == 0) {
        const cplx<R> t = cmul(x[0], twid<R, INV>(tw, k1 * 8 + a));
        if (h2) x[0] = t;
      } else {
        x[4 * kk + m] = cmul(x[4 * kk + m], twid<R, INV>(tw, k1 * 8 + a));
      }
    }
  __syncwarp();   // the group's reads of the previous exchange are done
#pragma unroll
  for (int kk = 0; kk < 2; ++kk)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int k1 = h2 + kk + 4 * m;
      xb[k1 * 8 + (a ^ (k1 & 7))] = x[4 * kk + m];
    }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = xb[l * 8 + (i ^ (l & 7))];
  dft_reg<R, INV, 8>(x);
}

// ---------------------------------------------------------------------------
// The layout a kernel works in: L lanes and E values per transform, G transforms per
// warp, TW table entries in shared memory, XB exchange entries per transform, the
// position pos(l, j) of a spectrum along the transformed direction, and none(j):
// element j of every lane lies outside the box.
//
//   warp layout   a warp per transform, exchanges by shuffles, and the two transforms
//                 of a pass in lockstep: the shorter chain of dependent operations.
//   group layout  (FP64 at N = 128) two transforms of 16 lanes per warp with 8 values
//                 per lane and one exchange through shared memory: 30% fewer
//                 instructions per transform, but half as many warps for the same
//                 columns.  The column passes of batched tangents use it.
// ---------------------------------------------------------------------------
template <typename R_, int N_, bool GROUP_ = false> struct Xf {
  static_assert(!GROUP_ || (sizeof(R_) == 8 && N_ == 128), "group layout: FP64, N = 128");
  using R = R_;
  static constexpr int N = N_;
  static constexpr bool GROUP = GROUP_;
  static constexpr int L = GROUP ? 16 : 32, E = N / L, G = 32 / L;
  static constexpr int TW = GROUP ? N : tw_smem(N);
  static constexpr int XB = GROUP ? N : 0;
  static constexpr int KMAX = (N - 1) / 3, K = KMAX + 1, M = 2 * KMAX + 1;
  // A column pass brings the operands of its algebra through shared memory (see Operands) in
  // FP64 at n = 128, where the rows of a stage would hold up to 128 registers of a lane. At
  // n = 64 (two values per lane) and in FP32 they fit into registers, and the shared room costs
  // more than it hides. Measured per call, staged -> in registers: tangents of 20 Lawson-RK4
  // steps, n = 64 FP64, batch 38 1.23 -> 1.13 ms; 24 steps of 32 states at n = 128 FP32, RK4
  // 1.77 -> 1.57, Lawson-RK6 3.78 -> 3.17; over both types, batches 1 to 192: tangents 0 to 7%,
  // cotangents 0 to 4% faster, state_vel at n = 64, batch 1 7.2 -> 7.3 us, batch 16 13.9 -> 9.6.
  static constexpr bool STAGED = !GROUP && N == 128 && sizeof(R) == 8;
  __device__ static __forceinline__ int pos(int l, int j) {
    if constexpr (GROUP) return l + L * j;
    else return spec_pos<N>(l, j);
  }
  __host__ __device__ static constexpr bool none(int j) { return GROUP && L * j > KMAX && L * j + L - 1 < N - KMAX; }
  // Shared entries of the tables and of the exchange buffers of W warps.
  __host__ __device__ static constexpr int smem(int W) { return TW + W * G * XB; }

  const cplx<R>* tw;   // tables (shared memory)
  cplx<R>* xb;         // the lane's exchange buffer
  int l;               // lane within the transform

  // `s` is the start of the shared region (tables, then the buffers); `warp` the
  // warp's index among those that transform.
  __device__ __forceinline__ Xf(cplx<R>* s, int warp) {
    const int lane = threadIdx.x & 31;
    tw = s; l = lane & (L - 1);
    xb = s + TW + (warp * G + lane / L) * XB;
  }
  // kx and box slot (-1 outside the box) of the lane's element j.
  __device__ __forceinline__ R kx(int j) const {
    if constexpr (GROUP) return (R)l + R(j < E / 2 ? L * j : L * j - N);
    else return (R)pos_to_k(spec_pos<N>(l, j), N);
  }
  __device__ __forceinline__ int slot(int j) const {
    if constexpr (GROUP) {
      const int p = l + L * j;
      if (j < E / 2) return p <= KMAX ? p : -1;
      return p >= N - KMAX ? p - N + M : -1;
    } else {
      return pos_to_slot(spec_pos<N>(l, j), N, KMAX, M);
    }
  }
  // Natural order -> spectral positions (column forward, row inverse) ...
  template <bool INV, bool ZBOX = false> __device__ __forceinline__ void to_spec(cplx<R> (&v)[E]) const {
    if constexpr (GROUP) fft_group16<R, INV, ZBOX>(v, tw, xb, l);
    else fft_dif<R, N, INV>(v, tw, l);
  }
  // ... and back.  ZBOX: the input vanishes outside the box.
  template <bool INV, bool ZBOX = false> __device__ __forceinline__ void from_spec(cplx<R> (&v)[E]) const {
    if constexpr (GROUP) fft_group16<R, INV, ZBOX>(v, tw, xb, l);
    else fft_dit<R, N, INV>(v, tw, l);
  }
  // Two transforms in lockstep (warp layout).
  template <bool INV> __device__ __forceinline__ void to_spec2(cplx<R> (&a)[E], cplx<R> (&b)[E]) const {
    fft_dif2<R, N, INV>(a, b, tw, l);
  }
  template <bool INV> __device__ __forceinline__ void from_spec2(cplx<R> (&a)[E], cplx<R> (&b)[E]) const {
    fft_dit2<R, N, INV>(a, b, tw, l);
  }
};

// Device table of (R, N): the shared entries of the warp layout, the uncurling
// multipliers (ky/k^2, -kx/k^2) / n^2 of every box mode [K][M] (mhd_jax.py:83-90; zero
// at (0,0); n^2 is a power of two, so the scale is exact), and the shared entries of the
// group layout where there is one.  The column passes divided for the multipliers at
// every mode, two FP64 divisions or about 40 instructions per mode and pass against one
// 16-byte load.  Built on the host when a context is created.
template <typename R, int N> struct XfTable {
  static constexpr bool GROUPS = sizeof(R) == 8 && N == 128;
  static constexpr int mu = tw_smem(N), group = mu + Xf<R, N>::K * Xf<R, N>::M, size = group + (GROUPS ? N : 0);
};
template <typename R, int N>
inline void xf_table(cplx<R>* img) {
  using T = XfTable<R, N>;
  using X = Xf<R, N>;
  const long double twopi = 6.283185307179586476925286766559005768L;
  auto w = [&](int k) {
    const long double a = twopi * (long double)(k % N) / (long double)N;
    return mk<R>((R)cosl(a), (R)(-sinl(a)));
  };
  cplx<R> half[N / 2];
  for (int k = 0; k < N / 2; ++k) half[k] = w(k);
  twiddle_image<cplx<R>, N>(half, img);
  const R inv_n2 = R(1) / (R(N) * R(N));
  for (int ky = 0; ky < X::K; ++ky)
    for (int s = 0; s < X::M; ++s) {
      const R rkx = (R)slot_to_kx(s, X::KMAX, X::M), rky = (R)ky, ksq = rkx * rkx + rky * rky;
      img[T::mu + ky * X::M + s] = ksq == R(0) ? mk<R>(R(0), R(0)) : mk<R>(rky / ksq * inv_n2, (-rkx) / ksq * inv_n2);
    }
  if (T::GROUPS)   // W_N^{l k} at k 8 + l, l < 8
    for (int k = 0; k < N / 8; ++k)
      for (int l = 0; l < 8; ++l) img[T::group + k * 8 + l] = w(k * l);
}

// Copy of the layout's tables into shared memory (cp.async: global -> shared without a
// register round trip); each thread waits for its own copies and the caller's
// __syncthreads makes them visible.
template <class X>
__device__ __forceinline__ void load_tables(cplx<typename X::R>* s, const cplx<typename X::R>* __restrict__ g) {
  using R = typename X::R;
  if (X::GROUP) g += XfTable<R, X::N>::group;
  for (int i = threadIdx.x; i < X::TW; i += blockDim.x) cp_async_c<R>(s + i, g + i);
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

}  // namespace ecs
