// tracker.cuh -- the homotopy path tracker for sm_100a.
//
// One sub-warp of W lanes (W = next power of two >= N, at least 4) tracks one
// path: lane r owns equation row r (its row of H_x lives in registers) and
// component r of the track.  The 32/W sub-warps of a warp run in lockstep
// through one warp-uniform loop (one path step per trip), so every shuffle and
// __syncwarp sees the full warp; a sub-warp whose path ends writes its
// endpoint and takes the next path from a global counter (work stealing).
//
// Per path step (reference GPU-HC/magmaHC/gpu-kernels/kernel_HC_Solver_P3P.cu:115-254,
// PH variant kernel_HC_Solver_trifocal_2op1p_30x30.cu:155-301):
//   end-zone clamp -> 4 RK stages (coefficients c_k(t) -> H_x, -H_t -> LU solve)
//   -> Newton corrector (H_x, H -> LU solve, success/infinity tests) -> step control.
//
// Arithmetic follows the oracle's operation order exactly (explicit fma,
// *_rn intrinsics so nothing else is contracted), so the FP64 tracker matches
// the oracle bit for bit.  Index tables are pre-compiled into term words
// (ghc_internal.h) and staged once per CTA in shared memory.
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>

#include <cstdint>
#include <type_traits>

#include "ghc_internal.h"

namespace ghc {
namespace dev {

constexpr unsigned kFull = 0xffffffffu;

template <typename R>
struct alignas(2 * sizeof(R)) cx {
  R re, im;
};

__device__ __forceinline__ double f_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float f_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double f_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float f_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double f_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float f_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double f_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float f_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double f_div(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float f_div(float a, float b) { return __fdiv_rn(a, b); }

template <typename R>
__device__ __forceinline__ cx<R>* view(unsigned char* p) {
  return reinterpret_cast<cx<R>*>(p);
}

template <typename R>
__device__ __forceinline__ cx<R> mk(R a, R b) {
  cx<R> r;
  r.re = a;
  r.im = b;
  return r;
}
template <typename R>
__device__ __forceinline__ cx<R> c_add(cx<R> a, cx<R> b) {
  return mk(f_add(a.re, b.re), f_add(a.im, b.im));
}
template <typename R>
__device__ __forceinline__ cx<R> c_sub(cx<R> a, cx<R> b) {
  return mk(f_sub(a.re, b.re), f_sub(a.im, b.im));
}
template <typename R>
__device__ __forceinline__ cx<R> c_scale(R s, cx<R> a) {
  return mk(f_mul(s, a.re), f_mul(s, a.im));
}
// a*b
template <typename R>
__device__ __forceinline__ cx<R> c_mul(cx<R> a, cx<R> b) {
  return mk(f_fma(a.re, b.re, -f_mul(a.im, b.im)), f_fma(a.re, b.im, f_mul(a.im, b.re)));
}
// c + a*b
template <typename R>
__device__ __forceinline__ cx<R> c_fma(cx<R> a, cx<R> b, cx<R> c) {
  return mk(f_fma(a.re, b.re, f_fma(-a.im, b.im, c.re)), f_fma(a.re, b.im, f_fma(a.im, b.re, c.im)));
}
// c - a*b
template <typename R>
__device__ __forceinline__ cx<R> c_fnma(cx<R> a, cx<R> b, cx<R> c) {
  return mk(f_fma(-a.re, b.re, f_fma(a.im, b.im, c.re)), f_fma(-a.re, b.im, f_fma(-a.im, b.re, c.im)));
}
// 1/b = conj(b) / |b|^2 with one correctly rounded reciprocal
__device__ __forceinline__ double f_rcp(double a) { return __drcp_rn(a); }
__device__ __forceinline__ float f_rcp(float a) { return __frcp_rn(a); }
template <typename R>
__device__ __forceinline__ cx<R> c_rcp(cx<R> b) {
  const R s = f_fma(b.re, b.re, f_mul(b.im, b.im));
  const R inv = f_rcp(s);
  return mk(f_mul(b.re, inv), -f_mul(b.im, inv));
}
template <typename R>
__device__ __forceinline__ R c_abs2(cx<R> a) {
  return f_fma(a.re, a.re, f_mul(a.im, a.im));
}
template <typename R, typename S>
__device__ __forceinline__ cx<R> c_cast(cx<S> a) {
  return mk((R)a.re, (R)a.im);
}

__device__ __forceinline__ double shfl_xor(double v, int off, int w) { return __shfl_xor_sync(kFull, v, off, w); }
__device__ __forceinline__ float shfl_xor(float v, int off, int w) { return __shfl_xor_sync(kFull, v, off, w); }

// Compiled tables staged in shared memory.  The straight-line term shapes (NV >= 0 variable slots)
// keep their terms there as packed words, decoded in about half the instructions of the compiled
// 64-bit term words (the scale needs no integer conversion, the first variable's address is one
// shift-add), for complex values of type R (B200: 5-point FP64 13.6 -> 13.2 ms, CY 95.4 -> 93.4,
// gen-3v-4pt 93.8 -> 91.8, the mix 60.9 -> 57.3):
//   lo  0.. 9  P2C coefficient index; PH: parameter index a (0..5) and b (6..11)
//   lo 12..22  H_x, balanced walk: where the entry's sum goes (slot * W + row); third variable (12..16)
//   lo 27..31  first variable
//   hi  .. 8   second variable as a byte offset (5 bits from bit 4, complex double; 3, complex float)
//   hi 13      H_x: the last term of its entry
//   hi 14..31  the integer scale as R: the upper bits of the double's upper word, or of the float
// The general shape (NV < 0) keeps the compiled words.
struct Tables {
  const uint2* hx_terms;
  const uint16_t* hx_off;
  const uint2* ht_terms;
  const uint2* ht_terms_hi;  // the terms packed for the state precision (mixed tracker's residual)
  const uint16_t* ht_off;
};

__device__ __forceinline__ uint64_t raw_word(uint2 w) { return (uint64_t)w.y << 32 | w.x; }
template <typename R>
constexpr unsigned kCxShift = sizeof(R) == 8 ? 4 : 3;  // log2 of a complex value's bytes

template <typename R, int KIND, int NV>
__device__ __forceinline__ uint2 pack_term(uint64_t w, int W) {
  if (NV < 0) return make_uint2((unsigned)w, (unsigned)(w >> 32));
  const unsigned s = sizeof(R) == 8 ? (unsigned)__double2hiint((double)term_scale(w))
                                    : __float_as_uint((float)term_scale(w));
  unsigned lo = KIND == KIND_P2C ? (unsigned)term_coef(w) : (unsigned)(term_pa(w) | term_pb(w) << 6);
  unsigned hi = s & 0xffffc000u;
  if (term_last(w)) hi |= 1u << 13;
  lo |= (unsigned)term_var(w, 0) << 27;
  if (NV >= 2) hi |= (unsigned)term_var(w, 1) << kCxShift<R>;
  if (NV >= 3) lo |= (unsigned)term_var(w, 2) << 12;
  else lo |= (unsigned)(term_dst_slot(w) * W + term_dst_row(w)) << 12;
  return make_uint2(lo, hi);
}
template <int NV>
__device__ __forceinline__ bool word_last(uint2 w) {
  return NV < 0 ? term_last(raw_word(w)) : (w.y & (1u << 13)) != 0u;
}
template <int NV>
__device__ __forceinline__ unsigned word_dst(uint2 w, int W) {
  if (NV < 0) return (unsigned)(term_dst_slot(raw_word(w)) * W + term_dst_row(raw_word(w)));
  return w.x >> 12 & 0x7ffu;
}
template <typename R, int NV>
__device__ __forceinline__ R word_scale(uint2 w) {
  if constexpr (NV < 0) return (R)term_scale(raw_word(w));
  else if constexpr (sizeof(R) == 8) return __hiloint2double((int)(w.y & 0xffffc000u), 0);
  else return __uint_as_float(w.y & 0xffffc000u);
}
template <typename R>
__device__ __forceinline__ cx<R> at(const unsigned char* base, unsigned off) {
  return *reinterpret_cast<const cx<R>*>(base + off);
}
// coefficient (P2C) or first / second parameter (PH) of a term, from an array of complex R
template <typename R, int KIND, int NV>
__device__ __forceinline__ cx<R> word_coef(uint2 w, const unsigned char* c) {
  if (NV < 0) return at<R>(c, (unsigned)(KIND == KIND_P2C ? term_coef(raw_word(w)) : term_pa(raw_word(w))) << kCxShift<R>);
  return at<R>(c, (w.x & (KIND == KIND_P2C ? 0x3ffu : 0x3fu)) << kCxShift<R>);
}
template <typename R, int NV>
__device__ __forceinline__ cx<R> word_coef_b(uint2 w, const unsigned char* c) {
  return at<R>(c, (NV < 0 ? (unsigned)term_pb(raw_word(w)) : w.x >> 6 & 0x3fu) << kCxShift<R>);
}

// acc += p * x[v0] * x[v1] ... over the term's variable slots (reference monomial term,
// dev-eval-indxing-P3P.cuh:70-118; slot N is the constant 1).  Every term of a table has
// the same number of slots: NV >= 0 fixes it at compile time (straight-line code), NV < 0
// reads it from the word.
template <typename R, int NV>
__device__ __forceinline__ cx<R> acc_term(cx<R> acc, cx<R> p, uint2 w, const unsigned char* xs) {
  static_assert(NV <= 3, "packed words hold three variables");
  if constexpr (NV == 0) {
    return c_add(acc, p);
  } else if constexpr (NV > 0) {
    const cx<R> x0 = at<R>(xs, w.x >> (27 - kCxShift<R>));
    if constexpr (NV == 1) return c_fma(p, x0, acc);
    p = c_mul(p, x0);
    const cx<R> x1 = at<R>(xs, w.y & (31u << kCxShift<R>));
    if constexpr (NV == 2) return c_fma(p, x1, acc);
    p = c_mul(p, x1);
    return c_fma(p, at<R>(xs, (w.x >> 12 & 31u) << kCxShift<R>), acc);
  } else {
    const uint64_t r = raw_word(w);
    const cx<R>* x = reinterpret_cast<const cx<R>*>(xs);
    const int nv = term_nv(r);
    if (nv == 0) return c_add(acc, p);
#pragma unroll 1
    for (int q = 0; q < nv - 1; ++q) p = c_mul(p, x[term_var(r, q)]);
    return c_fma(p, x[term_var(r, nv - 1)], acc);
  }
}

// complex entry of a table of doubles: one 16-byte load where the table is aligned to that (WIDE)
template <typename R, bool WIDE>
__device__ __forceinline__ cx<R> ldg_cx(const double* a) {
  if constexpr (WIDE) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(a));
    return mk((R)v.x, (R)v.y);
  } else {
    return mk((R)__ldg(a), (R)__ldg(a + 1));
  }
}
// polynomial with complex coefficients a[0..n] at t (Horner)
template <typename R, bool WIDE, int NN>
__device__ __forceinline__ cx<R> poly_at(const double* a, int n, R t) {
  if constexpr (NN >= 0) {  // all loads at once
    cx<R> v[NN + 1];
#pragma unroll
    for (int j = 0; j <= NN; ++j) v[j] = ldg_cx<R, WIDE>(a + 2 * j);
#pragma unroll
    for (int j = NN - 1; j >= 0; --j) v[NN] = mk(f_fma(v[NN].re, t, v[j].re), f_fma(v[NN].im, t, v[j].im));
    return v[NN];
  } else {
    cx<R> v = ldg_cx<R, WIDE>(a + 2 * n);
    for (int j = n - 1; j >= 0; --j) {
      const cx<R> w = ldg_cx<R, WIDE>(a + 2 * j);
      v = mk(f_fma(v.re, t, w.re), f_fma(v.im, t, w.im));
    }
    return v;
  }
}
// c_k(t), c'_k(t) for k = l, l + step, ... (reference eval_parameter_homotopy), computed in R and
// stored in RO; with HI the R values of c_k(t) are also kept in hi (the residual's copy).
// KK: the polynomials' degree K, or 0 for any.
template <typename R, typename RO, bool HI, bool WIDE, int KK>
__device__ __forceinline__ void coef_loop_p2c(const double* __restrict__ hx, const double* __restrict__ ht, int M,
                                              int K, R t, bool fresh, cx<RO>* c, cx<RO>* cp, cx<R>* hi, int l, int step) {
  const int n = KK > 0 ? KK : K;
  for (int k = l; k <= M; k += step) {
    const cx<R> v = poly_at<R, WIDE, (KK > 0 ? KK : -1)>(hx + 2 * (size_t)k * (n + 1), n, t);
    c[k] = c_cast<RO>(v);
    if (HI) hi[k] = v;
    if (KK != 1) cp[k] = n >= 1 ? c_cast<RO>(poly_at<R, WIDE, KK - 1>(ht + 2 * (size_t)k * n, n - 1, t)) : mk(RO(0), RO(0));
  }
  if (KK == 1 && fresh)  // constant in t: written for the path's first evaluation
    for (int k = l; k <= M; k += step) cp[k] = c_cast<RO>(ldg_cx<R, WIDE>(ht + 2 * (size_t)k));
}
// The lanes of a path read its tables entry by entry at a stride of K (+ 1) complex values, so every
// load touches most lines of the table: half as many loads (whole complex values) are half as many
// passes over them.  With the shorter path record: P3P one instance FP64 123 -> 105 us, 20,000 hypotheses
// 2.11 -> 1.88 ms, 5-point 12.3 -> 10.9, gen-3v-4pt 90.5 -> 84.8.  Higher degrees keep 8-byte loads: 16-byte
// ones there gained 1.5 to 3.5 % on 6-point rolling shutter and P4P (K = 3), nothing on distorted 2-view
// triangulation and TDOA, and cost 6-line 3-view 2.4 % in mixed precision.
template <typename R, typename RO, bool HI>
__device__ __forceinline__ void coef_eval_p2c(const double* __restrict__ hx, const double* __restrict__ ht, int M,
                                              int K, R t, bool fresh, cx<RO>* c, cx<RO>* cp, cx<R>* hi, int l, int step) {
  const bool wide = ((reinterpret_cast<uintptr_t>(hx) | reinterpret_cast<uintptr_t>(ht)) & 15) == 0;
  if (wide && K == 1) coef_loop_p2c<R, RO, HI, true, 1>(hx, ht, M, K, t, fresh, c, cp, hi, l, step);
  else if (wide && K == 2) coef_loop_p2c<R, RO, HI, true, 2>(hx, ht, M, K, t, fresh, c, cp, hi, l, step);
  else coef_loop_p2c<R, RO, HI, false, 0>(hx, ht, M, K, t, fresh, c, cp, hi, l, step);
}

// p(t) = p1 t + p0 (1-t) and, on a new path (fresh), the parameter differences (reference
// compute_param_homotopy), computed in R and stored in RO; with HI the R values of p(t) are also kept in hi
template <typename R, typename RO, bool HI, bool WIDE>
__device__ __forceinline__ void coef_loop_ph(const double* __restrict__ ps, const double* __restrict__ pt,
                                             const double* __restrict__ pd, int P, R t, bool fresh, cx<RO>* ph,
                                             cx<RO>* dp, cx<R>* hi, int l, int step) {
  const R u = f_sub(R(1), t);
  for (int k = l; k < P; k += step) {
    const cx<R> g = ldg_cx<R, WIDE>(pt + 2 * k), s = ldg_cx<R, WIDE>(ps + 2 * k);
    const cx<R> v = mk(f_fma(g.re, t, f_mul(s.re, u)), f_fma(g.im, t, f_mul(s.im, u)));
    ph[k] = c_cast<RO>(v);
    if (HI) hi[k] = v;
  }
  if (fresh) {
    for (int k = l; k <= P; k += step) dp[k] = mk((RO)__ldg(pd + 2 * k), (RO)__ldg(pd + 2 * k + 1));
    if (l == 0) {
      ph[P] = mk(RO(1), RO(0));
      if (HI) hi[P] = mk(R(1), R(0));
    }
  }
}
template <typename R, typename RO, bool HI>
__device__ __forceinline__ void coef_eval_ph(const double* __restrict__ ps, const double* __restrict__ pt,
                                             const double* __restrict__ pd, int P, R t, bool fresh, cx<RO>* ph,
                                             cx<RO>* dp, cx<R>* hi, int l, int step) {
  if (((reinterpret_cast<uintptr_t>(ps) | reinterpret_cast<uintptr_t>(pt)) & 15) == 0)
    coef_loop_ph<R, RO, HI, true>(ps, pt, pd, P, t, fresh, ph, dp, hi, l, step);
  else
    coef_loop_ph<R, RO, HI, false>(ps, pt, pd, P, t, fresh, ph, dp, hi, l, step);
}

// term value p (coefficient, or product of two homotopy parameters, times the integer scale)
template <typename R, int KIND, int NV>
__device__ __forceinline__ cx<R> term_coef_value(uint2 w, const unsigned char* ca) {
  const cx<R> p = c_scale(word_scale<R, NV>(w), word_coef<R, KIND, NV>(w, ca));
  if (KIND == KIND_P2C) return p;
  return c_mul(p, word_coef_b<R, NV>(w, ca));
}

// Row r of H_x into A.
//
// Flat (always above 16 unknowns, else when the problem's flat_eval is set):
// the row's terms are walked as one list (CSR row r, entry ends flagged in the term word),
// so a sub-warp spends max_r(terms of row r) iterations instead of
// sum_i max_r(terms of entry (r, i)).  The k-th non-zero entry of the row is
// staged in the sub-warp's scratch slot scr[k][r] (only as many slots as the
// fullest row has non-zero entries) and read back into registers through the
// lane's non-zero mask nz (entry i is in slot popc(nz & (2^i - 1))); every slot
// below the row's count is rewritten by every evaluation.  Balanced (walk 2): the
// entries are dealt to all W lanes at table-compile time by term count, a lane
// stores each finished sum into its row's slot, and the rows read their slots back
// after a sub-warp synchronisation (max over lanes instead of over rows: 65 -> 43
// iterations for the 5-point problem, whose rows hold 4..65 terms).  Entry-wise:
// one loop per column, straight into registers.  Every walk sums each entry in
// table order, as in the oracle.
template <int N>
constexpr bool kFlatAlways = N > 16;

// Term walks unrolled by 4: the loads of the next terms hide behind the arithmetic of the first
// (5-point FP64, 12 warps a SM: 14.2 ms rolled, 13.4 by 2, 13.2 by 4); above 16 unknowns the H_t walk
// only by 2 (30x30 FP64 113.3 against 118.9 ms).
template <int N>
constexpr int kUnrollHt = N > 16 ? 2 : 4;
// The mixed kernel's general H_x walk at 5 unknowns only by 2: by 4 the kernel spills, and its code, with
// the FP64 residual's general walk beside it, is longer than short lists repay (distorted 2-view
// triangulation, 18 terms a lane, 1,428 hypotheses 8.87 -> 8.70 ms; TDOA, 45 terms, 45.3 -> 44.6); the longer
// lists of the problems with 4 and 6 unknowns are better by 4 (PnP by quaternions 22.1 against 22.5,
// 6-line 3-view 731 against 737).
template <int N, int NVX, bool MIXED>
constexpr int kUnrollHx = MIXED && NVX < 0 && N == 5 ? 2 : 4;

// Row r of H (which = 0) or of -H_t (which = 1) from the H_t term table, in precision R
template <typename R, int N, int KIND, int NVT>
__device__ __forceinline__ cx<R> eval_rhs(const uint2* terms, const uint16_t* off, const unsigned char* ca,
                                          const unsigned char* cb, const unsigned char* xs, int r, bool live,
                                          int which) {
  cx<R> h = mk(R(0), R(0));
  if (live) {
    const uint2* wp = terms + r;
    const int len = off[r + 1] - off[r];
    const unsigned char* c0 = KIND == KIND_P2C && which ? cb : ca;
#pragma unroll(kUnrollHt<N>)
    for (int q = 0; q < len; ++q) {
      const uint2 w = wp[q * N];
      cx<R> p;
      if (KIND == KIND_P2C || !which) {
        p = term_coef_value<R, KIND, NVT>(w, c0);
      } else {
        const cx<R> u = c_fma(word_coef_b<R, NVT>(w, cb), word_coef<R, KIND, NVT>(w, ca),
                              c_mul(word_coef<R, KIND, NVT>(w, cb), word_coef_b<R, NVT>(w, ca)));
        p = c_scale(word_scale<R, NVT>(w), u);
      }
      h = acc_term<R, NVT>(h, p, w, xs);
    }
  }
  return which ? mk(-h.re, -h.im) : h;
}

template <typename R, int N, int W, int KIND, int NVX, int U>
__device__ __forceinline__ void eval_row(const Tables& tb, const unsigned char* ca, const unsigned char* xs, int r,
                                         bool live, cx<R> (&A)[N], int walk, uint2 seg, unsigned char* scr, unsigned nz) {
  // the row's k-th non-zero entry waits in slot k (W complex values each) until the row is read back
  auto read_back = [&]() {
    const cx<R>* sp = view<R>(scr) + r;
#pragma unroll
    for (int i = 0; i < N; ++i)
      A[i] = ((nz >> i) & 1u) ? sp[__popc(nz & ((1u << i) - 1u)) * W] : mk(R(0), R(0));
  };
  const int lanes = balanced_walk_built(N) ? tb.hx_off[N * N + 1] : kNoLanes;
  const bool balanced = balanced_walk_built(N) && walk == 2 && lanes != kNoLanes;
  if (!kFlatAlways<N> && walk == 0) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      cx<R> acc = mk(R(0), R(0));
      if (live) {
        const int base = tb.hx_off[r * N], j0 = tb.hx_off[r * N + i], j1 = tb.hx_off[r * N + i + 1];
        for (int j = j0; j < j1; ++j) {
          const uint2 w = tb.hx_terms[(j - base) * N + r];
          acc = acc_term<R, NVX>(acc, term_coef_value<R, KIND, NVX>(w, ca), w, xs);
        }
      }
      A[i] = acc;
    }
  } else if (balanced) {
    // this lane's share of the entries (every lane takes part); each finished sum goes into the slot of
    // its row, read back after the sub-warp synchronises
    const int len = (int)(seg.x >> 16);
    const uint2* wp = tb.hx_terms + r + (seg.x & 0xffffu) * W;  // (the staged section is the balanced one)
    cx<R> acc = mk(R(0), R(0));
#pragma unroll(U)
    for (int q = 0; q < len; ++q) {
      const uint2 w = wp[q * W];
      acc = acc_term<R, NVX>(acc, term_coef_value<R, KIND, NVX>(w, ca), w, xs);
      if (word_last<NVX>(w)) {
        view<R>(scr)[word_dst<NVX>(w, W)] = acc;
        acc = mk(R(0), R(0));
      }
    }
    __syncwarp(kFull);  // other lanes wrote this row's slots
    read_back();
  } else {
    if (live) {
      const int len = (int)(seg.x >> 16);
      const uint2* wp = tb.hx_terms + r + (seg.x & 0xffffu) * N;
      cx<R>* sp = view<R>(scr) + r + seg.y * W;
      cx<R> acc = mk(R(0), R(0));
#pragma unroll(U)
      for (int q = 0; q < len; ++q) {
        const uint2 w = wp[q * N];
        acc = acc_term<R, NVX>(acc, term_coef_value<R, KIND, NVX>(w, ca), w, xs);
        if (word_last<NVX>(w)) {  // the entry's sum is complete
          *sp = acc;
          sp += W;
          acc = mk(R(0), R(0));
        }
      }
    }
    __syncwarp(kFull);  // (a spread path's other sub-warps wrote slots of this row too)
    read_back();
  }
}

// Pivot key of a row for column i: magnitude |Re|+|Im| cut to its upper bits, position in the
// low 5 bits (largest key = largest cut magnitude, lowest position among equal ones).  Pivoted
// rows 0; a NaN at the current position wins, a NaN below never does.  The cut only speeds up the
// search: a near tie it gets wrong is found and redone on the full magnitudes (pivot_exact).
__device__ __forceinline__ unsigned mag_bits(double v) { return (unsigned)__double2hiint(v); }
__device__ __forceinline__ unsigned mag_bits(float v) { return __float_as_uint(v); }
template <typename R>
__device__ __forceinline__ unsigned pivot_key(R v, int pos, int i) {
  if (pos < i) return 0u;
  if (v != v) return (pos == i) ? (0xffffffe0u | (unsigned)(31 - pos)) : 0u;
  return ((mag_bits(v) >> 5) << 5) | (unsigned)(31 - pos);
}
__device__ __forceinline__ unsigned long long full_bits(double v) { return (unsigned long long)__double_as_longlong(v); }
__device__ __forceinline__ unsigned long long full_bits(float v) { return (unsigned long long)__float_as_uint(v); }

// compile-time loop: f(integral_constant<int, I>) for I in [B, E)
template <int B, int E, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (B < E) {
    f(std::integral_constant<int, B>{});
    static_for<B + 1, E>(f);
  }
}

// Partial-pivot LU + back substitution, one row per lane, rows in registers.  A zero pivot skips
// that column's elimination and leaves a non-finite solution, as in the reference.  Two forms, the
// operations of every entry in the oracle's order:
//   LU_GROUPED  columns in groups of lu_group(N), each group one rolled loop whose body eliminates
//               the row's first entry and shifts the row down by one, so that a column needs no
//               compile-time index: the code is one body per group instead of one per column.
//               The pivot rows stay in shared memory, where the back substitution finds them;
//               pivoted lanes go on computing values that nothing reads, so the update has no
//               branch.  What bounded the LU with every column unrolled was fetching its code
//               (gen-3v-4pt: 2.0 of 8.9 cycles per issue; grouped 0.2).  Measured when it took the
//               unrolled form's place (B200, default launch choice, groups of 2, 4 and 10 at N = 6,
//               12 and 30): gen-3v-4pt FP64 101.9 -> 92.8 ms (512 hypotheses), mixed 46.6 -> 39.0 (251),
//               CY 103.2 -> 96.8 (128), 30x30 FP64 126.8 -> 117.0 (48), mixed 86.8 -> 75.8 (37);
//               5-point equal (-0.4 %).
//   LU_SERIAL   (N <= 3) every lane of the sub-warp gathers the whole system through shared memory
//               and eliminates it in its registers, rows swapped by selects: no pivot search across
//               lanes and no broadcast per column, so a lone small system's solve is a short chain
//               (the single-instance P3P case is latency bound).
constexpr int LU_GROUPED = 0, LU_SERIAL = 1;
#ifndef GHC_LU_SERIAL_MAX_N
#define GHC_LU_SERIAL_MAX_N 3
#endif
template <int N>
constexpr int kLuForm = N <= GHC_LU_SERIAL_MAX_N ? LU_SERIAL : LU_GROUPED;
// Columns per group: a smaller group wastes fewer updates beyond the shrinking row (a group's columns
// all run at its first one's width), a larger one is less code and less shared memory.  B200, ms:
// N = 6 (five-point FP64) 10.64 at 1, 10.90 at 2, 11.21 at 6; N = 12 gen-3v-4pt FP64 83.5 at 3, 83.3 at
// 2, 83.8 at 4, 85.4 at 6, mixed 34.6, 35.1, 34.8, 36.9; N = 18 (6-point rolling shutter, one line, 187
// hypotheses) FP64 15.9 at 3, 15.7 at 2, 16.5 at 6, 17.1 at 9, FP32 11.2, 11.3, 11.5, 11.6, mixed 14.7, 14.8,
// 15.1, 15.5; N = 30 FP64 109.0 at 5, 112.0 at 6, 110.3 at 10, 114.1 at 3, FP32 67.0 at 5 and 6, 69.3 at 3,
// 71.8 at 10.  At N = 8, 10, 11 and 16 batches at 1, 2, 3 and 4 differ by up to 4 % either way (FP64 3-view
// triangulation, N = 8, 3.59, 3.64, 3.64, 3.65; 4-view, N = 11, 6.63, 6.60, 6.58, 6.71; 5-point full form,
// N = 16, 14.2, 14.4, 14.7, 14.8).
__host__ __device__ constexpr int lu_group(int N) { return N <= 6 ? 1 : N <= 18 ? 3 : 5; }
// stored pivot rows of a group that starts with rows of w entries: even stride (with the right-hand
// side at entry w), so that the back substitution's diagonal reads fall into different banks
__host__ __device__ constexpr int lu_row_stride(int w) { return (w + 2) & ~1; }
// offset of column i's stored pivot row
__host__ __device__ constexpr int lu_row_off(int N, int i) {
  int off = 0;
  for (int c = 0; c < N; c += lu_group(N)) {
    const int w = N - c;
    if (i < c + lu_group(N)) return off + (i - c) * lu_row_stride(w);
    off += lu_group(N) * lu_row_stride(w);
  }
  return off;
}
// complex values of the per-sub-warp solve scratch sx: the pivot rows with their right-hand sides,
// or, for the serial form, the whole system
__host__ __device__ constexpr int lu_scratch_len(int N) {
  return N <= GHC_LU_SERIAL_MAX_N ? N * (N + 1)
                                  : lu_row_off(N, N - 1) + lu_row_stride(N - (N - 1) / lu_group(N) * lu_group(N));
}

// Pivot position of column i by the reference's rule (dev-cgesv-batched-small.cuh:54-65): the
// largest |Re|+|Im| among the unpivoted rows, the lowest position among equal magnitudes, a NaN at
// position i kept and a NaN below never taken.  Sub-warps of 16 and 32 lanes: pivot_redux3 (below),
// exact in three warp reductions.  Narrower sub-warps, two steps:
//   pivot_fast   an integer max butterfly over pivot_key (one shuffle per level): the largest cut
//                magnitude, the lowest position among equal cut magnitudes;
//   cut_was_wrong  after the chosen row is broadcast, true on a lane whose row shares the winner's
//                cut magnitude but has a strictly larger full one -- the only way the cut choice
//                can differ from the exact one (equal full magnitudes are ordered by position in
//                both);
//   pivot_exact  the full magnitudes and the positions reduced as pairs, run (by the whole warp)
//                only when some lane saw cut_was_wrong.
template <typename R, int W>
__device__ __forceinline__ unsigned pivot_fast(unsigned key) {
  unsigned best = key;
#pragma unroll
  for (int off = W / 2; off > 0; off >>= 1) best = max(best, __shfl_xor_sync(kFull, best, off, W));
  return best;
}
// (magnitudes compared as bit patterns: non-negative values order like their bits, and a NaN --
// only a NaN below the current position can share a bucket -- merely sends the column to the exact
// reduction, which never takes it)
template <typename R>
__device__ __forceinline__ bool cut_was_wrong(R m, unsigned key, unsigned best, bool cand, R pm) {
  return cand && ((key ^ best) >> 5) == 0u && full_bits(m) > full_bits(pm);
}
template <typename R, int W>
__device__ __forceinline__ int pivot_exact(R m, bool cand, int pos, int i) {
  // (magnitude bits, position): non-negative magnitudes order as their bit patterns; a NaN at
  // position i first, a NaN below and the pivoted rows last
  unsigned long long mb = 0ull;
  int mp = 64;
  if (cand) {
    if (m == m) {
      mb = full_bits(m);
      mp = pos;
    } else if (pos == i) {
      mb = ~0ull;
      mp = pos;
    }
  }
#pragma unroll
  for (int off = W / 2; off > 0; off >>= 1) {
    const unsigned long long ob = __shfl_xor_sync(kFull, mb, off, W);
    const int op = __shfl_xor_sync(kFull, mp, off, W);
    if (ob > mb || (ob == mb && op < mp)) {
      mb = ob;
      mp = op;
    }
  }
  return mp;
}

// Warp reductions of the sub-warp (W = 16 or 32): max and min of a 32-bit value over the
// sub-warp's lanes; two sub-warps of 16 reduce at once, one by the operation, the other by the
// opposite operation on complemented values.
template <int W>
__device__ __forceinline__ unsigned subwarp_max(unsigned v) {
  static_assert(W == 16 || W == 32, "redux reductions need a sub-warp of 16 or 32");
  if constexpr (W == 32) {
    return __reduce_max_sync(kFull, v);
  } else {
    const bool upper = (threadIdx.x & 16u) != 0u;
    const unsigned lo = __reduce_max_sync(kFull, upper ? 0u : v);
    const unsigned hi = __reduce_min_sync(kFull, upper ? ~v : ~0u);
    return upper ? ~hi : lo;
  }
}
template <int W>
__device__ __forceinline__ unsigned subwarp_min(unsigned v) {
  static_assert(W == 16 || W == 32, "redux reductions need a sub-warp of 16 or 32");
  if constexpr (W == 32) {
    return __reduce_min_sync(kFull, v);
  } else {
    const bool upper = (threadIdx.x & 16u) != 0u;
    const unsigned lo = __reduce_min_sync(kFull, upper ? ~0u : v);
    const unsigned hi = __reduce_max_sync(kFull, upper ? ~v : 0u);
    return upper ? ~hi : lo;
  }
}
// The exact pivot position of column i in three sub-warp reductions (sub-warps of 16 or 32):
// the largest upper word of the candidates' magnitudes (shifted up by one so that a candidate
// with magnitude 0 still outranks a non-candidate; a NaN at position i above everything, a NaN
// below excluded), then the largest lower word among the candidates with that upper word, then
// the lowest position among those with both -- the reference's strict-> scan in position order.
// The candidate at position i always takes part, so some lane always wins.
template <typename R, int W>
__device__ __forceinline__ int pivot_redux3(R m, bool cand, int pos, int i) {
  const unsigned long long mb = full_bits(m);
  const unsigned hi = sizeof(R) == 8 ? (unsigned)(mb >> 32) : (unsigned)mb;
  unsigned khi = 0u;
  if (cand) khi = (m == m) ? hi + 1u : (pos == i ? 0xffffffffu : 0u);
  const unsigned top = subwarp_max<W>(khi);
  bool win = khi != 0u && khi == top;
  if constexpr (sizeof(R) == 8) {
    const unsigned lo = (unsigned)mb;
    const unsigned low = subwarp_max<W>(win ? lo : 0u);
    win = win && lo == low;
  }
  return (int)subwarp_min<W>(win ? (unsigned)pos : 63u);
}
template <int W>
constexpr bool kPivotRedux3 = W == 16 || W == 32;

// PivotRange: what one solve saw of its pivot magnitudes |U_ii| (|Re|+|Im|).  singular(): a zero
// pivot, unless column 0's magnitude was NaN (the oracle's running minimum then stays NaN).  With
// SPAN (the mixed tracker's conditioning test) also the smallest and largest magnitudes and whether
// any was NaN; without it only two flags stay live across the LU.
template <typename R, bool SPAN>
struct PivotRange {
  R lo = R(__builtin_huge_val()), hi = R(0);
  bool nan = false, zero = false, nan0 = false;
  __device__ __forceinline__ void add(bool first, R pm) {
    if (first) nan0 = pm != pm;
    zero = zero || pm == R(0);
    if constexpr (SPAN) {
      lo = pm < lo ? pm : lo;
      hi = pm > hi ? pm : hi;
      nan = nan || pm != pm;
    }
  }
  __device__ __forceinline__ bool singular() const { return zero && !nan0; }
};

// returns this lane's component of the solution (lane l < N: component l)
template <typename R, int N, int W, bool SPAN>
__device__ __forceinline__ cx<R> lu_solve_grouped(cx<R> (&A)[N], cx<R> b, int l, cx<R>* sx, cx<R>* sol,
                                                  PivotRange<R, SPAN>& rg) {
  constexpr int G = lu_group(N);
  int pos = l < N ? l : -1;  // the row's position; -1: pivoted (or no row)
  static_for<0, (N + G - 1) / G>([&](auto gc) {
    constexpr int c0 = decltype(gc)::value * G, w = N - c0, n = w < G ? w : G;
    cx<R>* px = sx + lu_row_off(N, c0);
#pragma unroll 1
    for (int i = c0; i < c0 + n; ++i, px += lu_row_stride(w)) {
      const R m = fabs(A[0].re) + fabs(A[0].im);
      const bool cand = pos >= i;
      // The group's later columns have shorter rows; leaving their last entries out (uniformly) spares
      // shared-memory traffic, which bounds FP64 up to 16 unknowns (gen-3v-4pt 91.9 -> 89.8 ms, CY
      // 93.9 -> 91.9; batches at N = 8, 10 and 11 equal, 5-point full form, N = 16, 14.5 -> 14.7, and one
      // instance there 4 to 7 % slower); in FP32 and at N = 30 the added branches cost more (mixed
      // 39.5 -> 40.9, 30x30 112.9 -> 118.2).
      constexpr bool kTrim = sizeof(R) == 8 && N > 6 && N <= 16;
      const int t = i - c0;
      auto has = [&](auto jc) {
        return !kTrim || decltype(jc)::value + n <= w || decltype(jc)::value < w - t;
      };
      auto store = [&]() {
        static_for<0, w>([&](auto jc) {
          if (has(jc)) px[decltype(jc)::value] = A[decltype(jc)::value];
        });
        px[w] = b;
      };
      int bp;
      unsigned key = 0u, best = 0u;
      if constexpr (kPivotRedux3<W>) {
        bp = pivot_redux3<R, W>(m, cand, pos, i);
      } else {
        key = cand ? pivot_key(m, pos, i) : 0u;
        best = pivot_fast<R, W>(key);
        bp = 31 - (int)(best & 31u);
      }
      if (pos == bp) store();
      __syncwarp(kFull);
      cx<R> p_i = px[0];
      R pm = fabs(p_i.re) + fabs(p_i.im);
      if (!kPivotRedux3<W> && __any_sync(kFull, cut_was_wrong(m, key, best, cand, pm))) {
        bp = pivot_exact<R, W>(m, cand, pos, i);
        __syncwarp(kFull);  // every lane has read the first choice
        if (pos == bp) store();
        __syncwarp(kFull);
        p_i = px[0];
        pm = fabs(p_i.re) + fabs(p_i.im);
      }
      rg.add(c0 == 0 && i == 0, pm);
      // (a zero pivot's reciprocal is NaN, as the oracle's c_rcp(0))
      const cx<R> rc = c_rcp(p_i);
      if (pos == bp) {
        sol[i] = rc;  // waits in the solution slot of its position until the back substitution
        pos = -1;
      } else if (pos == i) {
        pos = bp;
      }
      cx<R> f = c_mul(A[0], rc);
      if (__any_sync(kFull, pm == R(0))) {
        // Rare: a path of the warp skips the column.  Its update takes zero times a row of zeros from
        // every entry, which leaves them (a zero may lose its sign); the stored row is not needed, for
        // the NaN reciprocal makes its component NaN whatever the row holds.
        if (pm == R(0)) {
          f = mk(R(0), R(0));
          for (int k = l; k <= w; k += W) px[k] = f;
        }
        __syncwarp(kFull);
      }
      static_for<0, w - 1>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        if (has(std::integral_constant<int, j + 1>{})) A[j] = c_fnma(f, px[j + 1], A[j + 1]);
      });
      b = c_fnma(f, px[w], b);
    }
  });
  __syncwarp(kFull);  // the pivot rows and reciprocals are stored
  // back substitution: lane l takes the pivot row of position l
  const cx<R>* row = sx;
  int w = N;
  static_for<0, (N + G - 1) / G>([&](auto gc) {
    constexpr int c0 = decltype(gc)::value * G;
    if (l >= c0 && l < N) {
      row = sx + lu_row_off(N, c0) + (l - c0) * lu_row_stride(N - c0);
      w = N - c0;
    }
  });
  b = row[w];
  const cx<R> rc = l < N ? sol[l] : mk(R(0), R(0));
#pragma unroll 2
  for (int i = N - 1; i > 0; --i) {
    const cx<R> z = c_mul(b, rc);
    const cx<R> xi = mk(__shfl_sync(kFull, z.re, i, W), __shfl_sync(kFull, z.im, i, W));
    if (l < i) b = c_fnma(row[i - l], xi, b);
  }
  __syncwarp(kFull);  // the scratch may be written again
  return c_mul(b, rc);
}

// The serial form: the oracle's elimination (rows at positions, strict-> scan from position i,
// zero pivot skipping its column, back substitution by the stored reciprocals) run by every lane
// on its own copy of the system; returns component l of the solution in lane l < N.
template <typename R, int N, int W, bool SPAN>
__device__ __forceinline__ cx<R> lu_solve_serial(cx<R> (&A)[N], cx<R> b, int l, cx<R>* sx,
                                                 PivotRange<R, SPAN>& rg) {
  constexpr int C = N + 1;  // row length with the right-hand side
  if (l < N) {
    static_for<0, N>([&](auto jc) { sx[l * C + decltype(jc)::value] = A[decltype(jc)::value]; });
    sx[l * C + N] = b;
  }
  __syncwarp(kFull);
  cx<R> M[N][C];
  static_for<0, N>([&](auto rc_) {
    static_for<0, C>([&](auto jc) { M[decltype(rc_)::value][decltype(jc)::value] = sx[decltype(rc_)::value * C + decltype(jc)::value]; });
  });
  __syncwarp(kFull);  // every lane has its copy before the next solve rewrites sx
  cx<R> rcp[N];
  static_for<0, N>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    R best = fabs(M[i][i].re) + fabs(M[i][i].im);
    int bp = i;
    static_for<i + 1, N>([&](auto jc) {
      constexpr int j = decltype(jc)::value;
      const R v = fabs(M[j][i].re) + fabs(M[j][i].im);
      if (v > best) {
        best = v;
        bp = j;
      }
    });
    rg.add(i == 0, best);
    // the pivot row moves to position i, the row at position i to the pivot's position
    static_for<i + 1, N>([&](auto jc) {
      constexpr int j = decltype(jc)::value;
      if (bp == j) {
        static_for<i, C>([&](auto kc) {
          constexpr int k = decltype(kc)::value;
          const cx<R> t = M[i][k];
          M[i][k] = M[j][k];
          M[j][k] = t;
        });
      }
    });
    const bool zero = best == R(0);
    rcp[i] = c_rcp(M[i][i]);
    if (!zero) {
      static_for<i + 1, N>([&](auto rc_) {
        constexpr int r = decltype(rc_)::value;
        M[r][i] = c_mul(M[r][i], rcp[i]);
        static_for<i + 1, C>([&](auto jc) {
          constexpr int j = decltype(jc)::value;
          M[r][j] = c_fnma(M[r][i], M[i][j], M[r][j]);
        });
      });
    }
  });
  cx<R> z[N];
  static_for<0, N>([&](auto ic) {
    constexpr int i = N - 1 - decltype(ic)::value;
    z[i] = c_mul(M[i][N], rcp[i]);
    static_for<0, i>([&](auto rc_) {
      constexpr int r = decltype(rc_)::value;
      M[r][N] = c_fnma(M[r][i], z[i], M[r][N]);
    });
  });
  cx<R> mine = z[0];
  static_for<1, N>([&](auto jc) {
    if (l == decltype(jc)::value) mine = z[decltype(jc)::value];
  });
  return mine;
}

template <typename R, int N, int W, bool SPAN>
__device__ __forceinline__ cx<R> lu_solve(cx<R> (&A)[N], cx<R> b, int l, cx<R>* sx, cx<R>* sol,
                                          PivotRange<R, SPAN>& rg) {
  if constexpr (kLuForm<N> == LU_SERIAL) return lu_solve_serial<R, N, W>(A, b, l, sx, rg);
  else return lu_solve_grouped<R, N, W>(A, b, l, sx, sol, rg);
}
template <typename R, int N, int W>
__device__ __forceinline__ cx<R> lu_solve(cx<R> (&A)[N], cx<R> b, int l, cx<R>* sx, cx<R>* sol) {
  PivotRange<R, false> rg;
  return lu_solve<R, N, W>(A, b, l, sx, sol, rg);
}

// xor-butterfly sum over the NP = W lanes of the sub-warp (order = oracle tree_sum); the same bits in
// every lane, for a + b = b + a
template <typename R, int N, int W>
__device__ __forceinline__ R tree_sum(R v) {
  constexpr int NP = (N <= 1) ? 1 : (N <= 2) ? 2 : (N <= 4) ? 4 : (N <= 8) ? 8 : (N <= 16) ? 16 : 32;
  static_assert(NP == W, "every lane of the sub-warp is a leaf of the reduction tree");
#pragma unroll
  for (int off = NP / 2; off > 0; off >>= 1) v = f_add(v, shfl_xor(v, off, W));
  return v;
}

// per-sub-warp shared-memory views
struct SubMem {
  unsigned char* coefA;  // c_k(t)   or p(t)     [Mc]
  unsigned char* coefB;  // c'_k(t)  or p1 - p0  [Mc]
  unsigned char* xs;     // track [N+1]
  unsigned char* sx;     // solve scratch [lu_scratch_len(N)]: the pivot rows + rhs, or the whole system
  unsigned char* sol;    // pivot reciprocals [N]
  unsigned char* state;  // per lane: RK base point x0 [W], RK accumulator [W] (state precision)
  unsigned char* scr;    // H_x row scratch [slots][W] of the flat walks, in the solve scratch's place
  unsigned char* seg;    // per lane: the terms of its H_x walk, first | number << 16, and the first one's slot [W]
  unsigned char* rec;    // the path's scalar state while the sub-warp evaluates and solves [kRecBytes]
  unsigned char* coefH;  // mixed: c_k(t) or p(t) in state precision, for the residual H [Mc] (else null)
  unsigned char* xsH;    // mixed: the track in state precision [N+1] (else null)
  unsigned char* xst;    // the track in state precision: xsH when mixed, else xs
  unsigned nz;           // this lane's row: bit i set when H_x entry (row, i) has terms
  int walk;              // H_x walk: 0 entry-wise, 1 row-wise, 2 balanced
};
constexpr int kRecBytes = 80;

// bit i set when row r of H_x has terms in column i (0 for lanes beyond the rows)
template <int N>
__device__ __forceinline__ unsigned row_mask(const uint16_t* hx_off, int r) {
  unsigned m = 0u;
  if (r < N)
    for (int i = 0; i < N; ++i)
      if (hx_off[r * N + i + 1] > hx_off[r * N + i]) m |= 1u << i;
  return m;
}

// This lane's part of the H_x walk: all of its list (row l, or, balanced, the l-th share), or, for one of
// `parts` sub-warps that evaluate one path together, the part-th piece of it, cut between entries.
template <int N, int W, int NVX>
__device__ __forceinline__ uint2 walk_range(const Tables& tb, int walk, int l, int part, int parts) {
  const bool balanced = balanced_walk_built(N) && walk == 2 && tb.hx_off[N * N + 1] != kNoLanes;
  const int len = balanced ? tb.hx_off[N * N + 2 + l] : l < N ? tb.hx_off[l * N + N] - tb.hx_off[l * N] : 0;
  const int stride = balanced ? W : N;
  int first = len, end = len, slot = 0, slots = 0;
  for (int q = 0; q <= len; ++q) {  // q: a place where an entry begins (or the list ends)
    if (q > 0 && !word_last<NVX>(tb.hx_terms[(q - 1) * stride + l])) continue;
    if (q > 0) ++slots;
    if (first == len && q * parts >= len * part) {
      first = q;
      slot = slots;
    }
    if (q * parts >= len * (part + 1)) {
      end = q;
      break;
    }
  }
  return make_uint2((unsigned)first | (unsigned)(end - first) << 16, (unsigned)slot);
}

// Row l of H_x and the right-hand side (which = 1: -H_t, which = 0: H), term walk of table shape S
// (EvalShape), in the linear-algebra precision RL.  With a state precision R above RL (mixed), the
// corrector's H is evaluated in R from the R copies of the coefficients and the track, then rounded
// to RL for the solve: Newton then converges to the R-accurate root at a rate set by the RL solve.
template <typename R, typename RL, int N, int W, int KIND, int S>
__device__ __forceinline__ void eval_any(const Tables& tb, const SubMem& sm, int l, cx<RL> (&A)[N], cx<RL>& b,
                                         int which) {
  constexpr int NVX = shape_nvx(S);
  eval_row<RL, N, W, KIND, NVX, kUnrollHx<N, NVX, !std::is_same<R, RL>::value>>(
      tb, sm.coefA, sm.xs, l, l < N, A, sm.walk, reinterpret_cast<const uint2*>(sm.seg)[l], sm.scr, sm.nz);
  if constexpr (std::is_same<R, RL>::value) {
    b = eval_rhs<RL, N, KIND, shape_nvt(S)>(tb.ht_terms, tb.ht_off, sm.coefA, sm.coefB, sm.xs, l, l < N, which);
  } else {
    if (which)
      b = eval_rhs<RL, N, KIND, shape_nvt(S)>(tb.ht_terms, tb.ht_off, sm.coefA, sm.coefB, sm.xs, l, l < N, 1);
    else
      b = c_cast<RL>(eval_rhs<R, N, KIND, shape_nvt(S)>(tb.ht_terms_hi, tb.ht_off, sm.coefH, sm.coefH, sm.xsH, l,
                                                        l < N, 0));
  }
}

// one evaluation + solve in precision RL; returns this lane's solution component in R.  ill (mixed
// tracker, cond_limit > 0): the pivot magnitudes spanned more than cond_limit or one was NaN -- the
// RL solve is too ill-conditioned to keep Newton's contraction
template <typename R, typename RL, int N, int W, int KIND, int S>
__device__ __forceinline__ cx<R> eval_solve(const Tables& tb, const SubMem& sm, int l, int which, double cond_limit,
                                            bool& ill, bool& sing) {
  cx<RL> A[N];
  cx<RL> b;
  eval_any<R, RL, N, W, KIND, S>(tb, sm, l, A, b, which);
  constexpr bool kSpan = !std::is_same<R, RL>::value;  // only the mixed tracker tests conditioning
  PivotRange<RL, kSpan> rg;
  __syncwarp(kFull);  // the solve's scratch shares the row scratch's memory
  const cx<RL> z = lu_solve<RL, N, W>(A, b, l, view<RL>(sm.sx), view<RL>(sm.sol), rg);
  if constexpr (kSpan) ill = cond_limit > 0.0 && (rg.nan || !(rg.hi <= (RL)cond_limit * rg.lo));
  else ill = false;
  sing = rg.singular();
  return l < N ? c_cast<R>(z) : mk(R(0), R(0));
}
template <typename R, typename RL, int N, int W, int KIND, int S>
__device__ __forceinline__ cx<R> eval_solve(const Tables& tb, const SubMem& sm, int l, int which) {
  bool ill, sing;
  return eval_solve<R, RL, N, W, KIND, S>(tb, sm, l, which, 0.0, ill, sing);
}

// the track into shared memory: in RL for H_x and H_t, and (mixed) in R for the residual; its last
// slot, the constant 1 of the term tables, is written once (write_one)
template <typename R, typename RL, int N>
__device__ __forceinline__ void write_track(const SubMem& sm, int l, cx<R> x) {
  if (l < N) {
    view<RL>(sm.xs)[l] = c_cast<RL>(x);
    if constexpr (!std::is_same<R, RL>::value) view<R>(sm.xsH)[l] = x;
  }
}
template <typename R, typename RL, int N>
__device__ __forceinline__ void write_one(const SubMem& sm, int l) {
  if (l == 0) {
    view<RL>(sm.xs)[N] = mk(RL(1), RL(0));
    if constexpr (!std::is_same<R, RL>::value) view<R>(sm.xsH)[N] = mk(R(1), R(0));
  }
}

template <typename R, typename RL, int W, int KIND>
__device__ __forceinline__ void coef_eval(const TrackParams& p, const SubMem& sm, long long hyp, R t, bool fresh, int l, int step) {
  constexpr bool HI = !std::is_same<R, RL>::value;
  if (KIND == KIND_P2C) {
    coef_eval_p2c<R, RL, HI>(p.coef_hx + 2 * hyp * p.stride_hx, p.coef_ht + 2 * hyp * p.stride_ht, p.M, p.K, t, fresh,
                                view<RL>(sm.coefA), view<RL>(sm.coefB), view<R>(sm.coefH), l, step);
  } else {
    coef_eval_ph<R, RL, HI>(p.p_start, p.p_tgt + 2 * hyp * p.stride_p, p.p_diff + 2 * hyp * p.stride_p, p.P, t, fresh,
                               view<RL>(sm.coefA), view<RL>(sm.coefB), view<R>(sm.coefH), l, step);
  }
}

// term words that a CTA of table shape S stages (EVAL_IN_PLACE: none)
template <int S>
__host__ __device__ inline int hx_words(int walk, int n_hx, int n_rows) {
  return S == EVAL_IN_PLACE ? 0 : staged_words(walk, n_hx, n_rows);
}
template <int S>
__host__ __device__ inline int ht_words(int n_ht) {
  return S == EVAL_IN_PLACE ? 0 : n_ht;
}

// byte sizes of the shared-memory layout
__host__ __device__ inline size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }
__host__ __device__ inline size_t tables_bytes(int N, int n_hx, int n_ht, bool mixed) {
  return align16(8 * ((size_t)n_hx + (mixed ? 2 : 1) * (size_t)n_ht) + 2 * (size_t)(hx_off_len(N) + N + 1));
}
// Per sub-warp: the path record [kRecBytes], the lanes' walk ranges [W], then, in complex values of e bytes (linear-algebra
// precision): track [N+1], pivot reciprocals [N]; the lane state [2 W] and, when es != e (mixed), the
// state-precision track [N+1] in complex values of es bytes (state precision); the row scratch
// [slots W] (flat) in the same place as the solve scratch [lu_scratch_len(N)]; the coefficient buffers
// [2 Mc] and, mixed, the state-precision coefficients [Mc].  What the problem's tables do not size
// comes first, so its offsets are constants of the kernel.  An odd multiple of 16 bytes: equal places
// of two sub-warps never fall into the same banks; with 4 lanes three or five eighths of a bank row
// apart, so that the windows of four complex values which neighbouring sub-warps read overlap least
// (P3P FP64, 20,000 hypotheses: 1.80 ms at 48 bytes beyond a multiple of 128, 1.90 at 112, 2.03 at 64).
struct SubOffsets {
  size_t seg, coefA, coefB, xs, sx, sol, state, scr, coefH, xsH, bytes;
};
__host__ __device__ inline SubOffsets sub_offsets(int N, int Mc, int W, int slots, int e, int es) {
  const bool mixed = es != e;
  SubOffsets o;
  size_t off = kRecBytes;
  o.seg = off;
  off += 8 * (size_t)W;
  o.xs = off;
  off += (size_t)e * (N + 1);
  o.sol = off;
  off = align16(off + (N <= GHC_LU_SERIAL_MAX_N ? 0 : (size_t)e * N));
  o.state = off;
  off += (size_t)es * 2 * W;
  o.xsH = 0;
  if (mixed) {
    o.xsH = off;
    off += (size_t)es * (N + 1);
  }
  o.sx = o.scr = off;
  off += (size_t)e * (slots * W > lu_scratch_len(N) ? slots * W : lu_scratch_len(N));
  o.coefA = off;
  off += (size_t)e * Mc;
  o.coefB = off;
  off += (size_t)e * Mc;
  o.coefH = 0;
  if (mixed) {
    off = align16(off);
    o.coefH = off;
    off += (size_t)es * Mc;
  }
  o.bytes = align16(off) | 16;
  if (W == 4)
    while (o.bytes % 128 != 48 && o.bytes % 128 != 80) o.bytes += 16;
  return o;
}
__host__ __device__ inline size_t sub_bytes(int N, int Mc, int W, int slots, int e, int es) {
  return sub_offsets(N, Mc, W, slots, e, es).bytes;
}
template <typename R, typename RL>
__device__ __forceinline__ SubMem sub_layout(unsigned char* base, int N, int Mc, int W, int slots, bool flat) {
  const SubOffsets o = sub_offsets(N, Mc, W, flat ? slots : 0, (int)sizeof(cx<RL>), (int)sizeof(cx<R>));
  SubMem sm;
  sm.rec = base;
  sm.seg = base + o.seg;
  sm.coefA = base + o.coefA;
  sm.coefB = base + o.coefB;
  sm.xs = base + o.xs;
  sm.sx = base + o.sx;
  sm.sol = base + o.sol;
  sm.state = base + o.state;
  sm.scr = base + o.scr;
  const bool mixed = !std::is_same<R, RL>::value;
  sm.coefH = mixed ? base + o.coefH : nullptr;
  sm.xsH = mixed ? base + o.xsH : nullptr;
  sm.xst = mixed ? sm.xsH : sm.xs;
  return sm;
}

// complex entry idx of an array of doubles (f64) or floats, in precision R
template <typename R>
__device__ __forceinline__ cx<R> load_cx(const void* base, bool f64, long long idx) {
  if (f64) {
    const double* d = reinterpret_cast<const double*>(base) + 2 * idx;
    return mk((R)d[0], (R)d[1]);
  }
  const float* f = reinterpret_cast<const float*>(base) + 2 * idx;
  return mk((R)f[0], (R)f[1]);
}

// CTAs of 128 threads per SM the tracker asks the register allocator for: the row of H_x (N complex
// values) dominates the registers, so small systems afford more.  Two compiled variants per size and
// precision; the autotuner (ghc_autotune) picks one per problem.  Variant 0 is the best of B200 sweeps
// (autotuning off, 3..8 CTAs, ms): FP64 N = 3 (20,000 hypotheses) 2.14 at 6, 2.13 at 7, 2.26 at 4;
// N = 6 (2,048) 12.4 at 4, 13.1 at 3, 12.8 at 6; N = 12 (gen-3v-4pt, 512) 92.1 at 5, 94.5 at 4, 101 at
// 6; N = 30 (48) 113 at 3, 189 at 4 (spills).  FP32 N = 6 (1,000) 6.00 at 6, 6.11 at 8; N = 12 (200)
// 111.9 at 6, 113.0 at 5, 118.4 at 7; N = 30 72.6 at 4, 74.8 at 5, 79.1 at 3.  The mixed tracker (FP64
// state, FP32 linear algebra) N = 12 (251) 38.8 at 6, 38.7 at 5, 40.9 at 7; N = 30 73.3 at 4, 74.7 at
// 3, 158 at 5.  Variant 1 is the runner-up budget.
template <int N, typename R, typename RL, int V>
constexpr int track_min_blocks() {
  return !std::is_same<R, RL>::value
             ? (V == 0 ? (N <= 8 ? 6 : N <= 12 ? 6 : N <= 18 ? 4 : 4) : (N <= 8 ? 8 : N <= 12 ? 5 : N <= 18 ? 5 : 3))
         : V == 0 ? (sizeof(R) == 8 ? (N <= 4 ? 6 : N <= 8 ? 4 : N <= 12 ? 5 : 3)
                                    : (N <= 4 ? 8 : N <= 12 ? 6 : 4))
                  : (sizeof(R) == 8 ? (N <= 4 ? 8 : N <= 8 ? 6 : N <= 12 ? 4 : N <= 18 ? 4 : 2)
                                    : (N <= 4 ? 10 : N <= 8 ? 8 : 5));
}

template <typename R, typename RL, int N, int KIND, int S>
__device__ __forceinline__ Tables stage_tables(unsigned char* smem, const uint64_t* g_hx, const uint16_t* g_hxo,
                                               const uint64_t* g_ht, const uint16_t* g_hto, int n_hx, int n_rows,
                                               int n_ht, int walk) {
  constexpr bool mixed = !std::is_same<R, RL>::value;
  constexpr int W = subwarp_width(N), NVX = shape_nvx(S), NVT = shape_nvt(S);
  if (walk == 2 && n_rows < n_hx) g_hx += n_rows;
  n_hx = hx_words<S>(walk, n_hx, n_rows);
  n_ht = ht_words<S>(n_ht);
  uint2* s_hx = reinterpret_cast<uint2*>(smem);
  uint2* s_ht = s_hx + n_hx;
  uint2* s_hth = mixed ? s_ht + n_ht : s_ht;
  uint16_t* s_hxo = reinterpret_cast<uint16_t*>(s_hth + n_ht);
  uint16_t* s_hto = s_hxo + hx_off_len(N);
  for (int i = threadIdx.x; i < n_hx; i += blockDim.x) s_hx[i] = pack_term<RL, KIND, NVX>(__ldg(g_hx + i), W);
  for (int i = threadIdx.x; i < n_ht; i += blockDim.x) {
    const uint64_t w = __ldg(g_ht + i);
    s_ht[i] = pack_term<RL, KIND, NVT>(w, W);
    if constexpr (mixed) s_hth[i] = pack_term<R, KIND, NVT>(w, W);
  }
  for (int i = threadIdx.x; i < hx_off_len(N); i += blockDim.x) s_hxo[i] = __ldg(g_hxo + i);
  for (int i = threadIdx.x; i < N + 1; i += blockDim.x) s_hto[i] = __ldg(g_hto + i);
  __syncthreads();
  Tables t;
  if constexpr (S == EVAL_IN_PLACE) {
    t.hx_terms = reinterpret_cast<const uint2*>(g_hx);
    t.ht_terms = t.ht_terms_hi = reinterpret_cast<const uint2*>(g_ht);
  } else {
    t.hx_terms = s_hx;
    t.ht_terms = s_ht;
    t.ht_terms_hi = s_hth;
  }
  t.hx_off = s_hxo;
  t.ht_off = s_hto;
  return t;
}

// -------------------------------------------------------------------------------------------------
// the tracker kernel: state, step control and norms in precision R, H_x, H_t and the LU in RL
// (R = RL: the plain FP64 and FP32 trackers; R = double, RL = float: the mixed tracker, whose
// corrector evaluates its residual H in R, so its endpoints converge to FP64 accuracy)
//
// Each sub-warp runs its path as a small state machine (phase 0..3 = RK stage,
// 4 = Newton iteration).  One trip of the warp loop performs exactly one
// evaluate-and-solve for every sub-warp, whatever its phase, so the
// LU exists once in the code and sub-warps of one warp never wait on each
// other's corrector iterations.
//
// Handover (first phase of the mixed-precision mode: t_handover > 0 or
// fail_limit > 0): a path also stops when t reaches t_handover, after
// fail_limit consecutive failed steps, or when the corrector sees divergence,
// leaving its last accepted point, t and dt in endpoints / t_end / dt_end.
// A resuming launch (resume = 1) starts every item from track_in at t_in[i]
// with step dt_in[i] and the step / corrector counts already in steps / corr.
// -------------------------------------------------------------------------------------------------
// Most threads per CTA of a tracker instantiation.  Where the coefficient buffers of a path, not the
// registers, limit the paths on an SM (FP64 at 5 to 8 unknowns: 2.4 of 3.8 KB a path for the 75
// coefficients of the five-point problem), the launch may use CTAs of up to 256 threads: one copy of
// the tables serves more paths, and what shared memory remains is handed out in finer steps.
template <int N, typename R, typename RL, int V>
constexpr int track_block() {
  return track_min_blocks<N, R, RL, V>() % 2 == 0 && N > 4 && N <= 8 ? 256 : 128;
}
template <int N, typename R, typename RL, int V>
constexpr int track_ctas() {
  return track_min_blocks<N, R, RL, V>() * 128 / track_block<N, R, RL, V>();
}
// WK >= 0: the H_x walk is fixed at compile time (only that walk's code is in the kernel, which
// spares the register allocator the other walk's read-back: above 16 unknowns, where the row fills
// most of the registers); WK < 0: chosen at run time from p.flat_eval.
//
// track_body is the work of one CTA on the items of p: CTA number `cta` of the `n_cta` CTAs that
// serve p (first items static: one per sub-warp slot of the CTA; then the shared counter), or,
// as a `visitor` (a CTA of another bucket of a mixed launch whose own items are done), items
// from p's counter only.  smem: the CTA's dynamic shared memory.
template <typename R, typename RL, int N, int W, int KIND, int S, int WK>
__device__ __forceinline__ void track_body(const TrackParams& p, unsigned char* smem, long long cta, long long n_cta,
                                           bool visitor) {
  const int walk = WK >= 0 ? WK : ((kFlatAlways<N> && p.flat_eval == 0) ? 1 : p.flat_eval);
  const int n_hx = hx_words<S>(walk, p.n_hx_terms, p.n_hx_rows), n_ht = ht_words<S>(p.n_ht_terms);
  const Tables tb = stage_tables<R, RL, N, KIND, S>(smem, p.hx_terms, p.hx_off, p.ht_terms, p.ht_off, p.n_hx_terms,
                                                    p.n_hx_rows, p.n_ht_terms, walk);

  const int lane = threadIdx.x & 31;
  const int l = lane % W;
  const int g = threadIdx.x / W;
  const int Mc = (KIND == KIND_P2C) ? p.M + 1 : p.P + 1;
  const bool flat = walk != 0;
  SubMem sm = sub_layout<R, RL>(smem + tables_bytes(N, n_hx, n_ht, !std::is_same<R, RL>::value) +
                                    (size_t)g * sub_bytes(N, Mc, W, flat ? p.scr_slots : 0, (int)sizeof(cx<RL>),
                                                          (int)sizeof(cx<R>)),
                                N, Mc, W, p.scr_slots, flat);
  sm.nz = row_mask<N>(tb.hx_off, l);
  sm.walk = walk;
  write_one<R, RL, N>(sm, l);
  // Spread, all sub-warps of the warp have the same path: they share one copy of the coefficients and
  // of the row scratch, and each evaluates a part of both, which shortens the chain of a lone path
  // (B200, one instance: P3P FP64 107 -> 92 us, 5-point FP32 2.19 -> 1.57 ms).  What a sub-warp updates in place, and its solve, stay its own.
  reinterpret_cast<uint2*>(sm.seg)[l] =
      walk_range<N, W, shape_nvx(S)>(tb, walk, l, p.spread ? lane / W : 0, p.spread ? 32 / W : 1);
  if (p.spread) {
    const SubMem first = sub_layout<R, RL>(
        smem + tables_bytes(N, n_hx, n_ht, !std::is_same<R, RL>::value) +
            (size_t)(g - lane / W) * sub_bytes(N, Mc, W, flat ? p.scr_slots : 0, (int)sizeof(cx<RL>), (int)sizeof(cx<R>)),
        N, Mc, W, p.scr_slots, flat);
    sm.coefA = first.coefA;
    sm.coefB = first.coefB;
    sm.coefH = first.coefH;
    sm.scr = first.scr;
  }
  // this lane's RK base point x0 and accumulator sols live in shared memory (register relief)
  cx<R>& x0 = view<R>(sm.state)[l];
  cx<R>& sols = view<R>(sm.state)[W + l];

  // Paths go to sub-warps in order, or, when the launch has fewer paths than one wave of warps
  // (spread), one path to each warp: a lone instance then has no two paths in one warp, whose
  // phases would serialise each other's step logic.  The other sub-warps of the warp track the
  // same path in lockstep (identical work, so no divergence and no idle lanes computing on stale
  // shared memory); only the first one (primary) writes results and takes the next path.
  const int subs_per_cta = blockDim.x / W;
  const int slots_per_cta = p.spread ? (int)(blockDim.x / 32) : subs_per_cta;
  const long long n_sw = n_cta * slots_per_cta;
  const bool primary = !p.spread || lane < W;
  const int leader = lane - l;
  // handover rules (first phase of the mixed mode): only the mixed tracker's launch sets them
  constexpr bool kMixed = !std::is_same<R, RL>::value;
  const bool handover = kMixed && (p.t_handover > 0.0 || p.fail_limit > 0);
  const bool by_time = kMixed && p.t_handover > 0.0;
  const R t_hand = kMixed ? (R)p.t_handover : R(0);

  // per-path state (replicated across the sub-warp's lanes)
  long long item = p.spread ? cta * slots_per_cta + (threadIdx.x >> 5) : cta * subs_per_cta + g;
  if (visitor) {  // the first item from the counter too (the static ones belong to p's own CTAs)
    long long nxt = 0;
    if (l == 0 && primary) nxt = n_sw + (long long)atomicAdd(reinterpret_cast<unsigned*>(p.counter), 1u);
    item = __shfl_sync(kFull, nxt, p.spread ? 0 : leader);
  }
  bool alive = item < p.n_items;
  long long hyp = 0;
  cx<R> x = mk(R(0), R(0));
  R t0 = 0, dt = 0, t_step = 0, half = 0, dt_pre = 0;
  R coef_t = R(-1);  // the t at which this sub-warp's coefficient buffers hold c_k(t) (-1: none)
  bool end_zone = false, success = false, inf = false, finished = false;
  // mixed tracker only: a solve of this step was ill-conditioned, or the step fell below the floor: stop
  bool step_ill = false, ill_stop = false;
  bool step_sing = false, last_sing = false;  // a solve of this step / the last completed step had a zero pivot
  int nsucc = 0, step = 0, ncorr = 0, phase = 0, cit = 0, nfail = 0;
  const R dt_init = (KIND == KIND_PH) ? R(0.01) : R(0.05);

  // end-zone clamp and bookkeeping at the start of a step (kernel_HC_Solver_P3P.cu:121-134)
  auto prologue = [&]() {
    if (!end_zone && fabs(f_sub(R(1), t0)) <= R(0.0500001)) end_zone = true;
    if (end_zone) {
      const R rem = fabs(f_sub(R(1), t0));
      if (dt > rem) dt = rem;
    } else {
      const R edge = (KIND == KIND_PH) ? fabs(f_sub(R(0.95), t0)) : fabs(f_sub(f_sub(R(1), R(0.05)), t0));
      if (dt > edge) dt = edge;
    }
    dt_pre = dt;  // the step without the handover clamp: the next phase resumes with it
    if (by_time && dt > f_sub(t_hand, t0)) dt = f_sub(t_hand, t0);
    t_step = t0;
    half = f_mul(R(0.5), dt);
    phase = 0;
    cit = 0;
    step_ill = false;
    step_sing = false;
  };
  // the path stops before its next step (kernel_HC_Solver_P3P.cu:247-249, plus the handover rules)
  auto at_end = [&]() -> bool {
    return !(t0 < R(1) && f_sub(R(1), t0) > R(1e-7)) || step > p.max_steps ||
           (by_time && f_sub(t_hand, t0) <= R(1e-6)) || (kMixed && p.fail_limit > 0 && nfail >= p.fail_limit) ||
           (kMixed && ill_stop);
  };
  auto init_path = [&](long long it) {
    hyp = it / p.paths_per_hyp;
    const long long pidx = it % p.paths_per_hyp;
    if (l < N) {
      if (p.track_in) {
        x = load_cx<R>(p.track_in, (sizeof(R) == 8) != (p.track_other != 0), it * p.ld_track + l);
      } else {
        x = load_cx<R>(p.start_sols, (sizeof(R) == 8) != (p.start_other != 0), pidx * p.ld_start + l);
      }
    } else {
      x = mk(R(0), R(0));
    }
    x0 = x;
    sols = x;
    t0 = p.t_in ? (R)p.t_in[it] : R(0);
    coef_t = R(-1);  // a new path may belong to another hypothesis
    dt = p.dt_in ? (R)p.dt_in[it] : dt_init;
    dt_pre = dt;
    step = p.resume ? p.steps[it] : 0;
    ncorr = p.resume ? p.corr[it] : 0;
    end_zone = false;
    success = false;
    inf = false;
    nsucc = 0;
    nfail = 0;
    step_ill = ill_stop = step_sing = last_sing = false;
    finished = at_end();
    if (!finished) prologue();
  };
  if (alive) init_path(item);

  // The path's scalar state (the same in every lane of the sub-warp) and this lane's track
  // component wait in shared memory while the sub-warp evaluates and solves, so that no
  // register holds them across the LU (register relief; the evaluation's synchronisations keep the
  // compiler from forwarding them).  In as few and as wide accesses as they fit in.
  cx<R>* const rec_r = view<R>(sm.rec);                                             // 3 complex
  int4* const rec_i = reinterpret_cast<int4*>(sm.rec + kRecBytes - 32);
  uint2* const rec_u = reinterpret_cast<uint2*>(sm.rec + kRecBytes - 16);
  auto stash = [&]() {
    rec_r[0] = mk(t0, dt);
    rec_r[1] = mk(t_step, coef_t);
    rec_i[0] = make_int4(step, ncorr, cit, nsucc);
    rec_u[0] = make_uint2((unsigned)item, (unsigned)hyp);
    const unsigned f = (alive ? 1 : 0) | (finished ? 2 : 0) | (end_zone ? 4 : 0) | (success ? 8 : 0) | (inf ? 16 : 0) |
                       (step_ill ? 32 : 0) | (ill_stop ? 64 : 0) | (step_sing ? 128 : 0) | (last_sing ? 256 : 0) |
                       (unsigned)phase << 9;
    if (kMixed) {
      rec_r[2] = mk(dt_pre, R(0));
      rec_u[1] = make_uint2(f, (unsigned)nfail);
    } else {
      rec_u[1].x = f;
    }
  };
  auto unstash = [&]() {
    const cx<R> a = rec_r[0], b = rec_r[1];
    t0 = a.re;
    dt = a.im;
    t_step = b.re;
    coef_t = b.im;
    half = f_mul(R(0.5), dt);  // as the step's prologue set it (dt does not change within a step)
    const int4 n = rec_i[0];
    step = n.x;
    ncorr = n.y;
    cit = n.z;
    nsucc = n.w;
    const uint2 u = rec_u[0];
    item = u.x;
    hyp = u.y;
    const unsigned f = rec_u[1].x;
    if (kMixed) {
      dt_pre = rec_r[2].re;
      nfail = (int)rec_u[1].y;
    }
    phase = (int)(f >> 9);
    alive = f & 1;
    finished = (f >> 1) & 1;
    end_zone = (f >> 2) & 1;
    success = (f >> 3) & 1;
    inf = (f >> 4) & 1;
    step_ill = (f >> 5) & 1;
    ill_stop = (f >> 6) & 1;
    step_sing = (f >> 7) & 1;
    last_sing = (f >> 8) & 1;
    x = (l < N) ? view<R>(sm.xst)[l] : mk(R(0), R(0));
  };

  while (__any_sync(kFull, alive)) {
    const bool served = alive && !finished;
    const bool rk = served && phase < 4;
    const bool corr = served && phase == 4;
    // ---------------- coefficients c_k(t) of the RK stage; the corrector reuses the last stage's
    // (RK stages 2 and 3 share t + dt/2, and after an accepted step the next step starts at the t
    // of the last stage, whose coefficients are still in the buffers: evaluate only on a new t)
    if (rk && t0 != coef_t) {
      coef_eval<R, RL, W, KIND>(p, sm, hyp, t0, coef_t == R(-1), p.spread ? lane : l, p.spread ? 32 : W);
      coef_t = t0;
    }
    // ---------------- one evaluate-and-solve per sub-warp (predictor: -H_t, corrector: H)
    write_track<R, RL, N>(sm, l, x);
    __syncwarp(kFull);
    stash();  // (after the synchronisation: a lane may still be reading the last trip's record before it)
    bool ill = false, sing = false;
    const cx<R> v = eval_solve<R, RL, N, W, KIND, S>(tb, sm, l, rk ? 1 : 0, p.cond_limit, ill, sing);
    unstash();
    if (kMixed && served && ill) step_ill = true;
    if (served && sing) step_sing = true;
    // ---------------- corrector norms (kernel_HC_Solver_P3P.cu:204-219), all lanes take part
    R ns0 = 0, nc0 = 0;
    if (__any_sync(kFull, corr)) {
      const cx<R> xn = c_sub(x, v);
      const R ns = tree_sum<R, N, W>((corr && l < N) ? c_abs2(v) : R(0));
      const R nc = tree_sum<R, N, W>((corr && l < N) ? c_abs2(xn) : R(0));
      ns0 = ns;
      nc0 = nc;
    }
    // ---------------- per-sub-warp state update (no synchronisation below until the fetch)
    bool end_step = false;
    if (rk) {
      if (phase < 3) {
        const R a = f_mul(dt, phase == 0 ? R(1.0 / 6.0) : R(2.0 / 6.0));
        const R d = f_mul(dt, phase == 2 ? R(1.0) : R(0.5));
        sols = mk(f_fma(v.re, a, sols.re), f_fma(v.im, a, sols.im));
        x = mk(f_fma(v.re, d, x0.re), f_fma(v.im, d, x0.im));
        if (phase != 1) t0 = f_add(t0, half);
        ++phase;
      } else {
        const R a = f_mul(dt, R(1.0 / 6.0));
        sols = mk(f_fma(v.re, a, sols.re), f_fma(v.im, a, sols.im));
        x = sols;
        phase = 4;
        cit = 0;
        success = false;
        inf = false;
        if (p.max_corr <= 0) end_step = true;
      }
    } else if (corr) {
      x = c_sub(x, v);
      ++ncorr;
      ++cit;
      success = ((double)ns0 < p.corr_tol2 * (double)nc0);
      inf = ((double)nc0 > 1e14);
      end_step = inf || success || cit >= p.max_corr || (cit == 1 && (double)ns0 > p.first_tol2 * (double)nc0);
    }
    bool done = alive && finished;
    if (end_step) {
      // step control (kernel_HC_Solver_P3P.cu:225-249)
      if (inf) {
        if (handover) {  // hand the last accepted point over
          x = x0;
          t0 = t_step;
        }
        done = true;
      } else if (!success) {
        dt = f_mul(dt, R(0.5));
        x = x0;
        sols = x0;
        nsucc = 0;
        t0 = t_step;
        ++nfail;
      } else {
        nfail = 0;
        ++nsucc;
        x0 = x;
        sols = x;
        if (nsucc >= p.incr) {
          nsucc = 0;
          dt = f_mul(dt, R(2));
          if ((double)dt > p.dt_max) dt = (R)p.dt_max;
        }
      }
      ++step;
      if (kMixed && (step_ill || (p.dt_floor > 0.0 && (double)dt < p.dt_floor))) ill_stop = true;
      last_sing = step_sing;
      if (!done) done = at_end();
      if (done && !inf && by_time && f_sub(t_hand, t0) <= R(1e-6) && step <= p.max_steps &&
          dt < dt_pre)
        dt = dt_pre;
      if (!done) prologue();
    }

    // ---------------- finished paths: write out and take the next path
    if (!__any_sync(kFull, done)) continue;
    // (a non-finite track anywhere in the sub-warp; every lane takes part in the vote)
    const unsigned bad = __ballot_sync(kFull, l < N && !(isfinite(x.re) && isfinite(x.im)));
    const bool nonfinite = ((W == 32 ? bad : bad >> leader) & (W == 32 ? kFull : ((1u << (W & 31)) - 1u))) != 0u;
    if (done && primary) {
      R* ep = reinterpret_cast<R*>(p.endpoints) + 2 * item * p.ld_out;
      if (l < N) {
        ep[2 * l] = x.re;
        ep[2 * l + 1] = x.im;
      }
      if (l == 0) {
        const bool conv = (t0 >= R(1) || f_sub(R(1), t0) <= R(1e-7));
        if (p.conv) p.conv[item] = conv ? 1 : 0;
        if (p.infy) p.infy[item] = inf ? 1 : 0;
        if (p.status)
          p.status[item] = conv        ? ST_CONVERGED
                           : inf       ? ST_DIVERGED
                           : nonfinite ? ST_NONFINITE
                           : last_sing ? ST_SINGULAR
                                       : ST_STEP_CAP;
        if (p.steps) p.steps[item] = step;
        if (p.corr) p.corr[item] = ncorr;
        // a path handed over at the boundary resumes at exactly t_handover, not at its float t
        // (a float t just short of the boundary would put the next step just short of the end
        // zone, where the edge clamp shrinks dt to the gap)
        const bool boundary = by_time && !inf && f_sub(t_hand, t0) <= R(1e-6);
        if (p.t_end) p.t_end[item] = boundary ? p.t_handover : (double)t0;
        if (p.dt_end) p.dt_end[item] = (double)dt;
      }
    }
    long long nxt = 0;
    if (done && l == 0 && primary) nxt = n_sw + (long long)atomicAdd(reinterpret_cast<unsigned*>(p.counter), 1u);
    nxt = __shfl_sync(kFull, nxt, p.spread ? 0 : leader);
    if (done) {
      item = nxt;
      alive = item < p.n_items;
      if (alive) init_path(item);
    }
  }
}

template <typename R, typename RL, int N, int W, int KIND, int V, int S, int WK>
__global__ void __launch_bounds__((track_block<N, R, RL, V>()), (track_ctas<N, R, RL, V>())) track_kernel(const TrackParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  track_body<R, RL, N, W, KIND, S, WK>(p, smem, blockIdx.x, gridDim.x, false);
}

// -------------------------------------------------------------------------------------------------
// Newton polish at t = 1 and the residual |H(x,1)| (double); one sub-warp per item
// -------------------------------------------------------------------------------------------------
template <int N, int W, int KIND, int S>
__global__ void __launch_bounds__(128) polish_kernel(const PolishParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int walk = (kFlatAlways<N> && p.flat_eval == 0) ? 1 : p.flat_eval;
  const int n_hx = hx_words<S>(walk, p.n_hx_terms, p.n_hx_rows), n_ht = ht_words<S>(p.n_ht_terms);
  const Tables tb = stage_tables<double, double, N, KIND, S>(smem, p.hx_terms, p.hx_off, p.ht_terms, p.ht_off,
                                                             p.n_hx_terms, p.n_hx_rows, p.n_ht_terms, walk);
  const int lane = threadIdx.x & 31;
  const int l = lane % W;
  const int g = threadIdx.x / W;
  const int Mc = (KIND == KIND_P2C) ? p.M + 1 : p.P + 1;
  const bool flat = walk != 0;
  SubMem sm = sub_layout<double, double>(smem + tables_bytes(N, n_hx, n_ht, false) +
                                             (size_t)g * sub_bytes(N, Mc, W, flat ? p.scr_slots : 0, 16, 16),
                                         N, Mc, W, p.scr_slots, flat);
  sm.nz = row_mask<N>(tb.hx_off, l);
  sm.walk = walk;
  write_one<double, double, N>(sm, l);
  reinterpret_cast<uint2*>(sm.seg)[l] = walk_range<N, W, shape_nvx(S)>(tb, walk, l, 0, 1);
  const int subs_per_cta = blockDim.x / W;
  for (long long item0 = (long long)blockIdx.x * subs_per_cta; item0 < p.n_items;
       item0 += (long long)gridDim.x * subs_per_cta) {
    const long long item = item0 + g;
    const bool valid = item < p.n_items;
    const bool conv = valid && p.conv[item];
    const long long hyp = valid ? item / p.paths_per_hyp : 0;
    double* ep = p.endpoints + 2 * (valid ? item : 0) * p.ld;
    cx<double> x = (valid && l < N) ? mk(ep[2 * l], ep[2 * l + 1]) : mk(0.0, 0.0);
    if (conv) {
      if (KIND == KIND_P2C) {
        coef_eval_p2c<double, double, false>(p.coef_hx + 2 * hyp * p.stride_hx, p.coef_ht + 2 * hyp * p.stride_ht,
                                                p.M, p.K, 1.0, true, view<double>(sm.coefA), view<double>(sm.coefB),
                                                nullptr, l, W);
      } else {
        coef_eval_ph<double, double, false>(p.p_start, p.p_tgt + 2 * hyp * p.stride_p,
                                               p.p_diff + 2 * hyp * p.stride_p, p.P, 1.0, true, view<double>(sm.coefA),
                                               view<double>(sm.coefB), nullptr, l, W);
      }
    }
    __syncwarp(kFull);
    for (int it = 0; it < p.iters; ++it) {
      write_track<double, double, N>(sm, l, x);
      __syncwarp(kFull);
      const cx<double> d = eval_solve<double, double, N, W, KIND, S>(tb, sm, l, 0);
      if (conv) x = c_sub(x, d);
    }
    // residual |H(x,1)|
    write_track<double, double, N>(sm, l, x);
    __syncwarp(kFull);
    cx<double> A[N];
    cx<double> h;
    eval_any<double, double, N, W, KIND, S>(tb, sm, l, A, h, 0);
    const double s = tree_sum<double, N, W>(l < N ? c_abs2(h) : 0.0);
    if (valid) {
      if (conv && l < N) {
        ep[2 * l] = x.re;
        ep[2 * l + 1] = x.im;
      }
      if (l == 0 && p.resid) p.resid[item] = conv ? sqrt(s) : -1.0;
    }
    __syncwarp(kFull);
  }
}

}  // namespace dev
}  // namespace ghc
