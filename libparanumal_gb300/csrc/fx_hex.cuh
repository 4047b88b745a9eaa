// Building blocks of the FP64 hexahedral operators with block fixed-point contractions
// (fx64.cuh): the layout of an element in shared memory, the tables of D and D^T, and the
// derivatives of a whole element along its three directions. Used by the C0 operator
// (ax_hex.cu) and the interior-penalty operator (ipdg_hex.cu).
//
// One thread holds one line at a time: thread l of an element takes line l of the r, then
// of the s, then of the t direction. Line maxima, even/odd sums and all integers of a line are
// then the thread's own registers. The element is kept in three copies, each with the lines of
// one direction contiguous, so one piece of code with immediate offsets serves all three, in
// place.
//
// The GLL mirror symmetry D[N-i][N-m] = -D[i][m] (and D^T) halves the products:
// with e_m = q_m + q_{N-m}, o_m = q_m - q_{N-m} (m < H = Nq/2), outputs t and N-t are A + B
// and B - A, A = sum Dp[t][m] e_m, B = sum Dm[t][m] o_m, Dp/Dm[t][m] = (D[t][m] +- D[t][N-m])/2.
// It is used for a D that satisfies it exactly, as this library's does, and for Nq = 4, 8
// always; other matrices at other Nq are contracted row by row.
#pragma once

#include "fx64.cuh"
#include "l2_run.hpp"

namespace lpg {

// L2 prefetch of `bytes` (a multiple of 16) from global memory; skipped unless the address
// is 16-byte aligned, as the bulk prefetch requires
__device__ __forceinline__ void prefetch_l2_bulk(const void* gmem, unsigned bytes) {
  if (((uintptr_t)gmem & 15u) == 0 && (bytes & 15u) == 0)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_l2_run(const L2Run r) {
  if (r.bytes)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(r.lo), "r"((unsigned)r.bytes) : "memory");
}
// Barrier over the threads of one element where they are whole warps, else over the CTA;
// returns whether `any` was set by one of them. The barrier numbers are immediates: a number
// in a register reserves all 16 of a CTA's barriers, and an SM's 64 then hold only 4 CTAs.
template <int NQ, int EPB>
__device__ __forceinline__ bool ax_fx_sync(const int el, const bool any = false) {
  if constexpr ((NQ * NQ) % 32 == 0 && EPB == 2) {
    int r;
#define LPG_FX_BARRIER(id)                                                                              \
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.s32 p, %2, 0;\nbarrier.cta.red.or.pred q, " #id ", %1, p;\n" \
               "selp.s32 %0, 1, 0, q;\n}\n"                                                              \
               : "=r"(r)                                                                                \
               : "n"(NQ * NQ), "r"((int)any)                                                            \
               : "memory")
    if (el == 0) LPG_FX_BARRIER(1);
    else LPG_FX_BARRIER(2);
#undef LPG_FX_BARRIER
    return r != 0;
  } else {
    return __syncthreads_or(any);
  }
}

// EO: contract through the mirror symmetry (the caller vouches for D; Nq = 4 and 8 always do)
template <int NQ, bool EO_ = true>
struct FxLayout {
  static constexpr bool EO = EO_ || NQ == 4 || NQ == 8;
  static constexpr int NP = NQ * NQ * NQ, NL = NQ * NQ, H = NQ / 2, MID = NQ % 2;
  static constexpr int P = NQ | 1, PL = P * NQ;      // odd row pitch: conflict-free lines
  static constexpr int ROWS = EO ? H + MID : NQ;     // rows of a table
  static constexpr int RS = (NQ + 1) & ~1;           // their length, 16-byte aligned
  // Bits S (fx64.cuh) of a line value (FS) and a table entry (DS): as many as keep the halves
  // in 32 bits and, for any D, the sum of the middle quarters, Nq products of each kind (EO:
  // half as many per sum, of doubled line values e, o and doubled entries 2 Dp, 2 Dm), and the
  // sum of three transposed lines below 2^63.
  static constexpr int FS = !EO && NQ <= 3 ? 8 : 7;
  static constexpr int DS = EO ? (NQ <= 4 ? 8 : 7) : NQ == 2 ? 8 : NQ == 9 ? 6 : 7;
  static constexpr int EXP = 2088 + FS + DS + (EO ? 1 : 0);   // of fx_line's unit
  static constexpr int EPB = NL >= 128 ? 1 : (128 + NL / 2) / NL;   // about 128 threads
  static constexpr int NT = NL * EPB;
  // A line is left to FP64 where the magnitudes of all entries but the largest add up to less
  // than 2^-T of the power of two under the largest: the derivative at an interior GLL point
  // leaves the point's own value out (D[i][i] = 0), so the largest entry's own output is made of
  // the others alone. The largest error of an output relative to its terms is then at most 3
  // times that of an FP64 chain on lines and metric factors over 15 decades (without it, up to
  // 10^9 times), and below it for the metric of any usual element. N = 1: every entry of D counts
  // in both outputs. One line in FP64 holds up its element by 1 to 2 us, so T is the largest that
  // keeps the 3: with one less a problem of one wave has such a line and takes 5 to 8 % more (16^3,
  // N = 5 and 4; 10^3, N = 6). The test itself costs 1 to 3 % of large problems: 64^3, N = 7
  // 3.07 -> 3.17 ms; 31 x 23 x 29, N = 5 111.8 -> 112.9 us.
  static constexpr int T = NQ == 3 ? 8 : NQ == 4 ? 6 : NQ == 5 ? 5 : NQ == 6 ? 4 : 3;
  // resident CTAs per SM to compile for (registers): measured best of 5 to 10
  static constexpr int MINB = NQ == 9 ? 5 : NQ <= 4 ? 10 : 7;
};

// Table of D (trans = false) or D^T: row t holds 2 Dp[t][m], 2 Dm[t][m] (m < H) alternating,
// then twice the middle entry for odd Nq; without EO the row itself. eR: exponent of the row.
// The sums are formed in integers: rounded to FP64 they would perturb D (N = 6, smooth field:
// error 1e-14 instead of 6e-16).
template <int NQ, bool EO>
__device__ __forceinline__ fx_half fx_table_entry(const double* __restrict__ Dg, bool trans, int t, int c, int eR) {
  using L = FxLayout<NQ, EO>;
  const int rs = trans ? 1 : NQ, cs = trans ? NQ : 1;
  if constexpr (L::EO) {
    const int m = c >> 1;   // the middle entry: m = H, its own mirror
    const int64_t d0 = fx_from_double<L::DS + 1>(Dg[t * rs + m * cs], eR);
    const int64_t d1 = fx_from_double<L::DS + 1>(Dg[t * rs + (NQ - 1 - m) * cs], eR);
    return fx_split((c & 1) ? d0 - d1 : d0 + d1);
  } else {
    return fx_split(fx_from_double<L::DS + 1>(Dg[t * rs + c * cs], eR));
  }
}

// emit(t, sum_m table[t][m] q[m]) for the outputs t of one line, as integers in units of
// 2^(eL + eR[t] - EXP); key: of the line's largest entry, eL its exponent. false, and nothing
// emitted, where the line is left to FP64 (T).
template <int NQ, bool EO, typename F>
__device__ __forceinline__ bool fx_line(const double (&q)[NQ], const unsigned key, const fx_half* __restrict__ tab,
                                        F&& emit) {
  using L = FxLayout<NQ, EO>;
  constexpr int N = NQ - 1, H = L::H, SH = L::FS + 1;
  constexpr int HALF = (NQ << (SH - 3)) > 256 ? 1 : 0;   // NQ high words below 2^(21 + SH) add up within 32 bits
  int64_t f[NQ];
  unsigned sum = 0;
#pragma unroll
  for (int m = 0; m < NQ; ++m) {
    unsigned mag;
    f[m] = fx_from_double<SH>(q[m], (int)(key >> 20), mag);
    sum += mag >> HALF;
  }
  if constexpr (NQ > 2) {
    const unsigned top = ((key & 0xfffffu) | 0x100000u) << (SH - HALF);   // the largest, but for its lowest bits
    if (sum - top < 1u << (20 + SH - HALF - L::T)) return false;
  }
  fx_half x[NQ];
  if constexpr (L::EO) {
#pragma unroll
    for (int m = 0; m < H; ++m) {
      x[2 * m] = fx_split(f[m] + f[N - m]);
      x[2 * m + 1] = fx_split(f[m] - f[N - m]);
    }
    if constexpr (L::MID) x[2 * H] = fx_split(f[H]);
#pragma unroll
    for (int t = 0; t < H; ++t) {
      const int4* row = reinterpret_cast<const int4*>(tab + t * L::RS);
      fx_half dp[H + 1], dm[H];
#pragma unroll
      for (int m = 0; m < H; ++m) {
        const int4 v = row[m];
        dp[m] = {v.x, v.y};
        dm[m] = {v.z, v.w};
      }
      if constexpr (L::MID) dp[H] = tab[t * L::RS + 2 * H];
      fx_acc A(x[0], dp[0]), B(x[1], dm[0]);
#pragma unroll
      for (int m = 1; m < H + L::MID; ++m) A.cross(x[2 * m], dp[m]);
#pragma unroll
      for (int m = 1; m < H; ++m) B.cross(x[2 * m + 1], dm[m]);
      A.fold();
      B.fold();
#pragma unroll
      for (int m = 0; m < H + L::MID; ++m) A.high(x[2 * m], dp[m]);
#pragma unroll
      for (int m = 0; m < H; ++m) B.high(x[2 * m + 1], dm[m]);
      emit(t, A.v + B.v + 1);   // both were rounded down
      emit(N - t, B.v - A.v);
    }
    if constexpr (L::MID) {   // the middle output: its row is odd
      fx_acc B(0x40000000ll);
      fx_half dm[H];
#pragma unroll
      for (int m = 0; m < H; ++m) {
        dm[m] = tab[H * L::RS + 2 * m + 1];
        B.cross(x[2 * m + 1], dm[m]);
      }
      B.fold();
#pragma unroll
      for (int m = 0; m < H; ++m) B.high(x[2 * m + 1], dm[m]);
      emit(H, B.v);
    }
  } else {
#pragma unroll
    for (int m = 0; m < NQ; ++m) x[m] = fx_split(f[m]);
#pragma unroll
    for (int t = 0; t < NQ; ++t) {
      fx_acc A(0x40000000ll);   // rounds to nearest
      fx_half d[NQ];
#pragma unroll
      for (int m = 0; m < NQ; ++m) {
        d[m] = tab[t * L::RS + m];
        A.cross(x[m], d[m]);
      }
      A.fold();
#pragma unroll
      for (int m = 0; m < NQ; ++m) A.high(x[m], d[m]);
      emit(t, A.v);
    }
  }
  return true;
}

// a line of zeros (as the masked lines of Dirichlet faces are): no magnitude bit is set
template <int NQ>
__device__ __forceinline__ bool fx_zero(const double* v, const unsigned key) {
  int lo = 0;
#pragma unroll
  for (int m = 0; m < NQ; ++m) lo |= __double2loint(v[m]);
  return key == 0 && lo == 0;
}

// row of the table that output t of a line uses
template <int NQ, bool EO>
__device__ __forceinline__ constexpr int fx_row(int t) {
  return FxLayout<NQ, EO>::EO && t > NQ - 1 - t ? NQ - 1 - t : t;
}

// one element's three copies in shared memory, seen by thread l = a + NQ b
template <int NQ>
struct FxElement {
  using L = FxLayout<NQ>;   // EO does not matter here
  static constexpr int DOUBLES = 3 * L::PL * NQ;   // of an element
  double* S;
  int l, a, b;
  __device__ __forceinline__ FxElement(double* base, int l_) : S(base), l(l_), a(l_ % NQ), b(l_ / NQ) {}
  // line l of direction d
  __device__ __forceinline__ double* line(int d) const { return S + d * L::PL * NQ + b * L::PL + a * L::P; }
  // node (i, j, k) in the copies of direction r, s, t
  __device__ __forceinline__ double& r(int i, int j, int k) const { return S[k * L::PL + j * L::P + i]; }
  __device__ __forceinline__ double& s(int i, int j, int k) const { return S[L::PL * NQ + k * L::PL + i * L::P + j]; }
  __device__ __forceinline__ double& t(int i, int j, int k) const { return S[2 * L::PL * NQ + j * L::PL + i * L::P + k]; }
};

// tables of D and D^T with the exponents of their rows, by the threads of a CTA; true where
// every line is left to FP64: a row's largest entry lies outside [2^-63, 2^63], or an entry off
// the diagonal is 0 or below 2^-10 of it (a GLL matrix has 2^-6 and more), so that more than its
// own node's value can be missing in an output
template <int NQ, bool EO>
__device__ __forceinline__ bool fx_tables(const double* __restrict__ Dg, const int tid, const int threads,
                                          fx_half (&tab)[2][FxLayout<NQ, EO>::ROWS * FxLayout<NQ, EO>::RS],
                                          int (&ex)[2][FxLayout<NQ, EO>::ROWS], const bool gll) {
  using L = FxLayout<NQ, EO>;
  constexpr int TAB = L::ROWS * NQ;
  bool plain = false;
  for (int w = tid; w < 2 * TAB; w += threads) {
    const int tr = w / TAB, t = (w % TAB) / NQ, c = w % NQ;
    unsigned key = 0, least = 0x7fffffffu;
#pragma unroll
    for (int m = 0; m < NQ; ++m) {
      const unsigned k = fx_key(Dg[tr ? m * NQ + t : t * NQ + m]);
      key = max(key, k);
      if (!gll && (m != t || NQ == 2)) least = min(least, k);
    }
    const int eR = max((int)(key >> 20), 960) + (L::EO ? 1 : 0);   // 2 Dp, 2 Dm reach twice the row's maximum
    tab[tr][t * L::RS + c] = fx_table_entry<NQ, EO>(Dg, tr, t, c, eR);
    if (c == 0) ex[tr][t] = eR;
    plain |= eR > 1086 || (key >> 20) < 960 || (!gll && (int)(key >> 20) - (int)(least >> 20) > 10);
  }
  return plain;
}

// the copies of q become D_r q, D_s q, D_t q (directions d0 to d1 - 1 by this thread)
template <int NQ, bool EO>
__device__ __forceinline__ void fx_forward(const FxElement<NQ>& E, const fx_half* tab, const int* ex, const bool plain,
                                           const double* __restrict__ Dg, const int d0 = 0, const int d1 = 3) {
  using L = FxLayout<NQ, EO>;
#pragma unroll 1
  for (int d = d0; d < d1; ++d) {
    double* const o = E.line(d);
    double v[NQ];
    unsigned key = 0;
#pragma unroll
    for (int m = 0; m < NQ; ++m) {
      v[m] = o[m];
      key = max(key, fx_key(v[m]));
    }
    const int eL = (int)(key >> 20);
    asm volatile("" ::: "memory");   // keeps the table reads of all directions out of registers
    if (fx_ordinary(eL) && !plain && fx_line<NQ, EO>(v, key, tab, [&](int t, int64_t r) {
          o[t] = fx_to_double(r, fx_base(eL + ex[fx_row<NQ, EO>(t)] - (L::EXP - 1086)));
        }))
      continue;
    if (fx_zero<NQ>(o, key)) {
#pragma unroll
      for (int t = 0; t < NQ; ++t) o[t] = 0.0;
    } else {
#pragma unroll
      for (int m = 0; m < NQ; ++m) v[m] = o[m];   // not held over the conversion
#pragma unroll 1
      for (int t = 0; t < NQ; ++t) {
        double r = 0;
#pragma unroll
        for (int m = 0; m < NQ; ++m) r += Dg[t * NQ + m] * v[m];
        o[t] = r;
      }
    }
  }
}

// the copies (u_r, u_s, u_t) become D_r^T u_r, D_s^T u_s, D_t^T u_t as integers, with the
// exponents of the lines in x, -1 for a line kept as FP64 values; true if this thread kept one
template <int NQ, bool EO>
__device__ __forceinline__ bool fx_transposed(const FxElement<NQ>& E, const fx_half* tab, const bool plain,
                                              const double* __restrict__ Dg, int (&x)[3][FxLayout<NQ>::NL],
                                              const int d0 = 0, const int d1 = 3) {
  bool fp = false;
#pragma unroll 1
  for (int d = d0; d < d1; ++d) {
    double* const o = E.line(d);
    double v[NQ];
    unsigned key = 0;
#pragma unroll
    for (int m = 0; m < NQ; ++m) {
      v[m] = o[m];
      key = max(key, fx_key(v[m]));
    }
    const int eL = (int)(key >> 20);
    int xl = eL;
    asm volatile("" ::: "memory");
    if (fx_ordinary(eL) && !plain &&
        fx_line<NQ, EO>(v, key, tab, [&](int t, int64_t r) { o[t] = __longlong_as_double(r); })) {
    } else if (fx_zero<NQ>(o, key)) {
      xl = 128;
#pragma unroll
      for (int t = 0; t < NQ; ++t) o[t] = 0.0;
    } else {
      xl = -1;
      fp = true;
#pragma unroll
      for (int m = 0; m < NQ; ++m) v[m] = o[m];   // not held over the conversion
#pragma unroll 1
      for (int t = 0; t < NQ; ++t) {
        double r = 0;
#pragma unroll
        for (int m = 0; m < NQ; ++m) r += Dg[m * NQ + t] * v[m];
        o[t] = r;
      }
    }
    x[d][E.l] = xl;
  }
  return fp;
}

// sum of the three transposed parts at node (a, b, k); er, es: exponents of the rows a and b
// of D^T; fp: some line of the element was kept in FP64
template <int NQ, bool EO>
__device__ __forceinline__ double fx_node_sum(const FxElement<NQ>& E, const int k, const int (&x)[3][FxLayout<NQ>::NL],
                                              const int* ex, const int er, const int es, const bool fp) {
  using L = FxLayout<NQ, EO>;
  constexpr int OFF = L::EXP - 1086;
  const int lr = x[0][E.b + NQ * k], ls = x[1][E.a + NQ * k], lt = x[2][E.l];
  const int xr = lr + er, xs = ls + es, xt = lt + ex[fx_row<NQ, EO>(k)];
  const double vr = E.r(E.a, E.b, k), vs = E.s(E.a, E.b, k), vt = E.t(E.a, E.b, k);
  if (!fp || (lr | ls | lt) >= 0) {
    const int X = max(xr, max(xs, xt));
    const int64_t sum = fx_shr(__double_as_longlong(vr), X - xr) + fx_shr(__double_as_longlong(vs), X - xs) +
                        fx_shr(__double_as_longlong(vt), X - xt);
    return fx_to_double(sum, fx_base(X - OFF));
  }
  return (lr < 0 ? vr : fx_to_double(__double_as_longlong(vr), fx_base(xr - OFF))) +
         (ls < 0 ? vs : fx_to_double(__double_as_longlong(vs), fx_base(xs - OFF))) +
         (lt < 0 ? vt : fx_to_double(__double_as_longlong(vt), fx_base(xt - OFF)));
}

}  // namespace lpg
