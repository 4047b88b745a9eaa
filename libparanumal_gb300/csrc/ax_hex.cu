// Matrix-free screened-Poisson operator on hexahedra (sum-factorised, GLL collocation)
// with the gather-scatter assembly fused into the kernel.
//
// Same operator as ellipticPartialAxHex3D (solvers/elliptic/okl/ellipticAxHex3D.okl:156-295):
// the r, s and t derivatives of an element's lines, the metric product G*grad per node, the
// transposed derivatives and the mass term. Differences for GB300:
//   * lines are contracted by one thread each from line-contiguous copies in shared memory,
//     FP64 ones in block fixed point (ax_hex_fx_kernel, ax_hex_line_kernel);
//   * the assembled result is accumulated straight into Aq with atomics (the reference
//     writes AqL, then an ogs Gather kernel re-reads it);
//   * geometric-factor offsets are 64-bit (the reference's int offsets overflow at 112^3, N=7);
//   * per-element lambda; FP64, double-word, FP32 and BF16-storage kernels.
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "df64.cuh"
#include "fx_hex.cuh"
#include "lpg_common.cuh"
#include "lpg_internal.hpp"

namespace lpg {

enum { IN_GATHER = 0, IN_LOCAL = 1 };
enum { OUT_ASSEMBLE = 0, OUT_LOCAL = 1, OUT_LOCAL_SUB = 2 };

template <int NQ>
constexpr int elems_per_block() {
  return (256 / (NQ * NQ)) > 0 ? (256 / (NQ * NQ)) : 1;
}

// FP64 with direct contractions, one layer at a time: LPG_AX_FP64 = direct
template <int NQ, int INMODE, int OUTMODE>
__global__ void __launch_bounds__(NQ * NQ * elems_per_block<NQ>())
ax_hex_kernel(const int64_t Nelements, const int32_t* __restrict__ elementList,
              const int32_t* __restrict__ g2l, const double* __restrict__ ggeo, const int64_t geoStride,
              const double* __restrict__ wJ, const int64_t wJStride, const double* __restrict__ Dg,
              const double lambda, const double* __restrict__ lambdaE, const double* __restrict__ q,
              double* __restrict__ out, const double outScale) {
  constexpr int NP = NQ * NQ * NQ;
  constexpr int EPB = elems_per_block<NQ>();
  __shared__ double s_D[NQ][NQ];
  __shared__ double s_q[EPB][NQ][NQ];
  __shared__ double s_Gqr[EPB][NQ][NQ];
  __shared__ double s_Gqs[EPB][NQ][NQ];

  const int i = threadIdx.x, j = threadIdx.y, el = threadIdx.z;
  const int tid = i + NQ * (j + NQ * el);
  for (int t = tid; t < NQ * NQ; t += NQ * NQ * EPB) s_D[t / NQ][t % NQ] = Dg[t];

  int64_t e = (int64_t)blockIdx.x * EPB + el;
  const bool active = e < Nelements;
  if (active && elementList) e = elementList[e];
  if (!active) e = 0;

  double r_q[NQ], r_Aq[NQ];
  int32_t r_id[NQ];
  const int64_t nodeBase = e * NP + j * NQ + i;
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    r_Aq[k] = 0;
    if (INMODE == IN_GATHER) {
      const int32_t id = active ? __ldg(g2l + nodeBase + k * NQ * NQ) : -1;
      r_id[k] = id;
      r_q[k] = (id >= 0) ? q[id] : 0.0;
    } else {
      r_id[k] = 0;
      r_q[k] = active ? q[nodeBase + k * NQ * NQ] : 0.0;
    }
  }
  if (OUTMODE == OUT_ASSEMBLE && INMODE != IN_GATHER) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) r_id[k] = active ? __ldg(g2l + nodeBase + k * NQ * NQ) : -1;
  }
  const double lam = (lambdaE && active) ? lambdaE[e] : lambda;
  const double* gp = ggeo + e * geoStride + j * NQ + i;
  const double* wp = wJ + e * wJStride + j * NQ + i;
  __syncthreads();

#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    double G00 = 0, G01 = 0, G02 = 0, G11 = 0, G12 = 0, G22 = 0, GwJ = 0;
    if (active) {
      const int off = k * NQ * NQ;
      G00 = __ldg(gp + 0 * NP + off);
      G01 = __ldg(gp + 1 * NP + off);
      G02 = __ldg(gp + 2 * NP + off);
      G11 = __ldg(gp + 3 * NP + off);
      G12 = __ldg(gp + 4 * NP + off);
      G22 = __ldg(gp + 5 * NP + off);
      GwJ = __ldg(wp + off);
    }
    s_q[el][j][i] = r_q[k];
    double qt = 0;
#pragma unroll
    for (int m = 0; m < NQ; ++m) qt += s_D[k][m] * r_q[m];
    __syncthreads();

    double qr = 0, qs = 0;
#pragma unroll
    for (int m = 0; m < NQ; ++m) {
      qr += s_D[i][m] * s_q[el][j][m];
      qs += s_D[j][m] * s_q[el][m][i];
    }
    s_Gqs[el][j][i] = (G01 * qr + G11 * qs + G12 * qt);
    s_Gqr[el][j][i] = (G00 * qr + G01 * qs + G02 * qt);
    const double Gqt = (G02 * qr + G12 * qs + G22 * qt);
    double Auk = GwJ * lam * r_q[k];
    __syncthreads();

#pragma unroll
    for (int m = 0; m < NQ; ++m) {
      Auk += s_D[m][j] * s_Gqs[el][m][i];
      r_Aq[m] += s_D[k][m] * Gqt;
      Auk += s_D[m][i] * s_Gqr[el][j][m];
    }
    r_Aq[k] += Auk;
    __syncthreads();
  }

  if (!active) return;
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    if (OUTMODE == OUT_ASSEMBLE) {
      if (r_id[k] >= 0) atomicAdd(out + r_id[k], outScale * r_Aq[k]);
    } else if (OUTMODE == OUT_LOCAL) {
      out[nodeBase + k * NQ * NQ] = r_Aq[k];
    } else {
      out[nodeBase + k * NQ * NQ] -= r_Aq[k];
    }
  }
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <typename G> __device__ __forceinline__ float geo_to_float(G v);
template <> __device__ __forceinline__ float geo_to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float geo_to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// ---------------------------------------------------------------- FP32 line kernel
// FP32 vectors. One thread holds one line of an element in each direction: its t-line in
// registers, its r- and s-line through two line-contiguous copies of the element in shared
// memory, contracted in place; a row of D is read once for the three. Two passes (D, D^T) with
// the metric product between them, 4 barriers an element. Many small CTAs: while some wait for
// their loads, others compute. 48^3, N = 7 with FP32 factors moves 2.26 GB in 357 us, 0.93 of
// the measured copy rate (379 with the clearing of out); with BF16 factors shared memory bounds it (80 % of its cycles).
template <int NQ>
struct LineLayout {
  static constexpr int NP = NQ * NQ * NQ, NL = NQ * NQ;
  static constexpr bool VEC = NQ % 4 == 0;   // lines of whole 16-byte units
  // Line l of an element starts at P l. An odd pitch keeps the accesses to lines and to columns
  // free of bank conflicts; at Nq = 8 the two 16-byte halves of a line trade places in every
  // other group of four lines instead, and at Nq = 4 the elements of a warp lie 16 banks apart.
  static constexpr int P = VEC ? NQ : NQ | 1;
  static constexpr int ES = P * NL + (NQ == 4 ? 16 : 0);   // a copy of an element
  // threads of a CTA (at most, at least one element) and resident CTAs per SM to compile for: the
  // best of 64, 128 and 256 threads and of 3 to 18 CTAs. Larger against chosen, us: 100^3, N = 1
  // 73.5 / 66.2; 80^3, N = 2 122.6 / 109.1; 48^3, N = 4 114.1 / 109.9; smaller against chosen:
  // 40^3, N = 5 113.5 / 110.9; 30^3, N = 6 88.6 / 82.9; 24^3, N = 8 110.3 / 95.6
  static constexpr int CTA = VEC || NQ <= 3 ? 64 : NQ == 5 ? 128 : 256, EPB = CTA / NL, NT = NL * EPB;
  static constexpr int RD = (NQ + 3) & ~3;                 // row of D in shared memory, 16-byte multiple
  // (Nq = 8, with the mass term and without a copy: 48^3 383 us at 16, 401 at 14)
  static constexpr int minb(bool full) {
    return NQ == 8 && full ? 16 : VEC ? 14 : NQ <= 3 ? 12 : NQ == 5 ? 10 : NQ == 9 ? 3 : 4;
  }
  __device__ __forceinline__ static constexpr int at(int l, int m) { return P * l + (NQ == 8 ? m ^ (l & 4) : m); }
};

// COPY: the factors are copied to shared memory by 16-byte cp.async while q is gathered and
// differentiated, instead of asked for in L2 and read where they are used
template <int NQ, typename G, bool MASS, bool COPY>
__global__ void __launch_bounds__(LineLayout<NQ>::NT, LineLayout<NQ>::minb(MASS && !COPY))
ax_hex_line_kernel(const int64_t Nelements, const int32_t* __restrict__ elementList,
                   const int32_t* __restrict__ g2l, const G* __restrict__ ggeo, const int64_t geoStride,
                   const G* __restrict__ wJ, const int64_t wJStride, const float* __restrict__ Dg, const float lambda,
                   const float* __restrict__ lambdaE, const float* __restrict__ q, float* __restrict__ out,
                   const float outScale) {
  using L = LineLayout<NQ>;
  constexpr int NP = L::NP, NL = L::NL, EPB = L::EPB, RD = L::RD, ROWS = MASS ? 7 : 6;
  constexpr int ROW_BYTES = NP * (int)sizeof(G);
  constexpr bool REREAD = NQ == 8 && !COPY;   // the dofs are read again: fewer registers, more CTAs
  __shared__ __align__(16) float s_D[2][NQ * RD];   // D, D^T
  __shared__ __align__(16) float s_v[2][EPB * L::ES];
  __shared__ __align__(16) unsigned char s_g[COPY ? EPB * ROWS * ROW_BYTES : 16];
  const int tid = threadIdx.x, el = tid / NL, l = tid % NL, a = l % NQ, b = l / NQ;
  float* const vr = &s_v[0][el * L::ES];   // r-lines: line (k, b), entry a
  float* const vs = &s_v[1][el * L::ES];   // s-lines: line (k, a), entry b
  const G* const sg = reinterpret_cast<const G*>(s_g) + el * ROWS * NP + l;
  int64_t e = (int64_t)blockIdx.x * EPB + el;
  const bool active = e < Nelements;
  if (active && elementList) e = elementList[e];
  if (!active) e = 0;
  const int64_t nodeBase = e * NP + l;
  if constexpr (!COPY) {
    if ((MASS || NQ < 4) && !elementList && geoStride <= 7 * NP) {
      // one thread asks for the factors of the CTA's run of elements in L2
      if (tid == 0)
        prefetch_l2_run(l2_factor_run((uint64_t)(ggeo + e * geoStride), geoStride, (uint64_t)(wJ + e * wJStride), wJStride,
                                       NP, sizeof(G), Nelements - e < EPB ? Nelements - e : EPB, MASS));
    } else if (NQ >= 4 && l == 0 && active) {
      const uintptr_t lo = ((uintptr_t)(ggeo + e * geoStride) + 15) & ~(uintptr_t)15;
      const uintptr_t hi = (uintptr_t)(ggeo + e * geoStride + 6 * NP) & ~(uintptr_t)15;
      prefetch_l2_bulk((const void*)lo, (unsigned)(hi - lo));
      if constexpr (MASS) {
        const uintptr_t lw = ((uintptr_t)(wJ + e * wJStride) + 15) & ~(uintptr_t)15;
        const uintptr_t hw = (uintptr_t)(wJ + e * wJStride + NP) & ~(uintptr_t)15;
        prefetch_l2_bulk((const void*)lw, (unsigned)(hw - lw));
      }
    }
  }
  int32_t id[NQ];
#pragma unroll
  for (int k = 0; k < NQ; ++k) id[k] = active ? __ldg(g2l + nodeBase + k * NL) : -1;
  if constexpr (COPY) {
    if (active) {
      constexpr int C = ROW_BYTES / 16;
      unsigned char* const dst = s_g + el * ROWS * ROW_BYTES;
      const char* src = reinterpret_cast<const char*>(ggeo + e * geoStride);
      for (int c = l; c < 6 * C; c += NL) cp_async16(dst + 16 * c, src + 16 * c);
      if constexpr (MASS) {
        src = reinterpret_cast<const char*>(wJ + e * wJStride);
        for (int c = l; c < C; c += NL) cp_async16(dst + 16 * (6 * C + c), src + 16 * c);
      }
    }
    cp_async_commit();
  }
  for (int t = tid; t < NL; t += L::NT) {
    s_D[0][t / NQ * RD + t % NQ] = Dg[t];
    s_D[1][t / NQ * RD + t % NQ] = Dg[t % NQ * NQ + t / NQ];
  }
  float v0[NQ], vt[NQ];
#pragma unroll
  for (int k = 0; k < NQ; ++k) v0[k] = id[k] >= 0 ? q[id[k]] : 0.f;
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    vr[L::at(k * NQ + b, a)] = vs[L::at(k * NQ + a, b)] = v0[k];
    vt[k] = v0[k];
  }
  __syncthreads();
  auto lines = [&](const float* M) {   // r-line l, s-line l and the column vt times M
    float xr[NQ], xs[NQ], xt[NQ];
    if constexpr (L::VEC) {
#pragma unroll
      for (int c = 0; c < NQ; c += 4) {
        const float4 u = *reinterpret_cast<const float4*>(vr + L::at(l, c));
        const float4 w = *reinterpret_cast<const float4*>(vs + L::at(l, c));
        xr[c] = u.x; xr[c + 1] = u.y; xr[c + 2] = u.z; xr[c + 3] = u.w;
        xs[c] = w.x; xs[c + 1] = w.y; xs[c + 2] = w.z; xs[c + 3] = w.w;
      }
    } else {
#pragma unroll
      for (int m = 0; m < NQ; ++m) {
        xr[m] = vr[L::at(l, m)];
        xs[m] = vs[L::at(l, m)];
      }
    }
#pragma unroll
    for (int m = 0; m < NQ; ++m) xt[m] = vt[m];
    if constexpr (L::VEC) {
      float y[NQ];
#pragma unroll
      for (int c = 0; c < NQ; c += 4) {
        float yr[4], ys[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float r0 = 0.f, r1 = 0.f, s0 = 0.f, s1 = 0.f, t0 = 0.f, t1 = 0.f;
#pragma unroll
          for (int m = 0; m < NQ; m += 4) {
            const float4 d = *reinterpret_cast<const float4*>(M + (c + u) * NQ + m);
            r0 += d.x * xr[m]; r1 += d.y * xr[m + 1]; r0 += d.z * xr[m + 2]; r1 += d.w * xr[m + 3];
            s0 += d.x * xs[m]; s1 += d.y * xs[m + 1]; s0 += d.z * xs[m + 2]; s1 += d.w * xs[m + 3];
            t0 += d.x * xt[m]; t1 += d.y * xt[m + 1]; t0 += d.z * xt[m + 2]; t1 += d.w * xt[m + 3];
          }
          yr[u] = r0 + r1; ys[u] = s0 + s1; y[c + u] = t0 + t1;
        }
        *reinterpret_cast<float4*>(vr + L::at(l, c)) = make_float4(yr[0], yr[1], yr[2], yr[3]);
        *reinterpret_cast<float4*>(vs + L::at(l, c)) = make_float4(ys[0], ys[1], ys[2], ys[3]);
      }
#pragma unroll
      for (int k = 0; k < NQ; ++k) vt[k] = y[k];
      return;
    }
#pragma unroll
    for (int t = 0; t < NQ; ++t) {
      float r[2] = {0.f, 0.f}, s[2] = {0.f, 0.f}, u[2] = {0.f, 0.f};
#pragma unroll
      for (int c = 0; c < NQ; c += 4) {
        const float4 d4 = *reinterpret_cast<const float4*>(M + t * RD + c);
        const float d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
        for (int m = c; m < NQ && m < c + 4; ++m) {
          r[m & 1] += d[m - c] * xr[m];
          s[m & 1] += d[m - c] * xs[m];
          u[m & 1] += d[m - c] * xt[m];
        }
      }
      vr[L::at(l, t)] = r[0] + r[1];
      vs[L::at(l, t)] = s[0] + s[1];
      vt[t] = u[0] + u[1];
    }
  };
  lines(s_D[0]);
  const float lam = MASS && active ? (lambdaE ? lambdaE[e] : lambda) : 0.f;
  if constexpr (COPY) cp_async_wait<0>();
  __syncthreads();
  const G* const gp = ggeo + e * geoStride + l;
  const G* const wp = wJ + e * wJStride + l;
  if (active) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      float g[ROWS];
#pragma unroll
      for (int c = 0; c < ROWS; ++c)
        g[c] = COPY ? geo_to_float(sg[c * NP + k * NL]) : load_geo<float, G>(c == 6 ? wp + k * NL : gp + c * NP + k * NL);
      float &r = vr[L::at(k * NQ + b, a)], &s = vs[L::at(k * NQ + a, b)];
      const float qr = r, qs = s, qt = vt[k];
      r = g[0] * qr + g[1] * qs + g[2] * qt;
      s = g[1] * qr + g[3] * qs + g[4] * qt;
      vt[k] = g[2] * qr + g[4] * qs + g[5] * qt;
      if constexpr (MASS) v0[k] *= g[6] * lam;
    }
  }
  __syncthreads();
  lines(s_D[1]);
  __syncthreads();
  if (!active) return;
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    // the r and s parts and the mass term are added before the t part: two roundings fewer at the size
    // of the result where t gives most of it, the direction in which the kernels before this one
    // were best. Error of boxes 2.4 times as fine along t against theirs, with the mass term added
    // last -> now: N = 2 1.14 -> 1.00, N = 3 1.20 -> 1.07, N = 4 1.11 -> 1.01, N = 5 1.10 -> 1.00,
    // N = 7 1.05 -> 0.97; cubes N = 2 to 8 1.01 to 0.77. (The mass term as the start of the t sums: not
    // better, and 7 % slower at N = 7 for lack of registers.)
    float r = vr[L::at(k * NQ + b, a)] + vs[L::at(k * NQ + a, b)];
    if constexpr (MASS) r += v0[k];
    r = vt[k] + r;
    const int32_t g = REREAD ? __ldg(g2l + nodeBase + k * NL) : id[k];
    if (g >= 0) atomicAdd(out + g, outScale * r);
  }
}

// Barrier over the NQ*NQ threads of one element (named barrier 1 + el) when that is a
// whole number of warps, else over the CTA.
template <int NQ>
__device__ __forceinline__ void elem_sync(const int el) {
  if constexpr ((NQ * NQ) % 32 == 0) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(1 + el), "r"(NQ * NQ) : "memory");
  } else {
    __syncthreads();
  }
}

// ---------------------------------------------------------------- FP64 block fixed-point kernel
// The FP64 operator with its contractions in block fixed point (fx64.cuh). Every 1-D line
// of an element is converted once to 64-bit integers on the exponent of its largest entry,
// contracted with D (or D^T) by integer multiply-adds, and converted back; the metric
// product G . grad q and the mass term stay in FP64.
//
// The element sits in three line-contiguous FP64 copies in shared memory and every step works
// in place, with 4 barriers (fx_hex.cuh):
//   q three times;  then D_r q, D_s q, D_t q;  then the three rows of G . grad q;  then the
//   transposed derivatives as integers (exponents in s_x), summed on their common exponent.
// q is gathered again for the mass term.
//
// What bounds it (N = 7): the FP64 pipe, at the 9 FP64 operations a node of the metric product and
// 1 of the mass term against 50 of the FP64 kernel it replaced, closely followed by the integer
// pipe (shifts, logic and multiply-adds share 64 lanes a clock; 537 instructions a node in all): 64
// and 57 % busy, with barriers between the two. 48^3, N = 7: 1.36 ms (lambda = 0: 1.22) against
// 4.79 (4.70) of that kernel; 28^3, N = 5: 134 us against 406; 64^3, N = 3: 334 us against 1099;
// 20^3, N = 8: 199 us against 699. Measured and not kept at 48^3: L2 prefetch of a later element's
// factors (one wave ahead) 1.53 against 1.37 ms; eight CTAs per SM with swizzled instead of pitched
// lines 1.37 against 1.37 ms.
// MASS = false: lambda == 0 and no lambda field, the mass term and its wJ reads are left out
// UNIT: lambda == 1 without a lambda field, the mass term is wJ q
// flags: bit 31 the sign bit for out -= A q, bit 0 this library's D
// W = 3: three threads a line position, each with one direction of the derivatives and a third
// of the layers, for problems too small to fill the GPU otherwise
template <int NQ, int W>
struct FxThreads {
  using L = FxLayout<NQ>;
  static constexpr int EPB = W == 1 ? L::EPB : (L::NL * W >= 96 ? 1 : 96 / (L::NL * W));
  static constexpr int NT = L::NL * W * EPB, MINB = W == 1 ? L::MINB : 1;
};

template <int NQ, bool EO, int W, int INMODE, int OUTMODE, bool MASS, bool UNIT>
__global__ void __launch_bounds__(FxThreads<NQ, W>::NT, FxThreads<NQ, W>::MINB)
ax_hex_fx_kernel(const int64_t Nelements, const int32_t* __restrict__ elementList,
                 const int32_t* __restrict__ g2l, const double* __restrict__ ggeo, const int64_t geoStride,
                 const double* __restrict__ wJ, const int64_t wJStride, const double* __restrict__ Dg,
                 const double lambda, const double* __restrict__ lambdaE, const double* __restrict__ q,
                 double* __restrict__ out, const unsigned flags) {
  using L = FxLayout<NQ, EO>;
  constexpr int NP = L::NP, NL = L::NL, EPB = FxThreads<NQ, W>::EPB, KN = (NQ + W - 1) / W;
  extern __shared__ __align__(16) unsigned char fx_smem[];
  __shared__ __align__(16) fx_half s_tab[2][L::ROWS * L::RS];   // D, D^T
  __shared__ int s_e[2][L::ROWS];                   // biased exponents of their rows
  __shared__ int s_x[EPB][3][NL];                   // exponents of the transposed lines, -1: FP64 values
  const int tid = threadIdx.x, el = tid / (NL * W), l = tid % NL, w = W == 1 ? 0 : tid / NL % W;
  // this thread's layers w, w + W, ... (layer() is a constant for W = 1)
  auto layer = [&](int i) { return W == 1 ? i : w + W * i; };
  auto inside = [&](int i) { return W == 1 || NQ % W == 0 || w + W * i < NQ; };
  const FxElement<NQ> E(reinterpret_cast<double*>(fx_smem) + el * FxElement<NQ>::DOUBLES, l);

  int64_t e = (int64_t)blockIdx.x * EPB + el;
  const bool active = e < Nelements;
  if (active && elementList) e = elementList[e];
  if (!active) e = 0;
  const int64_t nodeBase = e * NP + l;
  // the factors are asked for in L2 by one thread: per element where a warp holds at most one,
  // else for the CTA's whole run of elements (one request per lane would be issued one by one:
  // 90^3, N = 1: 138 against 121 us)
  if constexpr (EPB <= 2) {
    if (active && l == 0 && w == 0) {
      prefetch_l2_bulk(ggeo + e * geoStride, 6 * NP * sizeof(double));
      if constexpr (MASS) prefetch_l2_bulk(wJ + e * wJStride, NP * sizeof(double));
    }
  } else if (tid == 0 && !elementList && geoStride <= 7 * NP) {
    const int64_t n = Nelements - e < EPB ? Nelements - e : EPB;
    prefetch_l2_run(l2_factor_run((uint64_t)(ggeo + e * geoStride), geoStride, (uint64_t)(wJ + e * wJStride), wJStride, NP,
                                   sizeof(double), n, MASS));
    if (MASS && wJStride == NP) prefetch_l2_bulk(wJ + e * NP, (unsigned)(n * NP * sizeof(double)));
  }
  bool plain;
  {
    double v[KN];
    if constexpr (INMODE == IN_GATHER) {
      int32_t id[KN];
#pragma unroll
      for (int i = 0; i < KN; ++i) id[i] = active && inside(i) ? __ldg(g2l + nodeBase + layer(i) * NL) : -1;
#pragma unroll
      for (int i = 0; i < KN; ++i) v[i] = id[i] >= 0 ? q[id[i]] : 0.0;
    } else {
#pragma unroll
      for (int i = 0; i < KN; ++i) v[i] = active && inside(i) ? q[nodeBase + layer(i) * NL] : 0.0;
    }
    plain = fx_tables<NQ, EO>(Dg, tid, FxThreads<NQ, W>::NT, s_tab, s_e, flags & 1);   // while the gather is in flight
#pragma unroll
    for (int i = 0; i < KN; ++i)
      if (inside(i)) E.r(E.a, E.b, layer(i)) = E.s(E.a, E.b, layer(i)) = E.t(E.a, E.b, layer(i)) = v[i];
  }
  plain = __syncthreads_or(plain);
  auto sync = [&](bool any) -> bool {
    if constexpr (W == 1) return ax_fx_sync<NQ, EPB>(el, any);
    else return __syncthreads_or(any);
  };
  const int d0 = W == 1 ? 0 : w, d1 = W == 1 ? 3 : w + 1;
  fx_forward<NQ, EO>(E, s_tab[0], s_e[0], plain, Dg, d0, d1);
  sync(false);

  // G . grad q
  {
    const double* gp = ggeo + e * geoStride + l;
#pragma unroll 4
    for (int i = 0; i < KN; ++i) {
      if (!inside(i)) break;
      const int k = layer(i);
      double G00 = 0, G01 = 0, G02 = 0, G11 = 0, G12 = 0, G22 = 0;
      if (active) {
        G00 = gp[0 * NP + k * NL]; G01 = gp[1 * NP + k * NL]; G02 = gp[2 * NP + k * NL];
        G11 = gp[3 * NP + k * NL]; G12 = gp[4 * NP + k * NL]; G22 = gp[5 * NP + k * NL];
      }
      double &ur = E.r(E.a, E.b, k), &us = E.s(E.a, E.b, k), &ut = E.t(E.a, E.b, k);
      const double qr = ur, qs = us, qt = ut;
      ur = G00 * qr + G01 * qs + G02 * qt;
      us = G01 * qr + G11 * qs + G12 * qt;
      ut = G02 * qr + G12 * qs + G22 * qt;
    }
  }
  sync(false);

  bool fp = fx_transposed<NQ, EO>(E, s_tab[1], plain, Dg, s_x[el], d0, d1);
  int32_t id[KN];   // in flight over the barrier
  if constexpr (OUTMODE == OUT_ASSEMBLE || (MASS && INMODE == IN_GATHER)) {
#pragma unroll
    for (int i = 0; i < KN; ++i) id[i] = active && inside(i) ? __ldg(g2l + nodeBase + layer(i) * NL) : -1;
  }
  fp = sync(fp);

  if (!active) return;
  const double lam = MASS ? (lambdaE ? lambdaE[e] : lambda) : 0.0;
  const double* wp = wJ + e * wJStride + l;
  const int er = s_e[1][fx_row<NQ, EO>(E.a)], es = s_e[1][fx_row<NQ, EO>(E.b)];
#pragma unroll
  for (int i = 0; i < KN; ++i) {
    if (!inside(i)) break;
    const int k = layer(i);
    double r = fx_node_sum<NQ, EO>(E, k, s_x[el], s_e[1], er, es, fp);
    if constexpr (MASS) {
      double v = 0.0;
      if constexpr (INMODE == IN_GATHER) v = id[i] >= 0 ? q[id[i]] : 0.0;
      else v = q[nodeBase + k * NL];
      r = fma(UNIT ? wp[k * NL] : wp[k * NL] * lam, v, r);
    }
    if constexpr (OUTMODE == OUT_ASSEMBLE) {
      if (id[i] >= 0)
        atomicAdd(out + id[i], __hiloint2double(__double2hiint(r) ^ (int)(flags & 0x80000000u), __double2loint(r)));
    } else if constexpr (OUTMODE == OUT_LOCAL) {
      out[nodeBase + k * NL] = r;
    } else {
      out[nodeBase + k * NL] -= r;
    }
  }
}

template <int NQ>
__device__ __forceinline__ int eo_row(const int jj) {
  const int lo = 2 * (jj >> 2) + (jj & 1);
  return (jj & 2) ? (NQ - 1 - lo) : lo;
}

template <int NQ>
__device__ __forceinline__ void eo_sync(const int el) {
  if constexpr ((NQ * NQ) % 32 == 0) elem_sync<NQ>(el);  // Nq = 8: the element's two warps
  else __syncwarp();                                    // Nq = 4: an element is half a warp
}

// ---------------------------------------------------------------- double-word variant
// Layer by layer, contracted through the mirror symmetry of D (even and odd parts of a line, its
// two halves exchanged by shuffles), every value held as a double-FP32 word (df64.cuh):
// FP64-accurate (48-bit significands, sums with absolute error of order 2^-48 times the
// magnitudes summed) on GB300's FP32 pipe, which runs ~64x the FP64 rate. q is read as
// FP64 and split with integer operations; the geometric factors come pre-split
// ([e][7][Np] hi/lo pairs, the same 8 bytes per value as FP64); each local result is
// rebuilt exactly as FP64 hi + lo (one FP64 add) and assembled with FP64 atomics.
// PFG: the geometric factors of layer k+1 are loaded into registers while layer k is
// computed, so their DRAM latency overlaps a whole layer's arithmetic
template <int NQ, bool PFG = false>
__global__ void __launch_bounds__(NQ * NQ * elems_per_block<NQ>(), (NQ == 4 ? 3 : 2))
ax_hex_dw_kernel(const int64_t Nelements, const int32_t* __restrict__ elementList,
                 const int32_t* __restrict__ g2l, const dw* __restrict__ ggeo, const int64_t geoStride,
                 const dw* __restrict__ wJ, const int64_t wJStride, const double* __restrict__ Dg,
                 const double lambda, const double* __restrict__ lambdaE, const double* __restrict__ q,
                 double* __restrict__ out) {
  static_assert(NQ == 4 || NQ == 8, "double-word kernel: Nq = 4 or 8");
  constexpr int NP = NQ * NQ * NQ, H = NQ / 2, N = NQ - 1;
  constexpr int EPB = elems_per_block<NQ>();
  __shared__ dw s_Dp[H][H], s_Dm[H][H], s_Tp[H][H], s_Tm[H][H];
  __shared__ dw s_R[EPB][NQ][NQ], s_S[EPB][NQ][NQ], s_dr[EPB][NQ][NQ], s_ds[EPB][NQ][NQ];
  __shared__ dw s_qt[NQ][NQ * NQ * EPB], s_gt[NQ][NQ * NQ * EPB];

  const int i = threadIdx.x, jj = threadIdx.y, el = threadIdx.z;
  const int j = eo_row<NQ>(jj);
  const int tid = i + NQ * (jj + NQ * el);
  for (int t = tid; t < H * H; t += NQ * NQ * EPB) {
    const int a = t / H, m = t % H;
    const double d0 = Dg[a * NQ + m], d1 = Dg[a * NQ + N - m];
    const double t0 = Dg[m * NQ + a], t1 = Dg[(N - m) * NQ + a];
    s_Dp[a][m] = dw_from_double(0.5 * (d0 + d1));
    s_Dm[a][m] = dw_from_double(0.5 * (d0 - d1));
    s_Tp[a][m] = dw_from_double(0.5 * (t0 + t1));
    s_Tm[a][m] = dw_from_double(0.5 * (t0 - t1));
  }

  int64_t e = (int64_t)blockIdx.x * EPB + el;
  const bool active = e < Nelements;
  if (active && elementList) e = elementList[e];
  if (!active) e = 0;

  dw r_q[NQ], r_Aq[NQ];
  int32_t r_id[NQ];
  const int64_t nodeBase = e * NP + j * NQ + i;
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    const int32_t id = active ? __ldg(g2l + nodeBase + k * NQ * NQ) : -1;
    r_id[k] = id;
    r_q[k] = dw_from_double((id >= 0) ? q[id] : 0.0);
  }
  const dw lam = dw_from_double((lambdaE && active) ? lambdaE[e] : lambda);
  const dw* gp = ggeo + e * geoStride + j * NQ + i;
  const dw* wp = wJ + e * wJStride + j * NQ + i;
  __syncthreads();

  {
    dw E[H], O[H];
#pragma unroll
    for (int m = 0; m < H; ++m) {
      E[m] = dw_add(r_q[m], r_q[N - m]);
      O[m] = dw_sub(r_q[m], r_q[N - m]);
    }
#pragma unroll
    for (int t = 0; t < H; ++t) {
      dw_acc A, B;
#pragma unroll
      for (int m = 0; m < H; ++m) {
        A.mac(s_Dp[t][m], E[m]);
        B.mac(s_Dm[t][m], O[m]);
      }
      const dw a = A.get(), b = B.get();
      s_qt[t][tid] = dw_add(a, b);
      s_qt[N - t][tid] = dw_sub(b, a);
    }
  }

  const bool rtask = i < H;
  const int pt = rtask ? i : i - H;
  dw* dst0 = rtask ? &s_dr[el][j][pt] : &s_ds[el][pt][j];
  dw* dst1 = rtask ? &s_dr[el][j][N - pt] : &s_ds[el][N - pt][j];
  const dw* line = rtask ? &s_R[el][j][0] : &s_S[el][j][0];
  const int slotR = (i < H) ? i : H + N - i, slotS = (j < H) ? j : H + N - j;
  const float sgnR = (i < H) ? 1.f : -1.f, sgnS = (j < H) ? 1.f : -1.f;

  const dw zero{0.f, 0.f};
  dw nG[7];   // next layer's factors (PFG)
  if constexpr (PFG) {
#pragma unroll
    for (int c = 0; c < 6; ++c) nG[c] = active ? gp[c * NP] : zero;
    nG[6] = active ? wp[0] : zero;
  }
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    const int off = k * NQ * NQ;
    dw G00, G01, G02, G11, G12, G22, GwJ;
    if constexpr (PFG) {
      G00 = nG[0]; G01 = nG[1]; G02 = nG[2]; G11 = nG[3]; G12 = nG[4]; G22 = nG[5]; GwJ = nG[6];
      if (k + 1 < NQ) {
        const int noff = off + NQ * NQ;
#pragma unroll
        for (int c = 0; c < 6; ++c) nG[c] = active ? gp[c * NP + noff] : zero;
        nG[6] = active ? wp[noff] : zero;
      }
    } else {
      G00 = active ? gp[0 * NP + off] : zero; G01 = active ? gp[1 * NP + off] : zero;
      G02 = active ? gp[2 * NP + off] : zero; G11 = active ? gp[3 * NP + off] : zero;
      G12 = active ? gp[4 * NP + off] : zero; G22 = active ? gp[5 * NP + off] : zero;
      GwJ = active ? wp[off] : zero;
    }
    const dw v = r_q[k];
    const dw pr = dw_shfl_xor(v, NQ - 1), ps = dw_shfl_xor(v, 2 * NQ);
    s_R[el][j][slotR] = dw_add(pr, dw_scale_sign(sgnR, v));
    s_S[el][i][slotS] = dw_add(ps, dw_scale_sign(sgnS, v));
    eo_sync<NQ>(el);
    {
      dw_acc A, B;
#pragma unroll
      for (int m = 0; m < H; ++m) {
        A.mac(s_Dp[pt][m], line[m]);
        B.mac(s_Dm[pt][m], line[H + m]);
      }
      const dw a = A.get(), b = B.get();
      *dst0 = dw_add(a, b);
      *dst1 = dw_sub(b, a);
    }
    eo_sync<NQ>(el);
    const dw qr = s_dr[el][j][i], qs = s_ds[el][j][i], qtk = s_qt[k][tid];
    dw_acc ar, as, at;
    ar.mac(G00, qr); ar.mac(G01, qs); ar.mac(G02, qtk);
    as.mac(G01, qr); as.mac(G11, qs); as.mac(G12, qtk);
    at.mac(G02, qr); at.mac(G12, qs); at.mac(G22, qtk);
    const dw Gqr = ar.get(), Gqs = as.get();
    s_gt[k][tid] = at.get();
    const dw mass = dw_mul(dw_mul(GwJ, lam), v);
    const dw pr2 = dw_shfl_xor(Gqr, NQ - 1), ps2 = dw_shfl_xor(Gqs, 2 * NQ);
    s_R[el][j][slotR] = dw_add(pr2, dw_scale_sign(sgnR, Gqr));
    s_S[el][i][slotS] = dw_add(ps2, dw_scale_sign(sgnS, Gqs));
    eo_sync<NQ>(el);
    {
      dw_acc A, B;
#pragma unroll
      for (int m = 0; m < H; ++m) {
        A.mac(s_Tp[pt][m], line[m]);
        B.mac(s_Tm[pt][m], line[H + m]);
      }
      const dw a = A.get(), b = B.get();
      *dst0 = dw_add(a, b);
      *dst1 = dw_sub(b, a);
    }
    eo_sync<NQ>(el);
    r_Aq[k] = dw_add(dw_add(mass, s_dr[el][j][i]), s_ds[el][j][i]);
  }

  {
    dw E[H], O[H];
#pragma unroll
    for (int m = 0; m < H; ++m) {
      const dw g0 = s_gt[m][tid], g1 = s_gt[N - m][tid];
      E[m] = dw_add(g0, g1);
      O[m] = dw_sub(g0, g1);
    }
#pragma unroll
    for (int t = 0; t < H; ++t) {
      dw_acc A, B;
#pragma unroll
      for (int m = 0; m < H; ++m) {
        A.mac(s_Tp[t][m], E[m]);
        B.mac(s_Tm[t][m], O[m]);
      }
      const dw a = A.get(), b = B.get();
      r_Aq[t] = dw_add(r_Aq[t], dw_add(a, b));
      r_Aq[N - t] = dw_add(r_Aq[N - t], dw_sub(b, a));
    }
  }

  if (!active) return;
#pragma unroll
  for (int k = 0; k < NQ; ++k)
    if (r_id[k] >= 0) atomicAdd(out + r_id[k], dw_to_double(r_Aq[k]));
}

// n double words from 16-byte aligned shared memory, two per 128-bit load
template <int n>
__device__ __forceinline__ void ld_dw4x2(const dw* src, dw* v) {
  const float4* p = reinterpret_cast<const float4*>(src);
#pragma unroll
  for (int t = 0; t < n / 2; ++t) {
    const float4 x = p[t];
    v[2 * t] = {x.x, x.y};
    v[2 * t + 1] = {x.z, x.w};
  }
}

// The N = 7 double-word kernel for four CTAs (32 warps) per SM, against two for the
// kernel above (64^3: 3.09 ms against 4.36 ms per application):
// - each thread's q pencil lives in shared memory (only the same thread reads it back),
//   and layer k's local result replaces its consumed t-derivative slot, so the thread
//   holds no pencils in registers (64 registers); dof indices are re-read at the end;
// - intermediate sums skip the renormalisation their consumers do not need (dw_add_u,
//   dw_acc::raw), sums start from their first product, and the +-1 of the even/odd line
//   values is folded into FMAs (~660 instructions per node against ~790);
// - line values and D rows are read from shared memory two double words per 128-bit load;
// - the layer loop is rolled (8x less code: instruction-cache misses were a stall with
//   four CTAs in different phases);
// - one thread per element asks L2 for the element's geometric factors (and wJ) in one
//   bulk prefetch each, so the per-layer loads of layers 1..N hit L2.
// Measured and not kept: the next layer's factors staged through shared memory with
// cp.async (more shared-memory traffic; slower at three CTAs per SM), a register prefetch
// (does not fit 64 registers). MASS = false: lambda == 0 and no lambda field, the mass term
// and its wJ reads are left out.
template <int NQ, bool MASS, bool UNIT = false>
__global__ void __launch_bounds__(NQ * NQ * elems_per_block<NQ>(), 4)
ax_hex_dw_lean_kernel(const int64_t Nelements, const int32_t* __restrict__ elementList,
                      const int32_t* __restrict__ g2l, const dw* __restrict__ ggeo, const int64_t geoStride,
                      const dw* __restrict__ wJ, const int64_t wJStride, const double* __restrict__ Dg,
                      const double lambda, const double* __restrict__ lambdaE, const double* __restrict__ q,
                      double* __restrict__ out) {
  static_assert(NQ == 8, "lean double-word kernel: Nq = 8");
  constexpr int NP = NQ * NQ * NQ, H = NQ / 2, N = NQ - 1;
  constexpr int EPB = elems_per_block<NQ>();
  constexpr int NT = NQ * NQ * EPB;
  __shared__ __align__(16) dw s_Dp[H][H], s_Dm[H][H], s_Tp[H][H], s_Tm[H][H];
  __shared__ __align__(16) dw s_R[EPB][NQ][NQ], s_S[EPB][NQ][NQ];
  __shared__ dw s_dr[EPB][NQ][NQ], s_ds[EPB][NQ][NQ];
  // s_q: layer k of the thread's q pencil until layer k reads it, then that layer's
  // t-contraction input G_t . grad q (the same thread writes and reads each slot)
  __shared__ dw s_q[NQ][NT], s_qt[NQ][NT];

  const int i = threadIdx.x, jj = threadIdx.y, el = threadIdx.z;
  const int j = eo_row<NQ>(jj);
  const int tid = i + NQ * (jj + NQ * el);
  for (int t = tid; t < H * H; t += NT) {
    const int a = t / H, m = t % H;
    const double d0 = Dg[a * NQ + m], d1 = Dg[a * NQ + N - m];
    const double t0 = Dg[m * NQ + a], t1 = Dg[(N - m) * NQ + a];
    s_Dp[a][m] = dw_from_double(0.5 * (d0 + d1));
    s_Dm[a][m] = dw_from_double(0.5 * (d0 - d1));
    s_Tp[a][m] = dw_from_double(0.5 * (t0 + t1));
    s_Tm[a][m] = dw_from_double(0.5 * (t0 - t1));
  }

  int64_t e = (int64_t)blockIdx.x * EPB + el;
  const bool active = e < Nelements;
  if (active && elementList) e = elementList[e];
  if (!active) e = 0;

  const int64_t nodeBase = e * NP + j * NQ + i;
  if (active && i == 0 && jj == 0) {
    prefetch_l2_bulk(ggeo + e * geoStride, 6 * NP * sizeof(dw));
    if constexpr (MASS) prefetch_l2_bulk(wJ + e * wJStride, NP * sizeof(dw));
  }
  {
    int32_t id[NQ];
#pragma unroll
    for (int k = 0; k < NQ; ++k) id[k] = active ? __ldg(g2l + nodeBase + k * NQ * NQ) : -1;
    double qv[NQ];
#pragma unroll
    for (int k = 0; k < NQ; ++k) qv[k] = (id[k] >= 0) ? q[id[k]] : 0.0;
#pragma unroll
    for (int k = 0; k < NQ; ++k) s_q[k][tid] = dw_from_double(qv[k]);
  }
  const dw lam = MASS ? dw_from_double((lambdaE && active) ? lambdaE[e] : lambda) : dw{0.f, 0.f};
  const dw* gp = ggeo + e * geoStride + j * NQ + i;
  const dw* wp = wJ + e * wJStride + j * NQ + i;
  __syncthreads();

  {
    dw E[H], O[H];
#pragma unroll
    for (int m = 0; m < H; ++m) {
      const dw q0 = s_q[m][tid], q1 = s_q[N - m][tid];
      E[m] = dw_add_u(q0, q1);
      O[m] = dw_add_u(q0, dw_neg(q1));
    }
#pragma unroll
    for (int t = 0; t < H; ++t) {
      dw_acc A(s_Dp[t][0], E[0]), B(s_Dm[t][0], O[0]);
#pragma unroll
      for (int m = 1; m < H; ++m) {
        A.mac(s_Dp[t][m], E[m]);
        B.mac(s_Dm[t][m], O[m]);
      }
      const dw a = A.raw(), b = B.raw();
      s_qt[t][tid] = dw_add_u(a, b);
      s_qt[N - t][tid] = dw_add_u(b, dw_neg(a));
    }
  }

  const bool rtask = i < H;
  const int pt = rtask ? i : i - H;
  dw* dst0 = rtask ? &s_dr[el][j][pt] : &s_ds[el][pt][j];
  dw* dst1 = rtask ? &s_dr[el][j][N - pt] : &s_ds[el][N - pt][j];
  const dw* line = rtask ? &s_R[el][j][0] : &s_S[el][j][0];
  const int slotR = (i < H) ? i : H + N - i, slotS = (j < H) ? j : H + N - j;
  const float sgnR = (i < H) ? 1.f : -1.f, sgnS = (j < H) ? 1.f : -1.f;

  const dw zero{0.f, 0.f};
  // the local result of layer k goes to s_qt[k] once layer k has read its t-derivative
#pragma unroll 1
  for (int k = 0; k < NQ; ++k) {
    const int off = k * NQ * NQ;
    const dw G00 = active ? gp[0 * NP + off] : zero, G01 = active ? gp[1 * NP + off] : zero;
    const dw G02 = active ? gp[2 * NP + off] : zero, G11 = active ? gp[3 * NP + off] : zero;
    const dw G12 = active ? gp[4 * NP + off] : zero, G22 = active ? gp[5 * NP + off] : zero;
    dw GwJ = zero;
    if constexpr (MASS) GwJ = active ? wp[off] : zero;
    const dw v = s_q[k][tid];
    const dw pr = dw_shfl_xor(v, NQ - 1), ps = dw_shfl_xor(v, 2 * NQ);
    s_R[el][j][slotR] = dw_add_sign_u(pr, sgnR, v);
    s_S[el][i][slotS] = dw_add_sign_u(ps, sgnS, v);
    eo_sync<NQ>(el);
    {
      dw L[NQ], Dp[H], Dm[H];
      ld_dw4x2<NQ>(line, L);
      ld_dw4x2<H>(&s_Dp[pt][0], Dp);
      ld_dw4x2<H>(&s_Dm[pt][0], Dm);
      dw_acc A(Dp[0], L[0]), B(Dm[0], L[H]);
#pragma unroll
      for (int m = 1; m < H; ++m) {
        A.mac(Dp[m], L[m]);
        B.mac(Dm[m], L[H + m]);
      }
      const dw a = A.raw(), b = B.raw();
      *dst0 = dw_add_u(a, b);
      *dst1 = dw_add_u(b, dw_neg(a));
    }
    eo_sync<NQ>(el);
    const dw qr = s_dr[el][j][i], qs = s_ds[el][j][i], qtk = s_qt[k][tid];
    dw_acc ar(G00, qr), as(G01, qr), at(G02, qr);
    ar.mac(G01, qs); ar.mac(G02, qtk);
    as.mac(G11, qs); as.mac(G12, qtk);
    at.mac(G12, qs); at.mac(G22, qtk);
    const dw Gqr = ar.raw(), Gqs = as.raw();
    s_q[k][tid] = at.raw();
    dw mass{0.f, 0.f};
    if constexpr (MASS && UNIT) mass = dw_mul(GwJ, v);   // lambda == 1: wJ q
    else if constexpr (MASS) mass = dw_mul(dw_mul(GwJ, lam), v);
    const dw pr2 = dw_shfl_xor(Gqr, NQ - 1), ps2 = dw_shfl_xor(Gqs, 2 * NQ);
    s_R[el][j][slotR] = dw_add_sign_u(pr2, sgnR, Gqr);
    s_S[el][i][slotS] = dw_add_sign_u(ps2, sgnS, Gqs);
    eo_sync<NQ>(el);
    {
      dw L[NQ], Tp[H], Tm[H];
      ld_dw4x2<NQ>(line, L);
      ld_dw4x2<H>(&s_Tp[pt][0], Tp);
      ld_dw4x2<H>(&s_Tm[pt][0], Tm);
      dw_acc A(Tp[0], L[0]), B(Tm[0], L[H]);
#pragma unroll
      for (int m = 1; m < H; ++m) {
        A.mac(Tp[m], L[m]);
        B.mac(Tm[m], L[H + m]);
      }
      const dw a = A.raw(), b = B.raw();
      *dst0 = dw_add_u(a, b);
      *dst1 = dw_add_u(b, dw_neg(a));
    }
    eo_sync<NQ>(el);
    if constexpr (MASS) s_qt[k][tid] = dw_add_u(dw_add_u(mass, s_dr[el][j][i]), s_ds[el][j][i]);
    else s_qt[k][tid] = dw_add_u(s_dr[el][j][i], s_ds[el][j][i]);
  }

  {
    dw E[H], O[H];
#pragma unroll
    for (int m = 0; m < H; ++m) {
      const dw g0 = s_q[m][tid], g1 = s_q[N - m][tid];
      E[m] = dw_add_u(g0, g1);
      O[m] = dw_add_u(g0, dw_neg(g1));
    }
#pragma unroll
    for (int t = 0; t < H; ++t) {
      dw_acc A(s_Tp[t][0], E[0]), B(s_Tm[t][0], O[0]);
#pragma unroll
      for (int m = 1; m < H; ++m) {
        A.mac(s_Tp[t][m], E[m]);
        B.mac(s_Tm[t][m], O[m]);
      }
      const dw a = A.raw(), b = B.raw();
      s_qt[t][tid] = dw_add_u(s_qt[t][tid], dw_add_u(a, b));
      s_qt[N - t][tid] = dw_add_u(s_qt[N - t][tid], dw_add_u(b, dw_neg(a)));
    }
  }

  if (!active) return;
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    const int32_t id = __ldg(g2l + nodeBase + k * NQ * NQ);
    if (id >= 0) atomicAdd(out + id, dw_to_double(s_qt[k][tid]));
  }
}

// Double-word operator for the degrees without an even-odd kernel (N = 1, 2, 4, 5, 6, 8):
// one thread per node, EPB elements per CTA (at least 128 threads), direct Nq-term
// contractions through shared memory, the same df64 building blocks and FP64 assembly.
template <int NQ>
constexpr int dw_generic_epb() {
  return (NQ * NQ * NQ >= 128) ? 1 : 128 / (NQ * NQ * NQ);
}

template <int NQ>
__global__ void __launch_bounds__(NQ * NQ * NQ * dw_generic_epb<NQ>())
ax_hex_dw_generic_kernel(const int64_t Nelements, const int32_t* __restrict__ elementList,
                         const int32_t* __restrict__ g2l, const dw* __restrict__ ggeo, const int64_t geoStride,
                         const dw* __restrict__ wJ, const int64_t wJStride, const double* __restrict__ Dg,
                         const double lambda, const double* __restrict__ lambdaE, const double* __restrict__ q,
                         double* __restrict__ out) {
  constexpr int NP = NQ * NQ * NQ, NFP = NQ * NQ, EPB = dw_generic_epb<NQ>();
  __shared__ dw s_D[NQ * NQ];
  __shared__ dw s_q[EPB][NP], s_r[EPB][NP], s_s[EPB][NP], s_t[EPB][NP];
  const int el = threadIdx.x / NP, n = threadIdx.x % NP;
  for (int t = threadIdx.x; t < NQ * NQ; t += blockDim.x) s_D[t] = dw_from_double(Dg[t]);
  int64_t e = (int64_t)blockIdx.x * EPB + el;
  const bool active = e < Nelements;
  if (active && elementList) e = elementList[e];
  if (!active) e = 0;
  const int32_t id = active ? g2l[e * NP + n] : -1;
  const dw qn = dw_from_double(id >= 0 ? q[id] : 0.0);
  s_q[el][n] = qn;
  __syncthreads();
  const int i = n % NQ, j = (n / NQ) % NQ, k = n / NFP;
  dw_acc ar, as, at;
#pragma unroll
  for (int m = 0; m < NQ; ++m) {
    ar.mac(s_D[i * NQ + m], s_q[el][m + j * NQ + k * NFP]);
    as.mac(s_D[j * NQ + m], s_q[el][i + m * NQ + k * NFP]);
    at.mac(s_D[k * NQ + m], s_q[el][i + j * NQ + m * NFP]);
  }
  const dw qr = ar.get(), qs = as.get(), qt = at.get();
  const dw* gp = ggeo + e * geoStride + n;
  const dw G00 = gp[0 * NP], G01 = gp[1 * NP], G02 = gp[2 * NP], G11 = gp[3 * NP], G12 = gp[4 * NP],
           G22 = gp[5 * NP];
  const dw GwJ = wJ[e * wJStride + n];
  const dw lam = dw_from_double((lambdaE && active) ? lambdaE[e] : lambda);
  {
    dw_acc gr, gs, gt;
    gr.mac(G00, qr); gr.mac(G01, qs); gr.mac(G02, qt);
    gs.mac(G01, qr); gs.mac(G11, qs); gs.mac(G12, qt);
    gt.mac(G02, qr); gt.mac(G12, qs); gt.mac(G22, qt);
    s_r[el][n] = gr.get();
    s_s[el][n] = gs.get();
    s_t[el][n] = gt.get();
  }
  const dw mass = dw_mul(dw_mul(GwJ, lam), qn);
  __syncthreads();
  dw_acc v;
  v.h = mass.h;
  v.l = mass.l;
#pragma unroll
  for (int p = 0; p < NQ; ++p) {
    v.mac(s_D[p * NQ + i], s_r[el][p + j * NQ + k * NFP]);
    v.mac(s_D[p * NQ + j], s_s[el][i + p * NQ + k * NFP]);
    v.mac(s_D[p * NQ + k], s_t[el][i + j * NQ + p * NFP]);
  }
  if (id >= 0) atomicAdd(out + id, dw_to_double(v.get()));
}

template <int NQ>
static int launch_dw_generic(const AxArgs<double, float2>& a, cudaStream_t s) {
  constexpr int EPB = dw_generic_epb<NQ>();
  const int64_t blocks = (a.Nelements + EPB - 1) / EPB;
  ax_hex_dw_generic_kernel<NQ><<<(unsigned)blocks, NQ * NQ * NQ * EPB, 0, s>>>(
      a.Nelements, a.elementList, a.g2l, reinterpret_cast<const dw*>(a.ggeo), a.geoStride,
      reinterpret_cast<const dw*>(a.wJ), a.wJStride, a.D, a.lambda, a.lambdaE, a.q, a.out);
  LPG_LAUNCH_CHECK("ax_hex_dw_generic_kernel");
  return LPG_OK;
}

// N = 7 double-word kernel: the four-CTA kernel (ax_hex_dw_lean_kernel). LPG_AX_DW =
// classic is a tuning override back to the two-CTA kernel with the register prefetch.
static bool dw7_classic() {
  static const bool v = [] {
    const char* ev = std::getenv("LPG_AX_DW");
    return ev && !std::strcmp(ev, "classic");
  }();
  return v;
}

int ax_hex_dw(const AxArgs<double, float2>& a, cudaStream_t s) {
  if (a.Nelements <= 0) return LPG_OK;
  if (a.N < 1 || a.N > 8) return set_error(LPG_ERR_UNSUPPORTED, "double-word operator: N must be 1..8");
  if (a.Nglobal > 0) LPG_CUDA_TRY(cudaMemsetAsync(a.out, 0, sizeof(double) * a.Nglobal, s));
  switch (a.N) {
    case 1: return launch_dw_generic<2>(a, s);
    case 2: return launch_dw_generic<3>(a, s);
    case 4: return launch_dw_generic<5>(a, s);
    case 5: return launch_dw_generic<6>(a, s);
    case 6: return launch_dw_generic<7>(a, s);
    case 8: return launch_dw_generic<9>(a, s);
    default: break;
  }
  if (a.N == 7) {
    const int64_t blocks = (a.Nelements + 3) / 4;
    const bool mass = a.lambdaE || a.lambda != 0.0;
#define LPG_DW_ARGS                                                                                   \
  a.Nelements, a.elementList, a.g2l, reinterpret_cast<const dw*>(a.ggeo), a.geoStride,               \
      reinterpret_cast<const dw*>(a.wJ), a.wJStride, a.D, a.lambda, a.lambdaE, a.q, a.out
    if (dw7_classic())
      ax_hex_dw_kernel<8, true><<<(unsigned)blocks, dim3(8, 8, 4), 0, s>>>(LPG_DW_ARGS);
    else if (mass && a.lambda == 1.0 && !a.lambdaE)
      ax_hex_dw_lean_kernel<8, true, true><<<(unsigned)blocks, dim3(8, 8, 4), 0, s>>>(LPG_DW_ARGS);
    else if (mass)
      ax_hex_dw_lean_kernel<8, true><<<(unsigned)blocks, dim3(8, 8, 4), 0, s>>>(LPG_DW_ARGS);
    else
      ax_hex_dw_lean_kernel<8, false><<<(unsigned)blocks, dim3(8, 8, 4), 0, s>>>(LPG_DW_ARGS);
#undef LPG_DW_ARGS
  } else {
    const int64_t blocks = (a.Nelements + 15) / 16;
    ax_hex_dw_kernel<4><<<(unsigned)blocks, dim3(4, 4, 16), 0, s>>>(
        a.Nelements, a.elementList, a.g2l, reinterpret_cast<const dw*>(a.ggeo), a.geoStride,
        reinterpret_cast<const dw*>(a.wJ), a.wJStride, a.D, a.lambda, a.lambdaE, a.q, a.out);
  }
  LPG_LAUNCH_CHECK("ax_hex_dw_kernel");
  return LPG_OK;
}

// LPG_AX_FP64 = direct: tuning override back to the direct-contraction FP64 kernel (ax_hex_kernel)
static bool fp64_direct_override() {
  static const bool direct = [] {
    const char* e = std::getenv("LPG_AX_FP64");
    return e && !std::strcmp(e, "direct");
  }();
  return direct;
}

template <int NQ, bool EO, int W, int INMODE, int OUTMODE, bool MASS, bool UNIT>
static int fx_config(KernelConfig* cfg, size_t* smem) {
  using L = FxThreads<NQ, W>;
  static PerDeviceConfig perDevice;   // per instantiation: dynamic shared memory opt-in, occupancy
  auto kern = ax_hex_fx_kernel<NQ, EO, W, INMODE, OUTMODE, MASS, UNIT>;
  const size_t bytes = sizeof(double) * FxElement<NQ>::DOUBLES * L::EPB;
  *smem = bytes;
  return perDevice.get(
      [&](int, KernelConfig& c) {
        LPG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
        LPG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c.ctasPerSM, kern, L::NT, bytes));
        return (int)LPG_OK;
      },
      cfg);
}

template <int NQ, bool EO, int W, int INMODE, int OUTMODE, bool MASS, bool UNIT>
static int launch_fx(const AxArgs<double, double>& a, cudaStream_t s) {
  using L = FxThreads<NQ, W>;
  KernelConfig cfg;
  size_t smem;
  const int rc = fx_config<NQ, EO, W, INMODE, OUTMODE, MASS, UNIT>(&cfg, &smem);
  if (rc) return rc;
  const int64_t blocks = (a.Nelements + L::EPB - 1) / L::EPB;
  if (blocks > 0x7fffffffLL) return set_error(LPG_ERR_INVALID, "ax: too many elements");
  ax_hex_fx_kernel<NQ, EO, W, INMODE, OUTMODE, MASS, UNIT><<<(unsigned)blocks, L::NT, smem, s>>>(
      a.Nelements, a.elementList, a.g2l, a.ggeo, a.geoStride, a.wJ, a.wJStride, a.D, a.lambda, a.lambdaE, a.q, a.out,
      (a.outScale < 0 ? 0x80000000u : 0u) | (a.mirrored ? 1u : 0u));
  LPG_LAUNCH_CHECK("ax_hex_fx_kernel");
  return LPG_OK;
}

template <int NQ, typename G>
static int launch_line(const AxArgs<float, G>& a, cudaStream_t s) {
  using L = LineLayout<NQ>;
  const int64_t blocks = (a.Nelements + L::EPB - 1) / L::EPB;
  if (blocks > 0x7fffffffLL) return set_error(LPG_ERR_INVALID, "ax: too many elements");
  auto go = [&](auto kern) {
    kern<<<(unsigned)blocks, L::NT, 0, s>>>(a.Nelements, a.elementList, a.g2l, a.ggeo, a.geoStride, a.wJ, a.wJStride,
                                            a.D, a.lambda, a.lambdaE, a.q, a.out, a.outScale);
  };
  const bool noMass = a.lambda == 0 && !a.lambdaE;
  // BF16 factors at Nq = 8, where they start on 16-byte boundaries, are copied: 48^3 322 us against
  // 357 read where they are used. FP32 factors need twice the shared memory, so fewer CTAs fit: 400
  // against 383.
  if constexpr (NQ == 8 && std::is_same<G, __nv_bfloat16>::value) {
    if (((uintptr_t)a.ggeo & 15) == 0 && ((uintptr_t)a.wJ & 15) == 0 && a.geoStride % 8 == 0 && a.wJStride % 8 == 0) {
      if (noMass) go(ax_hex_line_kernel<NQ, G, false, true>);
      else go(ax_hex_line_kernel<NQ, G, true, true>);
      LPG_LAUNCH_CHECK("ax_hex_line_kernel");
      return LPG_OK;
    }
  }
  if (noMass) go(ax_hex_line_kernel<NQ, G, false, false>);
  else go(ax_hex_line_kernel<NQ, G, true, false>);
  LPG_LAUNCH_CHECK("ax_hex_line_kernel");
  return LPG_OK;
}

// FP32 vectors. Measured against the kernels before this one, which copied a persistent CTA's
// next elements to shared memory (Nq = 4, 8) or read D once per direction (the other Nq), us.
// FP32 geometry: 100^3, N = 1 68.5 -> 66.2; 80^3, N = 2 118 -> 110; 100^3, N = 3 491 -> 411;
// 48^3, N = 4 119 -> 110; 40^3, N = 5 142 -> 110; 30^3, N = 6 100 -> 83; 48^3, N = 7 425 -> 379;
// 24^3, N = 8 113 -> 96. BF16 geometry: 60^3, N = 3 101 -> 87; 40^3, N = 5 120 -> 101; 48^3,
// N = 7 410 -> 323.
template <int NQ, int INMODE, int OUTMODE, typename G>
static int launch_ax(const AxArgs<float, G>& a, cudaStream_t s) {
  if constexpr (INMODE == IN_GATHER && OUTMODE == OUT_ASSEMBLE) {
    if (a.Nelements <= 0) return LPG_OK;
    return launch_line<NQ, G>(a, s);
  } else {
    return set_error(LPG_ERR_UNSUPPORTED, "ax: FP32 vectors are provided for the assembled operator only");
  }
}

template <int NQ, int INMODE, int OUTMODE>
static int launch_ax(const AxArgs<double, double>& a, cudaStream_t s) {
  if (a.Nelements <= 0) return LPG_OK;
  if (!fp64_direct_override()) {
    auto go = [&](auto eo) {
      constexpr bool EO = decltype(eo)::value;
      // Below 448 line positions an SM the GPU is not full and the time is that of one element:
      // three threads a position, each with one direction. Measured, one against three threads:
      // N = 7, 4^3 18.6 against 12.5 us, 10^3 29.1 against 25.0, 12^3 35.2 against 35.4, 16^3 73
      // against 79; N = 5, 8^3 17.6 against 13.6, 16^3 35.2 against 35.0; N = 3, 14^3 16.9
      // against 14.8, 20^3 23.0 against 24.9.
      if constexpr (OUTMODE == OUT_ASSEMBLE && EO) {
        KernelConfig cfg;
        size_t smem;
        const int rc = fx_config<NQ, EO, 1, INMODE, OUTMODE, true, false>(&cfg, &smem);
        if (rc) return rc;
        if (a.Nelements * (NQ * NQ) <= (int64_t)448 * cfg.numSMs) {
          if (a.lambda == 0.0 && !a.lambdaE) return launch_fx<NQ, EO, 3, INMODE, OUTMODE, false, false>(a, s);
          return launch_fx<NQ, EO, 3, INMODE, OUTMODE, true, false>(a, s);
        }
      }
      if (a.lambda == 0.0 && !a.lambdaE) return launch_fx<NQ, EO, 1, INMODE, OUTMODE, false, false>(a, s);
      if (a.lambda == 1.0 && !a.lambdaE) return launch_fx<NQ, EO, 1, INMODE, OUTMODE, true, true>(a, s);
      return launch_fx<NQ, EO, 1, INMODE, OUTMODE, true, false>(a, s);
    };
    // half the products where D is known to be mirrored (28^3, N = 5: 133 against 156 us;
    // 20^3, N = 8: 201 against 253 us)
    if constexpr (NQ != 4 && NQ != 8 && OUTMODE == OUT_ASSEMBLE)
      if (a.mirrored) return go(std::true_type{});
    return go(std::integral_constant<bool, NQ == 4 || NQ == 8>{});
  }
  constexpr int EPB = elems_per_block<NQ>();
  const int64_t blocks = (a.Nelements + EPB - 1) / EPB;
  if (blocks > 0x7fffffffLL) return set_error(LPG_ERR_INVALID, "ax: too many elements");
  ax_hex_kernel<NQ, INMODE, OUTMODE><<<(unsigned)blocks, dim3(NQ, NQ, EPB), 0, s>>>(
      a.Nelements, a.elementList, a.g2l, a.ggeo, a.geoStride, a.wJ, a.wJStride, a.D, a.lambda, a.lambdaE, a.q, a.out,
      a.outScale);
  LPG_LAUNCH_CHECK("ax_hex_kernel");
  return LPG_OK;
}

template <typename T, typename G, int INMODE, int OUTMODE>
static int dispatch_ax(const AxArgs<T, G>& a, cudaStream_t s) {
  switch (a.N) {
    case 1: return launch_ax<2, INMODE, OUTMODE>(a, s);
    case 2: return launch_ax<3, INMODE, OUTMODE>(a, s);
    case 3: return launch_ax<4, INMODE, OUTMODE>(a, s);
    case 4: return launch_ax<5, INMODE, OUTMODE>(a, s);
    case 5: return launch_ax<6, INMODE, OUTMODE>(a, s);
    case 6: return launch_ax<7, INMODE, OUTMODE>(a, s);
    case 7: return launch_ax<8, INMODE, OUTMODE>(a, s);
    case 8: return launch_ax<9, INMODE, OUTMODE>(a, s);
    default: return set_error(LPG_ERR_UNSUPPORTED, "ax: polynomial degree must be 1..8");
  }
}

template <typename T, typename G>
int ax_hex(const AxArgs<T, G>& a, AxMode mode, cudaStream_t s) {
  if (std::is_same<T, double>::value && a.outScale != T(1) && a.outScale != T(-1))
    return set_error(LPG_ERR_UNSUPPORTED, "ax: FP64 assembles A q or -A q");
  switch (mode) {
    case AxMode::Assemble: {
      if (a.Nglobal > 0) LPG_CUDA_TRY(cudaMemsetAsync(a.out, 0, sizeof(T) * a.Nglobal, s));
      return dispatch_ax<T, G, IN_GATHER, OUT_ASSEMBLE>(a, s);
    }
    case AxMode::AccumulateAssembled:
      return dispatch_ax<T, G, IN_GATHER, OUT_ASSEMBLE>(a, s);
    case AxMode::PartialLocal:
      return dispatch_ax<T, G, IN_GATHER, OUT_LOCAL>(a, s);
    case AxMode::LocalInSubtract:
      return dispatch_ax<T, G, IN_LOCAL, OUT_LOCAL_SUB>(a, s);
  }
  return set_error(LPG_ERR_INVALID, "ax: bad mode");
}

template <int NQ>
static int wave_elements(bool dw, bool mass) {
  int dev = 0, sms = 0, per = 0, epb = elems_per_block<NQ>();
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 1;
  cudaError_t e = cudaSuccess;
  if (dw) {
    if constexpr (NQ == 8)
      e = dw7_classic()
              ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, ax_hex_dw_kernel<8, true>, NQ * NQ * epb, 0)
              : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, ax_hex_dw_lean_kernel<8, true>, NQ * NQ * epb, 0);
    else
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, ax_hex_dw_kernel<NQ>, NQ * NQ * epb, 0);
  } else if (fp64_direct_override()) {
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, ax_hex_kernel<NQ, IN_GATHER, OUT_ASSEMBLE>,
                                                      NQ * NQ * epb, 0);
  } else {
    KernelConfig cfg;
    size_t smem;
    const int rc = mass ? fx_config<NQ, true, 1, IN_GATHER, OUT_ASSEMBLE, true, false>(&cfg, &smem)
                        : fx_config<NQ, true, 1, IN_GATHER, OUT_ASSEMBLE, false, false>(&cfg, &smem);
    per = rc ? 0 : cfg.ctasPerSM;
    epb = FxLayout<NQ>::EPB;
  }
  if (e != cudaSuccess || per < 1) {
    cudaGetLastError();
    return 1;
  }
  return sms * per * epb;
}

int ax_wave_elements(int N, bool dw, bool mass) {
  if (N == 7) return wave_elements<8>(dw, mass);
  if (N == 3) return wave_elements<4>(dw, mass);
  return 1;
}

template int ax_hex<double, double>(const AxArgs<double, double>&, AxMode, cudaStream_t);
template int ax_hex<float, float>(const AxArgs<float, float>&, AxMode, cudaStream_t);
template int ax_hex<float, __nv_bfloat16>(const AxArgs<float, __nv_bfloat16>&, AxMode, cudaStream_t);

}  // namespace lpg

using namespace lpg;

template <typename T, typename G>
static int ax_entry(int N, int64_t Nelements, const int32_t* elementList, const int32_t* g2l,
                    const G* ggeo, int64_t geoStride, const G* wJ, int64_t wJStride, const T* D,
                    T lambda, const T* lambdaE, const T* q, T* out, int64_t Nglobal, AxMode mode,
                    void* stream) {
  if (N < 1 || N > 8) return set_error(LPG_ERR_UNSUPPORTED, "polynomial degree must be 1..8");
  if (Nelements < 0 || !g2l || !ggeo || !wJ || !D || !q || !out)
    return set_error(LPG_ERR_INVALID, "ax: null pointer or negative size");
  const int64_t Np = (int64_t)(N + 1) * (N + 1) * (N + 1);
  if (geoStride < 6 * Np || wJStride < Np) return set_error(LPG_ERR_INVALID, "ax: stride too small");
  AxArgs<T, G> a;
  a.N = N; a.Nelements = Nelements; a.elementList = elementList; a.g2l = g2l;
  a.ggeo = ggeo; a.geoStride = geoStride; a.wJ = wJ; a.wJStride = wJStride; a.D = D;
  a.lambda = lambda; a.lambdaE = lambdaE; a.q = q; a.out = out; a.Nglobal = Nglobal;
  return ax_hex<T, G>(a, mode, as_stream(stream));
}

extern "C" int lpg_ax_hex_f64(int N, int64_t Nelements, const int32_t* elementList,
                              const int32_t* GlobalToLocal, const double* ggeo, int64_t geoStride,
                              const double* wJ, int64_t wJStride, const double* D, double lambda,
                              const double* lambdaE, const double* q, double* Aq, int64_t Nglobal,
                              void* stream) {
  return ax_entry<double, double>(N, Nelements, elementList, GlobalToLocal, ggeo, geoStride, wJ,
                                  wJStride, D, lambda, lambdaE, q, Aq, Nglobal, AxMode::Assemble,
                                  stream);
}

extern "C" int lpg_ax_hex_f32(int N, int64_t Nelements, const int32_t* elementList,
                              const int32_t* GlobalToLocal, const float* ggeo, int64_t geoStride,
                              const float* wJ, int64_t wJStride, const float* D, float lambda,
                              const float* lambdaE, const float* q, float* Aq, int64_t Nglobal,
                              void* stream) {
  return ax_entry<float, float>(N, Nelements, elementList, GlobalToLocal, ggeo, geoStride, wJ,
                                wJStride, D, lambda, lambdaE, q, Aq, Nglobal, AxMode::Assemble,
                                stream);
}

extern "C" int lpg_ax_hex_bf16g(int N, int64_t Nelements, const int32_t* elementList,
                                const int32_t* GlobalToLocal, const void* ggeo_bf16,
                                int64_t geoStride, const void* wJ_bf16, int64_t wJStride,
                                const float* D, float lambda, const float* lambdaE, const float* q,
                                float* Aq, int64_t Nglobal, void* stream) {
  return ax_entry<float, __nv_bfloat16>(
      N, Nelements, elementList, GlobalToLocal, (const __nv_bfloat16*)ggeo_bf16, geoStride,
      (const __nv_bfloat16*)wJ_bf16, wJStride, D, lambda, lambdaE, q, Aq, Nglobal,
      AxMode::Assemble, stream);
}

extern "C" int lpg_partial_ax_hex_f64(int N, int64_t Nelements, const int32_t* elementList,
                                      const int32_t* GlobalToLocal, const double* ggeo,
                                      int64_t geoStride, const double* wJ, int64_t wJStride,
                                      const double* D, double lambda, const double* lambdaE,
                                      const double* q, double* AqL, void* stream) {
  return ax_entry<double, double>(N, Nelements, elementList, GlobalToLocal, ggeo, geoStride, wJ,
                                  wJStride, D, lambda, lambdaE, q, AqL, 0, AxMode::PartialLocal,
                                  stream);
}
