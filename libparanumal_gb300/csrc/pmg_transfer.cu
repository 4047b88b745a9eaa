// p-multigrid transfers (tensor-product restriction / prolongation between GLL degrees).
//
// Restriction follows ellipticPartialPreconCoarsenHex3D
// (solvers/elliptic/okl/ellipticPreconCoarsenHex3D.okl:209-294) with the inverse-degree
// weighting (ellipticPreconMultiGridLevel.cpp:41-82) folded into the load and the coarse
// ogs Gather(Add, Trans) folded into the store (atomics). Prolongation follows
// ellipticPartialPreconProlongateHex3D (ellipticPreconProlongateHex3D.okl:216-301) with the
// Gather(NoTrans) + axpy folded into the store: the owning copy of each fine dof adds
// its value.
#include <type_traits>

#include "fx64.cuh"
#include "lpg_common.cuh"
#include "lpg_internal.hpp"

namespace lpg {

template <typename T>
__global__ void __launch_bounds__(256)
pmg_coarsen_kernel(const int NqF, const int NqC, const int32_t* __restrict__ g2lF,
                   const T* __restrict__ wF, const T* __restrict__ xF, const T* __restrict__ Pg,
                   const int32_t* __restrict__ g2lC, T* __restrict__ xC) {
  __shared__ T s_f[kMaxNq * kMaxNq * kMaxNq];
  __shared__ T s_cff[kMaxNq * kMaxNq * kMaxNq];
  __shared__ T s_ccf[kMaxNq * kMaxNq * kMaxNq];
  __shared__ T s_P[kMaxNq * kMaxNq];
  const int64_t e = blockIdx.x;
  const int NpF = NqF * NqF * NqF, NpC = NqC * NqC * NqC;
  for (int t = threadIdx.x; t < NqF * NqC; t += blockDim.x) s_P[t] = Pg[t];
  for (int t = threadIdx.x; t < NpF; t += blockDim.x) {
    const int32_t g = g2lF[e * NpF + t];
    s_f[t] = (g >= 0) ? wF[g] * xF[g] : T(0);
  }
  __syncthreads();
  // k: s_cff[k][j][i] = sum_m P[m][k] f[m][j][i]
  for (int t = threadIdx.x; t < NqC * NqF * NqF; t += blockDim.x) {
    const int i = t % NqF, j = (t / NqF) % NqF, k = t / (NqF * NqF);
    T r = 0;
    for (int m = 0; m < NqF; ++m) r += s_P[m * NqC + k] * s_f[m * NqF * NqF + j * NqF + i];
    s_cff[t] = r;
  }
  __syncthreads();
  // j: s_ccf[k][j][i] = sum_m P[m][j] cff[k][m][i]
  for (int t = threadIdx.x; t < NqC * NqC * NqF; t += blockDim.x) {
    const int i = t % NqF, j = (t / NqF) % NqC, k = t / (NqF * NqC);
    T r = 0;
    for (int m = 0; m < NqF; ++m) r += s_P[m * NqC + j] * s_cff[k * NqF * NqF + m * NqF + i];
    s_ccf[t] = r;
  }
  __syncthreads();
  // i: qc[k][j][i] = sum_m P[m][i] ccf[k][j][m]
  for (int t = threadIdx.x; t < NpC; t += blockDim.x) {
    const int i = t % NqC, j = (t / NqC) % NqC, k = t / (NqC * NqC);
    T r = 0;
    for (int m = 0; m < NqF; ++m) r += s_P[m * NqC + i] * s_ccf[k * NqC * NqF + j * NqF + m];
    const int32_t g = g2lC[e * NpC + t];
    if (g >= 0) atomicAdd(xC + g, r);
  }
}

// ---------------------------------------------------------------- transfers of fixed degrees
// Transfers between the node counts of the degree schedules (7 -> 3 -> 1 and the schedules
// that halve the dofs), one line of the element a thread and one direction after the other,
// through line-contiguous arrays in shared memory; several elements per CTA. Same sums as
// the generic kernels above (ellipticPreconCoarsenHex3D.okl:209-294,
// ellipticPreconProlongateHex3D.okl:216-301).
//
// FP64 contracts in block fixed point (fx64.cuh): with FP64 products the 7 <-> 3 transfers were
// bound by the FP64 pipe (8 operations a fine node). 20^3 elements, FP64, us before -> now:
// restriction 65.9 -> 31.5, prolongation 65.8 -> 31.0, 3 <-> 1 12.4 -> 11.4 and 10.4 -> 8.3; 32^3, FP32
// (strided shared-memory operands before): 65.2 -> 36.6, 85.1 -> 47.6, 10.5 -> 9.3, 13.0 -> 9.7.
// Now bound by the gathers: the prolongation of 20^3 in FP64 moves at least 85 MB in
// 31.0 us. All other pairs take the generic kernels.
template <int NQF, int NQC>
struct TransferLayout {
  static constexpr int NL = NQF * NQF, P = NQF | 1;        // fine lines; odd pitch of every line
  static constexpr int EPB = NL >= 128 ? 1 : 128 / NL, NT = NL * EPB;
  static constexpr int A = NQC * NQF * P, B = NL * P;      // array sizes of an element
};

// y[t] = sum_m M[t][m] x[m] by FMA, or through integers, with the table of M in shared memory
template <int NIN, int NOUT, typename T>
struct LineMatrix;

template <int NIN, int NOUT>
struct LineMatrix<NIN, NOUT, float> {
  float c[NOUT * NIN];
  __device__ __forceinline__ void fill(const float* M, int rs, int cs, int tid, int threads) {
    for (int w = tid; w < NOUT * NIN; w += threads) c[w] = M[w / NIN * rs + w % NIN * cs];
  }
  template <typename F>
  __device__ __forceinline__ void apply(const float (&x)[NIN], F&& emit) const {
#pragma unroll
    for (int t = 0; t < NOUT; ++t) {
      float r = 0.f;
#pragma unroll
      for (int m = 0; m < NIN; ++m) r += c[t * NIN + m] * x[m];
      emit(t, r);
    }
  }
};

// The end nodes (and the midpoints, where both degrees are even) are nodes of both levels:
// their rows of P are rows of the identity. Such values are passed on in FP64, and the integers
// hold the other entries only, so that every entry of a line counts in every sum and the error is
// relative to the terms of the sum (rows of P differ by 66 times at most among the others). A P
// of another kind is contracted in FP64.
template <int NIN, int NOUT>
struct LineMatrix<NIN, NOUT, double> {
  // bits of a value and of an entry (fx_hex.cuh, FxLayout): NIN products of each kind per sum
  static constexpr int FS = 7, DS = NIN >= 8 ? 6 : 7, RS = (NIN + 1) & ~1, OFF = 2088 + FS + DS - 1086;
  static constexpr bool UP = NIN < NOUT;   // prolongation
  static constexpr int LO = UP ? NIN : NOUT, HI = UP ? NOUT : NIN;
  fx_half tab[NOUT * RS];
  double c[NOUT * NIN];   // for lines left to FP64
  int ex[NOUT];
  // the coarse node at fine node i, or -1
  __host__ __device__ static constexpr int shared(int i) {
    return i == 0 ? 0 : i == HI - 1 ? LO - 1 : HI % 2 && LO % 2 && 2 * i == HI - 1 ? (LO - 1) / 2 : -1;
  }
  __device__ __forceinline__ void fill(const double* M, int rs, int cs, int tid, int threads) {
    for (int w = tid; w < NOUT * NIN; w += threads) {
      const int t = w / NIN, m = w % NIN;
      unsigned key = 0, least = 0x7fffffffu;
      bool nodal = true;
#pragma unroll
      for (int k = 0; k < NIN; ++k) {
        const double v = M[t * rs + k * cs];
        const int s = shared(UP ? t : k);
        if (s >= 0) nodal = nodal && v == (s == (UP ? k : t) ? 1.0 : 0.0);
        else least = min(least, fx_key(v));
        if (UP || s < 0) key = max(key, fx_key(v));
      }
      const int eR = max((int)(key >> 20), 960);
      c[w] = M[t * rs + m * cs];
      tab[t * RS + m] = fx_split(fx_from_double<DS + 1>(c[w], eR));
      if (m == 0) {
        const bool even = least == 0x7fffffffu || (int)(key >> 20) - (int)(least >> 20) <= 10;
        ex[t] = !nodal || !even || eR > 1086 || (key >> 20) < 960 ? -1 : eR;
      }
    }
  }
  template <typename F>
  __device__ __forceinline__ void apply(const double (&x)[NIN], F&& emit) const {
    unsigned key = 0, ends = 0;
    int lo = 0, plain = 0;
#pragma unroll
    for (int m = 0; m < NIN; ++m) {
      if (!UP && shared(m) >= 0) {
        ends = max(ends, fx_key(x[m]));
        continue;
      }
      key = max(key, fx_key(x[m]));
      lo |= __double2loint(x[m]);
    }
#pragma unroll
    for (int t = 0; t < NOUT; ++t) plain |= ex[t];
    const int eL = (int)(key >> 20);
    const bool zero = key == 0 && lo == 0;
    if ((zero || fx_ordinary(eL)) && ends < 0x7ff00000u && plain >= 0) {
      fx_half f[NIN];
#pragma unroll
      for (int m = 0; m < NIN; ++m)
        if (UP || shared(m) < 0) f[m] = fx_split(fx_from_double<FS + 1>(x[m], eL));
#pragma unroll
      for (int t = 0; t < NOUT; ++t) {
        if (UP && shared(t) >= 0) {
          emit(t, x[UP ? shared(t) : 0]);
          continue;
        }
        fx_acc A(0x40000000ll);
        fx_half d[NIN];
#pragma unroll
        for (int m = 0; m < NIN; ++m) {
          if (!UP && shared(m) >= 0) continue;
          d[m] = tab[t * RS + m];
          A.cross(f[m], d[m]);
        }
        A.fold();
#pragma unroll
        for (int m = 0; m < NIN; ++m)
          if (UP || shared(m) < 0) A.high(f[m], d[m]);
        double y = zero ? 0.0 : fx_to_double(A.v, fx_base(eL + ex[t] - OFF));
#pragma unroll
        for (int m = 0; m < NIN; ++m)
          if (!UP && shared(m) == t) y += x[m];
        emit(t, y);
      }
      return;
    }
#pragma unroll
    for (int t = 0; t < NOUT; ++t) {
      double r = 0;
#pragma unroll
      for (int m = 0; m < NIN; ++m) r += c[t * NIN + m] * x[m];
      emit(t, r);
    }
  }
};

template <int NQF, int NQC, typename T>
__global__ void __launch_bounds__(TransferLayout<NQF, NQC>::NT)
pmg_restrict_line_kernel(const int64_t E, const int32_t* __restrict__ g2lF, const T* __restrict__ wF,
                         const T* __restrict__ xF, const T* __restrict__ Pg, const int32_t* __restrict__ g2lC,
                         T* __restrict__ xC) {
  using L = TransferLayout<NQF, NQC>;
  constexpr int NL = L::NL, P = L::P, NPF = NQF * NL, NPC = NQC * NQC * NQC;
  __shared__ __align__(16) LineMatrix<NQF, NQC, T> R;   // rows of P^T
  __shared__ T s_u[L::EPB][L::A];                       // lines (kc, i) along j
  __shared__ T s_v[L::EPB][NQC * NQC * P];              // lines (kc, jc) along i
  const int tid = threadIdx.x, el = tid / NL, l = tid % NL;
  const int64_t e = (int64_t)blockIdx.x * L::EPB + el;
  const bool active = e < E;
  T x[NQF];
  {
    int32_t g[NQF];
#pragma unroll
    for (int k = 0; k < NQF; ++k) g[k] = active ? __ldg(g2lF + e * NPF + k * NL + l) : -1;
#pragma unroll
    for (int k = 0; k < NQF; ++k) x[k] = g[k] >= 0 ? wF[g[k]] * xF[g[k]] : T(0);
  }
  R.fill(Pg, 1, NQC, tid, L::NT);
  __syncthreads();
  {
    const int i = l % NQF, j = l / NQF;
    R.apply(x, [&](int kc, T u) { s_u[el][(kc * NQF + i) * P + j] = u; });
  }
  __syncthreads();
  if (l < NQC * NQF) {
    const int i = l % NQF, kc = l / NQF;
#pragma unroll
    for (int m = 0; m < NQF; ++m) x[m] = s_u[el][l * P + m];
    R.apply(x, [&](int jc, T v) { s_v[el][(kc * NQC + jc) * P + i] = v; });
  }
  __syncthreads();
  if (l < NQC * NQC && active) {
#pragma unroll
    for (int m = 0; m < NQF; ++m) x[m] = s_v[el][l * P + m];
    const int32_t* gC = g2lC + e * NPC + l * NQC;
    R.apply(x, [&](int ic, T c) {
      const int32_t g = gC[ic];
      if (g >= 0) atomicAdd(xC + g, c);
    });
  }
}

template <int NQF, int NQC, typename T>
__global__ void __launch_bounds__(TransferLayout<NQF, NQC>::NT)
pmg_prolong_line_kernel(const int64_t E, const int32_t* __restrict__ g2lC, const T* __restrict__ xC,
                        const T* __restrict__ Pg, const int32_t* __restrict__ g2lF,
                        const int32_t* __restrict__ ownerF, T* __restrict__ xF) {
  using L = TransferLayout<NQF, NQC>;
  constexpr int NL = L::NL, P = L::P, NPF = NQF * NL, NPC = NQC * NQC * NQC;
  __shared__ __align__(16) LineMatrix<NQC, NQF, T> I;
  __shared__ T s_c[L::EPB][L::B];                       // lines (kc, jc) along ic, then (i, j) along kc
  __shared__ T s_w[L::EPB][L::A];                       // lines (kc, i) along jc
  const int tid = threadIdx.x, el = tid / NL, l = tid % NL;
  const int64_t e = (int64_t)blockIdx.x * L::EPB + el;
  const bool active = e < E;
  for (int p = l; p < NPC; p += NL) {
    const int32_t g = active ? __ldg(g2lC + e * NPC + p) : -1;
    s_c[el][p / NQC * P + p % NQC] = g >= 0 ? xC[g] : T(0);
  }
  I.fill(Pg, NQC, 1, tid, L::NT);
  // this column's dofs and whether this copy owns them, in flight meanwhile
  int32_t g[NQF];
  const int32_t id0 = (int32_t)(e * NPF) + l;
#pragma unroll
  for (int k = 0; k < NQF; ++k) g[k] = active ? __ldg(g2lF + e * NPF + k * NL + l) : -1;
#pragma unroll
  for (int k = 0; k < NQF; ++k)
    if (g[k] >= 0 && __ldg(ownerF + g[k]) != id0 + k * NL) g[k] = -1;
  __syncthreads();
  T x[NQC];
  if (l < NQC * NQC) {
    const int jc = l % NQC, kc = l / NQC;
#pragma unroll
    for (int m = 0; m < NQC; ++m) x[m] = s_c[el][l * P + m];
    I.apply(x, [&](int a, T v) { s_w[el][(kc * NQF + a) * P + jc] = v; });
  }
  __syncthreads();
  if (l < NQC * NQF) {
    const int a = l % NQF, kc = l / NQF;
#pragma unroll
    for (int m = 0; m < NQC; ++m) x[m] = s_w[el][l * P + m];
    I.apply(x, [&](int b, T v) { s_c[el][(b * NQF + a) * P + kc] = v; });
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < NQC; ++m) x[m] = s_c[el][l * P + m];
  T old[NQF];
#pragma unroll
  for (int k = 0; k < NQF; ++k) old[k] = g[k] >= 0 ? xF[g[k]] : T(0);
  I.apply(x, [&](int k, T f) {
    if (g[k] >= 0) xF[g[k]] = old[k] + f;
  });
}

template <int NQF, int NQC, typename T>
static int launch_restrict(int64_t E, const int32_t* g2lF, const T* weightF, const T* xF, const T* P,
                           const int32_t* g2lC, T* xC, cudaStream_t s) {
  using L = TransferLayout<NQF, NQC>;
  pmg_restrict_line_kernel<NQF, NQC, T><<<(unsigned)((E + L::EPB - 1) / L::EPB), L::NT, 0, s>>>(E, g2lF, weightF, xF, P,
                                                                                              g2lC, xC);
  LPG_LAUNCH_CHECK("pmg_restrict_line_kernel");
  return LPG_OK;
}
template <int NQF, int NQC, typename T>
static int launch_prolong(int64_t E, const int32_t* g2lC, const T* xC, const T* P, const int32_t* g2lF,
                          const int32_t* ownerF, T* xF, cudaStream_t s) {
  using L = TransferLayout<NQF, NQC>;
  pmg_prolong_line_kernel<NQF, NQC, T><<<(unsigned)((E + L::EPB - 1) / L::EPB), L::NT, 0, s>>>(E, g2lC, xC, P, g2lF,
                                                                                             ownerF, xF);
  LPG_LAUNCH_CHECK("pmg_prolong_line_kernel");
  return LPG_OK;
}

// f(node counts per direction) for the degree pairs with kernels of their own
constexpr int kNoPair = 1;   // not a status
template <typename F>
static int for_pair(int Nf, int Nc, F&& f) {
#define LPG_PAIR(a, b) \
  if (Nf == a && Nc == b) return f(std::integral_constant<int, a + 1>{}, std::integral_constant<int, b + 1>{})
  LPG_PAIR(7, 3);
  LPG_PAIR(3, 1);
  LPG_PAIR(8, 6);
  LPG_PAIR(7, 5);
  LPG_PAIR(6, 4);
  LPG_PAIR(5, 3);
  LPG_PAIR(4, 2);
  LPG_PAIR(3, 2);
  LPG_PAIR(2, 1);
#undef LPG_PAIR
  return kNoPair;
}

template <typename T>
int pmg_coarsen(int Nf, int Nc, int64_t E, const int32_t* g2lF, const T* weightF, const T* xF,
                const T* P, const int32_t* g2lC, T* xC, int64_t NglobalC, cudaStream_t s) {
  if (Nf + 1 > kMaxNq || Nc < 1 || Nc > Nf) return set_error(LPG_ERR_UNSUPPORTED, "pmg_coarsen: bad degrees");
  LPG_CUDA_TRY(cudaMemsetAsync(xC, 0, sizeof(T) * NglobalC, s));
  if (E <= 0) return LPG_OK;
  const int rc = for_pair(Nf, Nc, [&](auto nf, auto nc) {
    return launch_restrict<decltype(nf)::value, decltype(nc)::value, T>(E, g2lF, weightF, xF, P, g2lC, xC, s);
  });
  if (rc != kNoPair) return rc;
  pmg_coarsen_kernel<T><<<(unsigned)E, 256, 0, s>>>(Nf + 1, Nc + 1, g2lF, weightF, xF, P, g2lC, xC);
  LPG_LAUNCH_CHECK("pmg_coarsen_kernel");
  return LPG_OK;
}

template <typename T>
__global__ void __launch_bounds__(256)
pmg_prolong_kernel(const int NqF, const int NqC, const int32_t* __restrict__ g2lC,
                   const T* __restrict__ xC, const T* __restrict__ Pg, const int32_t* __restrict__ g2lF,
                   const int32_t* __restrict__ ownerF, T* __restrict__ xF) {
  __shared__ T s_ccc[kMaxNq * kMaxNq * kMaxNq];
  __shared__ T s_ccf[kMaxNq * kMaxNq * kMaxNq];
  __shared__ T s_cff[kMaxNq * kMaxNq * kMaxNq];
  __shared__ T s_P[kMaxNq * kMaxNq];
  const int64_t e = blockIdx.x;
  const int NpF = NqF * NqF * NqF, NpC = NqC * NqC * NqC;
  for (int t = threadIdx.x; t < NqF * NqC; t += blockDim.x) s_P[t] = Pg[t];
  for (int t = threadIdx.x; t < NpC; t += blockDim.x) {
    const int32_t g = g2lC[e * NpC + t];
    s_ccc[t] = (g >= 0) ? xC[g] : T(0);
  }
  __syncthreads();
  // i: ccf[k][j][i] = sum_m P[i][m] ccc[k][j][m]
  for (int t = threadIdx.x; t < NqC * NqC * NqF; t += blockDim.x) {
    const int i = t % NqF, j = (t / NqF) % NqC, k = t / (NqF * NqC);
    T r = 0;
    for (int m = 0; m < NqC; ++m) r += s_P[i * NqC + m] * s_ccc[k * NqC * NqC + j * NqC + m];
    s_ccf[t] = r;
  }
  __syncthreads();
  // j: cff[k][j][i] = sum_m P[j][m] ccf[k][m][i]
  for (int t = threadIdx.x; t < NqC * NqF * NqF; t += blockDim.x) {
    const int i = t % NqF, j = (t / NqF) % NqF, k = t / (NqF * NqF);
    T r = 0;
    for (int m = 0; m < NqC; ++m) r += s_P[j * NqC + m] * s_ccf[k * NqC * NqF + m * NqF + i];
    s_cff[t] = r;
  }
  __syncthreads();
  // k: f[k][j][i] = sum_m P[k][m] cff[m][j][i]; the owning copy adds it to xF
  for (int t = threadIdx.x; t < NpF; t += blockDim.x) {
    const int i = t % NqF, j = (t / NqF) % NqF, k = t / (NqF * NqF);
    T r = 0;
    for (int m = 0; m < NqC; ++m) r += s_P[k * NqC + m] * s_cff[m * NqF * NqF + j * NqF + i];
    const int64_t id = e * NpF + t;
    const int32_t g = g2lF[id];
    if (g >= 0 && ownerF[g] == (int32_t)id) xF[g] += r;
  }
}

template <typename T>
int pmg_prolongate_map(int Nf, int Nc, int64_t E, const int32_t* g2lC, const T* xC, const T* P,
                       const int32_t* g2lF, const int32_t* ownerF, T* xF, cudaStream_t s) {
  if (Nf + 1 > kMaxNq || Nc < 1 || Nc > Nf) return set_error(LPG_ERR_UNSUPPORTED, "pmg_prolongate: bad degrees");
  if (E <= 0) return LPG_OK;
  const int rc = for_pair(Nf, Nc, [&](auto nf, auto nc) {
    return launch_prolong<decltype(nf)::value, decltype(nc)::value, T>(E, g2lC, xC, P, g2lF, ownerF, xF, s);
  });
  if (rc != kNoPair) return rc;
  pmg_prolong_kernel<T><<<(unsigned)E, 256, 0, s>>>(Nf + 1, Nc + 1, g2lC, xC, P, g2lF, ownerF, xF);
  LPG_LAUNCH_CHECK("pmg_prolong_kernel");
  return LPG_OK;
}

template int pmg_coarsen<double>(int, int, int64_t, const int32_t*, const double*, const double*, const double*,
                                 const int32_t*, double*, int64_t, cudaStream_t);
template int pmg_coarsen<float>(int, int, int64_t, const int32_t*, const float*, const float*, const float*,
                                const int32_t*, float*, int64_t, cudaStream_t);
template int pmg_prolongate_map<double>(int, int, int64_t, const int32_t*, const double*, const double*,
                                        const int32_t*, const int32_t*, double*, cudaStream_t);
template int pmg_prolongate_map<float>(int, int, int64_t, const int32_t*, const float*, const float*,
                                       const int32_t*, const int32_t*, float*, cudaStream_t);

}  // namespace lpg
