// (e) SIMP strain-energy sensitivities and the optimality-criteria update.
//
// The reference has neither (its modulus is linear in density,
// src/Solvers/GPUSolver.jl:254, and its update is a stress-ratio rule,
// src/Optimization/TopOpt.jl:211-482).  These kernels restate the published
// SIMP / OC method (Bendsoe & Sigmund; the OC update of Andreassen et al.
// 2011, "Efficient topology optimization in MATLAB using 88 lines of code"):
//   E_e  = Emin + rho_e^p (E0 - Emin)
//   ce_e = u_e^T K0 u_e           (K0 for E = 1)
//   c    = sum_e E_e ce_e,  dc_e = -p rho_e^(p-1) (E0 - Emin) ce_e
//   x_new = clamp(x * sqrt(-dc / (lambda dv)), max(0, x-move), min(1, x+move))
// with lambda found by bisection so that mean(x_new) = volfrac.  The element
// energy uses the same Hadamard-basis blocks as the operator: ce = u_hat^T B u_hat.
#include <algorithm>
#include <cmath>

#include "hexa_common.cuh"
#include "hexa_kernels.h"

namespace hexa {

static inline int topo_blocks(long long n) {
  long long b = (n + 255) / 256;
  if (b < 1) b = 1;
  if (b > 152 * 8) b = 152 * 8;
  return (int)b;
}

// rho^n for n >= 0: products with the rounding errors carried along (each by
// one FMA), rounded once at the end, so never further off than pow; 1 to 4 FP64
// instructions per factor against about 100 for pow, on a part that issues 2 per
// clock and SM.
template <int N>
__device__ __forceinline__ double powi(double r) {
  if (N == 0) return 1.0;
  double h = r, l = 0.0;
#pragma unroll
  for (int k = 1; k < N; ++k) {
    const double q = h * r;
    l = (k == N - 1 && N == 2) ? 0.0 : fma(l, r, fma(h, r, -q));
    h = q;
  }
  // a finite h by its bits: no FP64 comparison
  return (N <= 2 || (__double2hiint(h) & 0x7ff00000) == 0x7ff00000) ? h : h + l;
}
// N < 0: any exponent.
template <int N>
__device__ __forceinline__ double simp_pow(double r, double p) { return N < 0 ? pow(r, p) : powi<(N < 0 ? 0 : N)>(r); }
// The penalty when it is a whole number up to 6 (the published method's 3 and
// its continuation), else -1.
static int whole_penal(double p) { return (p >= 1.0 && p <= 6.0 && p == (double)(int)p) ? (int)p : -1; }

// 256x128x128, penalty 3: 74 us (FP64 issue, 9 instructions an element), 693 us
// through pow.
template <int N>
__global__ void simp_factors_kernel(const double* __restrict__ rho, double Emin, double E0, double penal,
                                    double* __restrict__ fac, long long n) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
    fac[e] = Emin + simp_pow<N>(rho[e], penal) * (E0 - Emin);
}
void launch_simp_factors(const double* rho, double Emin, double E0, double penal, double* fac, long long n,
                         cudaStream_t st) {
  const int b = topo_blocks(n);
  switch (whole_penal(penal)) {
#define HEXA_CASE(N) \
  case N: simp_factors_kernel<N><<<b, 256, 0, st>>>(rho, Emin, E0, penal, fac, n); break;
    HEXA_CASE(1) HEXA_CASE(2) HEXA_CASE(3) HEXA_CASE(4) HEXA_CASE(5) HEXA_CASE(6)
#undef HEXA_CASE
    default: simp_factors_kernel<-1><<<b, 256, 0, st>>>(rho, Emin, E0, penal, fac, n);
  }
}

// The element energy u_e^T K0 u_e as a sum over the modal classes (see ModalK)
// of symmetric 3x3 forms: class q couples component c of mode q ^ (1 << c).
// Off-diagonal entries doubled; a class of two bits splits into one component
// and a shear pair, whose 2x2 form is a square (a rotation has no energy).
struct EnergyK {
  double full[2][6];   // q = 0, 7: a00, 2a01, 2a02, a11, 2a12, a22
  double pair[3][3];   // q = 1, 2, 4 (bit d), without component d: a00, 2a01, a11
  double one[3];       // q = 7 ^ (1 << d): component d alone
  double shear[3][2];  // and the other two: (s0 u + s1 v)^2
};
static EnergyK energy_blocks(const ModalK<double>& K) {
  EnergyK E;
  for (int t = 0; t < 2; ++t) {
    const double(&B)[3][3] = K.B[t ? 7 : 0];
    E.full[t][0] = B[0][0], E.full[t][1] = B[0][1] + B[1][0], E.full[t][2] = B[0][2] + B[2][0];
    E.full[t][3] = B[1][1], E.full[t][4] = B[1][2] + B[2][1], E.full[t][5] = B[2][2];
  }
  for (int d = 0; d < 3; ++d) {
    const int u = d == 0 ? 1 : 0, v = d == 2 ? 1 : 2;
    const double(&P)[3][3] = K.B[1 << d];
    E.pair[d][0] = P[u][u], E.pair[d][1] = P[u][v] + P[v][u], E.pair[d][2] = P[v][v];
    const double(&S)[3][3] = K.B[7 ^ (1 << d)];
    E.one[d] = S[d][d];
    E.shear[d][0] = std::sqrt(S[u][u]);
    E.shear[d][1] = (S[u][v] < 0 ? -1.0 : 1.0) * std::sqrt(S[v][v]);
  }
  return E;
}

// A warp owns 32 element columns in x and marches through kz layers: the
// xy-butterflies of a node layer serve the elements on both sides of it, and
// the rigid translations (mode 0) are never formed.  About 100 FP64 instructions
// an element, against 215 with the three transforms, the unsymmetric products
// and pow per element; FP64 issue bound (85 % of
// the pipe).  256x128x128: 825 us, 1851 before.
// kz: kSensZ where that gives every SM eight items (256x128x128: 846 us a call,
// 856 in items of 6 layers), else fewer by the operator's chunk rule (starting
// an item costs a quarter of a layer): 48x24x24 57 us in items of 8 layers, 35 in
// items of two; 96x48x48 91 and 73 to 79 in items of 2 to 6.
constexpr int kSensZ = 16;
template <int N>
__global__ void __launch_bounds__(128) sens_kernel(Grid g, const __grid_constant__ EnergyK K,
                                                   const double* __restrict__ rho, const double* __restrict__ u,
                                                   double Emin, double E0, double penal, double* __restrict__ dc,
                                                   int kz, RedArgs red) {
  const int nbx = (g.nx + 31) / 32, nby = (g.ny + 3) / 4, nzc = (g.nz + kz - 1) / kz;
  const long long items = (long long)nbx * nby * nzc;
  const double dE = E0 - Emin, scale = -penal * dE;
  double acc[1] = {0.0};
  for (long long item = blockIdx.x; item < items; item += gridDim.x) {
    const int i = (int)(item % nbx) * 32 + threadIdx.x, j = (int)(item / nbx % nby) * 4 + threadIdx.y;
    const int k0 = (int)(item / nbx / nby) * kz, k1 = min(k0 + kz, g.nz);
    if (i >= g.nx || j >= g.ny) continue;
    const long long plane = 3LL * g.NX * g.NY;
    const double* col = u + 3 * ((long long)i + (long long)g.NX * j);
    double v[4][3];  // the next node layer's corners (dx + 2dy)
    auto load = [&](int k) {
      const double* p = col + plane * k;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        v[0][c] = __ldg(p + c), v[1][c] = __ldg(p + 3 + c);
        v[2][c] = __ldg(p + 3 * g.NX + c), v[3][c] = __ldg(p + 3 * g.NX + 3 + c);
      }
    };
    auto forward = [&](double (&m)[4][3]) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double a0 = v[0][c] + v[1][c], a1 = v[1][c] - v[0][c], b0 = v[2][c] + v[3][c], b1 = v[3][c] - v[2][c];
        m[0][c] = a0 + b0, m[1][c] = a1 + b1, m[2][c] = b0 - a0, m[3][c] = b1 - a1;
      }
    };
    double L[4][3];
    load(k0);
    forward(L);
    load(k0 + 1);
    const long long e0 = (long long)i + (long long)g.nx * j, ep = (long long)g.nx * g.ny;
    double rn = rho[e0 + ep * k0];
    for (int k = k0; k < k1; ++k) {
      double U[4][3];
      forward(U);
      const double r = rn;
      if (k + 1 < k1) {
        load(k + 2);
        rn = rho[e0 + ep * (k + 1)];
      }
      double h[8][3];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (m > 0) h[m][c] = L[m][c] + U[m][c];
          h[m + 4][c] = U[m][c] - L[m][c];
          L[m][c] = U[m][c];
        }
      double ce = 0.0;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int q = t ? 7 : 0;
        const double a = h[q ^ 1][0], b = h[q ^ 2][1], c = h[q ^ 4][2];
        ce = fma(a, fma(K.full[t][0], a, fma(K.full[t][1], b, K.full[t][2] * c)), ce);
        ce = fma(b, fma(K.full[t][3], b, K.full[t][4] * c), ce);
        ce = fma(c, K.full[t][5] * c, ce);
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int cu = d == 0 ? 1 : 0, cv = d == 2 ? 1 : 2;
        const int q = 1 << d, s = 7 ^ q;
        const double a = h[q ^ (1 << cu)][cu], b = h[q ^ (1 << cv)][cv];
        ce = fma(a, fma(K.pair[d][0], a, K.pair[d][1] * b), ce);
        ce = fma(b, K.pair[d][2] * b, ce);
        const double o = h[s ^ q][d], x = h[s ^ (1 << cu)][cu], y = h[s ^ (1 << cv)][cv];
        ce = fma(o, K.one[d] * o, ce);
        const double w = fma(K.shear[d][0], x, K.shear[d][1] * y);
        ce = fma(w, w, ce);
      }
      const double rp1 = simp_pow<(N < 0 ? -1 : N - 1)>(r, penal - 1.0);
      dc[e0 + ep * k] = scale * rp1 * ce;
      acc[0] = fma(fma(rp1 * r, dE, Emin), ce, acc[0]);
    }
  }
  block_reduce_finalize<1>(red, acc);
}
void launch_sensitivities(const Grid& g, const ModalK<double>& K, const double* rho, const double* u, double Emin,
                          double E0, double penal, double* dc, const RedArgs& red, cudaStream_t st) {
  const long long tiles = (long long)((g.nx + 31) / 32) * ((g.ny + 3) / 4);
  const bool many = tiles * ((g.nz + kSensZ - 1) / kSensZ) >= 152 * 8;
  const int kz = many ? kSensZ : std::min(kSensZ, op_chunk_layers(tiles, g.nz, 152, 0.25));
  const long long items = tiles * ((g.nz + kz - 1) / kz);
  const int b = (int)std::min<long long>(items, 152 * 8);
  const EnergyK E = energy_blocks(K);
  switch (whole_penal(penal)) {
#define HEXA_CASE(N) \
  case N: sens_kernel<N><<<b, dim3(32, 4), 0, st>>>(g, E, rho, u, Emin, E0, penal, dc, kz, red); break;
    HEXA_CASE(1) HEXA_CASE(2) HEXA_CASE(3) HEXA_CASE(4) HEXA_CASE(5) HEXA_CASE(6)
#undef HEXA_CASE
    default: sens_kernel<-1><<<b, dim3(32, 4), 0, st>>>(g, E, rho, u, Emin, E0, penal, dc, kz, red);
  }
}

__device__ __forceinline__ double oc_new(double x, double dc, double dv, double lam, double move) {
  const double be = x * sqrt(-dc / dv / lam);
  return fmax(0.0, fmax(x - move, fmin(1.0, fmin(x + move, be))));
}

// What the volume of the update needs per element.  The update of one element
// is clamp(x sqrt(-dc / dv) / sqrt(lambda), lo, hi): t = x sqrt(-dc / dv) and
// the limits do not depend on lambda, so the division and the square root
// (about 12 FP64 instructions each on a part that issues 2 FP64 instructions
// per clock and SM) are done once per element and not once per element and
// multiplier.  lo = max(0, x - move), hi = min(1, x + move); a t that is NaN
// (dc > 0) selects hi, as fmin / fmax do in oc_new.
struct OcElem {
  double t, lo, hi;
};
__device__ __forceinline__ OcElem oc_elem(double x, double dc, double dv, double move) {
  OcElem e;
  e.t = x * sqrt(-dc / dv);
  e.t = e.t <= 0.0 ? 0.0 : e.t;  // -0 and negative products give lo, a NaN stays
  e.lo = fmax(0.0, x - move);
  e.hi = fmax(0.0, fmin(1.0, x + move));
  return e;
}
// max(lo, min(hi, be)) on the bit patterns: every finite value here is >= 0,
// where doubles order as their bits, and a NaN of either sign lies above hi.
// Integer comparisons leave the FP64 pipe to the product and the sum.
__device__ __forceinline__ double oc_clamp(double be, double lo, double hi, bool* inside) {
  const unsigned long long b = __double_as_longlong(be), l = __double_as_longlong(lo), h = __double_as_longlong(hi);
  *inside = b < h && b > l;
  const double v = b < h ? be : hi;
  return b < l || h < l ? lo : v;
}

// Block sums of NS values per thread in a fixed order: the block's totals go
// to part[block * NS + q]; the last block (by ticket) returns true in all its
// threads with the totals over the blocks, added in block order, in tot.
template <int NS, typename A>
__device__ __forceinline__ bool oc_block_totals(A (&acc)[NS], double* __restrict__ part, unsigned* ticket,
                                                double* tot) {
  __shared__ A sw[8][NS];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    A v = acc[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == (q & 31)) sw[wid][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < NS) {
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += (double)sw[w][threadIdx.x];
    part[(long long)blockIdx.x * NS + threadIdx.x] = s;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  // the blocks in 256 / NS strided runs per value, then the runs in order
  constexpr int RUNS = 256 / NS;
  __shared__ double sr[NS][RUNS];
  const int q = threadIdx.x % NS, run = threadIdx.x / NS;
  if (run < RUNS) {
    double s = 0.0;
    for (unsigned b = run; b < gridDim.x; b += RUNS) s += ((volatile double*)part)[(long long)b * NS + q];
    sr[q][run] = s;
  }
  __syncthreads();
  if (threadIdx.x < NS) {
    double s = 0.0;
    for (int r = 0; r < RUNS; ++r) s += sr[threadIdx.x][r];
    tot[threadIdx.x] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) *ticket = 0u;
  return true;
}

// Per-element arrays of the search (24 B written per element) and the bracket
// of its root: the volume at kOcCand values of s = 1/sqrt(lambda), each twice
// the one before from lambda = 1e9 down, in FP32 (the FP64 pipe is 64 times
// narrower; the bracket is widened by a candidate on either side, so FP32's
// 1e-6 does not decide anything).  With the Newton steps below the update of
// 256x128x128 elements takes 0.69 ms; 16 passes that each evaluated 31
// multipliers of the bisection in FP64 (5.8 ms a pass, two divisions and a
// square root per multiplier) took 93.7 ms, with bitwise the same result.
constexpr int kOcCand = 32;
__global__ void __launch_bounds__(256) oc_prepare_kernel(const double* __restrict__ x, const double* __restrict__ dc,
                                                         const double* __restrict__ dv, long long n, double move,
                                                         double target, double* __restrict__ t,
                                                         double* __restrict__ lo, double* __restrict__ hi,
                                                         double* __restrict__ part, OcState* __restrict__ st) {
  const float s0 = 3.1622776e-5f;  // 1 / sqrt(1e9)
  float acc[kOcCand];
#pragma unroll
  for (int q = 0; q < kOcCand; ++q) acc[q] = 0.f;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const OcElem el = oc_elem(x[e], dc[e], dv[e], move);
    t[e] = el.t;
    lo[e] = el.lo;
    hi[e] = el.hi;
    const float l = (float)el.lo, h = (float)el.hi;
    float be = (float)el.t * s0;
#pragma unroll
    for (int q = 0; q < kOcCand; ++q) {
      acc[q] += fmaxf(l, fminf(h, be));  // NaN: h
      be += be;
    }
  }
  __shared__ double tot[kOcCand];
  if (!oc_block_totals<kOcCand, float>(acc, part, &st->ticket, tot) || threadIdx.x != 0) return;
  int k = 0;
  while (k < kOcCand && !(tot[k] > target)) ++k;
  const double s00 = 1.0 / sqrt(1e9);
  auto at = [&](int q) { return q < 0 ? 0.0 : s00 * exp2((double)q); };
  st->state = 0;
  // the volume at the upper multiplier exceeds the target, by more than FP32 sums
  // are off: so it does at every multiplier of the bisection, which ends there
  if (tot[0] > 1.001 * target) {
    st->root = 1e-150;
    st->state = 1;
    return;
  }
  if (k == kOcCand) {  // no multiplier of the range reaches the target (or NaN)
    st->state = 2;
    return;
  }
  st->s_lo = at(k - 2);
  st->s_hi = at(k + 1);
  const double v0 = k > 0 ? tot[k - 1] : 0.0;
  const double a = at(k - 1), b = at(k);
  double s = a + (target - v0) / (tot[k] - v0) * (b - a);
  if (!(s > st->s_lo && s < st->s_hi)) s = 0.5 * (st->s_lo + st->s_hi);
  st->s = s;
}

// One step of the search for V(s) = target: V and its slope at s in FP64, then
// a Newton step kept inside the bracket (V is piecewise linear and does not
// fall with s).  Done when the step is below 1e-10 s: the root is then
// s + step to the rounding of V itself, since between s and the root the
// elements change their branch by less than 1e-10 of their value.
__global__ void __launch_bounds__(256) oc_step_kernel(const double* __restrict__ t, const double* __restrict__ lo,
                                                      const double* __restrict__ hi, long long n, double target,
                                                      double* __restrict__ part, OcState* __restrict__ st) {
  if (*((volatile int*)&st->state) != 0) return;
  const double s = *((volatile double*)&st->s);
  double acc[2] = {0.0, 0.0};
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const double te = t[e];
    bool inside;
    acc[0] += oc_clamp(te * s, lo[e], hi[e], &inside);
    if (inside) acc[1] += te;
  }
  __shared__ double tot[2];
  if (!oc_block_totals<2, double>(acc, part, &st->ticket, tot) || threadIdx.x != 0) return;
  const double V = tot[0], slope = tot[1];
  if (V > target) st->s_hi = s;
  else st->s_lo = s;
  const double sn = s + (target - V) / slope;
  if (fabs(sn - s) <= 1e-10 * s) {
    st->root = sn;
    st->state = 1;
  } else {
    st->s = (sn > st->s_lo && sn < st->s_hi) ? sn : 0.5 * (st->s_lo + st->s_hi);
  }
}

void launch_oc_prepare(const double* x, const double* dc, const double* dv, long long n, double move, double target,
                       double* t, double* lo, double* hi, double* part, OcState* st, int nblocks, cudaStream_t s) {
  oc_prepare_kernel<<<nblocks, 256, 0, s>>>(x, dc, dv, n, move, target, t, lo, hi, part, st);
}
void launch_oc_step(const double* t, const double* lo, const double* hi, long long n, double target, double* part,
                    OcState* st, int nblocks, cudaStream_t s) {
  oc_step_kernel<<<nblocks, 256, 0, s>>>(t, lo, hi, n, target, part, st);
}

// Sum over elements of x_new(lambda_q) for nlam candidate multipliers; block
// partials [block][32] are summed in block order by the caller.  Only for
// volumes without a root in the search's range (a target that no multiplier
// reaches, NaN input).
__global__ void oc_volumes_kernel(const double* __restrict__ t, const double* __restrict__ lo,
                                  const double* __restrict__ hi, long long n, const double* __restrict__ lam, int nlam,
                                  double* __restrict__ partials) {
  __shared__ double sl[32];
  __shared__ double sw[8][32];
  if (threadIdx.x < nlam) sl[threadIdx.x] = 1.0 / sqrt(lam[threadIdx.x]);
  __syncthreads();
  double acc[32];
#pragma unroll
  for (int q = 0; q < 32; ++q) acc[q] = 0.0;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const double te = t[e], l = lo[e], h = hi[e];
    bool inside;
#pragma unroll
    for (int q = 0; q < 32; ++q)
      if (q < nlam) acc[q] += oc_clamp(te * sl[q], l, h, &inside);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 32; ++q) {
    double v = warp_sum(acc[q]);
    if (lane == q) sw[wid][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < nlam) {
    double v = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += sw[w][threadIdx.x];
    partials[(long long)blockIdx.x * 32 + threadIdx.x] = v;
  }
}
void launch_oc_volumes(const double* t, const double* lo, const double* hi, long long n, const double* lam, int nlam,
                       double* partials, int nblocks, cudaStream_t st) {
  oc_volumes_kernel<<<nblocks, 256, 0, st>>>(t, lo, hi, n, lam, nlam, partials);
}

__global__ void oc_apply_kernel(const double* __restrict__ x, const double* __restrict__ dc, const double* __restrict__ dv,
                                long long n, double lam, double move, double* __restrict__ xout) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
    xout[e] = oc_new(x[e], dc[e], dv[e], lam, move);
}
void launch_oc_apply(const double* x, const double* dc, const double* dv, long long n, double lam, double move,
                     double* xout, cudaStream_t st) {
  oc_apply_kernel<<<topo_blocks(n), 256, 0, st>>>(x, dc, dv, n, lam, move, xout);
}

}  // namespace hexa
