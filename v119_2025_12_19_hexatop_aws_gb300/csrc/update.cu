// Density update between SIMP solves: the stress-ratio proposal, the update
// statistics, the culling of the weakest low-density elements and the hard
// projection of TopologyOptimization.update_density!
// (src/Optimization/TopOpt.jl:211-482), on the device with no host round trip
// between the passes.
//
//  propose   proposed_e = original_e (protected) or
//            max((l1_e / l1_allowable) / E, min_density)      TopOpt.jl:254-263
//  update    per unprotected element: raw = max(filtered, min_density),
//            |min(raw, max_density) - old| summed, raw > min_density counted;
//            the clamp to max_density, the active count (protected elements by
//            their original density) and the cull candidates
//            (min_density < rho < threshold)                   TopOpt.jl:369-447
//  select    the k = floor(active * max_culling_ratio) smallest candidates,
//            ties by element index (Julia's stable sort! of the candidate
//            list), by a radix select over the 64-bit key
//            (float bits of rho << 32 | index): 11-bit digits from the top,
//            each a histogram whose last block picks the digit; the first comes
//            with the update pass, and a short list of ties ends it early
//                                                              TopOpt.jl:449-460
//  finish    culled -> min_density, the "hard" projection rho > min_density
//            -> 1, protected elements back to their original density
//                                                              TopOpt.jl:462-481
//
// Every float operation the reference rounds is one rounded operation here
// (__fdiv_rn; min/max are exact), so densities, counts and the culled set are
// bit-identical to the reference's on the same filtered field; the mean change
// is a sum whose order the reference itself leaves to its thread count.
#include <cuda_runtime.h>

#include <algorithm>

#include "hexa_common.cuh"
#include "hexa_kernels.h"

namespace hexa {

namespace {

constexpr int kUpdBlocks = 152 * 4;
constexpr int kUpdThreads = 256;
constexpr int kDigitBits = 11;
constexpr int kBins = 1 << kDigitBits;

__device__ __forceinline__ bool is_candidate(float d, float min_d, float thr) { return d > min_d && d < thr; }

__device__ __forceinline__ unsigned long long cull_key(float d, long long e) {
  return ((unsigned long long)__float_as_uint(d) << 32) | (unsigned long long)e;
}

__device__ __forceinline__ float proposal(float l1, float allow, float E, float min_d) {
  return fmaxf(__fdiv_rn(__fdiv_rn(l1, allow), E), min_d);
}

__global__ void propose_kernel(long long n, const float* __restrict__ l1, const uint8_t* __restrict__ prot,
                               const float* __restrict__ orig, float allow, float E, float min_d,
                               float* __restrict__ prop, UpdateState* __restrict__ s) {
  bool nan = false;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const float v = l1[e];
    nan |= (v != v);
    prop[e] = (prot && prot[e]) ? orig[e] : proposal(v, allow, E, min_d);
  }
  if (__any_sync(0xffffffffu, nan) && (threadIdx.x & 31) == 0) atomicOr(&s->nan_stress, 1);
}

__device__ __forceinline__ void digit_span(int pass, int* shift, int* width) {
  // passes from the top: bits [53,64), [42,53), [31,42), [20,31), [9,20), [0,9)
  const int top = 64 - kDigitBits * pass;
  *width = top >= kDigitBits ? kDigitBits : top;
  *shift = top - *width;
}

// True in every thread of the launch's last block (which resets the ticket).
__device__ __forceinline__ bool last_block(unsigned* ticket) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    if (last) *ticket = 0u;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// The last block of a digit pass: the bin that holds the remaining-th smallest
// key, by a scan over the bins (8 per thread); clears them for the next pass.
// When the float bits are settled (pass 2) and every key left in the bin is
// culled, the rest of the key is filled with ones and the selection is done.
__device__ __forceinline__ void pick_digit(int pass, UpdateState* s, unsigned long long* hist) {
  constexpr int PER = kBins / kUpdThreads;
  __shared__ unsigned long long wsum[kUpdThreads / 32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  unsigned long long c[PER], incl = 0;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    c[q] = ((volatile unsigned long long*)hist)[PER * t + q];
    incl += c[q];
  }
  const unsigned long long own = incl;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  unsigned long long excl = incl - own;
  for (int q = 0; q < w; ++q) excl += wsum[q];
  const unsigned long long rem = *((volatile unsigned long long*)&s->remaining);
  const bool search = *((volatile int*)&s->mode) == 2;
  int shift, width;
  digit_span(pass, &shift, &width);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    if (search && excl < rem && rem <= excl + c[q]) {
      s->prefix |= (unsigned long long)(PER * t + q) << shift;
      s->remaining = rem - excl;
      s->ties = c[q];
      if (pass == 2 && rem - excl == c[q]) {
        s->prefix |= (1ull << shift) - 1ull;
        s->done = 1;
      }
    }
    excl += c[q];
    hist[PER * t + q] = 0ull;
  }
}

// The update pass over src (the filtered field), or with FUSED over the
// proposal formed on the way from src = the stress norms (no filter in
// between: the proposal is neither written nor read, and the host does not wait
// for its NaN flag).  Per-block partial sums land in part[4 * blockIdx.x + ...]
// (change as FP64, three counts as unsigned 64-bit in the same double slots);
// the histogram of the selection's first digit is taken along.  The last block
// sums the partials in a fixed order, fixes the culling mode (0 none, 1 every
// candidate, 2 the k smallest keys) and picks the first digit: a thread summing
// 608 partials by itself had taken 101 us.
template <bool FUSED>
__global__ void __launch_bounds__(kUpdThreads) update_kernel(long long n, const float* __restrict__ old,
                                                             const float* __restrict__ src,
                                                             const uint8_t* __restrict__ prot,
                                                             const float* __restrict__ orig, float allow, float E,
                                                             float min_d, float max_d, float thr, float ratio,
                                                             float* __restrict__ out, double* __restrict__ part,
                                                             unsigned long long* __restrict__ hist,
                                                             UpdateState* __restrict__ s) {
  __shared__ unsigned int h[kBins];
  for (int i = threadIdx.x; i < kBins; i += kUpdThreads) h[i] = 0u;
  __syncthreads();
  double change = 0.0;
  unsigned long long act1 = 0, act2 = 0, cand = 0;
  bool nan = false;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const float f = src[e];
    nan |= (f != f);
    if (prot && prot[e]) {
      act2 += orig[e] > min_d;
      out[e] = old[e];  // restored to the original density at the end
      continue;
    }
    const float raw = FUSED ? proposal(f, allow, E, min_d) : fmaxf(f, min_d);
    change += (double)fabsf(fminf(raw, max_d) - old[e]);
    act1 += raw > min_d;
    const float d = fminf(raw, max_d);
    const bool live = d > min_d;
    act2 += live;
    if (live && d < thr) {
      ++cand;
      atomicAdd(&h[__float_as_uint(d) >> 21], 1u);  // key bits [53, 64)
    }
    out[e] = d;
  }
  if (__any_sync(0xffffffffu, nan) && (threadIdx.x & 31) == 0) atomicOr(FUSED ? &s->nan_stress : &s->nan_filtered, 1);
  __shared__ double sc[kUpdThreads / 32];
  __shared__ unsigned long long sa[3][kUpdThreads / 32];
  auto block_sums = [&]() {
    for (int o = 16; o > 0; o >>= 1) {
      change += __shfl_xor_sync(0xffffffffu, change, o);
      act1 += __shfl_xor_sync(0xffffffffu, act1, o);
      act2 += __shfl_xor_sync(0xffffffffu, act2, o);
      cand += __shfl_xor_sync(0xffffffffu, cand, o);
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) sc[w] = change, sa[0][w] = act1, sa[1][w] = act2, sa[2][w] = cand;
    __syncthreads();
    if (threadIdx.x == 0) {
      change = 0.0, act1 = act2 = cand = 0;
      for (int i = 0; i < kUpdThreads / 32; ++i) change += sc[i], act1 += sa[0][i], act2 += sa[1][i], cand += sa[2][i];
    }
  };
  block_sums();
  unsigned long long* pu = reinterpret_cast<unsigned long long*>(part);
  if (threadIdx.x == 0) {
    part[4 * blockIdx.x] = change;
    pu[4 * blockIdx.x + 1] = act1;
    pu[4 * blockIdx.x + 2] = act2;
    pu[4 * blockIdx.x + 3] = cand;
  }
  for (int i = threadIdx.x; i < kBins; i += kUpdThreads)
    if (h[i]) atomicAdd(&hist[i], (unsigned long long)h[i]);
  if (!last_block(&s->ticket)) return;
  change = 0.0, act1 = act2 = cand = 0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += kUpdThreads) {
    change += ((volatile double*)part)[4 * i];
    act1 += ((volatile unsigned long long*)pu)[4 * i + 1];
    act2 += ((volatile unsigned long long*)pu)[4 * i + 2];
    cand += ((volatile unsigned long long*)pu)[4 * i + 3];
  }
  __syncthreads();
  block_sums();
  if (threadIdx.x == 0) {
    s->change = change;
    s->active_updated = act1;
    s->active = act2;
    s->candidates = cand;
    // Int * Float32 is a Float32 product in Julia, floored to Int
    const unsigned long long allowed = (unsigned long long)floorf(__fmul_rn(__ull2float_rn(act2), ratio));
    s->allowed = allowed;
    s->mode = (cand <= allowed) ? 1 : (allowed > 0 ? 2 : 0);
    s->culled = (cand <= allowed) ? cand : allowed;
    s->prefix = 0ull;
    s->remaining = allowed;
    s->done = 0;
    s->ntie = 0u;
    s->mean_change = act1 > 0 ? __fdiv_rn((float)change, __ull2float_rn(act1)) : 0.0f;
    __threadfence();
  }
  __syncthreads();
  pick_digit(0, s, hist);
}

// One digit of the selection (pass >= 1): a histogram over the candidates that
// share the digits above, the pick in the last block.  Pass 3 starts on the
// element index; where at most kTies candidates share the float value that the
// cut falls on (a handful, unless the field has plateaus) it gathers their
// indices instead and settles the cut by rank, and the later passes return.
constexpr int kTies = 1024;
__global__ void __launch_bounds__(kUpdThreads) select_kernel(long long n, const float* __restrict__ d,
                                                             const uint8_t* __restrict__ prot, float min_d, float thr,
                                                             int pass, UpdateState* __restrict__ s,
                                                             unsigned long long* __restrict__ hist,
                                                             unsigned* __restrict__ tie) {
  if (s->mode != 2 || s->done) return;
  __shared__ unsigned int h[kBins];
  for (int i = threadIdx.x; i < kBins; i += kUpdThreads) h[i] = 0u;
  __syncthreads();
  int shift, width;
  digit_span(pass, &shift, &width);
  const int above = shift + width;  // bits at and above this position are fixed by the prefix
  const unsigned long long prefix = s->prefix;
  const bool gather = pass == 3 && s->ties <= kTies;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const float v = d[e];
    if (!is_candidate(v, min_d, thr)) continue;
    const unsigned long long key = cull_key(v, e);
    if ((key >> above) != (prefix >> above)) continue;
    if (prot && prot[e]) continue;
    if (gather) tie[atomicAdd(&s->ntie, 1u)] = (unsigned)e;
    else atomicAdd(&h[(key >> shift) & ((1u << width) - 1u)], 1u);
  }
  __syncthreads();
  if (!gather)
    for (int i = threadIdx.x; i < kBins; i += kUpdThreads)
      if (h[i]) atomicAdd(&hist[i], (unsigned long long)h[i]);
  if (!last_block(&s->ticket)) return;
  if (!gather) {
    pick_digit(pass, s, hist);
    return;
  }
  const unsigned m = (unsigned)s->ties;
  const unsigned long long rem = s->remaining;
  for (unsigned i = threadIdx.x; i < m; i += kUpdThreads) h[i] = ((volatile unsigned*)tie)[i];
  __syncthreads();
  for (unsigned i = threadIdx.x; i < m; i += kUpdThreads) {
    unsigned rank = 1;
    for (unsigned q = 0; q < m; ++q) rank += h[q] < h[i];
    if (rank == rem) {
      s->prefix = (prefix >> 32 << 32) | h[i];
      s->done = 1;
    }
  }
}

// Into res (which may be d): not where the stress field or the filtered field
// held a NaN, for which the caller has another answer.
__global__ void finish_kernel(long long n, const float* d, float* res, const uint8_t* __restrict__ prot,
                              const float* __restrict__ orig, float min_d, float thr, int hard,
                              const UpdateState* __restrict__ s) {
  if (s->nan_stress || s->nan_filtered) return;
  const int mode = s->mode;
  const unsigned long long kth = s->prefix;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    if (prot && prot[e]) {
      res[e] = orig[e];
      continue;
    }
    float v = d[e];
    if (is_candidate(v, min_d, thr) && (mode == 1 || (mode == 2 && cull_key(v, e) <= kth))) v = min_d;
    if (hard && v > min_d) v = 1.0f;
    res[e] = v;
  }
}

int grid_for(long long n) { return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 152LL * 16)); }

}  // namespace

void launch_propose(long long n, const float* l1, const uint8_t* prot, const float* orig, float allow, float E,
                    float min_d, float* prop, UpdateState* s, cudaStream_t st) {
  propose_kernel<<<grid_for(n), 256, 0, st>>>(n, l1, prot, orig, allow, E, min_d, prop, s);
}

int launch_update_cull(bool fused, long long n, const float* old, const float* src, const uint8_t* prot,
                       const float* orig, float allow, float E, float min_d, float max_d, float thr, float ratio,
                       int hard, float* work, float* res, double* part, unsigned long long* hist, unsigned* tie,
                       UpdateState* s, cudaStream_t st) {
  cudaMemsetAsync(hist, 0, kBins * sizeof(unsigned long long), st);
  if (fused)
    update_kernel<true><<<kUpdBlocks, kUpdThreads, 0, st>>>(n, old, src, prot, orig, allow, E, min_d, max_d, thr, ratio,
                                                            work, part, hist, s);
  else
    update_kernel<false><<<kUpdBlocks, kUpdThreads, 0, st>>>(n, old, src, prot, orig, allow, E, min_d, max_d, thr,
                                                             ratio, work, part, hist, s);
  constexpr int passes = (64 + kDigitBits - 1) / kDigitBits;
  const int blocks = std::min(grid_for(n), 152 * 8);
  for (int pass = 1; pass < passes; ++pass)
    select_kernel<<<blocks, kUpdThreads, 0, st>>>(n, work, prot, min_d, thr, pass, s, hist, tie);
  finish_kernel<<<grid_for(n), 256, 0, st>>>(n, work, res, prot, orig, min_d, thr, hard, s);
  return passes + 1;
}
int update_ties() { return kTies; }

size_t update_partials_doubles() { return 4 * (size_t)kUpdBlocks; }
int update_hist_bins() { return kBins; }

}  // namespace hexa
