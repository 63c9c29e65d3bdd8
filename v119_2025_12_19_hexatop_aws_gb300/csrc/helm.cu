// (d) Helmholtz PDE density filter on the structured grid.
//
// Replaces GPUHelmholtz.jl's path (src/Optimization/GPUHelmholtz.jl:59-266):
// the RHS scatter with atomics (:59-70) becomes a gather over the <= 8
// elements of each node; the 8 colour-batched element launches per matvec
// (:73-97, 155-172, 230-238) with a host-built sortperm colouring become one
// node-centric launch of the constant-coefficient element matrix
// Ae = R^2 Ke + Me (natural boundary: only elements inside the box count);
// the diagonal (:112-123) is analytic; the Jacobi-PCG loop (:208-260) keeps
// the reference's arithmetic but its dots and the every-10 convergence test run
// on the device; the element average (:99-110) is one gather pass.
//
// The element matrix of a brick depends only on which axes two corners differ
// in (8 weights w[m], bit d of m: axis d), so the row of a node is
//   y = sum_m w[m] prod_d (bit d of m ? S_d : c_d) x,
// S_d x = the sum of the two neighbours along axis d (zero past the grid) and
// c_d = the number of neighbours that exist (2 inside, 1 on a face): 16 FP64
// instructions a node against the 64 multiply-adds of the element-wise gather.
// FP64 issues 2 instructions per clock and SM on this part, so they set the
// FP64 filter's time.
#include <algorithm>

#include "hexa_common.cuh"
#include "hexa_kernels.h"

namespace hexa {

static inline int helm_blocks(long long n) {
  long long b = (n + 255) / 256;
  if (b < 1) b = 1;
  if (b > 152 * 8) b = 152 * 8;
  return (int)b;
}

template <typename T>
__global__ void helm_rhs_kernel(Grid g, const T* __restrict__ rho, T scale, T* __restrict__ b) {
  const long long nn = g.nnode();
  for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < nn; n += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(n % g.NX);
    const long long t = n / g.NX;
    const int j = (int)(t % g.NY), k = (int)(t / g.NY);
    T s = T(0);
    for (int dz = -1; dz <= 0; ++dz)
      for (int dy = -1; dy <= 0; ++dy)
        for (int dx = -1; dx <= 0; ++dx) {
          const int ei = i + dx, ej = j + dy, ek = k + dz;
          if (ei >= 0 && ei < g.nx && ej >= 0 && ej < g.ny && ek >= 0 && ek < g.nz)
            s += rho[(long long)ei + (long long)g.nx * ((long long)ej + (long long)g.ny * ek)] * scale;
        }
    b[n] = s;
  }
}
template <typename T>
void launch_helm_rhs(const Grid& g, const T* rho, T scale, T* b, cudaStream_t st) {
  helm_rhs_kernel<T><<<helm_blocks(g.nnode()), 256, 0, st>>>(g, rho, scale, b);
}

template <typename T>
struct HelmW {
  T w[8];        // weight of two corners that differ in the axes of m
  T p[4], z[4];  // of an inner node: own layer (c, S_x, S_y, S_xy), the layers above and below
};
// The quadrature's 8x8 matrix is symmetric under the brick's reflections up to
// rounding: the weight of m is the mean over the corner pairs.
template <typename T>
static HelmW<T> helm_weights(const HelmK& K) {
  HelmW<T> W;
  for (int m = 0; m < 8; ++m) {
    double s = 0.0;
    for (int c = 0; c < 8; ++c) s += K.A[c][c ^ m];
    W.w[m] = (T)(s / 8.0);
  }
  for (int m = 0; m < 4; ++m) {
    const T c = (T)(m == 0 ? 4 : (m == 3 ? 1 : 2));
    W.p[m] = T(2) * c * W.w[m];
    W.z[m] = c * W.w[m + 4];
  }
  return W;
}

__device__ __forceinline__ int on_face(int i, int n) { return (i == 0) | (i == n - 1); }
// v * 2^faces (-3 <= faces <= 3): a node on `faces` (0..3) faces of the box has 2^-faces of the
// inner nodes' diagonal.  Through the exponent bits, so that nothing is issued
// to the FP64 pipe.  Values whose exponent field could leave its range stay as
// they are: zeros and magnitudes below 2^-1019, which are nothing beside
// the terms they are added to, and non-finite values and magnitudes from 2^1021,
// whose squares have overflowed the PCG's sums anyway.
__device__ __forceinline__ float scale2(float v, int faces) { return v * __int_as_float((127 + faces) << 23); }
__device__ __forceinline__ double scale2(double v, int faces) {
  const int hi = __double2hiint(v);
  const bool in = (unsigned)(hi & 0x7ff00000) - 0x00400000u < 0x7f800000u;  // exponent field 4 .. 0x7fb
  return __hiloint2double(hi + (in ? faces * (1 << 20) : 0), __double2loint(v));
}

// ---- one grid: the PCG in two launches per iteration
//
// helm_dir_kernel: p = z + beta p_old, q = A p, p.q.  A CTA owns TX x TY node
// columns and marches through the layers of its z-chunk: each layer's p (tile
// and one node around it) is formed from r and p_old into shared memory, every
// thread takes its column's in-plane sums from there, and the layer below is
// finished with the z-neighbours' sums held in registers.  The search
// direction is formed where it is needed, so there is no z vector, no inverse
// diagonal vector and no pass of its own for p (p_old and p alternate, since
// neighbouring tiles read p_old).  The preconditioner is D^-1 times the inner
// nodes' diagonal, z = 2^faces r: a constant factor in z cancels in the
// iterates, and the common case needs no product.  On 256x128x128 in FP64 it
// takes 0.169 ms (FP64 pipe 81 % busy, 18 FP64 instructions a node) where the
// element-wise product and the p pass took 0.539 + 0.016 ms; with the update
// below the whole filter (10 iterations) went from 6.83 to 2.44 ms.
//
// Tile: the TX x TY columns that cover the grid's cross-section with the fewest
// threads (NX is often one more than a multiple of 32, so that 32-wide tiles
// would leave a ninth tile one column wide), a little in favour of small
// halos; a thread stages at most two nodes.  Chunk: the layer count for which
// the SM with the most items (of its layers, two halo layers and a start each)
// has the least to do: the FP64 pipe, which the CTAs of an SM share, sets the
// time.
constexpr int kHelmMaxBlocks = 152 * 16;
HelmPlan helm_plan(const Grid& g) {
  HelmPlan best{};
  double cost = 1e300;
  for (int tx = 2; tx <= 64; ++tx)
    for (int ty = 2; ty <= 64; ++ty) {
      const int thr = (tx * ty + 31) / 32 * 32;
      if (thr > 288 || thr < 128 || (tx + 2) * (ty + 2) > 2 * thr) continue;
      const double nx = (g.NX + tx - 1) / tx, ny = (g.NY + ty - 1) / ty;
      const double c = nx * ny * (thr + 0.5 * (tx + ty + 2));
      if (c < cost) {
        cost = c;
        best.tx = tx, best.ty = ty, best.threads = thr, best.ntx = (int)nx, best.nty = (int)ny;
        // whole warps with 2 * stage >= nodes (rounded up before the halving: a 53 x 5 tile has an odd 385)
        best.stage = (((tx + 2) * (ty + 2) + 1) / 2 + 31) / 32 * 32;
      }
    }
  const long long tiles = (long long)best.ntx * best.nty;
  cost = 1e300;
  for (int nch = 1; nch <= std::max(1, g.NZ / 2); ++nch) {
    const int kc = (g.NZ + nch - 1) / nch;
    const long long items = tiles * ((g.NZ + kc - 1) / kc);
    const double t = (double)((items + 151) / 152) * (kc + 2.5);
    if (t < cost) {
      cost = t;
      best.kchunk = kc;
      best.items = items;
    }
  }
  best.blocks = (int)std::min<long long>(best.items, kHelmMaxBlocks);
  return best;
}

// Index of the node that a position one past the grid mirrors (positions
// further out belong to no output and only have to be readable).
__device__ __forceinline__ int mirror(int i, int n) { return i < 0 ? 1 : (i >= n ? max(2 * n - 2 - i, 0) : i); }

// Faces without per-thread weights: with the neighbour past a face read as the
// mirrored one inside, the inner nodes' formula gives twice the row of a face
// node, per face.  All weights are then the same constants, and the result is
// scaled by 2^-faces through its exponent.
template <typename T>
__global__ void __launch_bounds__(288, 3) helm_dir_kernel(Grid g, HelmPlan pl, HelmW<T> W, const T* __restrict__ r,
                                                          const T* __restrict__ po, T* __restrict__ pn,
                                                          T* __restrict__ q, RedArgs red, const PcgScalars* s) {
  if (*((volatile const int*)&s->halt)) return;
  extern __shared__ __align__(16) unsigned char helm_smem[];
  const int tid = threadIdx.x, SX = pl.tx + 2, nslots = SX * (pl.ty + 2);
  T* const smem = reinterpret_cast<T*>(helm_smem);
  const bool first = s->iter == 0;  // no previous direction
  const T beta = first ? T(0) : (T)s->beta;
  const int tiles = pl.ntx * pl.nty;
  const long long plane = (long long)g.NX * g.NY;
  // the first warps stage two nodes per thread, the others none
  const int half = pl.stage;
  const bool stager = tid < half;
  const bool two = stager && tid + half < nslots;
  const int lx = tid % pl.tx, ly = tid / pl.tx, c = (lx + 1) + SX * (ly + 1);
  double sum = 0.0;
  for (long long item = blockIdx.x; item < pl.items; item += gridDim.x) {
    const int ch = (int)(item / tiles), tile = (int)(item - (long long)ch * tiles);
    const int i0 = (tile % pl.ntx) * pl.tx, j0 = (tile / pl.ntx) * pl.ty;
    const int k0 = ch * pl.kchunk, k1 = min(k0 + pl.kchunk, g.NZ);
    int off[2], fxy[2];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const int sl = tid + a * half;
      const int gi = mirror(i0 - 1 + sl % SX, g.NX), gj = mirror(j0 - 1 + sl / SX, g.NY);
      off[a] = gi + g.NX * gj;
      fxy[a] = on_face(gi, g.NX) + on_face(gj, g.NY);
    }
    const int i = i0 + lx, j = j0 + ly;
    const bool own = ly < pl.ty && i < g.NX && j < g.NY;
    const int col = own ? i + g.NX * j : 0, cf = on_face(i, g.NX) + on_face(j, g.NY);
    T rv[2], pv[2];
    auto load = [&](int k) {
      const long long base = plane * mirror(k, g.NZ);
      rv[0] = (r + base)[off[0]];
      if (two) rv[1] = (r + base)[off[1]];
      pv[0] = pv[1] = T(0);
      if (!first) {
        pv[0] = (po + base)[off[0]];
        if (two) pv[1] = (po + base)[off[1]];
      }
    };
    T G0 = T(0), Gm = T(0), Gp = T(0), pc = T(0);  // of layer k-1: in-plane sums, p; of layers k-2, k-1: z-weighted sums
    if (stager) load(k0 - 1);
    for (int k = k0 - 1; k <= k1; ++k) {
      T* buf = smem + ((k & 1) ? nslots : 0);
      if (stager) {
        const int fz = on_face(mirror(k, g.NZ), g.NZ);
        buf[tid] = fma(beta, pv[0], scale2(rv[0], fxy[0] + fz));
        if (two) buf[tid + half] = fma(beta, pv[1], scale2(rv[1], fxy[1] + fz));
        if (k < k1) load(k + 1);
      }
      __syncthreads();  // two buffers: the one rewritten next layer was read before this barrier
      if (own) {
        const T* u = buf + c;
        const T pk = u[0];
        const T sx = u[-1] + u[1], sy = u[-SX] + u[SX];
        const T sxy = (u[-SX - 1] + u[-SX + 1]) + (u[SX - 1] + u[SX + 1]);
        const T H1 = fma(W.z[0], pk, fma(W.z[1], sx, fma(W.z[2], sy, W.z[3] * sxy)));
        if (k > k0) {  // layer k-1 is complete
          const T y = scale2(G0 + (Gm + H1), -(cf + on_face(k - 1, g.NZ)));
          (q + plane * (k - 1))[col] = y;
          sum = fma((double)pc, (double)y, sum);
        }
        Gm = Gp;
        Gp = H1;
        if (k >= k0 && k < k1) {
          G0 = fma(W.p[0], pk, fma(W.p[1], sx, fma(W.p[2], sy, W.p[3] * sxy)));
          (pn + plane * k)[col] = pk;
          pc = pk;
        }
      }
    }
    __syncthreads();  // the next item writes either buffer
  }
  double v[1] = {sum};
  block_reduce_finalize<1>(red, v);
}
template <typename T>
void launch_helm_dir(const Grid& g, const HelmPlan& pl, const HelmK& K, const T* r, const T* po, T* pn, T* q,
                     const RedArgs& red, const PcgScalars* s, cudaStream_t st) {
  const size_t smem = 2 * sizeof(T) * (size_t)(pl.tx + 2) * (pl.ty + 2);
  helm_dir_kernel<T><<<pl.blocks, pl.threads, smem, st>>>(g, pl, helm_weights<T>(K), r, po, pn, q, red, s);
}

// x += alpha p, r -= alpha q, ||r||^2 and r.z in one pass.  A warp takes whole
// node rows: with z = 2^faces r the row's r.z is 2^(y and z faces) times its
// ||r||^2 plus the two end nodes' squares once more, so the inner loop is three
// FP64 instructions a node.  The squares of up to kHelmFlush terms are summed
// in T, then folded into FP64.  256x128x128 in FP64: 0.053 ms, 0.074 before
// (with a z vector and an inverse diagonal, 64 B a node instead of 48).
constexpr int kHelmFlush = 32;
template <typename T>
__global__ void __launch_bounds__(256) helm_update_kernel(Grid g, T* __restrict__ x, T* __restrict__ r,
                                                          const T* __restrict__ p, const T* __restrict__ q,
                                                          RedArgs red, const PcgScalars* s) {
  if (*((volatile const int*)&s->halt)) return;
  const bool first = s->iter == 0;  // x starts at zero
  const T alpha = (T)s->alpha;
  const int lane = threadIdx.x & 31;
  const long long rows = (long long)g.NY * g.NZ, nw = (long long)gridDim.x * (blockDim.x >> 5);
  double acc[2] = {0.0, 0.0};
  for (long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows; row += nw) {
    const int k = (int)(row / g.NY), j = (int)(row - (long long)k * g.NY);
    const long long base = row * g.NX;
    double rr = 0.0;
    T ends = T(0);
    for (int ib = lane; ib < g.NX; ib += 32 * kHelmFlush) {
      T part = T(0);
      const int ie = min(g.NX, ib - lane + 32 * kHelmFlush);
#pragma unroll 4
      for (int i = ib; i < ie; i += 32) {
        const long long n = base + i;
        const T pv = p[n], xv = first ? T(0) : x[n];
        const T ri = fma(-alpha, q[n], r[n]);
        x[n] = fma(alpha, pv, xv);
        r[n] = ri;
        part = fma(ri, ri, part);
        if (i == 0) ends = ri;  // lane 0's first node
      }
      rr += (double)part;
    }
    T rz = T(0);
    if (lane == 0) rz = ends * ends;
    if (lane == ((g.NX - 1) & 31)) {
      const T re = r[base + g.NX - 1];  // this thread's own last node
      rz = fma(re, re, rz);
    }
    acc[0] += rr;
    acc[1] += scale2(rr + (double)rz, on_face(j, g.NY) + on_face(k, g.NZ));
  }
  block_reduce_finalize<2, 256>(red, acc);
}
// One wave of warps with equal row counts (4 CTAs of 8 warps on each SM).
static int helm_update_blocks(const Grid& g) {
  const long long rows = (long long)g.NY * g.NZ, slots = 152 * 4 * 8;
  const long long per = (rows + slots - 1) / slots;
  return (int)(((rows + per - 1) / per + 7) / 8);
}
template <typename T>
void launch_helm_update(const Grid& g, T* x, T* r, const T* p, const T* q, const RedArgs& red, const PcgScalars* s,
                        cudaStream_t st) {
  helm_update_kernel<T><<<helm_update_blocks(g), 256, 0, st>>>(g, x, r, p, q, red, s);
}

// Right-hand side r = b (the element densities around a node times vol/8) and
// the sums b.b and b.z.  A thread marches kHelmZ nodes of its column and
// carries the sum of the four elements below.
constexpr int kHelmZ = 8;
template <typename T, typename TI>
__global__ void __launch_bounds__(128) helm_init_kernel(Grid g, const TI* __restrict__ rho, T scale,
                                                        T* __restrict__ r, RedArgs red) {
  const int nbx = (g.NX + 31) / 32, nby = (g.NY + 3) / 4, nzc = (g.NZ + kHelmZ - 1) / kHelmZ;
  const long long items = (long long)nbx * nby * nzc;
  double acc[2] = {0.0, 0.0};
  for (long long item = blockIdx.x; item < items; item += gridDim.x) {
    const int i = (int)(item % nbx) * 32 + threadIdx.x, j = (int)(item / nbx % nby) * 4 + threadIdx.y;
    const int k0 = (int)(item / nbx / nby) * kHelmZ;
    if (i >= g.NX || j >= g.NY) continue;
    const bool xl = i >= 1, xr = i < g.nx, yl = j >= 1, yr = j < g.ny;
    T e[kHelmZ + 1];
#pragma unroll
    for (int c = 0; c <= kHelmZ; ++c) {
      const int ek = k0 - 1 + c;
      const bool z = ek >= 0 && ek < g.nz;
      const TI* row = rho + (long long)g.nx * ((long long)(j - 1) + (long long)g.ny * ek) + i;
      const T e0 = (z && yl && xl) ? (T)row[-1] : T(0), e1 = (z && yl && xr) ? (T)row[0] : T(0);
      const T e2 = (z && yr && xl) ? (T)row[g.nx - 1] : T(0), e3 = (z && yr && xr) ? (T)row[g.nx] : T(0);
      e[c] = (e0 + e1) + (e2 + e3);
    }
    T part[2] = {T(0), T(0)};
#pragma unroll
    for (int c = 0; c < kHelmZ; ++c) {
      const int k = k0 + c;
      if (k >= g.NZ) break;
      const T b = (e[c] + e[c + 1]) * scale;
      r[(long long)i + (long long)g.NX * ((long long)j + (long long)g.NY * k)] = b;
      part[0] = fma(b, b, part[0]);
      const T bz = scale2(b, on_face(i, g.NX) + on_face(j, g.NY) + on_face(k, g.NZ));
      part[1] = fma(b, bz, part[1]);
    }
    acc[0] += (double)part[0], acc[1] += (double)part[1];
  }
  block_reduce_finalize<2>(red, acc);
}
static int helm_init_blocks(const Grid& g) {
  const long long items =
      (long long)((g.NX + 31) / 32) * ((g.NY + 3) / 4) * ((g.NZ + kHelmZ - 1) / kHelmZ);
  return (int)std::min<long long>(items, 152 * 8);
}
template <typename T, typename TI>
void launch_helm_init(const Grid& g, const HelmK& K, const TI* rho, T* r, const RedArgs& red, cudaStream_t st) {
  helm_init_kernel<T, TI><<<helm_init_blocks(g), dim3(32, 4), 0, st>>>(g, rho, (T)K.rhs_scale, r, red);
}
static_assert(kHelmPartials >= kHelmMaxBlocks && kHelmPartials >= 2 * 152 * 8, "partials of the filter's passes");

// Element mean of the nodal solution; each thread marches kHelmZ elements of
// its column and carries the sum of the four nodes below.
template <typename T, typename TO>
__global__ void __launch_bounds__(128) helm_mean_kernel(Grid g, const T* __restrict__ psi, TO* __restrict__ out) {
  const int nbx = (g.nx + 31) / 32, nby = (g.ny + 3) / 4, nzc = (g.nz + kHelmZ - 1) / kHelmZ;
  const long long items = (long long)nbx * nby * nzc;
  for (long long item = blockIdx.x; item < items; item += gridDim.x) {
    const int i = (int)(item % nbx) * 32 + threadIdx.x, j = (int)(item / nbx % nby) * 4 + threadIdx.y;
    const int k0 = (int)(item / nbx / nby) * kHelmZ;
    if (i >= g.nx || j >= g.ny) continue;
    T f[kHelmZ + 1];
#pragma unroll
    for (int c = 0; c <= kHelmZ; ++c) {
      const T* row = psi + (long long)i + (long long)g.NX * ((long long)j + (long long)g.NY * (k0 + c));
      f[c] = k0 + c < g.NZ ? (row[0] + row[1]) + (row[g.NX] + row[g.NX + 1]) : T(0);
    }
#pragma unroll
    for (int c = 0; c < kHelmZ; ++c)
      if (k0 + c < g.nz)
        out[(long long)i + (long long)g.nx * ((long long)j + (long long)g.ny * (k0 + c))] =
            (TO)((f[c] + f[c + 1]) * T(0.125));
  }
}
template <typename T, typename TO>
void launch_helm_mean(const Grid& g, const T* psi, TO* out, cudaStream_t st) {
  const long long items =
      (long long)((g.nx + 31) / 32) * ((g.ny + 3) / 4) * ((g.nz + kHelmZ - 1) / kHelmZ);
  helm_mean_kernel<T, TO><<<(int)std::min<long long>(items, 152 * 16), dim3(32, 4), 0, st>>>(g, psi, out);
}

// ---- batches: one thread per node, the 27 neighbours read through L1
template <typename T>
__device__ __forceinline__ double helm_apply_body(const Grid& g, const HelmW<T>& W, const T* __restrict__ x,
                                                  T* __restrict__ y, long long first, long long stride) {
  double acc = 0.0;
  const long long nn = g.nnode();
  for (long long n = first; n < nn; n += stride) {
    const int i = (int)(n % g.NX);
    const long long t = n / g.NX;
    const int j = (int)(t % g.NY), k = (int)(t / g.NY);
    const bool xl = i > 0, xr = i < g.nx, yl = j > 0, yr = j < g.ny;
    const T cx = xl && xr ? T(2) : T(1), cy = yl && yr ? T(2) : T(1), cz = (k > 0 && k < g.nz) ? T(2) : T(1);
    T c0 = T(0), f[4] = {T(0), T(0), T(0), T(0)}, z[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
    for (int dk = -1; dk <= 1; ++dk) {
      if (k + dk < 0 || k + dk >= g.NZ) continue;
      const T* u = x + n + (long long)g.NX * g.NY * dk;
      auto pair = [&](const T* v) { return (xl ? __ldg(v - 1) : T(0)) + (xr ? __ldg(v + 1) : T(0)); };
      const T c = __ldg(u), sx = pair(u);
      const T sy = (yl ? __ldg(u - g.NX) : T(0)) + (yr ? __ldg(u + g.NX) : T(0));
      const T sxy = (yl ? pair(u - g.NX) : T(0)) + (yr ? pair(u + g.NX) : T(0));
      if (dk == 0) c0 = c, f[0] = c, f[1] = sx, f[2] = sy, f[3] = sxy;
      else z[0] += c, z[1] += sx, z[2] += sy, z[3] += sxy;
    }
    T sum = cz * fma(W.w[0] * cx * cy, f[0], fma(W.w[1] * cy, f[1], fma(W.w[2] * cx, f[2], W.w[3] * f[3])));
    sum = fma(W.w[4] * cx * cy, z[0], fma(W.w[5] * cy, z[1], fma(W.w[6] * cx, z[2], fma(W.w[7], z[3], sum))));
    y[n] = sum;
    acc += (double)c0 * (double)sum;
  }
  return acc;
}

// Batch form over node vectors: instance I's nodes start at I.noff.
template <typename T>
__global__ void batch_helm_apply_kernel(const BatchInst* in, int ninst, HelmW<T> W, const T* __restrict__ x,
                                        T* __restrict__ y, RedArgs red, const PcgScalars* s) {
  int lo = 0, hi = ninst - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (in[mid].vblk0 <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const BatchInst& I = in[lo];
  if (s && *((volatile const int*)&s[I.id].halt)) return;
  double acc[1] = {helm_apply_body<T>(I.g, W, x + I.noff, y + I.noff,
                                      (long long)(blockIdx.x - I.vblk0) * blockDim.x + threadIdx.x,
                                      (long long)I.vnblk * blockDim.x)};
  block_reduce_finalize_at<1, 256>(red, acc, I.id, blockIdx.x, I.vnblk, I.vblk0, 1);
}
template <typename T>
void launch_batch_helm_apply_dot(const BatchInst* in, int ninst, int nblocks, const HelmK& K, const T* x, T* y,
                                 const RedArgs& red, const PcgScalars* s, cudaStream_t st) {
  batch_helm_apply_kernel<T><<<nblocks, 256, 0, st>>>(in, ninst, helm_weights<T>(K), x, y, red, s);
}

template <typename T>
__global__ void helm_dinv_kernel(Grid g, T dinv8, T* __restrict__ dinv) {
  const long long nn = g.nnode();
  for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < nn; n += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(n % g.NX);
    const long long t = n / g.NX;
    const int j = (int)(t % g.NY), k = (int)(t / g.NY);
    dinv[n] = scale2(dinv8, on_face(i, g.NX) + on_face(j, g.NY) + on_face(k, g.NZ));  // GPUHelmholtz.jl:153
  }
}
template <typename T>
void launch_helm_dinv(const Grid& g, const HelmK& K, T* dinv, cudaStream_t st) {
  helm_dinv_kernel<T><<<helm_blocks(g.nnode()), 256, 0, st>>>(g, (T)1 / (T(8) * helm_weights<T>(K).w[0]), dinv);
}

#define INST(T)                                                                                              \
  template void launch_helm_rhs<T>(const Grid&, const T*, T, T*, cudaStream_t);                              \
  template void launch_helm_dir<T>(const Grid&, const HelmPlan&, const HelmK&, const T*, const T*, T*, T*,   \
                                   const RedArgs&, const PcgScalars*, cudaStream_t);                         \
  template void launch_helm_update<T>(const Grid&, T*, T*, const T*, const T*, const RedArgs&,               \
                                      const PcgScalars*, cudaStream_t);                                      \
  template void launch_helm_init<T, double>(const Grid&, const HelmK&, const double*, T*, const RedArgs&,    \
                                            cudaStream_t);                                                   \
  template void launch_helm_init<T, float>(const Grid&, const HelmK&, const float*, T*, const RedArgs&,      \
                                           cudaStream_t);                                                    \
  template void launch_helm_mean<T, double>(const Grid&, const T*, double*, cudaStream_t);                   \
  template void launch_helm_mean<T, float>(const Grid&, const T*, float*, cudaStream_t);                     \
  template void launch_helm_dinv<T>(const Grid&, const HelmK&, T*, cudaStream_t);                            \
  template void launch_batch_helm_apply_dot<T>(const BatchInst*, int, int, const HelmK&, const T*, T*,       \
                                               const RedArgs&, const PcgScalars*, cudaStream_t);
INST(double)
INST(float)
#undef INST

}  // namespace hexa
