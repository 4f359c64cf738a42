// Krylov support: dots with the basis, orthogonalisation with the norm, null-space
// removal and the coarsest-level dense solve.  Every reduction is two-stage with
// a block count fixed by the size and a fixed summation tree, so their results do
// not depend on timing or on what else shares the GPU.
#include <algorithm>

#include "intmul.cuh"
#include "launch.cuh"

namespace cvb {

static long long g_launches = 0;
void count_launch(int n) { __atomic_add_fetch(&g_launches, (long long)n, __ATOMIC_RELAXED); }
long long launch_count() { return __atomic_load_n(&g_launches, __ATOMIC_RELAXED); }

static const int kRedThreads = 256;  // the reductions' kernels: four blocks an SM, all resident
static int g_red_blocks = 0;

int sm_count() {
  static int sms = 0;
  if (!sms) {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    sms = v > 0 ? v : 148;
  }
  return sms;
}

int reduce_blocks() {
  if (!g_red_blocks) g_red_blocks = sm_count() * 4;
  return g_red_blocks;
}

// ------------------------------------------------------------ reductions
// A kernel's NR sums over all its blocks.  Each thread's terms go through shared
// memory, a warp per sum, into partial[q][block]; the last block to arrive adds
// the partials, a warp per sum, and only its threads see the totals (tot, true
// returned).  The trees are fixed by the grid, so the totals do not depend on the
// order of arrival.  Few FP64 additions (12 a sum and warp-pair of a block, where
// a shuffle tree per warp makes 40): they share the pipe that bounds these
// kernels.  *counter is zero between launches.
template <int NR>
struct ReduceSmem {
  double v[NR][kRedThreads];
  double tot[NR];
  int last;
};
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
template <int NR>
__device__ __forceinline__ bool reduce_all(ReduceSmem<NR> &sm, const double (&acc)[NR], double *partial,
                                           unsigned *counter) {
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nb = gridDim.x;
#pragma unroll
  for (int q = 0; q < NR; q++) sm.v[q][t] = acc[q];
  __syncthreads();
  for (int q = wid; q < NR; q += kRedThreads / 32) {
    double v = sm.v[q][lane];
#pragma unroll
    for (int u = 1; u < kRedThreads / 32; u++) v += sm.v[q][lane + 32 * u];
    v = warp_sum(v);
    if (lane == 0) {
      __stcg(partial + (size_t)q * nb + blockIdx.x, v);
      __threadfence();
    }
  }
  __syncthreads();
  if (t == 0) sm.last = atomicAdd(counter, 1u) == (unsigned)nb - 1u;
  __syncthreads();
  if (!sm.last) return false;
  __threadfence();
  for (int q = wid; q < NR; q += kRedThreads / 32) {
    double v = 0.0;
    for (int b = lane; b < nb; b += 32) v += __ldcg(partial + (size_t)q * nb + b);
    v = warp_sum(v);
    if (lane == 0) sm.tot[q] = v;
  }
  if (t == 0) *counter = 0;
  __syncthreads();
  return true;
}

// Two cells a thread at least, so that a small problem's last block has few partials.
static unsigned red_grid(size_t n) {
  return (unsigned)std::min<size_t>(reduce_blocks(), (n + 2 * kRedThreads - 1) / (2 * kRedThreads));
}

// out[base + q] = V_{base + q} . w for NV vectors.  The vector count is a
// template parameter: predicated-off products would still occupy the FP64 pipe,
// which bounds this kernel on this part (six vectors on 4.4 M cells: 45 us of it).
template <int NV>
__global__ void __launch_bounds__(kRedThreads, 4) k_dots(const __grid_constant__ BasisList V, int base,
                                                      const double *__restrict__ w, size_t n, double *partial,
                                                      unsigned *counter, double *__restrict__ out) {
  dep_sync();
  constexpr int U = NV <= 2 ? 4 : NV <= 4 ? 2 : 1;
  __shared__ ReduceSmem<NV> sm;
  double acc[NV];
#pragma unroll
  for (int q = 0; q < NV; q++) acc[q] = 0.0;
  const size_t step = (size_t)gridDim.x * kRedThreads;
  size_t p = blockIdx.x * (size_t)kRedThreads + threadIdx.x;
  for (; p + (U - 1) * step < n; p += U * step) {
    double v[U][NV], wp[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      wp[u] = w[p + u * step];
#pragma unroll
      for (int q = 0; q < NV; q++) v[u][q] = V.v[base + q][p + u * step];
    }
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int q = 0; q < NV; q++) acc[q] = fma(v[u][q], wp[u], acc[q]);
  }
  for (; p < n; p += step) {
    const double wp = w[p];
#pragma unroll
    for (int q = 0; q < NV; q++) acc[q] = fma(V.v[base + q][p], wp, acc[q]);
  }
  if (reduce_all<NV>(sm, acc, partial, counter) && threadIdx.x < NV) out[base + threadIdx.x] = sm.tot[threadIdx.x];
}

template <int NV>
static void dots_chunk(const BasisList &V, int base, int cnt, const double *w, size_t n, double *partial,
                       unsigned *counter, double *out, cudaStream_t s) {
  if (cnt == NV)
    launch_dep(k_dots<NV>, red_grid(n), kRedThreads, 0, s, V, base, w, n, partial, counter, out);
  else if constexpr (NV > 1)
    dots_chunk<NV - 1>(V, base, cnt, w, n, partial, counter, out, s);
}
// Dots of w with V_0..V_{nv-1} into out, in chunks of up to 8 vectors (each chunk
// reads w once more).
void launch_dots(const BasisList &V, int nv, const double *w, size_t n, double *partial, unsigned *counter, double *out,
                 cudaStream_t s) {
  for (int base = 0; base < nv; base += 8)
    dots_chunk<8>(V, base, std::min(nv - base, 8), w, n, partial, counter, out, s);
}

// out[q] = sum_b partial[q][b], one block per q, fixed tree.
__global__ void k_finish(const double *__restrict__ partial, int nblocks, double *__restrict__ out,
                         const int *gate) {
  dep_sync();
  if (gated(gate)) return;
  __shared__ double sh[kRedThreads];
  int q = blockIdx.x;
  double v = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += kRedThreads) v += partial[(size_t)q * nblocks + b];
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = kRedThreads / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[q] = sh[0];
}
void launch_finish_sums(const double *partial, int nv, int nblocks, double *out, cudaStream_t s, const int *gate) {
  launch_dep(k_finish, nv, kRedThreads, 0, s, partial, nblocks, out, gate);
}

// What a norm's kernel leaves: out[0] = the sum of squares, out[1] = 1 / its root;
// the sum, after nh other scalars h, also in pinned host memory.
__device__ __forceinline__ void store_norm(double sum, double *out, const double *h, int nh, double *host) {
  const int t = threadIdx.x;
  if (t == 0) {
    out[0] = sum;
    out[1] = 1.0 / sqrt(sum);
    host[nh] = sum;
  }
  for (int q = t; q < nh; q += kRedThreads) host[q] = h[q];
}

// w -= sum_q h[q] V_q for 8 * octets + NR vectors, and the norm of w.  The
// remainder is a template parameter for the same reason as k_dots's count; each
// octet's loads come before its products.
template <int NR>
__global__ void __launch_bounds__(kRedThreads, 4) k_orthogonalise(double *__restrict__ w,
                                                               const __grid_constant__ BasisList V,
                                                               const double *__restrict__ h, int octets, size_t n,
                                                               double *partial, unsigned *counter, double *out,
                                                               double *host) {
  dep_sync();
  __shared__ ReduceSmem<1> sm;
  __shared__ double hs[kMaxBasis];
  const int nv = 8 * octets + NR;
  if (threadIdx.x < nv) hs[threadIdx.x] = h[threadIdx.x];
  __syncthreads();
  constexpr int U = NR <= 3 ? 2 : 1;
  double acc[1] = {0.0};
  const size_t step = (size_t)gridDim.x * kRedThreads;
  for (size_t p0 = blockIdx.x * (size_t)kRedThreads + threadIdx.x; p0 < n; p0 += U * step) {
    double x[U][NR], v[U];
    const bool two = U > 1 && p0 + step < n;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const size_t p = u && two ? p0 + step : p0;
      v[u] = w[p];
#pragma unroll
      for (int q = 0; q < NR; q++) x[u][q] = V.v[q][p];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (u && !two) break;
      const size_t p = p0 + u * step;
#pragma unroll
      for (int q = 0; q < NR; q++) v[u] = fma(-hs[q], x[u][q], v[u]);
      for (int o = 0; o < octets; o++) {
        const int b = NR + 8 * o;
        double y[8];
#pragma unroll
        for (int q = 0; q < 8; q++) y[q] = V.v[b + q][p];
#pragma unroll
        for (int q = 0; q < 8; q++) v[u] = fma(-hs[b + q], y[q], v[u]);
      }
      w[p] = v[u];
      acc[0] = fma(v[u], v[u], acc[0]);
    }
  }
  if (reduce_all<1>(sm, acc, partial, counter)) store_norm(sm.tot[0], out, hs, nv, host);
}
template <int NR>
static void orthogonalise(double *w, const BasisList &V, const double *h, int nv, size_t n, double *partial,
                          unsigned *counter, double *out, double *host, cudaStream_t s) {
  const int r = (nv - 1) % 8 + 1;
  if (r == NR)
    launch_dep(k_orthogonalise<NR>, red_grid(n), kRedThreads, 0, s, w, V, h, nv / 8 - (NR == 8), n, partial, counter,
               out, host);
  else if constexpr (NR > 1)
    orthogonalise<NR - 1>(w, V, h, nv, n, partial, counter, out, host, s);
}
void launch_orthogonalise(double *w, const BasisList &V, const double *h, int nv, size_t n, double *partial,
                          unsigned *counter, double *out, double *host, cudaStream_t s) {
  orthogonalise<8>(w, V, h, nv, n, partial, counter, out, host, s);
}

// The norm of v.
__global__ void __launch_bounds__(kRedThreads, 4) k_norm(const double *__restrict__ v, size_t n, double *partial,
                                                      unsigned *counter, double *out, double *host) {
  dep_sync();
  __shared__ ReduceSmem<1> sm;
  double acc[1] = {0.0};
  const size_t step = (size_t)gridDim.x * kRedThreads;
  for (size_t p0 = blockIdx.x * (size_t)kRedThreads + threadIdx.x; p0 < n; p0 += 4 * step) {
    double x[4];
#pragma unroll
    for (int u = 0; u < 4; u++) x[u] = p0 + u * step < n ? v[p0 + u * step] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (p0 + u * step < n) acc[0] = fma(x[u], x[u], acc[0]);
  }
  if (reduce_all<1>(sm, acc, partial, counter)) store_norm(sm.tot[0], out, nullptr, 0, host);
}
void launch_norm(const double *v, size_t n, double *partial, unsigned *counter, double *out, double *host,
                 cudaStream_t s) {
  launch_dep(k_norm, red_grid(n), kRedThreads, 0, s, v, n, partial, counter, out, host);
}

// dst = src *rcp (a norm's reciprocal), and with dst32 its FP32 copy (the next
// V-cycle's input in mixed precision): one FP64 operation a cell, the
// conversion on the integer pipe.
__global__ void __launch_bounds__(256) k_scale(double *__restrict__ dst, const double *__restrict__ src,
                                               const double *__restrict__ rcp, size_t n, float *__restrict__ dst32) {
  dep_sync();
  const double inv = *rcp;
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    const double v = src[p] * inv;
    dst[p] = v;
    if (dst32) dst32[p] = int_narrow(v);
  }
}
void launch_scale(double *dst, const double *src, const double *rcp, size_t n, float *dst32, cudaStream_t s) {
  launch_dep(k_scale, (unsigned)((n + 1023) / 1024), 256, 0, s, dst, src, rcp, n, dst32);
}

__global__ void k_reciprocal(const double *__restrict__ a, double *__restrict__ out, size_t n) {
  dep_sync();
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x)
    out[p] = 1.0 / a[p];
}
void launch_reciprocal(const double *a, double *out, size_t n, cudaStream_t s) {
  launch_dep(k_reciprocal, reduce_blocks(), 256, 0, s, a, out, n);
}

// x += sum_q y[q] Z_q for 8 * octets + NR vectors
template <int NR>
__global__ void __launch_bounds__(256) k_axpy_z(double *__restrict__ x, const __grid_constant__ BasisList Z,
                                                const __grid_constant__ BasisWeights y, int octets, size_t n) {
  dep_sync();
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    double z[NR];
    double v = x[p];
#pragma unroll
    for (int q = 0; q < NR; q++) z[q] = Z.v[q][p];
#pragma unroll
    for (int q = 0; q < NR; q++) v = fma(y.y[q], z[q], v);
    for (int o = 0; o < octets; o++) {
      const int b = NR + 8 * o;
      double u[8];
#pragma unroll
      for (int q = 0; q < 8; q++) u[q] = Z.v[b + q][p];
#pragma unroll
      for (int q = 0; q < 8; q++) v = fma(y.y[b + q], u[q], v);
    }
    x[p] = v;
  }
}
template <int NR>
static void axpy_z(double *x, const BasisList &Z, const BasisWeights &y, int nz, size_t n, cudaStream_t s) {
  if ((nz - 1) % 8 + 1 == NR)
    launch_dep(k_axpy_z<NR>, (unsigned)((n + 1023) / 1024), 256, 0, s, x, Z, y, nz / 8 - (NR == 8), n);
  else if constexpr (NR > 1)
    axpy_z<NR - 1>(x, Z, y, nz, n, s);
}
void launch_axpy_z(double *x, const BasisList &Z, const BasisWeights &y, int nz, size_t n, cudaStream_t s) {
  axpy_z<8>(x, Z, y, nz, n, s);
}

// ------------------------------------------------------------ null space, range
// The mean over the interior fluid cells (nvert < 0.1) of x (the null space,
// PoissonNullSpaceFunction, poisson.c:411-558), or of b / aj as b times the
// stored 1 / aj (the range projection), times `sign`, into *out: counted in an
// integer, four cells a step, so that a cell costs one FP64 operation.
template <bool RATIO>
__global__ void __launch_bounds__(kRedThreads, 4) k_fluid_mean(size_t n, const uint32_t *__restrict__ code,
                                                            const double *__restrict__ x,
                                                            const double *__restrict__ inv_aj, double sign,
                                                            double *partial, unsigned *counter, double *out) {
  dep_sync();
  __shared__ ReduceSmem<2> sm;
  double acc[2] = {0.0, 0.0};
  unsigned cnt = 0;
  const size_t step = (size_t)gridDim.x * kRedThreads;
  for (size_t p0 = blockIdx.x * (size_t)kRedThreads + threadIdx.x; p0 < n; p0 += 4 * step) {
    uint32_t c[4];
    double v[4], a[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const size_t p = p0 + u * step;
      c[u] = p < n ? code[p] : 0;
      v[u] = p < n ? x[p] : 0.0;
      a[u] = RATIO && p < n ? inv_aj[p] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (c[u] & CODE_FLUID) {
        acc[0] = RATIO ? fma(v[u], a[u], acc[0]) : acc[0] + v[u];
        cnt++;
      }
  }
  acc[1] = (double)cnt;
  if (reduce_all<2>(sm, acc, partial, counter) && threadIdx.x == 0)
    *out = sm.tot[1] > 0.0 ? sm.tot[0] / (sign * sm.tot[1]) : 0.0;
}
void launch_fluid_mean(const Geom &g, const uint32_t *code, const double *x, const double *inv_aj, double sign,
                       double *partial, unsigned *counter, double *out, cudaStream_t s) {
  if (inv_aj)
    launch_dep(k_fluid_mean<true>, red_grid(g.n()), kRedThreads, 0, s, g.n(), code, x, inv_aj, sign, partial, counter,
               out);
  else
    launch_dep(k_fluid_mean<false>, red_grid(g.n()), kRedThreads, 0, s, g.n(), code, x, inv_aj, sign, partial, counter,
               out);
}

// x += *shift on interior fluid cells; with zero_outside the ring and the
// non-fluid cells are set to zero.
__global__ void __launch_bounds__(256) k_add_fluid_const(size_t n, const uint32_t *__restrict__ code,
                                                         double *__restrict__ x, const double *__restrict__ shift,
                                                         int zero_outside) {
  dep_sync();
  const double c0 = *shift;
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    const uint32_t c = code[p];
    if (c & CODE_FLUID) x[p] += c0;
    if (zero_outside && (c & CODE_IDENTITY)) x[p] = 0.0;  // the ring and nvert > 0.1
  }
}
void launch_add_fluid_const(const Geom &g, const uint32_t *code, double *x, const double *shift, int zero_outside,
                            cudaStream_t s) {
  launch_dep(k_add_fluid_const, (unsigned)((g.n() + 1023) / 1024), 256, 0, s, g.n(), code, x, shift, zero_outside);
}

// The range projection b -= aj *mean on the fluid cells, and the norm of what is
// left (the mean goes to the host with it).
__global__ void __launch_bounds__(kRedThreads, 4) k_remove_mean(size_t n, const uint32_t *__restrict__ code,
                                                             const double *__restrict__ aj, double *__restrict__ b,
                                                             const double *__restrict__ mean, double *partial,
                                                             unsigned *counter, double *out, double *host) {
  dep_sync();
  __shared__ ReduceSmem<1> sm;
  const double c0 = *mean;
  double acc[1] = {0.0};
  const size_t step = (size_t)gridDim.x * kRedThreads;
  for (size_t p0 = blockIdx.x * (size_t)kRedThreads + threadIdx.x; p0 < n; p0 += 4 * step) {
    uint32_t c[4];
    double v[4], a[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const size_t p = p0 + u * step;
      c[u] = p < n ? code[p] : 0;
      v[u] = p < n ? b[p] : 0.0;
      a[u] = p < n ? aj[p] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (c[u] & CODE_FLUID) {
        v[u] -= a[u] * c0;
        b[p0 + u * step] = v[u];
      }
      if (p0 + u * step < n) acc[0] = fma(v[u], v[u], acc[0]);
    }
  }
  if (reduce_all<1>(sm, acc, partial, counter)) store_norm(sm.tot[0], out, mean, 1, host);
}
void launch_remove_mean(const Geom &g, const uint32_t *code, const double *aj, double *b, const double *mean,
                        double *partial, unsigned *counter, double *out, double *host, cudaStream_t s) {
  launch_dep(k_remove_mean, red_grid(g.n()), kRedThreads, 0, s, g.n(), code, aj, b, mean, partial, counter, out, host);
}

// Coarsest level: e = Minv r with a dense FP64 inverse over the cells idx[0..m),
// e = r on the identity cells idx[m..n).  A block first gathers r over the
// inverted cells into shared memory, in the inverse's column order and in FP64;
// its warps then take rows, each lane two adjacent columns per step with one
// 16-byte load of the row (rows are 16-byte aligned for even m) into two
// accumulators, four steps in flight, then a shuffle sum.  The inverse is the
// bulk of the bytes (8 m^2), read once per apply.  STAGED false (m beyond what
// shared memory holds): r is read through idx at every step instead.
template <typename T, bool STAGED>
__global__ void __launch_bounds__(256) k_dense(const double *__restrict__ M, const int *__restrict__ idx, int m, int n,
                                               const T *__restrict__ r, T *__restrict__ e, const int *gate) {
  extern __shared__ __align__(16) double rc[];
  dep_sync();
  if (gated(gate)) return;
  if (STAGED) {
    for (int c = threadIdx.x; c < m; c += blockDim.x) rc[c] = (double)r[idx[c]];
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  // rows dealt out block by block: every SM gets the same number of them
  for (int row = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; row < n; row += gridDim.x * nw) {
    if (row >= m) {
      if (lane == 0) e[idx[row]] = r[idx[row]];
      continue;
    }
    const double *Mr = M + (size_t)row * m;
    double s0 = 0.0, s1 = 0.0;
    if (STAGED && (m & 1) == 0) {
      const double2 *M2 = reinterpret_cast<const double2 *>(Mr);
      const double2 *R2 = reinterpret_cast<const double2 *>(rc);
#pragma unroll 4
      for (int c2 = lane; c2 < (m >> 1); c2 += 32) {
        const double2 v = __ldg(M2 + c2), x = R2[c2];
        s0 = fma(v.x, x.x, s0);
        s1 = fma(v.y, x.y, s1);
      }
    } else {
      for (int c = lane; c < m; c += 32) s0 = fma(__ldg(Mr + c), STAGED ? rc[c] : (double)r[idx[c]], s0);
    }
    double sum = s0 + s1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if (lane == 0) e[idx[row]] = (T)sum;
  }
}
template <typename T>
static void dense_apply(const LevelDev &C, const double *Minv, const T *r, T *e, cudaStream_t s, const int *gate) {
  constexpr int kMaxStaged = 8192;  // 64 KB of staged FP64 input
  const int n = (int)C.g.n();
  static PerDevice smem;
  allow_smem(smem, 8 * kMaxStaged, k_dense<T, true>);
  const int rows_per_block = 8, blocks = std::max(1, std::min((n + rows_per_block - 1) / rows_per_block, 4 * sm_count()));
  if (C.cm <= kMaxStaged)
    launch_dep(k_dense<T, true>, blocks, 256, sizeof(double) * (size_t)C.cm, s, Minv, C.cidx, C.cm, n, r, e, gate);
  else
    launch_dep(k_dense<T, false>, blocks, 256, 0, s, Minv, C.cidx, C.cm, n, r, e, gate);
}
void launch_dense_apply(const LevelDev &C, const double *Minv, const double *r, double *e, cudaStream_t s,
                        const int *gate) {
  dense_apply<double>(C, Minv, r, e, s, gate);
}
void launch_dense_apply_f32(const LevelDev &C, const double *Minv, const float *r, float *e, cudaStream_t s,
                            const int *gate) {
  dense_apply<float>(C, Minv, r, e, s, gate);
}

}  // namespace cvb
