// The kernels around the solve: PoissonRHS, VolumeFlux_rev, UpdatePressure and
// the flux correction of Projection.  Element-wise arithmetic keeps the
// reference's operation order (explicit round-to-nearest intrinsics, no fused
// multiply-add); reductions are two-stage and deterministic.
#include "cvb_internal.h"
#include "intmul.cuh"
#include "launch.cuh"

namespace cvb {

static const int kT = 256;
static inline unsigned nblk(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

__device__ __forceinline__ void block_sum2(double a, double b, double *partial, int nblocks) {
  __shared__ double sh[2][kT / 32];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  if (lane == 0) { sh[0][wid] = a; sh[1][wid] = b; }
  __syncthreads();
  if (threadIdx.x < 2) {
    double v = 0.0;
    for (int w = 0; w < kT / 32; w++) v += sh[threadIdx.x][w];
    partial[(size_t)threadIdx.x * nblocks + blockIdx.x] = v;
  }
}

// v > 0.1, the IEEE compare, on the integer pipe.
__device__ __forceinline__ bool above_01(double v) {
  const long long b = __double_as_longlong(v);
  return b > 0x3FB999999999999ALL && b <= 0x7FF0000000000000LL;
}

// ((-s / dt) aj) / st 1.5 of PoissonRHS: the divisions through the divisors'
// reciprocals (RCP: both are in quot_known's range), the products on the
// integer pipe where the operands allow.
__device__ __noinline__ double rhs_slow(double s, double aj, double dt, double st) {
  return __dmul_rn(__ddiv_rn(__dmul_rn(__ddiv_rn(-s, dt), aj), st), 1.5);
}
template <bool RCP>
__device__ __forceinline__ double rhs_value(double s, double aj, double dt, double rdt, double st, double rst) {
  if constexpr (RCP) {
    bool out = false;
    const IntMulB ab = int_split_b(aj, out);
    const IntMulA qa = int_split_a(quot_known(-s, dt, rdt), out);
    if (!out) {
      double v = int_mul(qa, ab);
      if (st != 1.0) v = quot_known(v, st, rst);
      const IntMulA va = int_split_a(v, out);
      if (!out) return int_mul(va, int_split_b(1.5));
    }
  }
  return rhs_slow(s, aj, dt, st);
}

// PoissonRHS (poisson.c:1531-1550) and, with SUM, its compatibility sum
// (1554-1566), which PoissonSolver_MG does not use.  Bound by the FP64 pipe: 192^3
// without the sum 0.64 ms with the five divisions, see rhs_value.
template <bool RCP, bool SUM>
__global__ void __launch_bounds__(kT) k_rhs(Geom g, const double *__restrict__ uc, const double *__restrict__ aj,
                                            const double *__restrict__ nv, double dt, double rdt, double st, double rst,
                                            double *__restrict__ b, double *partial) {
  dep_sync();
  double acc = 0.0;
  const unsigned n = (unsigned)g.n(), pl = g.mx * g.my;
  for (unsigned p = blockIdx.x * kT + threadIdx.x; p < n; p += gridDim.x * kT) {
    const int k = p / pl, ij = p - k * pl, j = ij / g.mx, i = ij - j * g.mx;
    double v;
    if (i == 0 || i == g.mx - 1 || j == 0 || j == g.my - 1 || k == 0 || k == g.mz - 1 || above_01(nv[p])) {
      v = 0.0;
    } else {
      const size_t q = p;
      double s = __dsub_rn(uc[3 * q], uc[3 * (q - 1)]);
      s = __dadd_rn(s, uc[3 * q + 1]);
      s = __dsub_rn(s, uc[3 * (q - g.mx) + 1]);
      s = __dadd_rn(s, uc[3 * q + 2]);
      s = __dsub_rn(s, uc[3 * (q - pl) + 2]);
      v = rhs_value<RCP>(s, aj[p], dt, rdt, st, rst);
    }
    b[p] = v;
    if (SUM) acc += __ddiv_rn(__dmul_rn(__ddiv_rn(v, aj[p]), dt), 1.5);
  }
  if (SUM) block_sum2(acc, 0.0, partial, gridDim.x);
}
// partial null: without the compatibility sum
void launch_poisson_rhs(const Geom &g, const double *ucont, const double *aj, const double *nvert, double dt,
                        double st, double *b, double *partial, cudaStream_t s) {
  const bool rcp = int_mul_factor(dt) && int_mul_factor(1.0 / dt) && int_mul_factor(st) && int_mul_factor(1.0 / st);
  auto go = [&](auto k, unsigned nb) {
    launch_dep(k, nb, kT, 0, s, g, ucont, aj, nvert, dt, 1.0 / dt, st, 1.0 / st, b, partial);
  };
  if (partial) rcp ? go(k_rhs<true, true>, reduce_blocks()) : go(k_rhs<false, true>, reduce_blocks());
  else rcp ? go(k_rhs<true, false>, nblk(g.n(), kT)) : go(k_rhs<false, false>, nblk(g.n(), kT));
}

// VolumeFlux_rev sums (poisson.c:3750-3798): flux and face area over the faces
// between fluid (nvert < 0.1) and IB-layer cells (1.1 < nvert < 1.5).
__device__ __forceinline__ bool is_ib(double v) { return v > 1.5 - 0.4 && v < 1.5; }
// None of a cell's faces is between fluid and an IB layer where it and its upper
// neighbours are +0, as nearly all are: told by their bits, without the FP64
// compares that bound these kernels.
__device__ __forceinline__ bool all_fluid(double a, double b, double c, double d) {
  return (__double_as_longlong(a) | __double_as_longlong(b) | __double_as_longlong(c) | __double_as_longlong(d)) == 0;
}
__global__ void __launch_bounds__(kT) k_ib_sums(Geom g, const double *__restrict__ uc, const double *__restrict__ a3,
                                                const double *__restrict__ nv, double *partial) {
  dep_sync();
  double f = 0.0, a = 0.0;
  const size_t n = g.n();
  const unsigned pl = g.mx * g.my;
  for (unsigned p = blockIdx.x * kT + threadIdx.x; p < (unsigned)n; p += gridDim.x * kT) {
    const int k = p / pl, ij = p - k * pl, j = ij / g.mx, i = ij - j * g.mx;
    if (i < 1 || i > g.mx - 2 || j < 1 || j > g.my - 2 || k < 1 || k > g.mz - 2) continue;
    double v = nv[p];
    double e = nv[p + 1], nn = nv[p + g.mx], t = nv[p + pl];
    if (all_fluid(v, e, nn, t)) continue;
    if (v < 0.1) {
      if (is_ib(e) && i < g.mx - 2) { f += uc[3 * (size_t)p]; a += a3[p]; }
      if (is_ib(nn) && j < g.my - 2) { f += uc[3 * (size_t)p + 1]; a += a3[n + p]; }
      if (is_ib(t) && k < g.mz - 2) { f += uc[3 * (size_t)p + 2]; a += a3[2 * n + p]; }
    }
    if (is_ib(v)) {
      if (e < 0.1 && i < g.mx - 2) { f -= uc[3 * (size_t)p]; a += a3[p]; }
      if (nn < 0.1 && j < g.my - 2) { f -= uc[3 * (size_t)p + 1]; a += a3[n + p]; }
      if (t < 0.1 && k < g.mz - 2) { f -= uc[3 * (size_t)p + 2]; a += a3[2 * n + p]; }
    }
  }
  block_sum2(f, a, partial, gridDim.x);
}
void launch_ib_sums(const Geom &g, const double *ucont, const double *csi, const double *eta, const double *zet,
                    const double *nvert, double *partial, cudaStream_t s) {
  (void)eta; (void)zet;  // csi points at the [3][N] face-area block
  launch_dep(k_ib_sums, reduce_blocks(), kT, 0, s, g, ucont, csi, nvert, partial);
}

// The uniform correction of VolumeFlux_rev (poisson.c:3810-3869).
__global__ void k_ib_correct(Geom g, double *__restrict__ uc, const double *__restrict__ a3,
                             const double *__restrict__ nv, const double *__restrict__ fa, double fis, int flg) {
  dep_sync();
  const size_t n = g.n();
  const unsigned pl = g.mx * g.my;
  for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < (unsigned)n; p += gridDim.x * blockDim.x) {
    const int k = p / pl, ij = p - k * pl, j = ij / g.mx, i = ij - j * g.mx;
    if (i < 1 || i > g.mx - 2 || j < 1 || j > g.my - 2 || k < 1 || k > g.mz - 2) continue;
    double v = nv[p];
    double e = nv[p + 1], nn = nv[p + g.mx], t = nv[p + pl];
    if (all_fluid(v, e, nn, t)) continue;
    const double flux = fa[0], area = fa[1];
    const double corr = area > 1.e-15 ? (flg ? __ddiv_rn(__dadd_rn(flux, fis), area) : __ddiv_rn(flux, area)) : 0.0;
    if (v < 0.1) {
      if (is_ib(e) && i < g.mx - 2) uc[3 * (size_t)p] = __dsub_rn(uc[3 * (size_t)p], __dmul_rn(a3[p], corr));
      if (is_ib(nn) && j < g.my - 2) uc[3 * (size_t)p + 1] = __dsub_rn(uc[3 * (size_t)p + 1], __dmul_rn(a3[n + p], corr));
      if (is_ib(t) && k < g.mz - 2) uc[3 * (size_t)p + 2] = __dsub_rn(uc[3 * (size_t)p + 2], __dmul_rn(a3[2 * n + p], corr));
    }
    if (is_ib(v)) {
      if (e < 0.1 && i < g.mx - 2) uc[3 * (size_t)p] = __dadd_rn(uc[3 * (size_t)p], __dmul_rn(a3[p], corr));
      if (nn < 0.1 && j < g.my - 2) uc[3 * (size_t)p + 1] = __dadd_rn(uc[3 * (size_t)p + 1], __dmul_rn(a3[n + p], corr));
      if (t < 0.1 && k < g.mz - 2) uc[3 * (size_t)p + 2] = __dadd_rn(uc[3 * (size_t)p + 2], __dmul_rn(a3[2 * n + p], corr));
    }
  }
}
void launch_ib_correct(const Geom &g, double *ucont, const double *csi, const double *eta, const double *zet,
                       const double *nvert, const double *flux_area, double flux_intp_sum, int flg, cudaStream_t s) {
  (void)eta; (void)zet;
  launch_dep(k_ib_correct, nblk(g.n(), kT), kT, 0, s, g, ucont, csi, nvert, flux_area, flux_intp_sum, flg);
}

// UpdatePressure (poisson.c:2945-3244): p += phi inside, then the periodic ring
// copies, in the reference's order: a first round restricted to interior
// tangential indices (x, y, z), a second round over whole ring planes (x, y, z).
__global__ void k_p_add(Geom g, double *__restrict__ p, const double *__restrict__ phi) {
  size_t n = g.n();
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(q % g.mx), j = (int)((q / g.mx) % g.my), k = (int)(q / ((size_t)g.mx * g.my));
    if (i >= 1 && i <= g.mx - 2 && j >= 1 && j <= g.my - 2 && k >= 1 && k <= g.mz - 2) p[q] = __dadd_rn(p[q], phi[q]);
  }
}
// axis 0: x ring (plane over j,k); 1: y; 2: z.  restricted: tangential interior only.
__global__ void k_ring_copy(Geom g, double *__restrict__ p, double *__restrict__ phi, int axis, int restricted) {
  int a = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y * blockDim.y + threadIdx.y;
  int na = axis == 0 ? g.my : g.mx, nb = axis == 2 ? g.my : g.mz;
  if (a >= na || b >= nb) return;
  if (restricted) {
    int ma = axis == 0 ? g.my : g.mx, mb = axis == 2 ? g.my : g.mz;
    if (a < 1 || a > ma - 2 || b < 1 || b > mb - 2) return;
  }
  size_t lo, lo_src, hi, hi_src;
  if (axis == 0) { lo = g.id(0, a, b); lo_src = g.id(g.mx - 2, a, b); hi = g.id(g.mx - 1, a, b); hi_src = g.id(1, a, b); }
  else if (axis == 1) { lo = g.id(a, 0, b); lo_src = g.id(a, g.my - 2, b); hi = g.id(a, g.my - 1, b); hi_src = g.id(a, 1, b); }
  else { lo = g.id(a, b, 0); lo_src = g.id(a, b, g.mz - 2); hi = g.id(a, b, g.mz - 1); hi_src = g.id(a, b, 1); }
  p[lo] = p[lo_src]; phi[lo] = phi[lo_src];
  p[hi] = p[hi_src]; phi[hi] = phi[hi_src];
}
void launch_update_pressure(const Geom &g, double *p, double *phi, cudaStream_t s) {
  k_p_add<<<nblk(g.n(), kT), kT, 0, s>>>(g, p, phi); count_launch();
  int per[3] = {g.px, g.py, g.pz};
  if (!(per[0] || per[1] || per[2])) return;
  for (int round = 0; round < 2; round++)
    for (int axis = 0; axis < 3; axis++) {
      if (!per[axis]) continue;
      int na = axis == 0 ? g.my : g.mx, nb = axis == 2 ? g.my : g.mz;
      dim3 blk(32, 8), grd(nblk(na, 32), nblk(nb, 8));
      k_ring_copy<<<grd, blk, 0, s>>>(g, p, phi, axis, round == 0); count_launch();
    }
}

__device__ __forceinline__ double dot3(const double *a, const double *b) {
  return __dadd_rn(__dadd_rn(__dmul_rn(a[0], b[0]), __dmul_rn(a[1], b[1])), __dmul_rn(a[2], b[2]));
}
struct ProjArgs {
  Geom g;
  const double *fm[9];  // ICsi IEta IZet JCsi JEta JZet KCsi KEta KZet (Cmpnts AoS)
  const double *aj[3];  // IAj, JAj, KAj
  const double *gram;   // the face metric products (k_face_gram), or null: formed from fm
  const double *nv, *ph;
  const uint32_t *code; // the operator's codes: the derivatives' forms
  double dt, st;
  double *uc;
};

// The pressure term of face d of cell p, ((f dt) st) / 1.5 with f = sum (dp_a
// (m_a . n)) J over the three directions a, m_n the face's own: with FP64
// multiplies and the division.
__device__ __noinline__ double proj_term_fp64(const ProjArgs &A, int d, size_t p, double d1, double d2, double d3) {
  const size_t n = A.g.n();
  const double dp[3] = {d1, d2, d3}, jac = A.aj[d][p];
  double t[3];
  for (int a = 0; a < 3; a++) {
    const double gr = A.gram ? A.gram[(3 * d + a) * n + p] : dot3(A.fm[3 * d + a] + 3 * p, A.fm[4 * d] + 3 * p);
    t[a] = __dmul_rn(__dmul_rn(dp[a], gr), jac);
  }
  const double f = __dadd_rn(__dadd_rn(t[0], t[1]), t[2]);
  return __ddiv_rn(__dmul_rn(__dmul_rn(f, A.dt), A.st), 1.5);
}

// Projection's correction of face d of cell p (poisson.c:2347-2870), between p
// and its neighbour o[d] up the direction; o, l: the offsets of its neighbours
// up and down the three directions, with the reference's periodic wrap for the
// ring faces' as for the others (none: the ring holds the images).  The
// tangential derivatives' forms (central, lower, upper, none) are those of the
// operator's cross terms, kept in its codes; all three share one expression.
// INT: the products on the integer pipe (gram, the Jacobians, dt and st in its
// range), the division by 1.5 as a product with its reciprocal and one
// correction: 2/3 rounds down by a third of a unit in its last place, so x times
// it, rounded, is within an ulp of the quotient, which the correction then
// rounds correctly (quot_known).
template <bool INT>
__device__ __forceinline__ void do_face(const ProjArgs &A, int d, unsigned p) {
  const Geom &g = A.g;
  const size_t n = g.n();
  const int st[3] = {1, g.mx, g.mx * g.my};
  const int sd = d == 0 ? st[0] : d == 1 ? st[1] : st[2];
  // both cells fluid: nvert, never negative, sums to zero only if both are
  if ((__double_as_longlong(A.nv[p]) | __double_as_longlong(A.nv[p + sd])) << 1) return;
  const uint32_t c = A.code[p];
  const double *P = A.ph + p;
  double dp[3];
  int which = 0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    if (a == d) {
      dp[a] = __dsub_rn(P[sd], P[0]);
      continue;
    }
    const int br = code_branch(c, d, which++), h = br == 2 ? 0 : st[a], l = br == 3 ? 0 : -st[a];
    dp[a] = br == 0 ? 0.0
                    : scale_down(__dsub_rn(__dsub_rn(__dadd_rn(P[h], P[sd + h]), P[l]), P[sd + l]), br == 1 ? 2 : 1);
  }
  double t = 0.0;
  bool fp64 = !INT;
  if constexpr (INT) {
    const IntMulB jac = int_split_b(A.aj[d][p]);
    const double *gr = A.gram + 3 * d * n + p;
    double f = 0.0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const double v = int_mul(int_split_a(int_mul(int_split_a(dp[a], fp64), int_split_b(gr[a * n])), fp64), jac);
      f = a == 0 ? v : __dadd_rn(f, v);
    }
    f = int_mul(int_split_a(f, fp64), int_split_b(A.dt));
    f = int_mul(int_split_a(f, fp64), int_split_b(A.st));
    // an ordinary f, or the division
    const unsigned h = (unsigned)__double2hiint(f) & 0x7fffffffu;
    fp64 = fp64 || h - (623u << 20) >= (800u << 20);
    t = __dmul_rn(f, 2.0 / 3.0);
    t = __fma_rn(__fma_rn(-1.5, t, f), 2.0 / 3.0, t);
  }
  if (fp64) t = proj_term_fp64(A, d, p, dp[0], dp[1], dp[2]);
  double *u = A.uc + 3 * (size_t)p + d;
  *u = __dsub_rn(*u, t);
}

// Interior faces: each cell updates its own three upper faces (a face belongs to
// exactly one cell, so there is no write conflict).  Bound by the FP64 pipe: 39
// operations a cell, about 150 with the metric products formed here, FP64
// products and divisions (2.48 ms at 192^3).
template <bool INT>
__global__ void __launch_bounds__(128) k_projection(const __grid_constant__ ProjArgs A) {
  dep_sync();
  const Geom &g = A.g;
  const unsigned p = blockIdx.x * blockDim.x + threadIdx.x, pl = g.mx * g.my;
  if (p >= (unsigned)g.n()) return;
  const int k = p / pl, ij = p - k * pl, j = ij / g.mx, i = ij - j * g.mx;
  if (i < 1 || i > g.mx - 2 || j < 1 || j > g.my - 2 || k < 1 || k > g.mz - 2) return;
#pragma unroll 1
  for (int d = 0; d < 3; d++) {
    const int last = d == 0 ? (g.px ? g.mx - 1 : g.mx - 2) - i
                            : d == 1 ? (g.py ? g.my - 1 : g.my - 2) - j : (g.pz ? g.mz - 1 : g.mz - 2) - k;
    if (last > 0) do_face<INT>(A, d, p);
  }
}
// The periodic ring faces (poisson.c:2600-2870): the face between ring cell 0 and cell 1.
template <bool INT>
__global__ void k_projection_ring(const __grid_constant__ ProjArgs A, int axis) {
  dep_sync();
  const Geom &g = A.g;
  int a = blockIdx.x * blockDim.x + threadIdx.x + 1, b = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (a > (axis == 0 ? g.my : g.mx) - 2 || b > (axis == 2 ? g.my : g.mz) - 2) return;
  do_face<INT>(A, axis, (unsigned)(axis == 0 ? g.id(0, a, b) : axis == 1 ? g.id(a, 0, b) : g.id(a, b, 0)));
}
// gram: k_face_gram's products, or null (formed from the metrics); tame: they
// and the metrics are in intmul.cuh's range; code: the finest level's codes
void launch_projection(const Geom &g, const double *const *fm, const double *iaj, const double *jaj,
                       const double *kaj, const double *gram, bool tame, const double *nvert, const uint32_t *code,
                       const double *phi, double dt, double st, double *ucont, cudaStream_t s) {
  ProjArgs A;
  A.g = g;
  for (int q = 0; q < 9; q++) A.fm[q] = fm[q];
  A.aj[0] = iaj; A.aj[1] = jaj; A.aj[2] = kaj;
  A.gram = gram; A.nv = nvert; A.code = code; A.ph = phi; A.dt = dt; A.st = st; A.uc = ucont;
  const bool whole = gram && tame && int_mul_factor(dt) && int_mul_factor(st);
  auto go = [&](auto k) { launch_dep(k, nblk(g.n(), 128), 128, 0, s, A); };
  whole ? go(k_projection<true>) : go(k_projection<false>);
  int per[3] = {g.px, g.py, g.pz};
  for (int axis = 0; axis < 3; axis++) {
    if (!per[axis]) continue;
    int na = axis == 0 ? g.my : g.mx, nb = axis == 2 ? g.my : g.mz;
    dim3 b2(32, 8), g2(nblk(na, 32), nblk(nb, 8));
    if (whole) launch_dep(k_projection_ring<true>, g2, b2, 0, s, A, axis);
    else launch_dep(k_projection_ring<false>, g2, b2, 0, s, A, axis);
  }
}

}  // namespace cvb
