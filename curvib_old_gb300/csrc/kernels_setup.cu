// Set-up kernels: face coefficients, switching codes, FP64 stencil weights,
// y-line Thomas factors and the immersed-boundary restriction of nvert.
// Run once per problem (or whenever nvert changes); the solve reuses the result.
#include <algorithm>
#include <vector>

#include "intmul.cuh"
#include "launch.cuh"
#include "row_swaps.h"

namespace cvb {

static inline unsigned nblk(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

// g11..g33 of PoissonLHSNew (poisson.c:699-735): (metric_b . metric_a) * face
// Jacobian, and their FP32 copies, in which each cross term carries the weight of
// its form (0 none, 1/4 central, 1/2 one-sided), so that the FP32 rows need no
// per-term selection (powers of two: that scaling is exact).  *cross is set where
// any FP32 cross term is not zero.
//
// Bound by the FP64 pipe: half of the products and the conversions are on the
// integer pipe (intmul.cuh; values beyond its range take FP64 multiplies).  At 96^3
// 103 us with all of them in FP64, and 33 us more for the copies made apart.
__device__ __noinline__ void gcoef_face_fp64(const double *const (&x)[3], const double *r, double j, double (&out)[3]) {
  for (int t = 0; t < 3; t++)
    out[t] = __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(x[t][0], r[0]), __dmul_rn(x[t][1], r[1])), __dmul_rn(x[t][2], r[2])), j);
}
__device__ __forceinline__ void gcoef_face(const double *const (&x)[3], const double *r, double j, double (&out)[3]) {
  bool wild = false;
  const double r0 = r[0];
  const IntMulB r1 = int_split_b(r[1], wild), r2 = int_split_b(r[2], wild), jb = int_split_b(j, wild);
#pragma unroll
  for (int t = 0; t < 3; t++) {
    const double s = __dadd_rn(__dadd_rn(__dmul_rn(x[t][0], r0), int_mul(int_split_a(x[t][1], wild), r1)),
                               int_mul(int_split_a(x[t][2], wild), r2));
    out[t] = int_mul(int_split_a(s, wild), jb);
  }
  if (wild) gcoef_face_fp64(x, r, j, out);
}
__global__ void __launch_bounds__(128) k_gcoef(Geom g, const __grid_constant__ FaceMetrics M,
                                               const uint32_t *__restrict__ code, double *__restrict__ g9,
                                               float *__restrict__ gf, int *__restrict__ cross) {
  const size_t n = g.n(), p = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const bool in = p < n;
  bool any = false;
  if (in) {
    const uint32_t c = code[p];
    const float wgt[4] = {0.0f, 0.25f, 0.5f, 0.5f};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double *x[3] = {M.m[d][0] + 3 * p, M.m[d][1] + 3 * p, M.m[d][2] + 3 * p};
      double v[3];
      gcoef_face(x, x[d], M.aj[d][p], v);
#pragma unroll
      for (int t = 0; t < 3; t++) {
        const int q = 3 * d + t, other = d == 0 ? t - 1 : d == 1 ? (t == 2) : t;  // the cross direction's place
        float f = int_narrow(v[t]);
        if (t != d) {
          f *= wgt[code_branch(c, d, other)];
          any = any || f != 0.0f;
        }
        g9[(size_t)q * n + p] = v[t];
        gf[(size_t)q * n + p] = f;
      }
    }
  }
  if (__any_sync(0xffffffffu, any) && (threadIdx.x & 31) == 0) *cross = 1;
}

void launch_gcoef(const Geom &g, const double *const *m, const double *iaj, const double *jaj, const double *kaj,
                  const uint32_t *code, double *g9, float *gf32, int *cross, cudaStream_t s) {
  FaceMetrics M;
  for (int q = 0; q < 9; q++) M.m[q / 3][q % 3] = m[q];
  M.aj[0] = iaj; M.aj[1] = jaj; M.aj[2] = kaj;
  k_gcoef<<<nblk(g.n(), 128), 128, 0, s>>>(g, M, code, g9, gf32, cross); count_launch();
}

// The cross-derivative form of poisson.c:793-1324 from the nvert sums of the two
// cells beside the face one step up/down the cross direction (against 0.1).
struct NvSum {
  bool gt, lt;
  __device__ __forceinline__ NvSum(double s) : gt(s > 0.1), lt(s < 0.1) {}
};
__device__ __forceinline__ int cross_branch(NvSum up, NvSum dn, int c, int m, int per) {
  if ((c == m - 2 && !per) || up.gt) return (dn.lt && (c != 1 || per)) ? 2 : 0;
  if ((c == 1 && !per) || dn.gt) return up.lt ? 3 : 0;
  return 1;
}

// Bound by the FP64 pipe where sums are formed and compared (24 of each a cell); a
// cell whose 19 values are all zero, the bulk of a flow, takes neither: its sums are
// zero.
__global__ void __launch_bounds__(256) k_codes(Geom g, const double *__restrict__ nv, uint32_t *__restrict__ code) {
  const int n = (int)g.n(), p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int mx = g.mx, my = g.my, mz = g.mz, pl = mx * my;
  const int k = p / pl, j = (p - k * pl) / mx, i = p - k * pl - j * mx;
  const bool inj = j >= 1 && j <= my - 2, ink = k >= 1 && k <= mz - 2, ini = i >= 1 && i <= mx - 2;
  uint32_t c = 0;
  auto form = [&](auto NV) {
    // upper-face cross branches, for every face some interior row can use
    if (inj && ink && i <= mx - 2) {  // E face of (i,j,k)
      c |= (uint32_t)cross_branch(NV(0, 1, 0) + NV(1, 1, 0), NV(0, -1, 0) + NV(1, -1, 0), j, my, g.py) << 8;
      c |= (uint32_t)cross_branch(NV(0, 0, 1) + NV(1, 0, 1), NV(0, 0, -1) + NV(1, 0, -1), k, mz, g.pz) << 10;
    }
    if (ini && ink && j <= my - 2) {  // N face
      c |= (uint32_t)cross_branch(NV(1, 0, 0) + NV(1, 1, 0), NV(-1, 0, 0) + NV(-1, 1, 0), i, mx, g.px) << 12;
      c |= (uint32_t)cross_branch(NV(0, 0, 1) + NV(0, 1, 1), NV(0, 0, -1) + NV(0, 1, -1), k, mz, g.pz) << 14;
    }
    if (ini && inj && k <= mz - 2) {  // T face
      c |= (uint32_t)cross_branch(NV(1, 0, 0) + NV(1, 0, 1), NV(-1, 0, 0) + NV(-1, 0, 1), i, mx, g.px) << 16;
      c |= (uint32_t)cross_branch(NV(0, 1, 0) + NV(0, 1, 1), NV(0, -1, 0) + NV(0, -1, 1), j, my, g.py) << 18;
    }
    if (!(ini && inj && ink) || NvSum(NV(0, 0, 0)).gt) {
      c |= CODE_IDENTITY;
    } else {
      const int x_end = g.px ? mx - 1 : mx - 2, x_str = g.px ? 0 : 1;
      const int y_end = g.py ? my - 1 : my - 2, y_str = g.py ? 0 : 1;
      const int z_end = g.pz ? mz - 1 : mz - 2, z_str = g.pz ? 0 : 1;
      if (NvSum(NV(1, 0, 0)).lt && i != x_end) c |= CODE_ACT_E;
      if (NvSum(NV(-1, 0, 0)).lt && i != x_str) c |= CODE_ACT_W;
      if (NvSum(NV(0, 1, 0)).lt && j != y_end) c |= CODE_ACT_N;
      if (NvSum(NV(0, -1, 0)).lt && j != y_str) c |= CODE_ACT_S;
      if (NvSum(NV(0, 0, 1)).lt && k != z_end) c |= CODE_ACT_T;
      if (NvSum(NV(0, 0, -1)).lt && k != z_str) c |= CODE_ACT_B;
    }
    if (NvSum(NV(0, 0, 0)).gt) c |= CODE_BLOCKED;
    if (ini && inj && ink && NvSum(NV(0, 0, 0)).lt) c |= CODE_FLUID;
  };
  bool open = ini && inj && ink;
  if (open) {
    const int o[19] = {0,       1,      -1,     mx,      -mx,     pl,      -pl,     1 + mx,  1 - mx, -1 + mx,
                       -1 - mx, 1 + pl, 1 - pl, -1 + pl, -1 - pl, mx + pl, mx - pl, pl - mx, -pl - mx};
    long long any = 0;
#pragma unroll
    for (int m = 0; m < 19; m++) any |= __double_as_longlong(nv[p + o[m]]);
    open = (any << 1) == 0;
  }
  if (open) form([](int, int, int) { return 0.0; });
  else form([&](int a, int b, int d) { return nv[p + a + b * mx + d * pl]; });
  code[p] = c;
}

__global__ void k_weight32(size_t n, const double *__restrict__ nv, float *__restrict__ w) {
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    double wt = 1.0 - nv[p];
    w[p] = (float)(wt > 0.0 ? wt : 0.0);
  }
}
void launch_weight32(const Geom &g, const double *nvert, float *wgt32, cudaStream_t s) {
  k_weight32<<<nblk(g.n(), 256) < 4096 ? nblk(g.n(), 256) : 4096, 256, 0, s>>>(g.n(), nvert, wgt32); count_launch();
}

void launch_codes(const Geom &g, const double *nvert, uint32_t *code, cudaStream_t s) {
  k_codes<<<nblk(g.n(), 256), 256, 0, s>>>(g, nvert, code); count_launch();
}

// The colour-split copies of a level's 7-point coefficients (row32_split).
__global__ void k_split_coef(Geom g, const float *__restrict__ gf, const float *__restrict__ aj,
                             const uint32_t *__restrict__ code, float *__restrict__ cs) {
  const size_t n = g.n(), S = SplitRow::count(g);
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(p % g.mx), j = (int)((p / g.mx) % g.my), k = (int)(p / ((size_t)g.mx * g.my));
    const size_t q = SplitRow::at(g, i, j, k);
    cs[q] = gf[p];
    cs[S + q] = gf[4 * n + p];
    cs[2 * S + q] = gf[8 * n + p];
    cs[3 * S + q] = aj[p];
    cs[4 * S + q] = __uint_as_float(code[p]);
  }
}
void launch_split_coef(const Geom &g, const float *gf32, const float *ajf32, const uint32_t *code, float *cs,
                       cudaStream_t s) {
  k_split_coef<<<nblk(g.n(), 256) < 4096 ? nblk(g.n(), 256) : 4096, 256, 0, s>>>(g, gf32, ajf32, code, cs);
  count_launch();
}

// One cross term into vol[] in the reference's order (see add_cross in the oracle).
__device__ __forceinline__ void add_cross(double *vol, int br, double gg, bool up, int P, int Q, int Pu,
                                          int Qu, int Pd, int Qd) {
  const double h = scale_down<1>(gg), q = scale_down<2>(gg);
  if (br == 2) {
    if (up) { vol[P] = __dadd_rn(vol[P], h); vol[Q] = __dadd_rn(vol[Q], h); vol[Pd] = __dsub_rn(vol[Pd], h); vol[Qd] = __dsub_rn(vol[Qd], h); }
    else { vol[P] = __dsub_rn(vol[P], h); vol[Q] = __dsub_rn(vol[Q], h); vol[Pd] = __dadd_rn(vol[Pd], h); vol[Qd] = __dadd_rn(vol[Qd], h); }
  } else if (br == 3) {
    if (up) { vol[Pu] = __dadd_rn(vol[Pu], h); vol[Qu] = __dadd_rn(vol[Qu], h); vol[P] = __dsub_rn(vol[P], h); vol[Q] = __dsub_rn(vol[Q], h); }
    else { vol[Pu] = __dsub_rn(vol[Pu], h); vol[Qu] = __dsub_rn(vol[Qu], h); vol[P] = __dadd_rn(vol[P], h); vol[Q] = __dadd_rn(vol[Q], h); }
  } else if (br == 1) {
    if (up) { vol[Pu] = __dadd_rn(vol[Pu], q); vol[Qu] = __dadd_rn(vol[Qu], q); vol[Pd] = __dsub_rn(vol[Pd], q); vol[Qd] = __dsub_rn(vol[Qd], q); }
    else { vol[Pu] = __dsub_rn(vol[Pu], q); vol[Qu] = __dsub_rn(vol[Qu], q); vol[Pd] = __dadd_rn(vol[Pd], q); vol[Qd] = __dadd_rn(vol[Qd], q); }
  }
}

// The 19 matrix entries of one row, accumulated exactly as PoissonLHSNew does
// (poisson.c:789-1327), so the stored weights equal the reference's assembled
// matrix bit for bit.  Bound by the FP64 pipe, which keeps the sums; the products
// are on the integer pipe (intmul.cuh).
__global__ void k_weights(Geom g, const double *__restrict__ g9, const double *__restrict__ aj,
                          const uint32_t *__restrict__ code, double *__restrict__ w, int *__restrict__ cross) {
  size_t n = g.n();
  bool any = false;  // an edge weight that is not zero
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    uint32_t c = code[p];
    if (c & CODE_IDENTITY) {
#pragma unroll
      for (int m = 0; m < NSLOT; m++) w[(size_t)m * n + p] = (m == CP) ? 1.0 : 0.0;
      continue;
    }
    const int i = (int)p % g.mx, j = (int)p / g.mx % g.my, k = (int)p / (g.mx * g.my);
    double vol[NSLOT];
#pragma unroll
    for (int m = 0; m < NSLOT; m++) vol[m] = 0.0;
    auto G = [&](int q, size_t at) { return g9[(size_t)q * n + at]; };
    size_t pw = g.id(i - 1, j, k), ps = g.id(i, j - 1, k), pb = g.id(i, j, k - 1);
    uint32_t cw = code[pw], cs = code[ps], cb = code[pb];
    if (c & CODE_ACT_E) {
      vol[CP] = __dsub_rn(vol[CP], G(0, p)); vol[EP] = __dadd_rn(vol[EP], G(0, p));
      add_cross(vol, code_branch(c, 0, 0), G(1, p), true, CP, EP, NP, NE, SP, SE);
      add_cross(vol, code_branch(c, 0, 1), G(2, p), true, CP, EP, TP, TE, BP, BE);
    }
    if (c & CODE_ACT_W) {
      vol[CP] = __dsub_rn(vol[CP], G(0, pw)); vol[WP] = __dadd_rn(vol[WP], G(0, pw));
      add_cross(vol, code_branch(cw, 0, 0), G(1, pw), false, CP, WP, NP, NW, SP, SW);
      add_cross(vol, code_branch(cw, 0, 1), G(2, pw), false, CP, WP, TP, TW, BP, BW);
    }
    if (c & CODE_ACT_N) {
      add_cross(vol, code_branch(c, 1, 0), G(3, p), true, CP, NP, EP, NE, WP, NW);
      vol[CP] = __dsub_rn(vol[CP], G(4, p)); vol[NP] = __dadd_rn(vol[NP], G(4, p));
      add_cross(vol, code_branch(c, 1, 1), G(5, p), true, CP, NP, TP, TN, BP, BN);
    }
    if (c & CODE_ACT_S) {
      add_cross(vol, code_branch(cs, 1, 0), G(3, ps), false, CP, SP, EP, SE, WP, SW);
      vol[CP] = __dsub_rn(vol[CP], G(4, ps)); vol[SP] = __dadd_rn(vol[SP], G(4, ps));
      add_cross(vol, code_branch(cs, 1, 1), G(5, ps), false, CP, SP, TP, TS, BP, BS);
    }
    if (c & CODE_ACT_T) {
      add_cross(vol, code_branch(c, 2, 0), G(6, p), true, CP, TP, EP, TE, WP, TW);
      add_cross(vol, code_branch(c, 2, 1), G(7, p), true, CP, TP, NP, TN, SP, TS);
      vol[CP] = __dsub_rn(vol[CP], G(8, p)); vol[TP] = __dadd_rn(vol[TP], G(8, p));
    }
    if (c & CODE_ACT_B) {
      add_cross(vol, code_branch(cb, 2, 0), G(6, pb), false, CP, BP, EP, BE, WP, BW);
      add_cross(vol, code_branch(cb, 2, 1), G(7, pb), false, CP, BP, NP, BN, SP, BS);
      vol[CP] = __dsub_rn(vol[CP], G(8, pb)); vol[BP] = __dadd_rn(vol[BP], G(8, pb));
    }
    const double a = -aj[p];
    bool wild = false;
    const IntMulB ab = int_split_b(a, wild);
    double r[NSLOT];
#pragma unroll
    for (int m = 0; m < NSLOT; m++) r[m] = int_mul(int_split_a(vol[m], wild), ab);
    if (wild) {
#pragma unroll
      for (int m = 0; m < NSLOT; m++) r[m] = __dmul_rn(vol[m], a);
    }
#pragma unroll
    for (int m = 0; m < NSLOT; m++) {
      w[(size_t)m * n + p] = r[m];
      if (m >= NE) any = any || (__double_as_longlong(r[m]) << 1) != 0;
    }
  }
  if (any) *cross = 1;
}

void launch_weights(const Geom &g, const double *g9, const double *aj, const uint32_t *code, double *w64, int *cross,
                    cudaStream_t s) {
  k_weights<<<nblk(g.n(), 128), 128, 0, s>>>(g, g9, aj, code, w64, cross); count_launch();
}

// Thomas factors of the in-line (j) part of each row: a_j = w[SP], m_j, c'_j.
// Couplings that wrap around a periodic y seam stay outside the line solve.
//
// A thread a line, a chain of one division a row: bound by that chain's latency, so
// rows are read four ahead of it and written four at a time.
__global__ void __launch_bounds__(32) k_line_factors(Geom g, const double *__restrict__ w, double *__restrict__ l64,
                                                     float *__restrict__ l32) {
  const size_t n = g.n();
  const LineFac F = LineFac::of(g);
  const int Q = F.Q, t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.mx * g.mz) return;
  const int i = t % g.mx, k = t / g.mx;
  const size_t base = F.line(i, k), col = g.id(i, 1, k);
  double an[4], bn[4], cn[4], cprev = 0.0;
  auto read = [&](int q0) {
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const bool in = q0 + u < g.my - 2;
      const size_t p = col + (size_t)(in ? q0 + u : 0) * g.mx;
      an[u] = in ? w[(size_t)SP * n + p] : 0.0;
      bn[u] = in ? w[(size_t)CP * n + p] : 0.0;
      cn[u] = in ? w[(size_t)NP * n + p] : 0.0;
    }
  };
  read(0);
  for (int q0 = 0; q0 < Q; q0 += 4) {
    double a[4], b[4], c[4], minv[4], cp[4];
#pragma unroll
    for (int u = 0; u < 4; u++) a[u] = an[u], b[u] = bn[u], c[u] = cn[u];
    if (q0 + 4 < Q) read(q0 + 4);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int j = q0 + u + 1;
      if (g.py && j == 1) a[u] = 0.0;
      if (g.py && j == g.my - 2) c[u] = 0.0;
      const double m = b[u] - a[u] * cprev;
      // an empty row (a fluid cell cut off from all its neighbours) has no
      // pivot: the sweep leaves it unchanged instead of dividing by zero; the
      // rows beyond the line (a = b = c = 0) pad the run with zeros likewise
      minv[u] = m != 0.0 ? 1.0 / m : 0.0;
      cprev = cp[u] = c[u] * minv[u];
    }
    const double *v[3] = {a, minv, cp};
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const size_t q = base + (size_t)r * Q + q0;
      reinterpret_cast<double2 *>(l64 + q)[0] = make_double2(v[r][0], v[r][1]);
      reinterpret_cast<double2 *>(l64 + q)[1] = make_double2(v[r][2], v[r][3]);
      *reinterpret_cast<float4 *>(l32 + q) = make_float4((float)v[r][0], (float)v[r][1], (float)v[r][2], (float)v[r][3]);
    }
  }
}

void launch_line_factors(const Geom &g, const double *w64, double *line64, float *line32,
                         cudaStream_t s) {
  int lines = g.mx * g.mz;
  k_line_factors<<<nblk(lines, 32), 32, 0, s>>>(g, w64, line64, line32); count_launch();
}

__global__ void k_to_f32(const double *__restrict__ a, float *__restrict__ b, size_t n) {
  dep_sync();
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x)
    b[p] = (float)a[p];
}
void launch_to_f32(const double *a, float *b, size_t n, cudaStream_t s) {
  launch_dep(k_to_f32, dim3(nblk(n, 256) < 4096 ? nblk(n, 256) : 4096), 256, 0, s, a, b, n);
}
// The FP32 V-cycle's result as the FP64 basis vector: the widening on the integer
// pipe, four cells a thread (17 + 35 MB on 4.4 M cells).
__global__ void __launch_bounds__(256) k_to_f64(const float *__restrict__ a, double *__restrict__ b, size_t n) {
  dep_sync();
  const size_t p = 4 * (blockIdx.x * (size_t)blockDim.x + threadIdx.x);
  if (p + 4 <= n) {  // both arrays are whole allocations: aligned
    const float4 f = *reinterpret_cast<const float4 *>(a + p);
    double2 *o = reinterpret_cast<double2 *>(b + p);
    o[0] = make_double2(int_widen(f.x), int_widen(f.y));
    o[1] = make_double2(int_widen(f.z), int_widen(f.w));
  } else {
    for (size_t q = p; q < n; q++) b[q] = int_widen(a[q]);
  }
}
void launch_f32_to_f64(const float *a, double *b, size_t n, cudaStream_t s) {
  launch_dep(k_to_f64, nblk((n + 3) / 4, 256), 256, 0, s, a, b, n);
}

// MyNvertRestriction (poisson.c:1662-1773): a coarse cell is blocked (1) when the
// product of its 8 children's nvert exceeds 0.1; then a fluid coarse cell pinched
// between blocked cells in all three directions is blocked too (second pass reads
// the first pass's result, as the reference's G2L copy does).
__global__ void k_nvert_pass1(Geom F, const double *__restrict__ nf, Geom C, int isc, int jsc, int ksc,
                              double *__restrict__ nc) {
  size_t n = C.n();
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(p % C.mx), j = (int)((p / C.mx) % C.my), k = (int)(p / ((size_t)C.mx * C.my));
    double v = 0.0;
    if (i >= 1 && i <= C.mx - 2 && j >= 1 && j <= C.my - 2 && k >= 1 && k <= C.mz - 2) {
      int ih = isc ? i : 2 * i, jh = jsc ? j : 2 * j, kh = ksc ? k : 2 * k;
      int ia = isc ? 0 : 1, ja = jsc ? 0 : 1, ka = ksc ? 0 : 1;
      auto N = [&](int a, int b, int c) { return nf[F.id(a, b, c)]; };
      double prod = N(ih, jh, kh) * N(ih - ia, jh, kh) * N(ih, jh - ja, kh) * N(ih, jh, kh - ka) *
                    N(ih - ia, jh - ja, kh) * N(ih - ia, jh, kh - ka) * N(ih, jh - ja, kh - ka) *
                    N(ih - ia, jh - ja, kh - ka);
      if (prod > 0.1) v = 1.0;
    }
    nc[p] = v;
  }
}
__global__ void k_nvert_pass2(Geom C, const double *__restrict__ snap, double *__restrict__ nc) {
  size_t n = C.n();
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(p % C.mx), j = (int)((p / C.mx) % C.my), k = (int)(p / ((size_t)C.mx * C.my));
    if (i >= 1 && i <= C.mx - 2 && j >= 1 && j <= C.my - 2 && k >= 1 && k <= C.mz - 2 && snap[p] < 0.1) {
      if (snap[C.id(i + 1, j, k)] + snap[C.id(i - 1, j, k)] > 1.1 &&
          snap[C.id(i, j + 1, k)] + snap[C.id(i, j - 1, k)] > 1.1 &&
          snap[C.id(i, j, k + 1)] + snap[C.id(i, j, k - 1)] > 1.1)
        nc[p] = 1.0;
    }
  }
}

void launch_nvert_restrict(const Geom &fine, const double *nvf, const Geom &coarse, int isc, int jsc,
                           int ksc, double *nvc, double *tmp, cudaStream_t s) {
  k_nvert_pass1<<<nblk(coarse.n(), 256), 256, 0, s>>>(fine, nvf, coarse, isc, jsc, ksc, tmp); count_launch();
  cudaMemcpyAsync(nvc, tmp, sizeof(double) * coarse.n(), cudaMemcpyDeviceToDevice, s);
  k_nvert_pass2<<<nblk(coarse.n(), 256), 256, 0, s>>>(coarse, tmp, nvc); count_launch();
}

}  // namespace cvb

namespace cvb {

// ------------------------------------------------------------------ dense inverse
// Gauss-Jordan inversion in place with partial pivoting, kGjW columns per step,
// for the coarsest level's matrix.  Step c0 takes the columns c0 .. c0 + w - 1:
//  - k_gj_panel (one block): LU elimination of those columns' rows from c0 down,
//    in shared memory, picks the pivot rows (the largest entry, the first of
//    equal ones, as column by column); the rows are swapped into place, the
//    pivot block D inverted, and the columns (the multipliers F) and the pivot
//    rows (B, the unit matrix in the panel's own columns) staged, so that no
//    thread of the next kernel reads what another writes;
//  - k_gj_update: R = D^-1 B replaces the pivot rows, and every other row
//    becomes its own (zero in the panel's columns) minus F R.
// The row swaps become column swaps of the result, undone by k_gj_unpermute
// from the composed column map.
//
// The update is bound by the FP64 pipe (n^3 multiply-adds in all), the panel by
// its n dependent steps on one SM.  Set-up of the coarsest solver, all in: 216
// unknowns 0.63 ms (3.8 inverted on the host), 1,024 6.6 ms, 4,096 170 ms (24 and
// 531 ms with one column a step: 2 n launches, n passes over the matrix, and
// the matrix formed on the host).
constexpr int kGjThreads = 1024, kGjW = 8;
// Panels of kGjW columns (64 bytes a row) of up to this many rows fit in shared
// memory; beyond, w shrinks.
constexpr int kGjSmemRows = 3200;

// The better pivot of two (magnitude as a bit pattern, row): the larger, the
// first of equal ones.  Magnitudes order as their patterns; a NaN counts as 0.
__device__ __forceinline__ unsigned long long gj_magnitude(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffULL;
  return b > 0x7ff0000000000000ULL ? 0 : b;
}
__device__ __forceinline__ void gj_better(unsigned long long &best, int &row, unsigned long long v, int r) {
  if (v > best || (v == best && r < row)) { best = v; row = r; }
}
__device__ __forceinline__ void gj_warp_best(unsigned long long &best, int &row) {
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_down_sync(0xffffffffu, best, o);
    const int r = __shfl_down_sync(0xffffffffu, row, o);
    gj_better(best, row, v, r);
  }
}

__global__ void __launch_bounds__(kGjThreads) k_gj_panel(double *__restrict__ A, int n, int c0, int w,
                                                         int *__restrict__ perm, double *__restrict__ F,
                                                         double *__restrict__ B, double *__restrict__ Dinv,
                                                         int *__restrict__ status) {
  extern __shared__ double S[];  // the panel's columns from row c0 down, [w][m | 1]
  __shared__ unsigned long long sv[32];
  __shared__ int si[32];
  __shared__ int piv[kGjW];
  __shared__ double rcp[kGjW];
  __shared__ double D[kGjW][2 * kGjW];
  dep_sync();
  if (*status) return;
  const int nt = blockDim.x, t = threadIdx.x, lane = t & 31, wid = t >> 5, m = n - c0, mp = m | 1;
#pragma unroll 4
  for (int e = t; e < m * kGjW; e += nt) {
    const int r = e / kGjW, q = e % kGjW;
    if (q < w) S[q * mp + r] = A[(size_t)(c0 + r) * n + c0 + q];
  }
  __syncthreads();
  unsigned long long best = 0;
  int row = m;
  for (int r = t; r < m; r += nt) gj_better(best, row, gj_magnitude(S[r]), r);
  for (int s = 0; s < w; s++) {
    gj_warp_best(best, row);
    if (lane == 0) { sv[wid] = best; si[wid] = row; }
    __syncthreads();
    if (wid == 0) {
      best = lane < nt / 32 ? sv[lane] : 0;
      row = lane < nt / 32 ? si[lane] : m;
      gj_warp_best(best, row);
      if (lane == 0) {
        piv[s] = best > 0 ? row : -1;
        if (best > 0) rcp[s] = 1.0 / S[s * mp + row];
      }
    }
    __syncthreads();
    const int p = piv[s];
    if (p < 0) {
      if (t == 0) *status = 1;
      return;
    }
    if (p != s) {
      if (t < w) {
        const double v = S[t * mp + s];
        S[t * mp + s] = S[t * mp + p];
        S[t * mp + p] = v;
      }
      __syncthreads();
    }
    // eliminate, and look for the next column's pivot on the way
    best = 0;
    row = m;
    if (s + 1 < w)
      for (int r = s + 1 + t; r < m; r += nt) {
        const double f = -S[s * mp + r] * rcp[s];
        for (int q = s + 1; q < w; q++) {
          const double v = fma(f, S[q * mp + s], S[q * mp + r]);
          S[q * mp + r] = v;
          if (q == s + 1) gj_better(best, row, gj_magnitude(v), r);
        }
      }
    __syncthreads();
  }
  if (t < w) perm[c0 + t] = c0 + piv[t];
  bool moved = false;
  for (int s = 0; s < w; s++) moved = moved || piv[s] != s;
  if (moved) {
    for (int q = t; q < n; q += nt)
      for (int s = 0; s < w; s++) {
        const int p = piv[s];
        if (p == s) continue;
        const double v = A[(size_t)(c0 + s) * n + q];
        A[(size_t)(c0 + s) * n + q] = A[(size_t)(c0 + p) * n + q];
        A[(size_t)(c0 + p) * n + q] = v;
      }
    __syncthreads();
  }
#pragma unroll 4
  for (int e = t; e < n * kGjW; e += nt) {
    const int r = e / kGjW, q = e % kGjW;
    F[e] = q < w ? A[(size_t)r * n + c0 + q] : 0.0;
  }
  for (int s = 0; s < kGjW; s++)
    for (int q = t; q < n; q += nt)
      B[(size_t)s * n + q] =
          q >= c0 && q < c0 + w ? (q - c0 == s ? 1.0 : 0.0) : s < w ? A[(size_t)(c0 + s) * n + q] : 0.0;
  // D and its inverse: Gauss-Jordan beside the unit matrix, in the order of the
  // pivots just found, whose reciprocals are at hand; the unit matrix beyond w
  const int r = t / (2 * kGjW), q = t % (2 * kGjW);
  const bool mine = t < kGjW * 2 * kGjW;
  double d = 0.0;
  if (mine) {
    d = q < kGjW ? (r < w && q < w ? A[(size_t)(c0 + r) * n + c0 + q] : (r == q ? 1.0 : 0.0))
                 : (q - kGjW == r ? 1.0 : 0.0);
    D[r][q] = d;
  }
  __syncthreads();
  for (int s = 0; s < w; s++) {
    if (mine) {
      const double pr = D[s][q] * rcp[s];
      d = r == s ? pr : fma(-D[r][s], pr, d);
    }
    __syncthreads();
    if (mine) D[r][q] = d;
    __syncthreads();
  }
  if (t < kGjW * kGjW) Dinv[t] = D[t / kGjW][kGjW + t % kGjW];
}

// A T x T tile per block, (T / 16)^2 entries a thread (columns 16 apart).
template <int T>
__global__ void __launch_bounds__(256) k_gj_update(double *__restrict__ A, int n, int c0, int w,
                                                   const double *__restrict__ F, const double *__restrict__ B,
                                                   const double *__restrict__ Dinv, const int *__restrict__ status) {
  constexpr int E = T / 16;
  __shared__ double sR[kGjW][T], sF[T][kGjW + 1], sD[kGjW * kGjW];
  dep_sync();
  if (*status) return;
  const int t = threadIdx.x, q0 = blockIdx.x * T, r0 = blockIdx.y * T;
  if (t < kGjW * kGjW) sD[t] = Dinv[t];
  for (int e = t; e < T * kGjW; e += 256) {
    const int r = e / kGjW;
    sF[r][e % kGjW] = r0 + r < n ? F[(size_t)r0 * kGjW + e] : 0.0;
  }
  __syncthreads();
  for (int e = t; e < kGjW * T; e += 256) {
    const int s = e / T, q = e % T;
    double v = 0.0;
    if (q0 + q < n)
      for (int u = 0; u < kGjW; u++) v = fma(sD[s * kGjW + u], B[(size_t)u * n + q0 + q], v);
    sR[s][q] = v;
  }
  __syncthreads();
  const int tx = t % 16, ty = t / 16;
  double acc[E][E];
#pragma unroll
  for (int a = 0; a < E; a++)
#pragma unroll
    for (int b = 0; b < E; b++) {
      const int r = r0 + ty * E + a, q = q0 + tx + 16 * b;
      acc[a][b] = r < n && q < n && !(q >= c0 && q < c0 + w) ? A[(size_t)r * n + q] : 0.0;
    }
#pragma unroll
  for (int s = 0; s < kGjW; s++) {
    double f[E], p[E];
#pragma unroll
    for (int a = 0; a < E; a++) f[a] = sF[ty * E + a][s];
#pragma unroll
    for (int b = 0; b < E; b++) p[b] = sR[s][tx + 16 * b];
#pragma unroll
    for (int a = 0; a < E; a++)
#pragma unroll
      for (int b = 0; b < E; b++) acc[a][b] = fma(-f[a], p[b], acc[a][b]);
  }
#pragma unroll
  for (int a = 0; a < E; a++)
#pragma unroll
    for (int b = 0; b < E; b++) {
      const int r = r0 + ty * E + a, q = q0 + tx + 16 * b;
      if (r < n && q < n) A[(size_t)r * n + q] = r >= c0 && r < c0 + w ? sR[r - c0][tx + 16 * b] : acc[a][b];
    }
}

__global__ void k_gj_unpermute(const double *__restrict__ A, int n, const int *__restrict__ colmap,
                               double *__restrict__ out) {
  const size_t nn = (size_t)n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < nn; e += (size_t)gridDim.x * blockDim.x) {
    int r = (int)(e / n), q = (int)(e % n);
    out[e] = A[(size_t)r * n + colmap[q]];
  }
}

size_t dense_inverse_doubles(int n) { return 2 * (size_t)kGjW * n + kGjW * kGjW; }

// Inverts the n x n row-major A (device, overwritten) into out (device).
// perm / colmap are n ints, work dense_inverse_doubles(n) doubles, status one
// int (device).  Returns false if a pivot column was all zero (a singular
// matrix), or a kernel did not run (the CUDA error stays for the caller).
bool device_dense_inverse(double *A, int n, double *out, int *perm, int *colmap, double *work, int *status,
                          cudaStream_t s) {
  static PerDevice smem;
  allow_smem(smem, kGjSmemRows * kGjW * 8, k_gj_panel);
  double *F = work, *B = F + (size_t)kGjW * n, *Dinv = B + (size_t)kGjW * n;
  cudaMemsetAsync(status, 0, sizeof(int), s);
  cudaMemsetAsync(perm, 0xff, sizeof(int) * n, s);  // -1: no row
  // the largest tile that still gives every SM a block (216 unknowns: 16 blocks of
  // 64 x 64 12 us a step)
  const unsigned tile = n >= 64 * 12 ? 64 : n >= 32 * 12 ? 32 : 16, tiles = (n + tile - 1) / tile;
  for (int c0 = 0; c0 < n;) {
    int w = kGjW;
    while (w > 1 && (long long)((n - c0) | 1) * w > (long long)kGjSmemRows * kGjW) w--;
    if (w > n - c0) w = n - c0;
    // fewer warps meet at a step's barriers where a row a thread takes fewer
    const int threads = std::min(kGjThreads, std::max(256, (n - c0 + 31) / 32 * 32));
    launch_dep(k_gj_panel, 1, threads, sizeof(double) * (size_t)((n - c0) | 1) * w, s, A, n, c0, w, perm, F, B, Dinv,
               status);
    auto update = [&](auto k) {
      launch_dep(k, dim3(tiles, tiles), 256, 0, s, A, n, c0, w, (const double *)F, (const double *)B,
                 (const double *)Dinv, (const int *)status);
    };
    if (tile == 64) update(k_gj_update<64>);
    else if (tile == 32) update(k_gj_update<32>);
    else update(k_gj_update<16>);
    c0 += w;
  }
  if (cudaPeekAtLastError() != cudaSuccess) return false;  // a launch failed
  int h_status = 0;
  std::vector<int> h_perm(n), map(n);
  cudaMemcpyAsync(&h_status, status, sizeof(int), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(h_perm.data(), perm, sizeof(int) * n, cudaMemcpyDeviceToHost, s);
  if (cudaStreamSynchronize(s) != cudaSuccess || h_status) return false;
  if (!undo_row_swaps(h_perm.data(), n, map.data())) return false;
  cudaMemcpyAsync(colmap, map.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s);
  const unsigned eb = (unsigned)std::min<size_t>(((size_t)n * n + 255) / 256, (size_t)152 * 16);
  k_gj_unpermute<<<eb, 256, 0, s>>>(A, n, colmap, out); count_launch();
  return cudaStreamSynchronize(s) == cudaSuccess;
}

// The coarsest level's dense matrix: row r of the m inverted cells idx[r] holds
// the level's 19 weights at its neighbours' columns (cols; -1: a neighbour that
// is not inverted, whose weight is zero) and sv0 / sv1 more at every column of
// its own fluid region; a row with no region is an identity row.
__global__ void __launch_bounds__(256) k_coarse_fill(int m, const int *__restrict__ region, double sv0, double sv1,
                                                     double *__restrict__ A) {
  dep_sync();
  const size_t mm = (size_t)m * m;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < mm; e += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(e / m), q = (int)(e % m), reg = region[r];
    A[e] = reg >= 0 && reg == region[q] ? (reg ? sv1 : sv0) : 0.0;
  }
}
__global__ void __launch_bounds__(128) k_coarse_rows(int m, int n, const int *__restrict__ idx,
                                                     const int *__restrict__ region, const int *__restrict__ cols,
                                                     const double *__restrict__ w, double *__restrict__ A) {
  dep_sync();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= m) return;
  if (region[r] < 0) {
    A[(size_t)r * m + r] = 1.0;
    return;
  }
  const int p = idx[r];
  for (int q = 0; q < NSLOT; q++) {
    const int c = cols[r * NSLOT + q];
    if (c >= 0) A[(size_t)r * m + c] += w[(size_t)q * n + p];
  }
}
void launch_coarse_matrix(int m, int n, const int *idx, const int *region, const int *cols, double sv0, double sv1,
                          const double *w64, double *A, cudaStream_t s) {
  const size_t mm = (size_t)m * m;
  launch_dep(k_coarse_fill, dim3((unsigned)std::min<size_t>((mm + 255) / 256, (size_t)152 * 16)), 256, 0, s, m, region,
             sv0, sv1, A);
  launch_dep(k_coarse_rows, dim3((m + 127) / 128), 128, 0, s, m, n, idx, region, cols, w64, A);
}

}  // namespace cvb
