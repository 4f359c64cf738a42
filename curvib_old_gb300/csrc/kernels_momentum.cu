// The momentum right-hand side of the fractional step on the finest level, for
// boxes with no periodic face: Viscous (rhs.c:1947-2566, laminar), FormFunction1
// (rhs.c:2567-3351) and CalcRHS (implicitsolver.c:6449-6713).  FP64, one thread
// per cell.  This file is compiled without multiply-add contraction
// (--fmad=false, build.py), so every product and sum rounds on its own in the
// order the expressions are written -- the reference's C order -- and the
// results equal the reference's bit for bit.
#include "cvb_internal.h"
#include "intmul.cuh"
#include "launch.cuh"

namespace cvb {

namespace {

inline unsigned blocks_for(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

// v > 0.5 && v < 7, on the integer pipe (the kernels here are bound by the
// FP64 one).  As signed 64-bit integers, the bit patterns of doubles of one
// sign compare as the values do; every value with the sign bit (negatives, -0,
// a NaN) lies below 0.5's pattern, and a NaN without it above 7's, so the
// result is the two comparisons', NaN included.
__device__ __forceinline__ bool visc_blocked(double v) {
  const long long b = __double_as_longlong(v);
  return b > 0x3FE0000000000000LL && b < 0x401C000000000000LL;
}

// v > c and v < c for c = 0.1, on the integer pipe.  For c > 0: a pattern
// above c's is a larger positive value, +inf, or a NaN without the sign bit
// (above +inf's pattern), which compares false; a pattern below c's is a
// smaller value of either sign, or a NaN with the sign bit (between -inf's
// pattern and 0 as signed integers), which compares false.
constexpr long long kBits01 = 0x3FB999999999999ALL, kBitsInf = 0x7FF0000000000000LL,
                    kBitsNegInf = (long long)0xFFF0000000000000ULL;
__device__ __forceinline__ bool gt_01(double v) {
  const long long b = __double_as_longlong(v);
  return b > kBits01 && b <= kBitsInf;
}
__device__ __forceinline__ bool lt_01(double v) {
  const long long b = __double_as_longlong(v);
  return b < kBits01 && !(b > kBitsNegInf && b < 0);
}

}  // namespace

namespace {

// One face of Viscous: the differences of ucat across face d of cell P into
// D[t][c] (t the direction), one-sided along its two tangential directions
// next to cells with nvert in (0.5, 7).
__device__ __forceinline__ void visc_differences(const long (&st)[3], int d, long sd, long P,
                                                 const double *__restrict__ nv, const double *__restrict__ ucat,
                                                 double (&D)[3][3]) {
#pragma unroll
  for (int t = 0; t < 3; t++) {
    if (t == d) {
#pragma unroll
      for (int c = 0; c < 3; c++) D[t][c] = ucat[3 * (P + sd) + c] - ucat[3 * P + c];
      continue;
    }
    const long s = st[t];
    const bool up = visc_blocked(nv[P + s]) || visc_blocked(nv[P + sd + s]);
    const bool dn = visc_blocked(nv[P - s]) || visc_blocked(nv[P + sd - s]);
    // one expression for the three forms, on the cells each takes
    const long h = up ? 0 : s, l = !up && dn ? 0 : -s;
    const int half = up || dn;
#pragma unroll
    for (int c = 0; c < 3; c++) {
#define U(off) ucat[3 * (P + (off)) + c]
      D[t][c] = scale_down(U(sd + h) + U(h) - U(sd + l) - U(l), half ? 1 : 2);
#undef U
    }
  }
}

// The flux of face d of cell P from its differences, with FP64 multiplies.
__device__ __noinline__ void visc_flux_fp64(const FaceMetrics &M, int d, long P, size_t n,
                                            const double *__restrict__ gram, double nu, const double (&D)[3][3],
                                            double (&v)[3]) {
  const double *m0 = M.m[d][0] + 3 * P, *m1 = M.m[d][1] + 3 * P, *m2 = M.m[d][2] + 3 * P, *nd = M.m[d][d] + 3 * P;
  const double *g = gram + (size_t)(3 * d) * n + P;
  const double ajc = M.aj[d][P];
  for (int c = 0; c < 3; c++) {
    double r[3];
    for (int q = 0; q < 3; q++) r[q] = D[0][q] * m0[c] + D[1][q] * m1[c] + D[2][q] * m2[c];
    v[c] = 0;
    v[c] += (g[0] * D[0][c] + g[n] * D[1][c] + g[2 * n] * D[2][c] + r[0] * nd[0] + r[1] * nd[1] + r[2] * nd[2]) *
            ajc * (nu);
  }
}

}  // namespace

// The viscous flux of every face (rhs.c:2056-2487): face d of cell P, between P
// and P + e_d, into fp[(3 d + c) N + P].  Bound by the FP64 pipe: of a face's
// 105 operations (21 sums for the differences, 45 for r, 39 for the flux) the
// 51 products go to the integer pipe (INT: intmul.cuh, for grids whose metrics
// are in its range), beside the 54 sums, and the leading 0 + v of the
// reference's accumulation, which only turns -0 into +0, to an integer compare.
// A face with a value out of that range takes the FP64 multiplies.  Viscous on
// the 192^3 box: 4.68 ms with FP64 multiplies, 2.83 ms so (the sums alone keep
// the FP64 pipe busy for 1.9 ms).  Four blocks per SM (128 registers): three
// (148 registers, nothing limited) 3.15 ms, five (spills) 2.88 ms.
template <bool INT>
__global__ void __launch_bounds__(128, 4) k_visc_faces(Geom g, const double *__restrict__ nv,
                                                       const double *__restrict__ ucat,
                                                       const __grid_constant__ FaceMetrics M,
                                                       const double *__restrict__ gram, double nu,
                                                       double *__restrict__ fp) {
  dep_sync();
  const size_t n = g.n();
  const long st[3] = {1, g.mx, (long)g.mx * g.my};
  const size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int pl = g.mx * g.my, k = (int)e / pl, j = ((int)e - k * pl) / g.mx, i = (int)e - k * pl - j * g.mx;
  const long P = (long)e;
  const FaceDirs dirs = FaceDirs::of_block();
  // the directions one after another, not unrolled: three copies of the
  // products' code would not fit the instruction cache
#pragma unroll 1
  for (int d = dirs.first; d < dirs.end; d++) {
    const bool in = i <= g.mx - 2 && j <= g.my - 2 && k <= g.mz - 2 && (d == 0 || i >= 1) && (d == 1 || j >= 1) &&
                    (d == 2 || k >= 1);
    if (!in) continue;
    double D[3][3], v[3];
    visc_differences(st, d, d == 0 ? st[0] : d == 1 ? st[1] : st[2], P, nv, ucat, D);
    bool fp64 = !INT;
    if constexpr (INT) {
      IntMulA Da[3][3];
      IntMulB Nb[3];
#pragma unroll
      for (int t = 0; t < 3; t++)
#pragma unroll
        for (int c = 0; c < 3; c++) Da[t][c] = int_split_a(D[t][c], fp64);
      {
        IntMulB Gb[3];
#pragma unroll
        for (int t = 0; t < 3; t++) Gb[t] = int_split_b(gram[(size_t)(3 * d + t) * n + e]);
#pragma unroll
        for (int c = 0; c < 3; c++)
          v[c] = int_mul(Da[0][c], Gb[0]) + int_mul(Da[1][c], Gb[1]) + int_mul(Da[2][c], Gb[2]);
      }
#pragma unroll
      for (int t = 0; t < 3; t++) Nb[t] = int_split_b(M.m[d][d][3 * P + t]);
      const IntMulB ajc = int_split_b(M.aj[d][P]), nub = int_split_b(nu);
#pragma unroll
      for (int c = 0; c < 3; c++) {
        IntMulB Mb[3];
#pragma unroll
        for (int t = 0; t < 3; t++) Mb[t] = int_split_b(M.m[d][t][3 * P + c]);
        double s = c == 0 ? v[0] : c == 1 ? v[1] : v[2];
#pragma unroll
        for (int t = 0; t < 3; t++) {
          const double r = int_mul(Da[0][t], Mb[0]) + int_mul(Da[1][t], Mb[1]) + int_mul(Da[2][t], Mb[2]);
          s = s + int_mul(int_split_a(r, fp64), Nb[t]);
        }
        s = int_mul(int_split_a(s, fp64), ajc);
        s = int_mul(int_split_a(s, fp64), nub);
        // 0 + s
        if (__double_as_longlong(s) == (long long)0x8000000000000000ULL) s = 0.;
        if (c == 0) v[0] = s;
        else if (c == 1) v[1] = s;
        else v[2] = s;
      }
    }
    if (fp64) visc_flux_fp64(M, d, P, n, gram, nu, D, v);
#pragma unroll
    for (int c = 0; c < 3; c++) fp[(size_t)(3 * d + c) * n + e] = v[c];
  }
}

// Component c of visc at interior cell e: the flux differences over the cell
// (rhs.c:2490-2511).
__device__ __forceinline__ double visc_cell(const Geom &g, const double *__restrict__ fp, size_t e, int c) {
  const size_t n = g.n(), w = e - 1, s = e - g.mx, b = e - (size_t)g.mx * g.my;
  return fp[(size_t)c * n + e] - fp[(size_t)c * n + w] + fp[(size_t)(3 + c) * n + e] - fp[(size_t)(3 + c) * n + s] +
         fp[(size_t)(6 + c) * n + e] - fp[(size_t)(6 + c) * n + b];
}

// visc, 0 on the ring (the reference's VecSet before the loops).
__global__ void k_visc_div(Geom g, const double *__restrict__ fp, double *__restrict__ visc) {
  dep_sync();
  const size_t n = g.n();
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(e % g.mx), j = (int)((e / g.mx) % g.my), k = (int)(e / ((size_t)g.mx * g.my));
    const bool in = i >= 1 && i <= g.mx - 2 && j >= 1 && j <= g.my - 2 && k >= 1 && k <= g.mz - 2;
    for (int c = 0; c < 3; c++) visc[3 * e + c] = in ? visc_cell(g, fp, e, c) : 0.0;
  }
}

// The metric products the viscous flux and FormFunction1's pressure gradient
// both form on every face (rhs.c's g11, g21, g31 of the face): gram[(3 d + a)
// N + P] = M[d][a] . M[d][d] at cell P (x, y, z products summed in that
// order, as the two kernels wrote them).  They depend on the grid alone, so
// they are formed once per grid and read back, the same values bit for bit.
// *wild counts the metrics, Jacobians and products that intmul.cuh's products
// do not take: neither zero nor within its range of exponents.
__global__ void k_face_gram(Geom g, FaceMetrics M, double *__restrict__ gram, int *__restrict__ wild) {
  const size_t n = g.n();
  const int m[3] = {g.mx, g.my, g.mz};
  bool out = false;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const int q[3] = {(int)(e % g.mx), (int)((e / g.mx) % g.my), (int)(e / ((size_t)g.mx * g.my))};
    for (int d = 0; d < 3; d++) {
      bool face = q[d] <= m[d] - 2;  // a face k_visc_faces forms
      for (int t = 0; t < 3; t++)
        if (t != d) face = face && q[t] >= 1 && q[t] <= m[t] - 2;
      auto look = [&](double v) {
        if (face) int_split_a(v, out);
      };
      const double *nd = M.m[d][d] + 3 * e;
      for (int a = 0; a < 3; a++) {
        const double *mm = M.m[d][a] + 3 * e;
        const double v = mm[0] * nd[0] + mm[1] * nd[1] + mm[2] * nd[2];
        gram[(size_t)(3 * d + a) * n + e] = v;
        look(v);
        for (int c = 0; c < 3; c++) look(mm[c]);
      }
      look(M.aj[d][e]);
    }
  }
  if (out) atomicAdd(wild, 1);
}

void launch_face_gram(const Geom &g, const double *const *fm, const double *iaj, const double *jaj,
                      const double *kaj, double *gram, int *wild, cudaStream_t s) {
  FaceMetrics M;
  for (int d = 0; d < 3; d++)
    for (int a = 0; a < 3; a++) M.m[d][a] = fm[3 * d + a];
  M.aj[0] = iaj; M.aj[1] = jaj; M.aj[2] = kaj;
  k_face_gram<<<blocks_for(g.n(), 256), 256, 0, s>>>(g, M, gram, wild); count_launch();
}

// tame: the grid's metrics are all in intmul.cuh's range (k_face_gram).  visc
// null: the face fluxes fp alone.
void launch_viscous(const Geom &g, const double *nvert, const double *ucat, const double *const *fm,
                    const double *iaj, const double *jaj, const double *kaj, const double *gram, bool tame, double nu,
                    double *fp, double *visc, cudaStream_t s) {
  FaceMetrics M;
  for (int d = 0; d < 3; d++)
    for (int a = 0; a < 3; a++) M.m[d][a] = fm[3 * d + a];
  M.aj[0] = iaj; M.aj[1] = jaj; M.aj[2] = kaj;
  const dim3 nb(blocks_for(g.n(), 128), face_split(blocks_for(g.n(), 128)));
  if (tame && int_mul_factor(nu)) launch_dep(k_visc_faces<true>, nb, 128, 0, s, g, nvert, ucat, M, gram, nu, fp);
  else launch_dep(k_visc_faces<false>, nb, 128, 0, s, g, nvert, ucat, M, gram, nu, fp);
  if (visc) launch_dep(k_visc_div, blocks_for(g.n(), 256), 256, 0, s, g, (const double *)fp, visc);
}

// ------------------------------------------------------------- FormFunction1
// rct: the contravariant form of rc = visc - conv at the cell centres
// (rhs.c:2682-2700), interior cells; the ring stays 0 (a new vector).  visc is
// formed here from Viscous's face fluxes fp (k_visc_div's differences), so it
// is not written and read back.  Bound by the FP64 pipe: 33 sums a cell, the
// 12 products on the integer pipe (INT).  At 192^3 0.49 ms, with k_visc_div
// and FP64 products 0.66 ms.
template <bool INT>
__device__ __forceinline__ void rct_cell(const Geom &g, const double (&rc)[3], const double *__restrict__ csi,
                                         const double *__restrict__ eta, const double *__restrict__ zet, double a,
                                         long P, bool &fp64, double (&out)[3]) {
  const long st[3] = {1, g.mx, (long)g.mx * g.my};
  const double *m[3] = {csi, eta, zet};
  IntMulA Rc[3];
  if constexpr (INT)
    for (int c = 0; c < 3; c++) Rc[c] = int_split_a(rc[c], fp64);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double mean[3];
#pragma unroll
    for (int c = 0; c < 3; c++) mean[c] = scale_down<1>(m[d][3 * P + c] + m[d][3 * (P - st[d]) + c]);
    if constexpr (INT) {
      const double s = int_mul(Rc[0], int_split_b(mean[0], fp64)) + int_mul(Rc[1], int_split_b(mean[1], fp64)) +
                       int_mul(Rc[2], int_split_b(mean[2], fp64));
      out[d] = int_mul(int_split_a(s, fp64), int_split_b(a, fp64));
    } else {
      out[d] = a * (mean[0] * rc[0] + mean[1] * rc[1] + mean[2] * rc[2]);
    }
  }
}
__device__ __noinline__ void rct_cell_fp64(const Geom &g, const double (&rc)[3], const double *__restrict__ csi,
                                           const double *__restrict__ eta, const double *__restrict__ zet, double a,
                                           long P, double (&out)[3]) {
  bool unused = false;
  rct_cell<false>(g, rc, csi, eta, zet, a, P, unused, out);
}

__global__ void __launch_bounds__(128) k_ff1_rct(const __grid_constant__ Geom g, const double *__restrict__ conv,
                                                 const double *__restrict__ fp, const double *__restrict__ csi,
                                                 const double *__restrict__ eta, const double *__restrict__ zet,
                                                 const double *__restrict__ aj, double *__restrict__ rct) {
  dep_sync();
  const size_t n = g.n();
  const size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int pl = g.mx * g.my, k = (int)e / pl, j = ((int)e - k * pl) / g.mx, i = (int)e - k * pl - j * g.mx;
  double out[3] = {0., 0., 0.};
  if (i >= 1 && i <= g.mx - 2 && j >= 1 && j <= g.my - 2 && k >= 1 && k <= g.mz - 2) {
    double rc[3];
#pragma unroll
    for (int c = 0; c < 3; c++) rc[c] = -1.0 * conv[3 * e + c] + visc_cell(g, fp, e, c);
    const double a = aj[e];
    bool fp64 = false;
    rct_cell<true>(g, rc, csi, eta, zet, a, (long)e, fp64, out);
    if (fp64) rct_cell_fp64(g, rc, csi, eta, zet, a, (long)e, out);
  }
#pragma unroll
  for (int c = 0; c < 3; c++) rct[3 * e + c] = out[c];
}

namespace {

// The sum of two nvert values (finite, >= 0): nearly all are +0, whose sum
// needs no FP64 add.
__device__ __noinline__ double nv_sum_slow(double a, double b) { return a + b; }
__device__ __forceinline__ double nv_sum(double a, double b) {
  if ((__double_as_longlong(a) | __double_as_longlong(b)) == 0) return 0.;
  return nv_sum_slow(a, b);
}

// One tangential pressure derivative of face d of cell P (rhs.c:2803-2849 and
// its siblings, walled boxes); false where the reference assigns nothing.
__device__ __forceinline__ bool ff_dp(const double *__restrict__ nv, const double *__restrict__ p, long P, long sd,
                                      long s, int q, int m, double &val) {
  const double up = nv_sum(nv[P + s], nv[P + sd + s]), dn = nv_sum(nv[P - s], nv[P + sd - s]);
  // upper (the cells above are blocked or beyond the wall), lower, or central:
  // one expression on the cells each takes
  const bool upper = q == m - 2 || gt_01(up), lower = !upper && (q == 1 || gt_01(dn));
  if (upper ? !(lt_01(dn) && q != 1) : lower && !lt_01(up)) return false;
  const long h = upper ? 0 : s, l = lower ? 0 : -s;
  val = scale_down(p[P + h] + p[P + sd + h] - p[P + l] - p[P + sd + l], upper || lower ? 1 : 2);
  return true;
}

// What the cell before (i, j, k) in the reference's loop order leaves in its
// derivative variables dpde, dpdz: its z-section's (dpde from its branch, else
// its y section's p[j+1] - p[j]); 0 before the first cell.  Its final dpdc is
// assigned again by the next cell's x section before any use.
__device__ __noinline__ void ff_previous(const Geom &g, const double *__restrict__ nv, const double *__restrict__ p,
                                         int i, int j, int k, double &de, double &dz) {
  de = dz = 0.0;
  i--;
  if (i < 1) { i = g.mx - 2; j--; }
  if (j < 1) { j = g.my - 2; k--; }
  if (k < 1) return;
  const long sy = g.mx, sz = (long)g.mx * g.my, Q = ((long)k * g.my + j) * g.mx + i;
  if (!ff_dp(nv, p, Q, sz, sy, j, g.my, de)) de = p[Q + sy] - p[Q];
  dz = p[Q + sz] - p[Q];
}

// What stands in derivative t of cell P at face d where d's own branch assigns
// nothing: the sections before it in the cell, then the previous cell.
__device__ __noinline__ double ff_carried(const Geom &g, const double *__restrict__ nv, const double *__restrict__ p,
                                          int i, int j, int k, int d, int t) {
  const long st[3] = {1, g.mx, (long)g.mx * g.my}, P = k * st[2] + j * st[1] + i;
  const int q = t == 0 ? i : t == 1 ? j : k, m = t == 0 ? g.mx : t == 1 ? g.my : g.mz;
  for (int b = d - 1; b >= 0; b--) {
    double v;
    if (t == b) return p[P + st[b]] - p[P];
    if (ff_dp(nv, p, P, st[b], st[t], q, m, v)) return v;
  }
  double de, dz;
  ff_previous(g, nv, p, i, j, k, de, dz);
  return t == 1 ? de : dz;
}

// The pressure gradient through a face, (dp . gram) aj, with FP64 multiplies.
__device__ __noinline__ double ff_gradient_fp64(double d0, double d1, double d2, const double *__restrict__ gr,
                                                size_t n, double aj) {
  return (d0 * gr[0] + d1 * gr[n] + d2 * gr[2 * n]) * aj;
}
// ... and the time term: 1.5 u - 2 u_o + 0.5 u_rm1 or u - u_o, times a, on
// top of r.
__device__ __noinline__ double ff_time_fp64(double r, double u, double uo, double urm, int bdf2, double a) {
  double du;
  if (bdf2) {
    du = u;
    du *= 1.5;
    du += -2. * uo;
    du += 0.5 * urm;
  } else {
    du = -1. * uo + u;
  }
  r += a * du;
  return r;
}

}  // namespace

// CalcRHS's part of k_ff1_faces.
struct CalcRhsArgs {
  const double *uc, *uo, *urm;  // Ucont, Ucont_o, Ucont_rm1
  int bdf2;
  double a;    // -1 / dt
  int mz_end;  // mz - 3, or mz - 2 with a convective outflow (bctype[5] 8)
};

// The face values of FormFunction1 (rhs.c:2760-3222) and its blocked-face masks
// (rhs.c:3225-3262) on the interior cells.  The reference keeps the three
// derivative variables across its loop: where a branch assigns nothing the
// value of the previous assignment stands.  Within a cell that is the previous
// section's value; entering a cell it is what the previous cell in loop order
// (k, j, i ascending over the interior) left (ff_previous).
//
// CALC: then CalcRHS (implicitsolver.c:6519-6713) in the same pass: rhs -= dU /
// dt over every entry of the box (second-order backward dU = 1.5 u - 2 u_o +
// 0.5 u_rm1, or u - u_o on the first step), the faces next to blocked cells
// and the walls zeroed, the convective-outflow term on the last k face
// (bctype[5] 8), then the reference's six boundary loops, which zero the ring
// except on the box's last row in each direction.
//
// Bound by the FP64 pipe: 42 sums a cell; the 15 products go to the integer
// pipe (INT: intmul.cuh; gram and the Jacobians in its range), the sums of
// nvert and the previous cell's values are formed only where they are needed,
// and the one-sided differences beside walls share the central ones' expression
// (a warp of a row's end ran both).  At 192^3 0.74 ms with CalcRHS, in two
// kernels with FP64 products 1.25 ms.  Eight blocks per SM (64 registers): six
// 0.88 ms, seven 0.79 ms.
template <bool INT, bool CALC>
__global__ void __launch_bounds__(128, 8) k_ff1_faces(const __grid_constant__ Geom g, const double *__restrict__ nv,
                                                   const double *__restrict__ p, const double *__restrict__ rct,
                                                   const __grid_constant__ FaceMetrics M,
                                                   const double *__restrict__ gram, CalcRhsArgs A,
                                                   double *__restrict__ rhs) {
  dep_sync();
  const size_t n = g.n();
  const int mx = g.mx, my = g.my, mz = g.mz;
  const long st[3] = {1, mx, (long)mx * my};
  const size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int pl = mx * my, k = (int)e / pl, j = ((int)e - k * pl) / mx, i = (int)e - k * pl - j * mx;
  const bool in = i >= 1 && i <= mx - 2 && j >= 1 && j <= my - 2 && k >= 1 && k <= mz - 2;
  if (!CALC && !in) return;
  const long P = (long)e;
  const bool solid = in && gt_01(nv[P]);
  const FaceDirs dirs = FaceDirs::of_block();
#pragma unroll 1
  for (int d = dirs.first; d < dirs.end; d++) {
    const long sd = d == 0 ? st[0] : d == 1 ? st[1] : st[2];
    double v = 0.;
    if (in) {
      double dp[3];
#pragma unroll
      for (int t = 0; t < 3; t++) {
        if (t == d) dp[t] = p[P + sd] - p[P];
        else if (!ff_dp(nv, p, P, sd, st[t], t == 0 ? i : t == 1 ? j : k, t == 0 ? mx : t == 1 ? my : mz, dp[t]))
          dp[t] = ff_carried(g, nv, p, i, j, k, d, t);
      }
      // (csi . nd, eta . nd, zet . nd) of face d, from k_face_gram
      const double *gr = gram + (size_t)(3 * d) * n + P;
      v = scale_down<1>(rct[3 * P + d] + rct[3 * (P + sd) + d]);
      bool fp64 = !INT;
      double gradient = 0.;
      if constexpr (INT) {
        const double s = int_mul(int_split_a(dp[0], fp64), int_split_b(gr[0])) +
                         int_mul(int_split_a(dp[1], fp64), int_split_b(gr[n])) +
                         int_mul(int_split_a(dp[2], fp64), int_split_b(gr[2 * n]));
        gradient = int_mul(int_split_a(s, fp64), int_split_b(M.aj[d][P]));
      }
      if (fp64) gradient = ff_gradient_fp64(dp[0], dp[1], dp[2], gr, n, M.aj[d][P]);
      v -= gradient;
      if (solid || gt_01(nv[P + sd])) v = 0;
    }
    const size_t q = 3 * e + d;
    if constexpr (CALC) {
      if (!in) v = rhs[q];
      const double u = A.uc[q], uo = A.uo[q], urm = A.bdf2 ? A.urm[q] : 0.;
      bool fp64 = !INT;
      double r = v;
      if constexpr (INT) {
        double du;
        if (A.bdf2) {
          du = int_mul(int_split_a(u, fp64), int_split_b(1.5));
          du += int_mul(int_split_a(uo, fp64), int_split_b(-2.));
          du += scale_down<1>(urm);
        } else {
          du = -1. * uo + u;
        }
        r += int_mul(int_split_a(du, fp64), int_split_b(A.a));
      }
      if (fp64) r = ff_time_fp64(v, u, uo, urm, A.bdf2, A.a);
      if (in) {
        const int lim = d == 0 ? i - (mx - 3) : d == 1 ? j - (my - 3) : k - A.mz_end;
        if (lim > 0 || gt_01(nv_sum(nv[P], nv[P + sd]))) r = 0.;
        if (d == 2 && A.mz_end == mz - 2 && k == mz - 2) r += 0.8 * (u - A.uc[3 * (P - st[2]) + 2]);
      }
      // the six boundary loops (each covers its face minus the last row of the
      // other two directions)
      const bool kin = k < mz - 1, jin = j < my - 1, iin = i < mx - 1;
      const bool all = ((i == 0 || i == mx - 1) && kin && jin) || ((j == 0 || j == my - 1) && kin && iin) ||
                       ((k == 0 || k == mz - 1) && jin && iin);
      const bool own = d == 0 ? i == mx - 2 && kin && jin : d == 1 ? j == my - 2 && kin && iin : k == mz - 2 && jin && iin;
      v = all || own ? 0. : r;
    }
    rhs[q] = v;
  }
}

// FormFunction1 after its Contra2Cart, Convection (conv) and Viscous (fp, its
// face fluxes); with calc, CalcRHS's part on top.
void launch_form_function1(const Geom &g, const double *nvert, const double *p, const double *conv,
                           const double *fp, const double *csi, const double *eta, const double *zet,
                           const double *aj, const double *const *fm, const double *iaj, const double *jaj,
                           const double *kaj, const double *gram, bool tame, const MomentumTime *calc, double *rct,
                           double *rhs, cudaStream_t s) {
  FaceMetrics M;
  for (int d = 0; d < 3; d++)
    for (int a = 0; a < 3; a++) M.m[d][a] = fm[3 * d + a];
  M.aj[0] = iaj; M.aj[1] = jaj; M.aj[2] = kaj;
  CalcRhsArgs A = {};
  if (calc) A = {calc->ucont, calc->ucont_o, calc->ucont_rm1, calc->bdf2, calc->neg_inv_dt, calc->mz_end};
  const unsigned nb = blocks_for(g.n(), 128);
  launch_dep(k_ff1_rct, nb, 128, 0, s, g, conv, fp, csi, eta, zet, aj, rct);
  auto go = [&](auto kern) {
    launch_dep(kern, dim3(nb, face_split(nb)), 128, 0, s, g, nvert, p, (const double *)rct, M, gram, A, rhs);
  };
  const bool whole = tame && (!calc || int_mul_factor(calc->neg_inv_dt));
  if (calc) whole ? go(k_ff1_faces<true, true>) : go(k_ff1_faces<false, true>);
  else whole ? go(k_ff1_faces<true, false>) : go(k_ff1_faces<false, false>);
}

// ------------------------------------------------------------------- ImpRK
// One Runge-Kutta stage's update (implicitsolver.c:7156, VecWAXPY): u = a rhs
// + pu over every entry; then, with inflow (an inlet on k = 0: k_inflow's
// terms), what the InflowFlux that follows leaves in Ucont, its Ucont.z above
// fluid cells.  The inlet's ubcs stay as the first InflowFlux of the call
// left them: they depend on the grid, nvert and the profile alone.
__global__ void __launch_bounds__(256) k_imp_waxpy(Geom g, double a, const double *__restrict__ rhs,
                                                   const double *__restrict__ pu, const double *__restrict__ nv,
                                                   const double *__restrict__ inflow, double *__restrict__ u) {
  dep_sync();
  const size_t n = 3 * g.n(), plane = (size_t)g.mx * g.my;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    double v = a * rhs[e] + pu[e];
    if (inflow && e < 3 * plane && e % 3 == 2) {
      const int q = (int)(e / 3), j = q / g.mx, i = q - j * g.mx;
      if (i >= 1 && i <= g.mx - 2 && j >= 1 && j <= g.my - 2 && nv[q + plane] < 0.1)
        v = inflow[(j - 1) * (g.mx - 2) + i - 1];
    }
    u[e] = v;
  }
}

// The two infinity norms ImpRK takes after its stages (implicitsolver.c:
// 7183-7200): |rhs| and |pu - u| (VecWAXPY(dU, -1, u, pu)), or |rhs| alone
// when pu is null.  The largest |x| is exact in any order; non-negative
// doubles order as their bit patterns, so every maximum is an integer one (FP64
// comparisons took 44 us at 96^3), the blocks' by atomicMax into out[0..1] (zeroed
// by the host).  NaN entries are passed
// over, as a comparison-based maximum passes them.
__device__ __forceinline__ void imp_max(unsigned long long &m, double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffULL;
  if (b > m && b <= 0x7ff0000000000000ULL) m = b;
}
__global__ void __launch_bounds__(256) k_imp_norms(size_t n, const double *__restrict__ rhs,
                                                   const double *__restrict__ pu, const double *__restrict__ u,
                                                   unsigned long long *out) {
  unsigned long long mf = 0, md = 0;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    imp_max(mf, rhs[e]);
    if (pu) imp_max(md, -1. * u[e] + pu[e]);
  }
  for (int o = 16; o; o >>= 1) {
    mf = max(mf, __shfl_xor_sync(0xffffffffu, mf, o));
    md = max(md, __shfl_xor_sync(0xffffffffu, md, o));
  }
  __shared__ unsigned long long sf[8], sd[8];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { sf[w] = mf; sd[w] = md; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); q++) mf = max(mf, sf[q]), md = max(md, sd[q]);
    atomicMax(out, mf);
    if (pu) atomicMax(out + 1, md);
  }
}

// ------------------------------------------------------------- InflowFlux
// The reference adds a plane's flux and area terms one after another in its
// (j, i) loop.  A chain of dependent FP64 adds is slow on this GPU (one
// thread, about 70 cycles an add: 2.5 ms for a 192 x 192 plane), so the
// kernel below writes the terms, in that order, for the host to add (as
// k_outlet_plane does); cells the reference skips carry +0.0, which leaves a
// sum that started at +0.0 as it was.
//
// The shaped inlet speeds (bcs.c:152-192) at face cell (i, j): the mean of
// its four nodes of the k = 0 node plane (coor0, [my][mx][3]) less the centre
// (cmy, cmz); profile 2 a parabola across y in [0, 4.1] peaking at 1.5, 4 a
// pipe of radius 0.5 peaking at 2, 7 a parabola across y in [-0.5, 0.5]
// peaking at 1.5.  Each product and sum rounded on its own, in the
// reference's order.
__device__ double inlet_shaped(int profile, const double *__restrict__ coor0, int mx, int i, int j, double cmy,
                               double cmz) {
  const double *a = coor0 + 3 * ((size_t)j * mx + i), *b = coor0 + 3 * ((size_t)(j - 1) * mx + i);
  const double *c = coor0 + 3 * ((size_t)j * mx + i - 1), *d = coor0 + 3 * ((size_t)(j - 1) * mx + i - 1);
  const double yc = (a[1] + b[1] + c[1] + d[1]) * 0.25 - cmy;
  const double zc = (a[2] + b[2] + c[2] + d[2]) * 0.25 - cmz;
  const double H = 4.1, Umax = 1.5;
  if (profile == 2) return __ddiv_rn(4. * Umax * yc * (H - yc), H * H);
  if (profile == 4) {
    const double r = __dsqrt_rn(zc * zc + yc * yc);
    return r > 0.5 ? 0. : 2. * (1. - 4. * r * r);
  }
  return 1.5 * (1. - 4. * yc * yc);
}

// InflowFlux on the k = 0 face (bcs.c:148-236): above a fluid cell, ubcs =
// uin zet / |zet| (in the reference's order .y, .z, .x, each its own
// quotient) and Ucont.z = uin |zet|, |zet| summed z, y, x; the face's flux
// terms into terms[(j - 1)(mx - 2) + i - 1].  uin is the constant speed; with
// coor0 set the shaped profile's at the cell, with uin_cell set the speed the
// host formed for the cell (at the terms' index).
__global__ void k_inflow(Geom g, const double *__restrict__ nv, const double *__restrict__ zet, double uin,
                         const double *__restrict__ coor0, int profile, double cmy, double cmz,
                         const double *__restrict__ uin_cell, double *__restrict__ uc, double *__restrict__ ub,
                         double *__restrict__ terms) {
  const int ni = g.mx - 2, n = ni * (g.my - 2);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int i = 1 + t % ni, j = 1 + t / ni;
  const size_t q = (size_t)j * g.mx + i;
  double term = 0.;
  if (nv[q + (size_t)g.mx * g.my] < 0.1) {
    if (uin_cell) uin = uin_cell[t];
    else if (coor0) uin = inlet_shaped(profile, coor0, g.mx, i, j, cmy, cmz);
    const double *z = zet + 3 * q;
    const double a = __dsqrt_rn(z[2] * z[2] + z[1] * z[1] + z[0] * z[0]);
    ub[3 * q + 1] = __ddiv_rn(uin * z[1], a);
    ub[3 * q + 2] = __ddiv_rn(uin * z[2], a);
    ub[3 * q + 0] = __ddiv_rn(uin * z[0], a);
    uc[3 * q + 2] = uin * a;
    term = uc[3 * q + 2];
  }
  terms[t] = term;
}

void launch_inflow(const Geom &g, const double *nvert, const double *zet, double uin, const double *coor0,
                   int profile, double cmy, double cmz, const double *uin_cell, double *ucont, double *ubcs,
                   double *terms, cudaStream_t s) {
  const int n = (g.mx - 2) * (g.my - 2);
  k_inflow<<<blocks_for(n, 256), 256, 0, s>>>(g, nvert, zet, uin, coor0, profile, cmy, cmz, uin_cell, ucont, ubcs,
                                              terms);
  count_launch();
}

void launch_imp_waxpy(const Geom &g, double a, const double *rhs, const double *pu, const double *nvert,
                      const double *inflow, double *u, cudaStream_t s) {
  launch_dep(k_imp_waxpy, blocks_for(3 * g.n(), 256), 256, 0, s, g, a, rhs, pu, nvert, inflow, u);
}

void launch_imp_norms(size_t n, const double *rhs, const double *pu, const double *u, unsigned long long *out,
                      cudaStream_t s) {
  cudaMemsetAsync(out, 0, 2 * sizeof(unsigned long long), s);
  // grid-stride over a few blocks per SM, so that few atomics meet
  const unsigned nb = blocks_for(n, 256) < 2432u ? blocks_for(n, 256) : 2432u;
  k_imp_norms<<<nb, 256, 0, s>>>(n, rhs, pu, u, out);
  count_launch();
}

}  // namespace cvb
