// Internal declarations shared by the CUDA kernels and the host library.
// Grid layout everywhere: one level is the reference's DMDA box [mz][my][mx],
// i fastest, boundary ring included (mx = IM+1 for IM nodes).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace cvb {

// Kernel launches issued by this library (all contexts), for measurement.
void count_launch(int n = 1);
long long launch_count();

// Stencil slots, in the order of the reference's PoissonLHSNew (poisson.c:576-594).
enum Slot { CP, EP, WP, NP, SP, TP, BP, NE, SE, NW, SW, TN, BN, TS, BS, TE, BE, TW, BW, NSLOT };

// Per-cell switching code (built once from nvert by build_codes):
//   bit 0       identity row (boundary ring, or nvert > 0.1)
//   bits 1..6   face active from this row's side: E, W, N, S, T, B
//   bit 7       blocked: nvert > 0.1 (read by the grid transfers)
//   bit 20      fluid: interior and nvert < 0.1
//   bits 8..19  cross-derivative form for this cell's three upper faces, 2 bits each:
//               E: (j, k)  N: (i, k)  T: (i, j)   0 none, 1 central, 2 lower, 3 upper
// A lower face (W/S/B) of a row is the upper face of its lower neighbour, so a
// row reads that neighbour's code for it.
enum : uint32_t {
  CODE_IDENTITY = 1u,
  CODE_BLOCKED = 1u << 7,  // nvert > 0.1 (IB or solid), any cell
  CODE_FLUID = 1u << 20,   // interior cell with nvert < 0.1 (the null space's and range projection's cells)
  CODE_ACT_E = 1u << 1, CODE_ACT_W = 1u << 2, CODE_ACT_N = 1u << 3,
  CODE_ACT_S = 1u << 4, CODE_ACT_T = 1u << 5, CODE_ACT_B = 1u << 6,
};
__host__ __device__ inline int code_branch(uint32_t c, int face, int which) {
  return (c >> (8 + 4 * face + 2 * which)) & 3u;  // face 0=E,1=N,2=T; which 0/1
}

struct Geom {
  int mx, my, mz;
  int px, py, pz;  // periodic directions (bctype 7)
  __host__ __device__ size_t n() const { return (size_t)mx * my * mz; }
  __host__ __device__ size_t id(int i, int j, int k) const {
    return ((size_t)k * my + j) * mx + i;
  }
  // neighbour index with the reference's periodic wrap of column indices
  __host__ __device__ int iu(int i) const { return (px && i == mx - 2) ? 1 : i + 1; }
  __host__ __device__ int id_(int i) const { return (px && i == 1) ? mx - 2 : i - 1; }
  __host__ __device__ int ju(int j) const { return (py && j == my - 2) ? 1 : j + 1; }
  __host__ __device__ int jd(int j) const { return (py && j == 1) ? my - 2 : j - 1; }
  __host__ __device__ int ku(int k) const { return (pz && k == mz - 2) ? 1 : k + 1; }
  __host__ __device__ int kd(int k) const { return (pz && k == 1) ? mz - 2 : k - 1; }
};

// Thomas factors in global memory, line by line: line (i, k) holds a_j, 1/m_j
// and c'_j for j = 1..my-2 as three runs of Q = my-2 rounded up to 4 values
// (zero-padded), so that a line's factors are 16-byte aligned and contiguous.
// Lines are ordered by plane k, then zebra colour (i + k) % 2, then i / 2: the
// lines of one colour in one plane -- the tile of a zebra line solve -- follow
// one another.
struct LineFac {
  int nt, Q;
  __host__ __device__ static LineFac of(const Geom &g) {
    LineFac f;
    f.nt = (g.mx + 1) >> 1;
    f.Q = (g.my - 2 + 3) & ~3;
    return f;
  }
  __host__ __device__ size_t line(int i, int k) const {
    return (((size_t)k * 2 + ((i + k) & 1)) * nt + (i >> 1)) * 3 * (size_t)Q;
  }
  __host__ __device__ size_t count(const Geom &g) const { return (size_t)g.mz * 2 * nt * 3 * Q; }
};

// Colour-split rows: the cells of zebra colour (i + k) % 2 == c of row (j, k)
// at c * half + i / 2 of a row of 2 * half slots.  A zebra half-sweep passes
// its residual to the line solves in this layout, so that the lines of one
// colour are adjacent in memory.
struct SplitRow {
  __host__ __device__ static int half(const Geom &g) { return (g.mx + 1) >> 1; }
  __host__ __device__ static size_t count(const Geom &g) { return (size_t)g.my * g.mz * 2 * half(g); }
  __host__ __device__ static int at(const Geom &g, int i, int j, int k) {
    const int h = half(g);
    return (k * g.my + j) * 2 * h + ((i + k) & 1) * h + (i >> 1);
  }
};

// Device data of one multigrid level.
struct LevelDev {
  Geom g;
  int isc, jsc, ksc;     // semi-coarsening flags of this level (GridRestriction)
  double *nvert;         // [N]
  uint32_t *code;        // [N]
  double *w64;           // [19][N] FP64 stencil weights (rows scaled by -aj; identity rows CP=1)
  float *gf32;           // [9][N]  FP32 face coefficients g11..g33, cross terms pre-scaled by form weight
  float *ajf32;          // [N]
  float *wgt32;          // [N]    restriction weight max(0, 1 - nvert), rounded to float
  float *line32;         // y-line Thomas factors (a_j, 1/m_j, c'_j) in FP32, LineFac layout
  float *cs32;           // levels without FP32 cross terms: g11, g22, g33, aj and the code (its bits)
                         // in colour-split rows ([5][SplitRow::count]) for the zebra residual; else null
  double *line64;        // ... in FP64
  // colour-split rows for the one-thread-per-line relaxation (kernels_lines.cu; null: not formed): m, beta,
  // -c of each row, and without cross terms the seven weights times -m
  double *lf64, *lw64;
  // work vectors of this level (the finest level's b/x live in the solver)
  double *r64, *e64, *t64;  // FP64 V-cycle vectors
  float *r32, *e32, *t32;   // FP32 V-cycle vectors
  int sweep32, sweep64;     // line-sweep variant chosen at set-up: 0 fused, 1 split
  // the operator has cross-derivative terms (FP32 flux form / FP64 edge
  // weights); 0 on an orthogonal grid, where the kernels read 7 points
  int cross32, cross64;
  int zfuse32, zfuse64;     // zebra variant chosen at set-up: 0 two kernels per half-sweep, 1 one
                            // (in place without cross terms, else out of place)
  int ztma32;               // FP32 zebra half-sweep with TMA-staged tiles (kernels_tma.cu): the
                            // row pairs per chunk (4, 8, 16) the autotuner chose, 0 off
  int zlines64;             // FP64 zebra half-sweep with one thread per line (kernels_lines.cu), chosen at set-up
  int ztw32;                // lines per block of the FP32 zebra line-solve tiles (4 or 8; 0: 8)
  // coarsest level only: the densely inverted cells (first cm of cidx) and the
  // identity ones (the rest of cidx)
  const int *cidx;
  int cm;
  // When set, every kernel launched for this level returns at once while *gate
  // is non-zero: an FGMRES iteration issued ahead of the host's convergence
  // check turns into no-ops once the previous iteration has converged.
  const int *gate;
};

__device__ __forceinline__ bool gated(const int *gate) { return gate && *gate; }

// Whether a level's operator in precision T has cross-derivative terms.
template <typename T>
__host__ __device__ inline bool has_cross(const LevelDev &L) {
  return sizeof(T) == 4 ? L.cross32 != 0 : L.cross64 != 0;
}

// The fused zebra half-sweep's condition (see zebra_fused_body): no
// cross-derivative terms, and colours kept apart across periodic seams.
template <typename T>
__host__ __device__ inline bool zebra_fusable(const LevelDev &L) {
  return !has_cross<T>(L) && (!L.g.px || (L.g.mx & 1) == 0) && (!L.g.pz || (L.g.mz & 1) == 0);
}


// The longest lines the tile and line kernels take (their shared memory).
constexpr int kMaxFusedRows = 400;

// --- kernel launchers (defined in the .cu files) ---------------------------
// setup
// The face metrics of a level, by value in a kernel's parameters.
struct FaceMetrics {
  const double *m[3][3];  // [face direction][csi, eta, zet] Cmpnts arrays
  const double *aj[3];    // IAj, JAj, KAj
};
// after launch_codes; gf32: the FP32 copies, cross terms scaled by their form's
// weight; *cross = 1 where one is not zero (zeroed by the caller)
void launch_gcoef(const Geom &g, const double *const *metric /*9 Cmpnts fields: I(csi,eta,zet) J.. K..*/,
                  const double *iaj, const double *jaj, const double *kaj, const uint32_t *code, double *g9 /*[9][N]*/,
                  float *gf32 /*[9][N]*/, int *cross, cudaStream_t s);
void launch_codes(const Geom &g, const double *nvert, uint32_t *code, cudaStream_t s);
// wgt32 = (float) max(0, 1 - nvert)
void launch_weight32(const Geom &g, const double *nvert, float *wgt32, cudaStream_t s);
// *cross = 1 where an edge weight is not zero (zeroed by the caller)
void launch_weights(const Geom &g, const double *g9, const double *aj, const uint32_t *code, double *w64, int *cross,
                    cudaStream_t s);
void launch_line_factors(const Geom &g, const double *w64, double *line64, float *line32,
                         cudaStream_t s);
void launch_to_f32(const double *a, float *b, size_t n, cudaStream_t s);
void launch_nvert_restrict(const Geom &fine, const double *nvf, const Geom &coarse, int isc, int jsc,
                           int ksc, double *nvc, double *tmp, cudaStream_t s);

// operator / smoother / transfers (T = float or double)
template <typename T>
void launch_apply(const LevelDev &L, const T *x, T *y, cudaStream_t s);
template <typename T>
void launch_residual(const LevelDev &L, const T *b, const T *x, T *r, cudaStream_t s);
template <typename T>
void launch_line_smooth(const LevelDev &L, const T *b, const T *x, T *xnew, T omega, int zero_guess,
                        cudaStream_t s);
// The FP32 zebra half-sweep of one colour in place with TMA-staged tiles of
// rp row pairs (kernels_tma.cu); false when the level does not allow it.
bool zebra_tma_ok(const LevelDev &L);
bool launch_zebra_tma(const LevelDev &L, const float *b, float *x, float omega, int color, int rp, cudaStream_t s);
// 1 if a TMA kernel's bounded wait gave up since the last call (cleared), 0 if
// not, -1 on a CUDA error; synchronises the stream.
int tma_timeout_take(cudaStream_t s);
// zebra half-sweep of one color, in place (res: scratch for the residual)
template <typename T>
void launch_zebra_half(const LevelDev &L, const T *b, T *x, T *res, T omega, int color, bool zero, cudaStream_t s);
// one zebra sweep (both colours) on x; tmp: a level-sized buffer for the
// out-of-place one-kernel form; zero_first: x is zero on entry
template <typename T>
void launch_zebra_sweep(const LevelDev &L, const T *b, T *x, T *tmp, T *res, T omega, bool zero_first, cudaStream_t s);
// restriction of xf into xc; zero_c, when set, is zeroed over the coarse grid too
template <typename T>
void launch_restrict(const LevelDev &F, const LevelDev &C, const T *xf, T *xc, cudaStream_t s, T *zero_c = nullptr);
template <typename T>
void launch_prolong_add(const LevelDev &C, const LevelDev &F, const T *xc, T *xf, cudaStream_t s);

// mixed-precision glue: FP64 operator on an FP32-stored vector
void launch_f32_to_f64(const float *a, double *b, size_t n, cudaStream_t s);

// Krylov support (deterministic two-stage reductions)
int reduce_blocks();
int sm_count();
// Pointers and weights of a Krylov basis, by value in a kernel's parameters.
constexpr int kMaxBasis = 65;
struct BasisList {
  const double *v[kMaxBasis];
};
struct BasisWeights {
  double y[kMaxBasis];
};
// The reductions below finish in their last block (partial: reduce_blocks()
// doubles a sum; *counter zero before and after) and leave their scalars on the
// device: out[0 .. nv) the dots with V; a norm's out[0] its square and out[1] its
// reciprocal, the square also in pinned host memory.
void launch_dots(const BasisList &V, int nv, const double *w, size_t n, double *partial, unsigned *counter, double *out,
                 cudaStream_t s);
void launch_finish_sums(const double *partial, int nv, int nblocks, double *out, cudaStream_t s,
                        const int *gate = nullptr);
// w -= sum h_q V_q and the norm of w; host[0 .. nv) = h, host[nv] = |w|^2
void launch_orthogonalise(double *w, const BasisList &V, const double *h, int nv, size_t n, double *partial,
                          unsigned *counter, double *out, double *host, cudaStream_t s);
void launch_norm(const double *v, size_t n, double *partial, unsigned *counter, double *out, double *host,
                 cudaStream_t s);
// dst = src * *rcp (and, with dst32, its FP32 copy)
void launch_scale(double *dst, const double *src, const double *rcp, size_t n, float *dst32, cudaStream_t s);
// cs[5][SplitRow::count] = g11, g22, g33 (gf32 slots 0, 4, 8), aj and the code's
// bits, each cell at its colour-split position
void launch_split_coef(const Geom &g, const float *gf32, const float *ajf32, const uint32_t *code, float *cs,
                       cudaStream_t s);
// out = 1 / a, element by element (correctly rounded)
void launch_reciprocal(const double *a, double *out, size_t n, cudaStream_t s);
void launch_axpy_z(double *x, const BasisList &Z, const BasisWeights &y, int nz, size_t n, cudaStream_t s);
// the mean over the fluid cells of x, or with inv_aj of x inv_aj, over sign,
// into *out (device); x += *shift there
void launch_fluid_mean(const Geom &g, const uint32_t *code, const double *x, const double *inv_aj, double sign,
                       double *partial, unsigned *counter, double *out, cudaStream_t s);
void launch_add_fluid_const(const Geom &g, const uint32_t *code, double *x, const double *shift, int zero_outside,
                            cudaStream_t s);
// range projection of a right-hand side, b -= aj *mean on the fluid cells, and
// the norm of the result; host[0] = *mean, host[1] = |b|^2
void launch_remove_mean(const Geom &g, const uint32_t *code, const double *aj, double *b, const double *mean,
                        double *partial, unsigned *counter, double *out, double *host, cudaStream_t s);

// In-place Gauss-Jordan inverse of the n x n row-major A on the device into
// out (kernels_setup.cu); false for a singular matrix.  Work arrays: perm and
// colmap n ints, work dense_inverse_doubles(n) doubles, status one int.
size_t dense_inverse_doubles(int n);
bool device_dense_inverse(double *A, int n, double *out, int *perm, int *colmap, double *work, int *status,
                          cudaStream_t s);
// The coarsest level's m x m matrix over the cells idx[0 .. m) of its n:
// region[r] the row's fluid region (-1: an identity row), cols[19 r ..] its
// neighbours' columns, sv0 / sv1 added over each region's block
void launch_coarse_matrix(int m, int n, const int *idx, const int *region, const int *cols, double sv0, double sv1,
                          const double *w64, double *A, cudaStream_t s);
// coarsest solve e = M^-1 r on C.cidx[0..C.cm), e = r on the other cells
void launch_dense_apply(const LevelDev &C, const double *Minv, const double *r, double *e, cudaStream_t s,
                        const int *gate = nullptr);
void launch_dense_apply_f32(const LevelDev &C, const double *Minv, const float *r, float *e, cudaStream_t s,
                            const int *gate = nullptr);

// projection-path kernels (FP64)
void launch_poisson_rhs(const Geom &g, const double *ucont, const double *aj, const double *nvert,
                        double dt, double st, double *b, double *partial, cudaStream_t s);
void launch_ib_sums(const Geom &g, const double *ucont, const double *csi, const double *eta,
                    const double *zet, const double *nvert, double *partial, cudaStream_t s);
void launch_ib_correct(const Geom &g, double *ucont, const double *csi, const double *eta,
                       const double *zet, const double *nvert, const double *flux_area,
                       double flux_intp_sum, int flg, cudaStream_t s);
void launch_update_pressure(const Geom &g, double *p, double *phi, cudaStream_t s);
void launch_projection(const Geom &g, const double *const *fm /*I,J,K csi/eta/zet*/, const double *iaj,
                       const double *jaj, const double *kaj, const double *gram, bool tame, const double *nvert,
                       const uint32_t *code, const double *phi, double dt, double st, double *ucont, cudaStream_t s);
// Immersed-body classification (kernels_ibm.cu).  The body's bounding box is
// cut into kIbmBuckets^3 buckets (ibm.c:4213); a ray from a cell centre walks
// one bucket column upward.
constexpr int kIbmBuckets = 40, kIbmMaxHits = 32, kIbmMaxTries = 64;
struct IbmArgs {
  Geom g;
  double min[3], max[3], dc[3];  // bounding box and bucket size
  const int *col_start;          // bucket column (i, k) = k * kIbmBuckets + i -> its entries
  const int2 *col_ent;           // (triangle, end of the triangle's bucket range in j)
  const double *tri;             // per triangle: v0, v1 - v0, v2 - v0, unit normal (12 doubles)
  const double *offsets;         // ray offset of seeds 1 .. tries (randomdirection's s)
  int tries;
  const double *cent;            // cell centres, [mz][my][mx][3]
  double *nvert;                 // [mz][my][mx], updated in place
  const double *nvert_o;         // the previous step's nvert
  int ibi, nbodies;
  int *failed;                   // set when a cell found no usable ray
};
// Work arrays of the search: per interior cell its bucket column (key) and
// the cell list sorted by column (list); per column its count, start and fill;
// per cell of the box a byte marking inside cells (in4).
struct IbmWork {
  int *key, *list, *count, *start, *fill, *total;
  unsigned char *in4;
};
// The search; tmp is one more [mz][my][mx] array.  The result is left in tmp.
void launch_ibm_search(const IbmArgs &A, const IbmWork &W, double *tmp, cudaStream_t s);

// The grid's Contra2Cart factors (launch_c2c_factors: 10 N doubles, and the
// determinants' reciprocals where there was room for them) and whether all of them
// are there and in intmul.cuh's range
struct C2cFactors {
  const double *fac, *rcp;
  bool tame;
};
void launch_contra2cart(const Geom &g, const C2cFactors &F, const double *nvert, const double *ucont, double *ucat,
                        cudaStream_t s, int k0 = 1, int nk = -1);
void launch_c2c_factors(const Geom &g, const double *csi, const double *eta, const double *zet, double *fac,
                        double *rcp, int *wild, cudaStream_t s);
// max |div| and its first box index into out_v / out_i (device); pv / pi
// hold 1024 partial pairs
void launch_divergence(const Geom &g, const double *ucont, const double *aj, const double *nvert, double *pv,
                       long long *pi, double *out_v, long long *out_i, cudaStream_t s);
void launch_convection(const Geom &g, const double *ucont, const double *ucat, const double *nvert, int central,
                       double *fp, double *conv, cudaStream_t s);
void launch_metrics_divergence(const Geom &g, const double *csi, const double *eta, const double *zet,
                               const double *aj, double *pv, long long *pi, double *out_v, long long *out_i,
                               cudaStream_t s);
// The momentum right-hand side (kernels_momentum.cu), boxes with no periodic
// face.  fm: the nine face-metric arrays (I, J, K x csi, eta, zet); fp: 9 N
// doubles of scratch; rct: 3 N doubles of scratch.
// gram: the 9 N face metric products of launch_face_gram (formed once per grid)
void launch_face_gram(const Geom &g, const double *const *fm, const double *iaj, const double *jaj,
                      const double *kaj, double *gram, int *wild, cudaStream_t s);
void launch_viscous(const Geom &g, const double *nvert, const double *ucat, const double *const *fm,
                    const double *iaj, const double *jaj, const double *kaj, const double *gram, bool tame, double nu,
                    double *fp, double *visc, cudaStream_t s);
// CalcRHS's time term, on top of FormFunction1
struct MomentumTime {
  const double *ucont, *ucont_o, *ucont_rm1;
  int bdf2;
  double neg_inv_dt;
  int mz_end;
};
void launch_form_function1(const Geom &g, const double *nvert, const double *p, const double *conv,
                           const double *fp, const double *csi, const double *eta, const double *zet,
                           const double *aj, const double *const *fm, const double *iaj, const double *jaj,
                           const double *kaj, const double *gram, bool tame, const MomentumTime *calc, double *rct,
                           double *rhs, cudaStream_t s);
// bc: the level's bctype[6]; the host has refused the types it does not cover.
// cent: the cell centres ([N][3]) an annulus face needs; u_bc: the rheology
// plates' velocity.  Returns whether any face's type writes ubcs
bool launch_ghost_node_velocity(const Geom &g, const int *bc, const double *csi, const double *eta,
                                const double *zet, double *ubcs, double *ucat, cudaStream_t s,
                                const double *cent = nullptr, double u_bc = 0.);
// FormBCS with walls on the x and y faces: the ghost faces' interior cells and
// the 12 edge averages of ucat and p, as its last pass leaves them
void launch_form_ring(const Geom &g, const double *ubcs, double *ucat, double *p, cudaStream_t s);
// The outlet's passes (bctype[5] 4) on the last interior k plane: with apply
// the flux correction by ratio and Contra2Cart of the plane; with want_terms
// (always without apply) its flux terms in the reference's loop order into
// terms[0 .. n2), with want_area the area terms into terms[n2 .. 2 n2)
void launch_outlet_plane(const Geom &g, const double *zet, const C2cFactors &F, const double *nvert, bool apply,
                         double ratio, bool want_terms, bool want_area, double *ucont, double *ubcs, double *ucat,
                         double *terms, cudaStream_t s);
// InflowFlux on an inlet k = 0 face with a constant speed uin: ubcs and
// Ucont.z there, and the face's flux terms in the reference's loop order into
// terms ((mx - 2)(my - 2) doubles) for the host to add
void launch_inflow(const Geom &g, const double *nvert, const double *zet, double uin, const double *coor0,
                   int profile, double cmy, double cmz, const double *uin_cell, double *ucont, double *ubcs,
                   double *terms, cudaStream_t s);
// ImpRK's stage update u = a rhs + pu, with inflow (an inlet: launch_inflow's
// terms) its Ucont.z on the inlet too; and its two infinity norms (|rhs|,
// |pu - u|; pu null: |rhs| only) as bit patterns into out[0..1] (device)
void launch_imp_waxpy(const Geom &g, double a, const double *rhs, const double *pu, const double *nvert,
                      const double *inflow, double *u, cudaStream_t s);
void launch_imp_norms(size_t n, const double *rhs, const double *pu, const double *u, unsigned long long *out,
                      cudaStream_t s);

// --- FP64 y-line relaxation, one thread per line (kernels_lines.cu)
// Tiles of 32 lines of one colour in a plane, and the fewest tiles of a colour
// in a level that can take it: two for each of 152 SMs.
inline int line_tiles_x(const Geom &g) { return ((g.mx - 1) / 2 + 31) / 32; }
constexpr int kLineTiles = 304, kLineBlocks = 4, kLineAhead = 8;
inline bool lines_fit(const Geom &g) {
  return g.my - 2 <= kMaxFusedRows && (long long)line_tiles_x(g) * (g.mz - 2) >= kLineTiles;
}
// A block's shared memory: a tile's rows, in steps of kLineAhead.
inline size_t lines_smem(const Geom &g) {
  return sizeof(double) * 32 * (size_t)((g.my - 2 + kLineAhead - 1) / kLineAhead * kLineAhead);
}
// Whether a level that can take it does.  A rule on the shape, not a time: its results
// differ from the tile kernels' by rounding, and a solve's bits must not depend on what
// else ran while the set-up timed its kernels.  What decides is how much of the blocks
// that run at a time have a line for every lane (fill): a tile takes as long for one
// line as for 32, and a second round of blocks as long as the first.  The shorter the
// lines, the more the tile kernels' scans cost them, up to 56 rows because the scans take
// 64 rows' time.  A sweep's time against the faster tile form's, 7- and 19-point levels
// of 304 to 1,840 tiles where the rule takes it and where not: 16 to 32 rows 0.22 ..
// 0.89 and 0.70 .. 1.07, 40 to 56 rows 0.55 .. 1.00 and 1.00 .. 1.01, 64 and more 0.68 ..
// 1.03 (median 0.91; 1.07 at 392 rows in two rounds) and 0.90 .. 1.44 (median 1.07).
inline bool lines_pay(const Geom &g) {
  const long long tiles = (long long)line_tiles_x(g) * (g.mz - 2), lines = (long long)((g.mx - 1) / 2) * (g.mz - 2);
  const long long per_sm = 228 * 1024 / (long long)(lines_smem(g) + 1024);
  const long long blocks = (per_sm < kLineBlocks ? per_sm : kLineBlocks) * sm_count();
  const long long rounds = (tiles + blocks - 1) / blocks;
  const double fill = (double)lines / (32.0 * blocks * rounds);
  const int rows = g.my - 2;
  if (rows <= 32) return fill >= 0.2;
  if (rows <= 56) return fill >= 0.35;
  return fill >= 0.6 || (rounds == 1 && fill >= 0.5);
}
// lf (and, with lw, the scaled weights of a level without cross terms) from
// the level's weights and Thomas factors
void launch_line_rows(const Geom &g, const double *w64, const double *line64, double *lf, double *lw, cudaStream_t s);
// one colour: fused, a half-sweep of x in place (xnew == x) for the right-hand
// side r (zebra_fusable levels); else the line solves of the residual r
// (rsplit: in colour-split rows), x null for a zero guess
void launch_lines(const LevelDev &L, bool fused, const double *r, const double *x, double *xnew, double omega,
                  int color, int rsplit, cudaStream_t s);

// --- a V-cycle's small levels in two kernels (kernels_tail.cu)
constexpr int kTailLevels = 3;
// how many of the levels 1, 2, ... they take (below the finest level)
template <typename T>
int tail_levels(const LevelDev *L, int nlevels);
// v: each level's right-hand side, correction, scratch and residual; up false:
// from the right-hand side of level n to that of level 0; up true: from level 0's
// correction to level n's
template <typename T>
void launch_tail(const LevelDev *L, T *const (*v)[4], int n, int pre, int post, T omega, bool up, cudaStream_t s);

}  // namespace cvb
