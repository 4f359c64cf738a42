// The FP64 y-line relaxation with one thread per line: a zebra half-sweep of a
// 7-point level in one kernel, and the line solves of a given residual.
//
// A block takes 32 lines of one colour, two cells apart in i, at one plane, a
// lane each.  Its eight warps form the rows' right-hand sides m r (m the Thomas
// pivots' reciprocals) row by row into shared memory, one warp runs the two
// recurrences of all 32 lines, and the eight write x + omega d.  The recurrences
// cost two multiply-adds a row, d_j = m_j r_j + beta_j d_{j-1} with beta = -m a
// and x_j = d_j - c_j x_{j+1}, where the warp-parallel scan of line_solve_body
// costs about thirteen: each lane composes its rows' maps, five shuffle steps
// combine them, and the rows are replayed.  The FP64 pipe bounds the half-sweep
// on GB300 (two operations per SM per clock, 64 clocks of latency), and it
// takes 11 operations a cell this way, about 24 that way.
//
// A line's chain of dependent operations is long, so this pays only where every
// SM has a few tiles to overlap: a sweep of the channel's finest level (512
// tiles, 4.4 M cells) took 153 us against 216 (one kernel with scans), of the
// distorted 192^3 box (576 tiles, after a residual kernel) 508 against 663; at
// 96^3 (192 tiles) it took 109 against 96, and on smaller levels twice as long.
// Levels with fewer than kLineTiles tiles cannot take it, lines_pay says which
// others do.  In FP32, whose pipe does not bound the sweep, it was slower everywhere
// (95 against 62 us on the channel's finest level).  Eight warps and four blocks
// per SM (64 registers): four warps 165 us, three blocks 226, six blocks 244.
//
// All per-line arrays lie in colour-split rows (SplitRow): the lanes of a warp
// read consecutive values, and a half-sweep reads its own colour's alone.
//  - lf64: m, beta and -c of every row ([3][SplitRow::count]);
//  - lw64 (levels without cross-derivative terms): the seven weights times -m,
//    so that m r is m b and seven multiply-adds; an identity row's are its 1.
#include "stencil_body.cuh"

namespace cvb {

// lf and lw from a level's weights and Thomas factors.
__global__ void __launch_bounds__(256) k_line_rows(Geom g, const double *__restrict__ w, const double *__restrict__ l64,
                                                   double *__restrict__ lf, double *__restrict__ lw) {
  const size_t n = g.n(), S = SplitRow::count(g);
  const LineFac F = LineFac::of(g);
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(p % g.mx), j = (int)((p / g.mx) % g.my), k = (int)(p / ((size_t)g.mx * g.my));
    if (j < 1 || j > g.my - 2) continue;
    const double *f = l64 + F.line(i, k) + (j - 1);
    const double a = f[0], m = f[F.Q], c = f[2 * (size_t)F.Q];
    const size_t q = SplitRow::at(g, i, j, k);
    lf[q] = m;
    lf[S + q] = -m * a;
    lf[2 * S + q] = -c;
    if (lw)
#pragma unroll
      for (int s = CP; s <= BP; s++) lw[s * S + q] = -m * w[s * n + p];
  }
}
void launch_line_rows(const Geom &g, const double *w64, const double *line64, double *lf, double *lw, cudaStream_t s) {
  const size_t nb = (g.n() + 255) / 256;
  k_line_rows<<<(unsigned)(nb < 8192 ? nb : 8192), 256, 0, s>>>(g, w64, line64, lf, lw);
  count_launch();
}

constexpr int kLineWarps = 8;

// The recurrences of a warp's 32 lines: sr[32 (j - 1) + lane] holds m r, then
// d, then the solution; np rows, the nr of the lines rounded up to a multiple
// of kAhead, zero beyond.  be and cn: the lane's beta and -c, `pitch` apart row
// to row, in flight kAhead rows before they are used (nx: the first beta's).
constexpr int kAhead = kLineAhead;
__device__ __forceinline__ void rows_ahead(double (&nx)[kAhead], const double *__restrict__ f, int pitch, int j0, int nr) {
#pragma unroll
  for (int u = 0; u < kAhead; u++) nx[u] = j0 + u >= 0 && j0 + u < nr ? __ldg(f + (size_t)(j0 + u) * pitch) : 0.0;
}
__device__ __forceinline__ void lanes_solve(double *sr, double (&nx)[kAhead], const double *__restrict__ be,
                                            const double *__restrict__ cn, int pitch, int nr, int np, int lane) {
  double cu[kAhead], d = 0.0;
  for (int j0 = 0; j0 < np; j0 += kAhead) {
    double *r = sr + 32 * j0 + lane, v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; u++) { cu[u] = nx[u]; v[u] = r[32 * u]; }
    if (j0 + kAhead < np) rows_ahead(nx, be, pitch, j0 + kAhead, nr);
    else rows_ahead(nx, cn, pitch, j0, nr);
#pragma unroll
    for (int u = 0; u < kAhead; u++) r[32 * u] = d = fma(cu[u], d, v[u]);
  }
  d = 0.0;
  for (int j0 = np - kAhead; j0 >= 0; j0 -= kAhead) {
    double *r = sr + 32 * j0 + lane, v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; u++) { cu[u] = nx[u]; v[u] = r[32 * u]; }
    rows_ahead(nx, cn, pitch, j0 - kAhead, nr);
#pragma unroll
    for (int u = kAhead - 1; u >= 0; u--) r[32 * u] = d = fma(cu[u], d, v[u]);
  }
}

// FUSED: one half-sweep of x in place on a level without cross-derivative
// terms whose colours the seams keep apart (zebra_fusable): the rows read cells
// of the other colour and of their own line alone.  Otherwise the line solves
// of the residual r (rsplit: in colour-split rows, else in the caller's
// layout), xnew = x + omega d on the colour's lines, or omega d with x null.
template <bool FUSED>
__global__ void __launch_bounds__(32 * kLineWarps, kLineBlocks) k_lines(const __grid_constant__ LevelDev L,
                                                              const double *__restrict__ r, const double *x,
                                                              double *xnew, double omega, int color, int rsplit) {
  dep_sync();
  if (gated(L.gate)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *sr = reinterpret_cast<double *>(smem_raw);
  constexpr int NW = kLineWarps;
  const Geom &g = L.g;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, k = blockIdx.y + 1, nr = g.my - 2;
  const int h = SplitRow::half(g), pitch = 2 * h;
  const size_t S = SplitRow::count(g);
  const int i = (((color + k) & 1) ? 1 : 2) + 2 * (blockIdx.x * 32 + lane);
  const bool on = i <= g.mx - 2;
  const int p0 = (k * g.my + 1) * g.mx + i, q0 = SplitRow::at(g, on ? i : 1, 1, k);  // row j = 1
  const double *lf = L.lf64 + q0, *lw = L.lw64 + q0;
  if (on) {
    const int oe = g.px && i == g.mx - 2 ? -(g.mx - 3) : 1, ow = g.px && i == 1 ? g.mx - 3 : -1;
    const int pl = g.mx * g.my, ot = g.pz && k == g.mz - 2 ? -(g.mz - 3) * pl : pl,
              ob = g.pz && k == 1 ? (g.mz - 3) * pl : -pl;
#pragma unroll 4
    for (int j = w; j < nr; j += NW) {
      const int p = p0 + j * g.mx;
      const double m = __ldg(lf + (size_t)j * pitch);
      double v;
      if constexpr (FUSED) {
        const int on_ = g.py && j == nr - 1 ? -(nr - 1) * g.mx : g.mx, os = g.py && j == 0 ? (nr - 1) * g.mx : -g.mx;
        const double *wp = lw + (size_t)j * pitch;
        v = m * r[p];
        v = fma(__ldg(wp + EP * S), x[p + oe], v);
        v = fma(__ldg(wp + WP * S), x[p + ow], v);
        v = fma(__ldg(wp + TP * S), x[p + ot], v);
        v = fma(__ldg(wp + BP * S), x[p + ob], v);
        v = fma(__ldg(wp + NP * S), x[p + on_], v);
        v = fma(__ldg(wp + SP * S), x[p + os], v);
        v = fma(__ldg(wp + CP * S), x[p], v);
      } else {
        v = m * (rsplit ? r[q0 + (size_t)j * pitch] : r[p]);
      }
      sr[32 * j + lane] = v;
    }
  }
  // the solving warp in turn, so that neighbouring blocks' use different
  // schedulers
  const int np = (nr + kAhead - 1) / kAhead * kAhead;
  for (int j = nr + w; j < np; j += NW) sr[32 * j + lane] = 0.0;
  const bool solver = on && w == ((blockIdx.x + blockIdx.y) & (NW - 1));
  double nx[kAhead];
  if (solver) rows_ahead(nx, lf + S, pitch, 0, nr);
  __syncthreads();
  if (solver) lanes_solve(sr, nx, lf + S, lf + 2 * S, pitch, nr, np, lane);
  __syncthreads();
  if (on)
#pragma unroll 4
    for (int j = w; j < nr; j += NW) {
      const int p = p0 + j * g.mx;
      const double d = sr[32 * j + lane];
      xnew[p] = x ? fma(omega, d, x[p]) : omega * d;
    }
}

void launch_lines(const LevelDev &L, bool fused, const double *r, const double *x, double *xnew, double omega, int color,
                  int rsplit, cudaStream_t s) {
  static PerDevice attr;
  allow_smem(attr, 200 * 1024, k_lines<true>, k_lines<false>);
  const dim3 grd(line_tiles_x(L.g), L.g.mz - 2);
  const size_t smem = lines_smem(L.g);
  const int nt = 32 * kLineWarps;
  if (fused) launch_dep(k_lines<true>, grd, nt, smem, s, L, r, x, xnew, omega, color, rsplit);
  else launch_dep(k_lines<false>, grd, nt, smem, s, L, r, x, xnew, omega, color, rsplit);
}

}  // namespace cvb
