// The V-cycle's small levels in two kernels: everything from the first sweep on
// the tail's finest level down to the coarsest right-hand side, and everything
// from the coarsest solution back up to the last sweep there.
//
// On levels of a few thousand cells each of a cycle's eleven passes a level is
// bound by its launch and by one chain of latencies, not by its work.  Here one
// cluster of 16 blocks, 512 threads each, runs the passes one after another with
// a cluster barrier between them; the vectors stay in the L2 cache.
#include "stencil_body.cuh"

namespace cvb {

constexpr int kTailCtas = 16, kTailGroups = 4, kTailUnits = kTailCtas * kTailGroups;

template <typename T>
struct TailArgs {
  LevelDev L[kTailLevels + 1];  // [0]: the level below the tail
  T *v[kTailLevels + 1][4];     // each level's right-hand side, correction, scratch, residual
  int n;                        // levels 1 .. n, the finest last
  int pre, post;
  T omega;
};

// tiles of four lines of either colour in a plane
__host__ __device__ inline int tail_tiles(const Geom &g) { return ((g.mx - 1) / 2 + 3) / 4; }

// Every thread of the cluster: its earlier writes are visible to the others' later reads.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// the 128 threads of one group of a block
__device__ __forceinline__ void group_barrier() {
  asm volatile("bar.sync %0, %1;" ::"r"((int)threadIdx.y + 1), "n"(kFlat) : "memory");
}

// A row's coefficients in registers: row32 and row64 (stencil_body.cuh) with the
// loads apart from the arithmetic, operation for operation.  (Those two written with
// these took a third more registers, and the 19-point residual of a colour at 128^3
// 31 us for 27.)
template <bool X>
struct Row32 {
  float g11, g22, g33, w11, s22, b33, aj;
  float g12, g13, g21, g23, g31, g32, w12, w13, s21, s23, b31, b32;  // cross terms (X only)
  uint32_t c, cw, cs, cb;
  __device__ __forceinline__ void load_codes(const Geom &g, const uint32_t *__restrict__ code, int p) {
    c = __ldg(code + p);
    if constexpr (X) {
      cw = __ldg(code + p - 1); cs = __ldg(code + p - g.mx); cb = __ldg(code + p - g.mx * g.my);
    }
  }
  __device__ __forceinline__ void load(const Geom &g, const float *__restrict__ gf, const float *__restrict__ ajf,
                                       int p, int n) {
    const int pw = p - 1, ps = p - g.mx, pb = p - g.mx * g.my;  // lower neighbours (never wrapped)
    g11 = __ldg(gf + p);
    if constexpr (X) { g12 = __ldg(gf + n + p); g13 = __ldg(gf + 2 * n + p); g21 = __ldg(gf + 3 * n + p); }
    g22 = __ldg(gf + 4 * n + p);
    if constexpr (X) { g23 = __ldg(gf + 5 * n + p); g31 = __ldg(gf + 6 * n + p); g32 = __ldg(gf + 7 * n + p); }
    g33 = __ldg(gf + 8 * n + p);
    w11 = __ldg(gf + pw);
    if constexpr (X) { w12 = __ldg(gf + n + pw); w13 = __ldg(gf + 2 * n + pw); s21 = __ldg(gf + 3 * n + ps); }
    s22 = __ldg(gf + 4 * n + ps);
    if constexpr (X) { s23 = __ldg(gf + 5 * n + ps); b31 = __ldg(gf + 6 * n + pb); b32 = __ldg(gf + 7 * n + pb); }
    b33 = __ldg(gf + 8 * n + pb);
    aj = __ldg(ajf + p);
  }
  __device__ __forceinline__ float apply(const Star<float> &s) const {
    float fe = g11 * (s.E - s.P), fw = w11 * (s.P - s.W), fn = g22 * (s.N - s.P);
    float fs = s22 * (s.P - s.S), ft = g33 * (s.Tt - s.P), fb = b33 * (s.P - s.B);
    if constexpr (X) {
      fe = fe + cross32(code_branch(c, 0, 0), g12, s.N + s.NE, s.P + s.E, s.S + s.SE) +
           cross32(code_branch(c, 0, 1), g13, s.Tt + s.TE, s.P + s.E, s.B + s.BE);
      fw = fw + cross32(code_branch(cw, 0, 0), w12, s.NW + s.N, s.W + s.P, s.SW + s.S) +
           cross32(code_branch(cw, 0, 1), w13, s.TW + s.Tt, s.W + s.P, s.BW + s.B);
      fn = fn + cross32(code_branch(c, 1, 0), g21, s.E + s.NE, s.P + s.N, s.W + s.NW) +
           cross32(code_branch(c, 1, 1), g23, s.Tt + s.TN, s.P + s.N, s.B + s.BN);
      fs = fs + cross32(code_branch(cs, 1, 0), s21, s.SE + s.E, s.S + s.P, s.SW + s.W) +
           cross32(code_branch(cs, 1, 1), s23, s.TS + s.Tt, s.S + s.P, s.BS + s.B);
      ft = ft + cross32(code_branch(c, 2, 0), g31, s.E + s.TE, s.P + s.Tt, s.W + s.TW) +
           cross32(code_branch(c, 2, 1), g32, s.N + s.TN, s.P + s.Tt, s.S + s.TS);
      fb = fb + cross32(code_branch(cb, 2, 0), b31, s.BE + s.E, s.B + s.P, s.BW + s.W) +
           cross32(code_branch(cb, 2, 1), b32, s.BN + s.N, s.B + s.P, s.BS + s.S);
    }
    float acc = act(c, CODE_ACT_E) * fe - act(c, CODE_ACT_W) * fw + act(c, CODE_ACT_N) * fn -
                act(c, CODE_ACT_S) * fs + act(c, CODE_ACT_T) * ft - act(c, CODE_ACT_B) * fb;
    return (c & CODE_IDENTITY) ? s.P : -aj * acc;
  }
};
template <bool X>
struct Row64 {
  double w[X ? 19 : 7];
  uint32_t c;
  __device__ __forceinline__ void load_codes(const uint32_t *__restrict__ code, int p) { c = __ldg(code + p); }
  __device__ __forceinline__ void load(const double *__restrict__ w64, int p, int n) {
#pragma unroll
    for (int m = 0; m < (X ? 19 : 7); m++) w[m] = __ldg(w64 + p + (size_t)m * n);
  }
  __device__ __forceinline__ double apply(const Star<double> &s) const {
    double r = w[CP] * s.P;
    r = fma(w[EP], s.E, r); r = fma(w[WP], s.W, r);
    r = fma(w[NP], s.N, r); r = fma(w[SP], s.S, r);
    r = fma(w[TP], s.Tt, r); r = fma(w[BP], s.B, r);
    if constexpr (X) {
      r = fma(w[NE], s.NE, r); r = fma(w[SE], s.SE, r); r = fma(w[NW], s.NW, r); r = fma(w[SW], s.SW, r);
      r = fma(w[TN], s.TN, r); r = fma(w[BN], s.BN, r); r = fma(w[TS], s.TS, r); r = fma(w[BS], s.BS, r);
      r = fma(w[TE], s.TE, r); r = fma(w[BE], s.BE, r); r = fma(w[TW], s.TW, r); r = fma(w[BW], s.BW, r);
    }
    return (c & CODE_IDENTITY) ? s.P : r;
  }
};
template <bool X>
__device__ __forceinline__ void tail_load(Row32<X> &r, const LevelDev &L, int p) {
  r.load_codes(L.g, L.code, p);
  r.load(L.g, L.gf32, L.ajf32, p, (int)L.g.n());
}
template <bool X>
__device__ __forceinline__ void tail_load(Row64<X> &r, const LevelDev &L, int p) {
  r.load_codes(L.code, p);
  r.load(L.w64, p, (int)L.g.n());
}
template <typename T>
struct TailTypes;
template <>
struct TailTypes<float> {
  template <bool X>
  using Row = Row32<X>;
  __device__ static const float *fac(const LevelDev &L) { return L.line32; }
};
template <>
struct TailTypes<double> {
  template <bool X>
  using Row = Row64<X>;
  __device__ static const double *fac(const LevelDev &L) { return L.line64; }
};

// What a group keeps of its tile through a level's passes: four lines of each
// colour at one k (columns 2 tile .. 2 tile + 1 of four), a thread one cell of each
// colour with its row's coefficients and right-hand side, a warp one line of each
// colour with a row's Thomas factors a lane.  In registers: the barrier empties the
// L1 cache, and reading them again from the L2 took more than the sweep itself (the
// passes of a 19-point level of 16^3 cells 2.4 us each).
template <typename T, bool X>
struct TailTile {
  using Row = typename TailTypes<T>::template Row<X>;
  Row row[2];
  T b[2], fa[2], fm[2], fc[2];
  int p[2];
  Off o[2];
  bool ok[2];
  bool any;  // the group has a tile

  __device__ __forceinline__ void load(const LevelDev &L, const T *bv, int unit) {
    const Geom &g = L.g;
    const int t = threadIdx.x, tx = t & 3, j = (t >> 2) + 1, warp = t >> 5, lane = t & 31;
    const int nt = tail_tiles(g);
    any = unit < nt * (g.mz - 2);
    const int k = unit / nt + 1, tile = unit - (k - 1) * nt;
    const LineFac F = LineFac::of(g);
    const T *fac = TailTypes<T>::fac(L);
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int first = (c + k) & 1 ? 1 : 2, i = first + 2 * (4 * tile + tx), il = first + 2 * (4 * tile + warp);
      ok[c] = any && i <= g.mx - 2 && j <= g.my - 2;
      p[c] = ok[c] ? (k * g.my + j) * g.mx + i : 0;
      fa[c] = fm[c] = fc[c] = b[c] = T(0);
      if (any && il <= g.mx - 2 && lane < g.my - 2) {
        const T *f = fac + F.line(il, k) + lane;
        fa[c] = __ldg(f);
        fm[c] = __ldg(f + F.Q);
        fc[c] = __ldg(f + 2 * F.Q);
      }
      if (ok[c]) {
        o[c] = offsets(g, i, j, k);
        b[c] = bv[p[c]];
        tail_load(row[c], L, p[c]);
      }
    }
  }
  __device__ __forceinline__ T residual(const T *x, int c, T &xo) const {
    const Star<T> s = load_star<T>(x, p[c], o[c]);
    xo = s.P;
    return b[c] - row[c].apply(s);
  }
  // One half-sweep, xin -> xout.  In place for zebra_fusable levels; else the
  // thread's cell of the other colour is copied.  zero: x is zero, xin is not read
  // and the other colour's cells are zeroed.
  template <int C>
  __device__ __forceinline__ void half(const T *xin, T *xout, T omega, bool zero, T *sm) const {
    if (!any) return;
    const int t = threadIdx.x, tx = t & 3, ty = t >> 2, warp = t >> 5, lane = t & 31;
    const bool copy = xin != xout && ok[1 - C];
    T r = T(0), xo = T(0), other = T(0);
    if (copy && !zero) other = xin[p[1 - C]];
    if (ok[C]) r = zero ? b[C] : residual(xin, C, xo);
    sm[tx * 33 + ty] = r;
    group_barrier();
    // d = m (r - a d_prev), then e = d - c e_next, as scans of affine maps over the lanes
    T B = -fm[C] * fa[C], G = fm[C] * sm[warp * 33 + lane];
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const T Bp = __shfl_up_sync(0xffffffffu, B, s), Gp = __shfl_up_sync(0xffffffffu, G, s);
      if (lane >= s) { G = B * Gp + G; B = B * Bp; }
    }
    B = -fc[C];
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const T Bn = __shfl_down_sync(0xffffffffu, B, s), Gn = __shfl_down_sync(0xffffffffu, G, s);
      if (lane + s < 32) { G = B * Gn + G; B = B * Bn; }
    }
    sm[warp * 33 + lane] = G;
    group_barrier();
    if (ok[C]) xout[p[C]] = xo + omega * sm[tx * 33 + ty];
    if (copy) xout[p[1 - C]] = other;
  }
  __device__ __forceinline__ void sweep(const LevelDev &L, T *x, T *tmp, T omega, bool zero, T *sm) const {
    T *mid = zebra_fusable<T>(L) ? x : tmp;
    half<0>(zero ? nullptr : x, mid, omega, zero, sm);
    cluster_barrier();
    half<1>(mid, x, omega, false, sm);
    cluster_barrier();
  }
};

template <typename T, bool X, bool UP>
__global__ void __launch_bounds__(kFlat *kTailGroups) k_tail(const __grid_constant__ TailArgs<T> A) {
  __shared__ T smem[kTailGroups][4 * 33];
  dep_sync();
  if (gated(A.L[A.n].gate)) return;
  const int unit = threadIdx.y * kTailCtas + blockIdx.x;
  T *sm = smem[threadIdx.y];
  TailTile<T, X> tile;
  if constexpr (!UP) {
    for (int l = A.n; l >= 1; l--) {
      const LevelDev &L = A.L[l], &C = A.L[l - 1];
      T *x = A.v[l][1], *tmp = A.v[l][2], *res = A.v[l][3];
      tile.load(L, A.v[l][0], unit);
      // the ring stays zero in both copies of x
      const int mx = L.g.mx, my = L.g.my, mz = L.g.mz, pl = mx * my, n = (int)L.g.n();
      for (int q = unit * kFlat + threadIdx.x; q < n; q += kTailUnits * kFlat) {
        const int k = q / pl, j = (q - k * pl) / mx, i = q - k * pl - j * mx;
        if (i < 1 || i > mx - 2 || j < 1 || j > my - 2 || k < 1 || k > mz - 2) x[q] = tmp[q] = T(0);
      }
      for (int q = 0; q < A.pre; q++) tile.sweep(L, x, tmp, A.omega, q == 0, sm);
#pragma unroll
      for (int c = 0; c < 2; c++) {
        T xo;
        if (tile.ok[c]) res[tile.p[c]] = tile.residual(x, c, xo);
      }
      cluster_barrier();
      const int pb = plane_blocks(C.g);
      for (int v = unit; v < pb * C.g.mz; v += kTailUnits) restrict_body<T>(L, C, res, A.v[l - 1][0], v % pb, 0, v / pb);
      if (l > 1) cluster_barrier();
    }
  } else {
    for (int l = 1; l <= A.n; l++) {
      const LevelDev &L = A.L[l], &C = A.L[l - 1];
      T *x = A.v[l][1], *tmp = A.v[l][2];
      const ProlongGrid P = ProlongGrid::of(L);
      for (int v = unit; v < P.gx * P.gz; v += kTailUnits)
        prolong_body<T>(C, L, A.v[l - 1][1], x, v % P.gx, 0, v / P.gx);
      tile.load(L, A.v[l][0], unit);
      cluster_barrier();
      for (int q = 0; q < A.post; q++) tile.sweep(L, x, tmp, A.omega, false, sm);
    }
  }
}

template <typename T>
static cudaLaunchConfig_t tail_config(cudaLaunchAttribute (&at)[2], cudaStream_t s) {
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kTailCtas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(kTailCtas);
  c.blockDim = dim3(kFlat, kTailGroups);
  c.stream = s;
  c.attrs = at;
  c.numAttrs = pdl_enabled() ? 2 : 1;
  return c;
}

// Whether the current device takes these clusters (16 blocks are beyond the portable eight).
template <typename T>
static bool tail_runs() {
  void (*ks[4])(TailArgs<T>) = {k_tail<T, false, false>, k_tail<T, false, true>, k_tail<T, true, false>,
                                k_tail<T, true, true>};
  for (auto k : ks) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t c = tail_config<T>(at, nullptr);
    c.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k, &c) != cudaSuccess || clusters < 1) {
      cudaGetLastError();
      return false;
    }
  }
  return true;
}

template <typename T>
int tail_levels(const LevelDev *L, int nlevels) {
  static PerDevice attr;
  const bool runs = attr.get(current_device(), tail_runs<T>);
  int n = 0;
  while (runs && n < kTailLevels && n + 1 < nlevels - 1) {
    const Geom &g = L[n + 1].g;
    if (g.my - 2 > 32 || tail_tiles(g) * (g.mz - 2) > kTailUnits) break;
    n++;
  }
  return n;
}
template int tail_levels<float>(const LevelDev *, int);
template int tail_levels<double>(const LevelDev *, int);

template <typename T>
void launch_tail(const LevelDev *L, T *const (*v)[4], int n, int pre, int post, T omega, bool up, cudaStream_t s) {
  TailArgs<T> A;
  bool cross = false;
  for (int l = 0; l <= n; l++) {
    A.L[l] = L[l];
    for (int q = 0; q < 4; q++) A.v[l][q] = v[l][q];
    cross = cross || (l > 0 && has_cross<T>(L[l]));
  }
  A.n = n;
  A.pre = pre;
  A.post = post;
  A.omega = omega;
  cudaLaunchAttribute at[2];
  const cudaLaunchConfig_t c = tail_config<T>(at, s);
  if (up) cudaLaunchKernelEx(&c, cross ? k_tail<T, true, true> : k_tail<T, false, true>, A);
  else cudaLaunchKernelEx(&c, cross ? k_tail<T, true, false> : k_tail<T, false, false>, A);
  count_launch();
}
template void launch_tail<float>(const LevelDev *, float *const (*)[4], int, int, int, float, bool, cudaStream_t);
template void launch_tail<double>(const LevelDev *, double *const (*)[4], int, int, int, double, bool, cudaStream_t);

}  // namespace cvb
