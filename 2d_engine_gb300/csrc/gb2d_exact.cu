// FP64 kernels that reproduce the reference's own FP64 CPU arithmetic: ghost
// fills, WENO5 advection and reinitialisation sweeps, ENO3 velocity advection,
// curvature, ghost-fluid Poisson assembly and the GFM velocity update.
// Built with --fmad=false: every multiply and add rounds separately, in the
// reference's association order, so results match it bit for bit (the sine of
// the smeared Heaviside is the only libm call and may differ in the last ulp).
// The "mixed" advection variants (FP32 flux evaluation, FP64 state) live here
// too so that they share the loaders.
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "gb2d_internal.cuh"
#include "gb2d_schemes.cuh"

namespace gb2d {

namespace {

inline unsigned blocks_for(size_t n, int threads = kThreads) { return (unsigned)((n + threads - 1) / threads); }

// x * y >= 0 as IEEE evaluates it.  When both are normal and finite and the
// product's exponent keeps it above the subnormal range, only the signs decide;
// zeros, subnormals, infinities, NaN and products that may round to zero take
// the FP64 multiply.
__device__ __forceinline__ bool prod_ge0(double x, double y) {
  const unsigned bx = words(x).hi, by = words(y).hi;
  const int ex = (int)((bx >> 20) & 0x7ff), ey = (int)((by >> 20) & 0x7ff);
  if (ex != 0 && ey != 0 && ex != 0x7ff && ey != 0x7ff && ex + ey >= 972) return (int)(bx ^ by) >= 0;
  return plain_mul(x, y) >= 0;
}


// FillGhostCellsFrom (FIELD_STRUCTURE_2D.h:374-449): interior copied, each ghost
// layer copies the second interior line, corners untouched.
__global__ void k_fill_ghost_copy(double* dst_a, int gd, const double* __restrict__ src_a, int gs, int nI, int nJ, int g) {
  pdl_enter();
  DField d = dfield(dst_a, gd, nI, nJ);
  DField s = dfield((double*)src_a, gs, nI, nJ);
  GB_FOR_IJ(ii, jj, nI + 2 * g, nJ + 2 * g) {
    int i = ii - g, j = jj - g;
    bool in_i = i >= 0 && i < nI, in_j = j >= 0 && j < nJ;
    if (in_i && in_j)
      GB_AT(d, i, j) = GB_AT(s, i, j);
    else if (in_j)
      GB_AT(d, i, j) = GB_AT(s, i < 0 ? 1 : nI - 2, j);
    else if (in_i)
      GB_AT(d, i, j) = GB_AT(s, i, j < 0 ? 1 : nJ - 2);
  }
}

// FillGhostCellsContinuousDerivativesFrom(phi, true, tid) on the field itself
// (FIELD_STRUCTURE_2D.h:641-716).  One thread per boundary line keeps the
// reference's layer order: left/bottom outermost first (the outer layer reads
// the previous inner value), right/top innermost first.
__global__ void k_extrapolate(double* a, int g, int nI, int nJ) {
  pdl_enter();
  DField f = dfield(a, g, nI, nJ);
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nJ) {
    int j = t;
    for (int i = -g; i <= -1; ++i) GB_AT(f, i, j) = 2.0 * GB_AT(f, i + 1, j) - GB_AT(f, i + 2, j);
    for (int i = nI; i <= nI - 1 + g; ++i) GB_AT(f, i, j) = 2.0 * GB_AT(f, i - 1, j) - GB_AT(f, i - 2, j);
  }
  if (t < nI) {
    int i = t;
    for (int j = nJ; j <= nJ - 1 + g; ++j) GB_AT(f, i, j) = 2.0 * GB_AT(f, i, j - 1) - GB_AT(f, i, j - 2);
    for (int j = -g; j <= -1; ++j) GB_AT(f, i, j) = 2.0 * GB_AT(f, i, j + 1) - GB_AT(f, i, j + 2);
  }
}

// Reads of the WENO scratch copy (scalar_field_ghost, ghost 3) synthesised from
// phi's interior: ghost layers hold the second interior line.
__device__ __forceinline__ void gather_x(const DField& s, int i, int j, double q[7]) {
  const int nI = s.nI;
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    int ii = i - 3 + k;
    ii = ii < 0 ? 1 : (ii >= nI ? nI - 2 : ii);
    q[k] = __ldg(&GB_AT(s, ii, j));
  }
}
__device__ __forceinline__ void gather_y(const DField& s, int i, int j, double q[7]) {
  const int nJ = s.nJ;
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    int jj = j - 3 + k;
    jj = jj < 0 ? 1 : (jj >= nJ ? nJ - 2 : jj);
    q[k] = __ldg(&GB_AT(s, i, jj));
  }
}

struct LSArgs {
  int ni, nj;
  double odx, ody, eps;
  float odx_f, ody_f, eps_f;  // the same in FP32 for the FP32 flux path
  int fast_f;                 // FP32 epsilon is in mx_sign's range
  int fast;                   // epsilon is in weno5_side_fast's range (and dx in [2^-300, 2^300], for dtau s h)
  int row0, rows;             // the launch's first tile row; tile rows of the grid (row `rows` copies the ghost ring)
};

// Reads phi's interior at (i, j), where positions outside it hold the second interior
// line as in the reference's ghost-filled scratch copy (scalar_field_ghost, ghost 3).
__device__ __forceinline__ double ghosted(const DField& s, int i, int j) {
  i = i < 0 ? 1 : (i >= s.nI ? s.nI - 2 : i);
  j = j < 0 ? 1 : (j >= s.nJ ? s.nJ - 2 : j);
  return __ldg(&GB_AT(s, i, j));
}

// One tile of the exact FP64 sweeps: kExX x kExY nodes with every WENO first difference
// o (q[k+1] - q[k]) formed once (12 per node when each node forms its own, 2.8 to 3.4
// here); dxs[r][c + k] is difference k of node (c, r) along x, dys[r + k][c] along y.
constexpr int kExX = 32, kExY = 4;
struct ExactTile {
  double ph[kExY + 6][kExX + 6];
  double dxs[kExY][kExX + 5], dys[kExY + 5][kExX];
};

// Stages the tile at (i0, j0); true in every thread where all differences are in
// weno5_side_fast's range.
__device__ __forceinline__ bool stage_exact(ExactTile& t, const DField& src, const LSArgs& a, int i0, int j0) {
  constexpr int NT = 2 * kExX * kExY, SW = kExX + 6, DW = kExX + 5;
  const int tid = threadIdx.x;
  for (int k = tid; k < SW * (kExY + 6); k += NT) t.ph[k / SW][k % SW] = ghosted(src, i0 - 3 + k % SW, j0 - 3 + k / SW);
  __syncthreads();
  bool ok = true;
  for (int k = tid; k < kExY * DW; k += NT) {
    const int c = k % DW, r = k / DW;
    const double d = a.odx * (t.ph[r + 3][c + 1] - t.ph[r + 3][c]);
    ok = ok && weno5_in_range(d);
    t.dxs[r][c] = d;
  }
  for (int k = tid; k < (kExY + 5) * kExX; k += NT) {
    const int c = k % kExX, r = k / kExX;
    const double d = a.ody * (t.ph[r + 1][c + 3] - t.ph[r][c + 3]);
    ok = ok && weno5_in_range(d);
    t.dys[r][c] = d;
  }
  return __syncthreads_and(ok && a.fast);
}

// Difference k (0..5) of node (c, r) along direction dir (0: x, 1: y).
__device__ __forceinline__ double ex_diff(const ExactTile& t, int dir, int c, int r, int k) {
  return dir == 0 ? t.dxs[r][c + k] : t.dys[r + k][c];
}
// One-sided derivative of node (c, r): side 0 the minus, side 1 the plus one.
template <bool FAST>
__device__ __forceinline__ double ex_side(const ExactTile& t, int dir, int c, int r, int side, double eps) {
  const double* d = dir == 0 ? &t.dxs[r][c] : &t.dys[r][c];
  const int st = dir == 0 ? 1 : kExX, first = side ? 5 * st : 0, step = side ? -st : st;
  const double a1 = d[first], a2 = d[first + step], a3 = d[first + 2 * step], a4 = d[first + 3 * step], a5 = d[first + 4 * step];
  if (FAST) return weno5_side_fast(a1, a2, a3, a4, a5, eps);
  return weno5_side<double>(a1, a2, a3, a4, a5, eps);
}
// g g, or 0 for |g| < 2^-400; |g| < 2^500.
__device__ __forceinline__ double sqr_flush(double g) {
  return ((words(g).hi >> 20) & 0x7ffu) < 1023u - 400u ? 0.0 : mul_rn(g, g);
}
// Out of line: the general forms serve differences outside the fast range only.
__device__ __noinline__ double ex_side_general(const ExactTile& t, int dir, int c, int r, int side, double eps) {
  return ex_side<false>(t, dir, c, r, side, eps);
}

// Copies src's ghost ring (width 2) to dst, a block's threads each taking every
// n-th element from the first-th.
__device__ __forceinline__ void copy_ring(const DField& src, const DField& dst, int first, int n) {
  const int W = src.nI + 4, rows = 4 * W, total = rows + 4 * src.nJ;
  for (int k = first; k < total; k += n) {
    int i, j;
    if (k < rows) {
      const int y = k / W;
      i = k - y * W - 2;
      j = y < 2 ? y - 2 : src.nJ + y - 2;
    } else {
      const int y = (k - rows) >> 2, x = (k - rows) & 3;
      i = x < 2 ? x - 2 : src.nI + x - 2;
      j = y;
    }
    GB_AT(dst, i, j) = GB_AT(src, i, j);
  }
}

// WENO5th (ADVECTION_METHOD_2D.h:508-663) for the node-grid level set: writes
// dst's interior from src, copies src's ghost ring (the sweep leaves phi's own
// ghosts to the caller's extrapolation).
// The exact FP64 sweep, bound by the FP64 pipe: each node evaluates the upwind side
// only (one WENO derivative per direction instead of two), from differences formed
// once per tile, the x and y directions on two threads.  The grid's last block row
// copies the ghost ring.
__global__ void __launch_bounds__(2 * kExX* kExY) k_weno5_advect_exact(const double* __restrict__ src_a, double* __restrict__ dst_a,
                                                                     const double* __restrict__ ua_a, const double* __restrict__ va_a,
                                                                     LSArgs a, DtArg dt_arg) {
  pdl_enter();
  constexpr int NN = kExX * kExY;
  __shared__ ExactTile t;
  __shared__ double vfy[NN];
  const DField src = dfield((double*)src_a, 2, a.ni, a.nj), dst = dfield(dst_a, 2, a.ni, a.nj);
  const int by = a.row0 + (int)blockIdx.y;
  if (by == a.rows) {
    copy_ring(src, dst, blockIdx.x * (2 * NN) + threadIdx.x, gridDim.x * (2 * NN));
    return;
  }
  const int i0 = (int)blockIdx.x * kExX, j0 = by * kExY;
  const bool fast = stage_exact(t, src, a, i0, j0);
  const int node = threadIdx.x & (NN - 1), dir = threadIdx.x / NN;
  const int c = node & (kExX - 1), r = node / kExX, i = i0 + c, j = j0 + r;
  const bool in = i < a.ni && j < a.nj;
  double wf = 0;  // u fx or v fy
  if (in) {
    const DField ua = dfield((double*)ua_a, 3, a.ni + 1, a.nj), va = dfield((double*)va_a, 3, a.ni, a.nj + 1);
    const double w = dir == 0 ? (__ldg(&GB_AT(ua, i + 1, j)) + __ldg(&GB_AT(ua, i, j))) * 0.5
                              : (__ldg(&GB_AT(va, i, j + 1)) + __ldg(&GB_AT(va, i, j))) * 0.5;
    const int side = gtz(w) ? 0 : 1;
    wf = w * (fast ? ex_side<true>(t, dir, c, r, side, a.eps) : ex_side_general(t, dir, c, r, side, a.eps));
  }
  if (dir == 1) vfy[node] = wf;
  __syncthreads();
  if (in && dir == 0) GB_AT(dst, i, j) = t.ph[r + 3][c + 3] - dt_arg.get() * (wf + vfy[node]);
}

// The plain FP64 forms of the assembly's expressions, for operands outside the fast forms'
// ranges (out of line, as plain_mul).
__device__ __noinline__ double plain_mul4(double a, double b, double c, double d) { return a * b * c * d; }
__device__ __noinline__ double plain_sign(double p, double dx2) { return p / sqrt(p * p + dx2); }
__device__ __noinline__ double plain_div(double odx, double du, double ody, double dv, double one_over_dt) {
  return (odx * du + ody * dv) * one_over_dt;
}
__device__ __noinline__ double plain_beta(double vc, double vn, double ac, double an) {
  return vc * vn * (an + ac) / (vc * an + vn * ac);
}

// Sign function of Reinitialization (EULERIAN_FLUID_SOLVER_2D.h:2431-2435).  dx2 = dx dx.
__global__ void k_reinit_sign(const double* __restrict__ phi_a, double* __restrict__ S, int ni, int nj, double dx2) {
  pdl_enter();
  DField phi = dfield((double*)phi_a, 2, ni, nj);
  const bool fast = mid_range<400>(dx2) && !is_zero(dx2);
  GB_FOR_IJ(i, j, ni, nj) {
    const size_t t = (size_t)j * ni + i;
    const double p = GB_AT(phi, i, j);
    if (fast && mid_range<200>(p)) {  // the same value: one FP64 addition, the rest on the integer pipes
      const Words w = words(div_pos(absd(p), sqrt_rn(mul_rn(p, p) + dx2)));
      S[t] = is_zero(p) ? p : from_words(w.lo, w.hi | (words(p).hi & 0x80000000u));
    } else {
      S[t] = plain_sign(p, dx2);
    }
  }
}

// WENO5thReinitialization (ADVECTION_METHOD_2D.h:1401-1658), the mixed form.
__global__ void k_reinit_sweep_mixed(const double* __restrict__ src_a, double* __restrict__ dst_a, const double* __restrict__ S, LSArgs a,
                                     double dtau) {
  pdl_enter();
  int ni = a.ni, nj = a.nj;
  int W = ni + 4, H = nj + 4;
  int ix = blockIdx.x * blockDim.x + threadIdx.x, jy = blockIdx.y * blockDim.y + threadIdx.y;
  if (ix >= W || jy >= H) return;
  int i = ix - 2, j = jy - 2;
  DField src = dfield((double*)src_a, 2, ni, nj), dst = dfield(dst_a, 2, ni, nj);
  double old = GB_AT(src, i, j);
  if (i < 0 || j < 0 || i >= ni || j >= nj) {
    GB_AT(dst, i, j) = old;
    return;
  }
  double q[7];
  double out = old;
  float mx, px, my, py, h;
  gather_x(src, i, j, q);
  weno5_pair_f32(q, a.odx_f, a.eps_f, mx, px);
  gather_y(src, i, j, q);
  weno5_pair_f32(q, a.ody_f, a.eps_f, my, py);
  double s = __ldg(&S[i + (size_t)j * ni]);
  if (godunov_h<float>(narrow(s), mx, px, my, py, h)) out = old - dtau * s * widen(h);
  GB_AT(dst, i, j) = out;
}

// Godunov choice of one direction from certain signs of s and of the one-sided
// derivatives (godunov_h's cases): 0 the minus side, 1 the plus side, 2 neither
// (rarefaction), 3 both values are needed (a shock, or a sign that is not certain).
// With |s| >= 2^-100 and derivatives above weno5_sign's margin no product s m
// underflows, so the products' signs are the signs' products.
__device__ __forceinline__ int godunov_case(int ss, int sm, int sp) {
  const int a = ss * sm, b = ss * sp;
  return a > 0 && b > 0 ? 0 : a < 0 && b < 0 ? 1 : a < 0 && b > 0 ? 2 : 3;
}

// The exact FP64 sweep, bound by the FP64 and integer pipes: a node's update uses one
// of its two one-sided derivatives per direction (or neither, in a rarefaction), and
// which one follows from their signs.  FP32 evaluations of the candidate stencils
// settle the signs almost everywhere; a thread evaluates the chosen side of one
// direction of its node exactly, and the few that need both values (shocks, flat
// directions) put the second evaluation on the block's list, which the block works
// off densely.  The update has the bits of evaluating all four derivatives.  A block row
// after the tiles', where the launch has one, copies src's ghost ring (needed until both
// buffers of the sweeps hold it).
// One level-set TVD-RK3 with its 75 sweeps at 512^2: 22.6 ms with four derivatives per
// node in FP64 divisions and products (578 FP64 instructions per node), 6.4 ms with the
// chosen sides, the differences shared and the divisions on the integer pipes (160), 3.5
// ms with every product there too (74).  The FP64 pipe is half busy then and the wait for
// dependent results shows: 5 blocks of 48 registers per SM 3.44 ms, 4 of 64 3.62, 3 of 79
// 3.97.  Tiles of 32 x 8 nodes are 3% slower, and 1.3 times as slow on small grids, where
// they leave SMs idle; 32 x 2 ones are no faster there.
__global__ void __launch_bounds__(2 * kExX * kExY, 5) k_reinit_sweep_exact(const double* __restrict__ src_a, double* __restrict__ dst_a,
                                                                     const double* __restrict__ S, LSArgs a, double dtau) {
  pdl_enter();
  constexpr int NN = kExX * kExY, NT = 2 * NN;  // nodes and threads: thread dir NN + node
  __shared__ ExactTile t;
  __shared__ double plus[NT], dy_own[NN];
  __shared__ unsigned short list[NT];
  __shared__ signed char dy_pick[NN];
  __shared__ int count;
  const DField src = dfield((double*)src_a, 2, a.ni, a.nj), dst = dfield(dst_a, 2, a.ni, a.nj);
  const int by = a.row0 + (int)blockIdx.y;
  if (by == a.rows) {
    copy_ring(src, dst, blockIdx.x * NT + threadIdx.x, gridDim.x * NT);
    return;
  }
  const int tid = threadIdx.x, i0 = (int)blockIdx.x * kExX, j0 = by * kExY;
  if (tid == 0) count = 0;
  const bool fast = stage_exact(t, src, a, i0, j0);
  const int node = tid & (NN - 1), dir = tid / NN, c = node & (kExX - 1), r = node / kExX, i = i0 + c, j = j0 + r;
  const bool in = i < a.ni && j < a.nj;
  const double s = in ? __ldg(&S[i + (size_t)j * a.ni]) : 0.0;
  const long long smag = mag_bits(s);
  // 2^-100 <= |s| < 2^100: S is the caller's in gb2d_reinit_sweep_apply, and mul_rn below takes
  // finite operands whose product stays in the normal range (dtau is in [2^-331, 2^300], |h| below 2^106).
  const bool sfast = smag >= ((1023LL - 100) << 52) && smag < ((1023LL + 100) << 52);
  int pick = in ? 3 : 2;
  if (in && fast && sfast) {
    float d[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) d[k] = narrow(ex_diff(t, dir, c, r, k));
    pick = godunov_case((int)words(s).hi < 0 ? -1 : 1, weno5_sign(d[0], d[1], d[2], d[3], d[4]), weno5_sign(d[5], d[4], d[3], d[2], d[1]));
  }
  if (in && fast && pick == 3) list[atomicAdd(&count, 1)] = (unsigned short)tid;
  __syncthreads();
  double own = 0;
  if (fast) {
    const int n = count, rounds = 1 + (n + NT - 1) / NT;
#pragma unroll 1
    for (int k = 0; k < rounds; ++k) {
      const int m = (k - 1) * NT + tid;
      const int item = k == 0 ? tid : m < n ? (int)list[m] : 0;
      if (k == 0 ? pick == 2 : m >= n) continue;
      const int nd = item & (NN - 1), side = k == 0 ? pick == 1 : 1;
      const double f = ex_side<true>(t, item / NN, nd & (kExX - 1), nd / kExX, side, a.eps);
      if (k == 0) own = f;
      else plus[item] = f;
    }
    __syncthreads();
  } else if (in) {
    own = ex_side_general(t, dir, c, r, 0, a.eps);
    plus[tid] = ex_side_general(t, dir, c, r, 1, a.eps);
  }
  if (in && pick == 3) {
    const double p = plus[tid];
    pick = godunov_pick(s, own, p, dir == 0);
    if (pick == 1) own = p;
  }
  if (dir == 1) {
    dy_own[node] = own;
    dy_pick[node] = (signed char)pick;
  }
  __syncthreads();
  if (!in || dir == 1) return;
  const double old = t.ph[r + 3][c + 3], gy = dy_own[node];
  const int ypick = dy_pick[node];
  if (pick < 0 || ypick < 0) {
    GB_AT(dst, i, j) = old;
    return;
  }
  double h = -1.0;
  if (fast && sfast) {  // the same values: |g| < 2^-400 changes neither the sum's root nor h
    const double g2 = (pick != 2 ? sqr_flush(own) : 0.0) + (ypick != 2 ? sqr_flush(gy) : 0.0);
    if (pick != 2 || ypick != 2) h = sqrt_rn(g2) - 1.0;
    GB_AT(dst, i, j) = old - mul_rn(mul_rn(s, dtau), h);
    return;
  }
  if (pick != 2 && ypick != 2)
    h = sqrt(own * own + gy * gy) - 1.0;
  else if (pick != 2)
    h = sqrt(own * own) - 1.0;
  else if (ypick != 2)
    h = sqrt(gy * gy) - 1.0;
  GB_AT(dst, i, j) = old - dtau * s * h;
}

// One tile of the mixed sweeps: kMxX x kMxY nodes with every WENO first difference formed
// once in FP64 (2.8 per node instead of 12; FP64 issue is scarce), narrowed to FP32 and
// scaled; the same values as the per-node gathers.  dxs[r][c + k] is difference k of node
// (c, r) along x, dys[r + k][c] along y.  Threads (kMxX, kMxY).
constexpr int kMxX = 32, kMxY = 8;
struct MixedTile {
  double ph[kMxY + 6][kMxX + 6];
  float dxs[kMxY][kMxX + 5], dys[kMxY + 5][kMxX];
};
// True in every thread where every difference is below 1e30 (false for NaN), so that
// weno5_side_f32's exact doublings do not overflow.
__device__ __forceinline__ bool stage_mixed(MixedTile& t, const DField& src, const LSArgs& a, int i0, int j0) {
  constexpr int NT = kMxX * kMxY;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kMxX + tx;
#pragma unroll
  for (int y = ty; y < kMxY + 6; y += kMxY) t.ph[y][tx] = ghosted(src, i0 - 3 + tx, j0 - 3 + y);
  for (int k = tid; k < (kMxY + 6) * 6; k += NT) t.ph[k / 6][kMxX + k % 6] = ghosted(src, i0 - 3 + kMxX + k % 6, j0 - 3 + k / 6);
  __syncthreads();
  bool ok = true;
  auto put = [&](float& f, double d, float o) {
    f = narrow(d) * o;
    ok = ok && fabsf(f) < 1e30f;
  };
  put(t.dxs[ty][tx], t.ph[ty + 3][tx + 1] - t.ph[ty + 3][tx], a.odx_f);
  if (tid < kMxY * 5) {
    const int r = tid / 5, c = kMxX + tid % 5;
    put(t.dxs[r][c], t.ph[r + 3][c + 1] - t.ph[r + 3][c], a.odx_f);
  }
#pragma unroll
  for (int r = ty; r < kMxY + 5; r += kMxY) put(t.dys[r][tx], t.ph[r + 1][tx + 3] - t.ph[r][tx + 3], a.ody_f);
  return __syncthreads_and(ok && a.fast_f);
}
// The six differences of node (c, r) along dir (0: x, 1: y), and its one-sided derivative
// from them: side 0 the minus, side 1 the plus one.
__device__ __forceinline__ void mx_load(const MixedTile& t, int dir, int c, int r, float d[6]) {
  const float* q = dir == 0 ? &t.dxs[r][c] : &t.dys[r][c];
  const int st = dir == 0 ? 1 : kMxX;
#pragma unroll
  for (int k = 0; k < 6; ++k) d[k] = q[k * st];
}
template <bool FAST>
__device__ __forceinline__ float mx_side(const float d[6], bool plus, float eps) {
  const float a1 = plus ? d[5] : d[0], a2 = plus ? d[4] : d[1], a3 = plus ? d[3] : d[2], a4 = plus ? d[2] : d[3], a5 = plus ? d[1] : d[4];
  return FAST ? weno5_side_f32(a1, a2, a3, a4, a5, eps) : weno5_side<float>(a1, a2, a3, a4, a5, eps);
}
__device__ __noinline__ float mx_side_general(const MixedTile& t, int dir, int c, int r, bool plus, float eps) {
  float d[6];
  mx_load(t, dir, c, r, d);
  return mx_side<false>(d, plus, eps);
}
// The common sign of both one-sided derivatives from their six differences, or 0 where it
// is not certain: with all six between lo and hi, six times each candidate stencil lies
// above 13 lo - 7 hi (lo > 0), and a derivative is a convex combination of its candidates.
// The bounds keep the FP32 evaluation's rounding (relative 1e-6) and its range out of
// question: 1e-15 < |d| < 1e8 with epsilon in [1e-15, 1e8] neither overflows a weight nor
// underflows a derivative times |s| >= 1e-12.  (min.NaN, max.NaN: a NaN makes every test
// false.)
__device__ __forceinline__ int mx_sign(const float d[6]) {
  float lo, hi, t;
  asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(t) : "f"(d[0]), "f"(d[1]), "f"(d[2]));
  asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(t) : "f"(t), "f"(d[3]), "f"(d[4]));
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(lo) : "f"(t), "f"(d[5]));
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(t) : "f"(d[0]), "f"(d[1]), "f"(d[2]));
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(t) : "f"(t), "f"(d[3]), "f"(d[4]));
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(hi) : "f"(t), "f"(d[5]));
  const bool neg = hi < 0.0f;
  const float small = neg ? -hi : lo, large = neg ? -lo : hi;  // of the magnitudes, where all signs agree
  return small > 1e-15f && large < 1e8f && 13.0f * small > 7.01f * large ? (neg ? -1 : 1) : 0;
}

// WENO5th (ADVECTION_METHOD_2D.h:508-663), the mixed form: the upwind side only, from the
// tile's differences.  The grid's last block row copies the ghost ring.
__global__ void __launch_bounds__(kMxX* kMxY, 8) k_weno5_advect_mixed(const double* __restrict__ src_a, double* __restrict__ dst_a,
                                                                   const double* __restrict__ ua_a, const double* __restrict__ va_a,
                                                                   LSArgs a, DtArg dt_arg) {
  constexpr int NT = kMxX * kMxY;
  pdl_enter();
  __shared__ MixedTile t;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const DField src = dfield((double*)src_a, 2, a.ni, a.nj), dst = dfield(dst_a, 2, a.ni, a.nj);
  const int by = a.row0 + (int)blockIdx.y;
  if (by == a.rows) {
    copy_ring(src, dst, blockIdx.x * NT + ty * kMxX + tx, gridDim.x * NT);
    return;
  }
  const int i0 = (int)blockIdx.x * kMxX, j0 = by * kMxY, i = i0 + tx, j = j0 + ty;
  const bool fast = stage_mixed(t, src, a, i0, j0);
  if (i >= a.ni || j >= a.nj) return;
  const DField ua = dfield((double*)ua_a, 3, a.ni + 1, a.nj), va = dfield((double*)va_a, 3, a.ni, a.nj + 1);
  const double u = (__ldg(&GB_AT(ua, i + 1, j)) + __ldg(&GB_AT(ua, i, j))) * 0.5;
  const double v = (__ldg(&GB_AT(va, i, j + 1)) + __ldg(&GB_AT(va, i, j))) * 0.5;
  const bool px = !gtz(u), py = !gtz(v);
  float fx32, fy32;
  if (fast) {
    float d[6];
    mx_load(t, 0, tx, ty, d);
    fx32 = mx_side<true>(d, px, a.eps_f);
    mx_load(t, 1, tx, ty, d);
    fy32 = mx_side<true>(d, py, a.eps_f);
  } else {
    fx32 = mx_side_general(t, 0, tx, ty, px, a.eps_f);
    fy32 = mx_side_general(t, 1, tx, ty, py, a.eps_f);
  }
  const double fx = widen(fx32), fy = widen(fy32);
  GB_AT(dst, i, j) = t.ph[ty + 3][tx + 3] - dt_arg.get() * (u * fx + v * fy);
}

// The mixed reinit sweep, bound by instruction issue.  Where the sign of a direction's
// derivatives is certain (almost everywhere) the update uses one of the two, and only that
// one is evaluated; the other nodes put the second evaluation on the block's list, which
// the block works off densely.  The results equal k_reinit_sweep_mixed's bit for bit.
// ring: the grid's last block row copies src's ghost ring.
// Level-set TVD-RK3 with its 75 sweeps at 1024^2: 1.98 ms with four derivatives per node
// (703 instructions a node), 1.64 ms with the chosen ones, 1.55 ms with the six differences
// of a direction read once and weno5_side_f32 (507), 1.43 ms with 8 blocks per SM instead
// of 6 (32 registers; staging, FP64 differences and evaluation of different blocks overlap).
// Tiles of 32 x 16: 1.72 ms, of 32 x 4: 1.57.
__global__ void __launch_bounds__(kMxX* kMxY, 8) k_reinit_sweep_tiled(const double* __restrict__ src_a, double* __restrict__ dst_a,
                                                                   const double* __restrict__ S, LSArgs a, double dtau, int ring) {
  constexpr int NT = kMxX * kMxY;
  pdl_enter();
  __shared__ MixedTile t;
  __shared__ float plus[2 * NT];
  __shared__ unsigned short list[2 * NT];
  __shared__ int count;
  const int ni = a.ni, nj = a.nj, tx = threadIdx.x, ty = threadIdx.y, tid = ty * kMxX + tx;
  const DField src = dfield((double*)src_a, 2, ni, nj), dst = dfield(dst_a, 2, ni, nj);
  if (ring && blockIdx.y == gridDim.y - 1) {
    copy_ring(src, dst, blockIdx.x * NT + tid, gridDim.x * NT);
    return;
  }
  if (tid == 0) count = 0;
  const int i0 = (int)blockIdx.x * kMxX, j0 = (int)blockIdx.y * kMxY, i = i0 + tx, j = j0 + ty;
  const bool fast = stage_mixed(t, src, a, i0, j0);
  const bool in = i < ni && j < nj;
  const double sv = in ? __ldg(&S[i + (size_t)j * ni]) : 0.0;
  const float s = narrow(sv);
  int xs = 3, ys = 3;  // 0: the minus side, 1: the plus side, 3: both are needed
  float gx = 0, gy = 0;
  int n = 0;
  if (fast) {
    float dx[6], dy[6];
    mx_load(t, 0, tx, ty, dx);
    mx_load(t, 1, tx, ty, dy);
    const int ss = s >= 1e-12f ? 1 : s <= -1e-12f ? -1 : 0;
    const int sx = ss * mx_sign(dx), sy = ss * mx_sign(dy);
    xs = sx > 0 ? 0 : sx < 0 ? 1 : 3;
    ys = sy > 0 ? 0 : sy < 0 ? 1 : 3;
    if (in && xs == 3) list[atomicAdd(&count, 1)] = (unsigned short)tid;
    if (in && ys == 3) list[atomicAdd(&count, 1)] = (unsigned short)(NT + tid);
    gx = mx_side<true>(dx, xs == 1, a.eps_f);
    gy = mx_side<true>(dy, ys == 1, a.eps_f);
    __syncthreads();
    n = count;
    for (int k = tid; k < n; k += NT) {
      const int item = list[k], nd = item & (NT - 1);
      mx_load(t, item / NT, nd & (kMxX - 1), nd / kMxX, dx);
      plus[item] = mx_side<true>(dx, true, a.eps_f);
    }
  } else {
    gx = mx_side_general(t, 0, tx, ty, false, a.eps_f);
    gy = mx_side_general(t, 1, tx, ty, false, a.eps_f);
    plus[tid] = mx_side_general(t, 0, tx, ty, true, a.eps_f);
    plus[NT + tid] = mx_side_general(t, 1, tx, ty, true, a.eps_f);
  }
  if (n > 0) __syncthreads();
  if (!in) return;
  const double old = t.ph[ty + 3][tx + 3];
  if (xs == 3) {
    const float p = plus[tid];
    xs = godunov_pick(s, gx, p, true);
    gx = xs == 0 ? gx : p;
  }
  if (ys == 3) {
    const float p = plus[NT + tid];
    ys = godunov_pick(s, gy, p, false);
    gy = ys == 0 ? gy : p;
  }
  double out = old;
  if (xs >= 0 && ys >= 0) {
    float h;
    if (xs != 2 && ys != 2)
      h = sqrtf(gx * gx + gy * gy) - 1.0f;
    else if (xs != 2)
      h = sqrtf(gx * gx) - 1.0f;
    else if (ys != 2)
      h = sqrtf(gy * gy) - 1.0f;
    else
      h = -1.0f;
    out = old - dtau * sv * widen(h);
  }
  GB_AT(dst, i, j) = out;
}

// Shu-Osher blend of the TVD-RK3 stages (EULERIAN_FLUID_SOLVER_2D.h:1706-1741): interior only.
__global__ void k_blend(const double* __restrict__ keep_a, double* phi_a, int ni, int nj, double c0, double c1) {
  pdl_enter();
  DField keep = dfield((double*)keep_a, 2, ni, nj), phi = dfield(phi_a, 2, ni, nj);
  GB_FOR_IJ(i, j, ni, nj) {
    GB_AT(phi, i, j) = mul_wide(GB_AT(keep, i, j), c0) + c1 * GB_AT(phi, i, j);
  }
}

struct EnoArgs {
  int ni, nj;
  Space xs, ys;
  double o3[2][2];  // 1/(3h) of x and y for the x-face grid [0] and the y-face grid [1], host IEEE quotients
  // FP32 path, per face grid: 1/h, 1/(2h), 1/(3h), h for x ([0..3]) and y ([4..7])
  float xs_f[8], ys_f[8];
  int fast;  // cell sizes in [2^-30, 2^30]
  int row0;  // the launch's first tile row
};

// x / 4, exact but for subnormal results, without the FP64 pipe.
__device__ __forceinline__ double quarter(double x) {
  const Words w = words(x);
  const unsigned e = (w.hi >> 20) & 0x7ffu;
  if (e > 2u && e < 0x7ffu) return from_words(w.lo, w.hi - (2u << 20));
  return is_zero(x) ? x : plain_mul(x, 0.25);
}

// One tile of one MAC component, kEnX x kEnY faces: its values q (ghost-filled copy,
// ghost 3) and along each direction the first, second and third divided differences, each
// formed once (a face of its own forms 6 + 5 + 4 of them per direction, all shared with
// its neighbours): entry k of face c is element c + k.
constexpr int kEnX = 32, kEnY = 8;
template <typename R>
struct EnoTile {
  double q[kEnY + 6][kEnX + 6];
  R x1[kEnY][kEnX + 5], x2[kEnY][kEnX + 4], x3[kEnY][kEnX + 3];
  R y1[kEnY + 5][kEnX], y2[kEnY + 4][kEnX], y3[kEnY + 3][kEnX];
};
__device__ __forceinline__ float eno_first(double d, float o) { return narrow(d) * o; }
__device__ __forceinline__ double eno_first(double d, double o) { return mul_rn(o, d); }
__device__ __forceinline__ float eno_next(float d, float o) { return o * d; }
__device__ __forceinline__ double eno_next(double d, double o) { return mul_rn(o, d); }
// d1 + (a t + c d3 h h) of the chosen formula (eno3_select's, in its order of operations;
// doubling is exact).
__device__ __forceinline__ float eno_value(float d1, float d2, float d3, float h, bool plus, bool twice) {
  const float t = d2 * h, a = plus ? d1 - t : d1 + t, x = (twice ? 2.0f * d3 : d3) * h * h;
  return twice ? a + x : a - x;
}
__device__ __forceinline__ double eno_value(double d1, double d2, double d3, double h, bool plus, bool twice) {
  const double t = mul_rn(d2, h), a = d1 + (plus ? negd(t) : t);
  return __fma_rn(twice ? 2.0 : -1.0, mul_rn(mul_rn(d3, h), h), a);
}
// One one-sided derivative (eno3_select): first differences at e1 (stride st), second at e2, third at e3.
template <typename R>
__device__ __forceinline__ R eno_side(const R* e1, const R* e2, const R* e3, int st, R h, bool plus) {
  const R a2 = e2[(plus ? 2 : 1) * st], b2 = e2[(plus ? 3 : 2) * st];
  const bool near = mag_le(a2, b2);             // the second difference on the minus side is the smaller
  const int k = (plus ? 1 : 0) + (near ? 0 : 1);  // the third differences k, k + 1 compete
  const R a3 = e3[k * st], b3 = e3[(k + 1) * st];
  return eno_value(e1[(plus ? 3 : 2) * st], near ? a2 : b2, mag_le(a3, b3) ? a3 : b3, h, plus, near != plus);
}
// The plain forms, for a tile with differences outside mid_range<200>.
__device__ __noinline__ double eno_side_plain(const double* q, int st, double o, double o2, double o3, double h, bool plus) {
  double v[7], dm, dp;
  for (int k = 0; k < 7; ++k) v[k] = q[k * st];
  eno3_pair(v, o, o2, o3, h, dm, dp);
  return plus ? dp : dm;
}
__device__ __noinline__ double eno_update_plain(double out, double dt, double uu, double fx, double vv, double fy) {
  return out - dt * (uu * fx + vv * fy);
}

// ENO3rd on both MAC components (ADVECTION_METHOD_2D.h:2038-2231) as called by
// Solve_Velocity (ADVECTION_2D.cpp:83-122): both read only the advecting copies
// UA/VA (already refreshed from U/V), so one launch updates U (blockIdx.z = 0) and V (1).
// MIXED: divided differences and the ENO selection in FP32 (first differences,
// face velocities and the update in FP64).  The exact form is bound by the FP64 and
// integer pipes: a face evaluates the upwind derivative only, its products run on the
// integer pipes, and the divided differences are shared (15 FP64 instructions a face
// instead of 90): 501 -> 71 us at 1000 x 750; the mixed form 363 -> 195 us at 2048^2.
template <bool MIXED>
__global__ void __launch_bounds__(kEnX* kEnY) k_eno3(double* __restrict__ u_a, double* __restrict__ v_a, const double* __restrict__ ua_a,
                                                     const double* __restrict__ va_a, EnoArgs a, DtArg dt_arg) {
  using R = typename std::conditional<MIXED, float, double>::type;
  constexpr int NT = kEnX * kEnY;
  pdl_enter();
  __shared__ EnoTile<R> t;
  const bool xc = blockIdx.z == 0;
  const int nI = a.ni + (xc ? 1 : 0), nJ = a.nj + (xc ? 0 : 1);
  const int i0 = (int)blockIdx.x * kEnX, j0 = (a.row0 + (int)blockIdx.y) * kEnY;
  if (i0 >= nI || j0 >= nJ) return;
  const DField ua = dfield((double*)ua_a, 3, a.ni + 1, a.nj), va = dfield((double*)va_a, 3, a.ni, a.nj + 1);
  const DField& g = xc ? ua : va;
  const Space& s = xc ? a.xs : a.ys;
  const float* sf = xc ? a.xs_f : a.ys_f;
  const double *o3 = a.o3[xc ? 0 : 1];
  R ox, ox2, ox3, hx, oy, oy2, oy3, hy;
  if constexpr (MIXED) {
    ox = sf[0], ox2 = sf[1], ox3 = sf[2], hx = sf[3], oy = sf[4], oy2 = sf[5], oy3 = sf[6], hy = sf[7];
  } else {
    ox = s.odx, ox2 = s.o2dx, ox3 = o3[0], hx = s.dx, oy = s.ody, oy2 = s.o2dy, oy3 = o3[1], hy = s.dy;
  }
  const int tid = threadIdx.x, tx = tid & (kEnX - 1), ty = tid / kEnX;
  for (int k = tid; k < (kEnY + 6) * (kEnX + 6); k += NT) {
    const int y = k / (kEnX + 6), x = k - y * (kEnX + 6), i = i0 - 3 + x, j = j0 - 3 + y;
    t.q[y][x] = __ldg(&GB_AT(g, i < nI + 3 ? i : nI + 2, j < nJ + 3 ? j : nJ + 2));
  }
  __syncthreads();
  bool ok = true;
  for (int k = tid; k < kEnY * (kEnX + 5); k += NT) {
    const int r = k / (kEnX + 5), c = k - r * (kEnX + 5);
    const double d = t.q[r + 3][c + 1] - t.q[r + 3][c];
    if (!MIXED) ok = ok && mid_range<200>(d);
    t.x1[r][c] = eno_first(d, ox);
  }
  for (int k = tid; k < (kEnY + 5) * kEnX; k += NT) {
    const int r = k / kEnX, c = k - r * kEnX;
    const double d = t.q[r + 1][c + 3] - t.q[r][c + 3];
    if (!MIXED) ok = ok && mid_range<200>(d);
    t.y1[r][c] = eno_first(d, oy);
  }
  const bool fast = __syncthreads_and(MIXED || (ok && a.fast));
  for (int k = tid; k < kEnY * (kEnX + 4); k += NT) {
    const int r = k / (kEnX + 4), c = k - r * (kEnX + 4);
    t.x2[r][c] = eno_next(t.x1[r][c + 1] - t.x1[r][c], ox2);
  }
  for (int k = tid; k < (kEnY + 4) * kEnX; k += NT) {
    const int r = k / kEnX, c = k - r * kEnX;
    t.y2[r][c] = eno_next(t.y1[r + 1][c] - t.y1[r][c], oy2);
  }
  __syncthreads();
  for (int k = tid; k < kEnY * (kEnX + 3); k += NT) {
    const int r = k / (kEnX + 3), c = k - r * (kEnX + 3);
    t.x3[r][c] = eno_next(t.x2[r][c + 1] - t.x2[r][c], ox3);
  }
  for (int k = tid; k < (kEnY + 3) * kEnX; k += NT) {
    const int r = k / kEnX, c = k - r * kEnX;
    t.y3[r][c] = eno_next(t.y2[r + 1][c] - t.y2[r][c], oy3);
  }
  __syncthreads();
  const int i = i0 + tx, j = j0 + ty;
  if (i >= nI || j >= nJ) return;
  double uu, vv;
  if (xc) {
    uu = t.q[ty + 3][tx + 3];
    vv = quarter(GB_AT(va, i, j) + GB_AT(va, i, j + 1) + GB_AT(va, i - 1, j) + GB_AT(va, i - 1, j + 1));
  } else {
    uu = quarter(GB_AT(ua, i, j - 1) + GB_AT(ua, i + 1, j - 1) + GB_AT(ua, i, j) + GB_AT(ua, i + 1, j));
    vv = t.q[ty + 3][tx + 3];
  }
  const bool px = !gtz(uu), py = !gtz(vv);
  const double dt = dt_arg.get();
  const DField out = xc ? dfield(u_a, 2, nI, nJ) : dfield(v_a, 2, nI, nJ);
  double fx, fy;
  if (fast) {
    fx = widen(eno_side(&t.x1[ty][tx], &t.x2[ty][tx], &t.x3[ty][tx], 1, hx, px));
    fy = widen(eno_side(&t.y1[ty][tx], &t.y2[ty][tx], &t.y3[ty][tx], kEnX, hy, py));
  } else {
    fx = eno_side_plain(&t.q[ty + 3][tx], 1, s.odx, s.o2dx, o3[0], s.dx, px);
    fy = eno_side_plain(&t.q[ty][tx + 3], kEnX + 6, s.ody, s.o2dy, o3[1], s.dy, py);
  }
  // FP32 derivatives (zero or above 2^-126) and exact ones (zero or above 2^-500) keep the
  // products normal for these velocities and steps.
  if (fast && mid_range<300>(uu) && mid_range<300>(vv) && mid_range<100>(dt) && mid_range<500>(fx) && mid_range<500>(fy))
    GB_AT(out, i, j) = GB_AT(out, i, j) - mul_wide(mul_rn(uu, fx) + mul_rn(vv, fy), dt);
  else
    GB_AT(out, i, j) = eno_update_plain(GB_AT(out, i, j), dt, uu, fx, vv, fy);
}

// A node's curvature in the plain FP64 forms (LEVELSET_2D.h:898-990); `zero` where the
// denominator vanishes with the central and with the one-sided differences.
struct Curv {
  double k;
  bool zero;
};
__device__ __noinline__ Curv plain_curvature(double c, double l, double r, double b, double tp, double dxy, const Space& s) {
  double px = (r - l) * s.o2dx;
  double py = (tp - b) * s.o2dy;
  const double pxx = (r - 2 * c + l) * s.odx2;
  const double pyy = (tp - 2 * c + b) * s.ody2;
  const double pxy = dxy * s.o2dx * s.o2dy;
  for (int k = 0; k < 2; ++k) {
    const double mag = sqrt(px * px + py * py);
    const double deno = mag * mag * mag;
    if ((__double_as_longlong(deno) & kAbsBits) != 0) {  // deno != 0 (NaN included)
      const double od = 1.0 / deno;
      return Curv{-(px * px * pyy - 2.0 * px * py * pxy + py * py * pxx) * od, false};
    }
    px = (r - c) * s.odx;
    py = (tp - c) * s.ody;
  }
  return Curv{0.0, true};
}

// ComputeCurvaturesThread with curvature_by_levelset (LEVELSET_2D.h:898-990);
// phi's ghosts must already be extrapolated.
__global__ void k_curvature(const double* __restrict__ phi_a, double* __restrict__ kappa, int ni, int nj, Space s, int* flag) {
  DField phi = dfield((double*)phi_a, 2, ni, nj);
  const double tol = s.dx < s.dy ? s.odx : s.ody;  // 1 / min(dx, dy), taken on the host
  const bool fast = mid_range<30>(s.odx) && mid_range<30>(s.ody);
  GB_FOR_IJ(i, j, ni, nj) {
    const size_t t = (size_t)j * ni + i;
    const double c = GB_AT(phi, i, j), l = GB_AT(phi, i - 1, j), r = GB_AT(phi, i + 1, j), b = GB_AT(phi, i, j - 1), tp = GB_AT(phi, i, j + 1);
    // r - 2 c as one FMA: doubling is exact (where 2 c overflows, the plain form is taken)
    const double dx = r - l, dy = tp - b, dxx = __fma_rn(-2.0, c, r) + l, dyy = __fma_rn(-2.0, c, tp) + b;
    const double dxy = GB_AT(phi, i + 1, j + 1) - GB_AT(phi, i + 1, j - 1) - GB_AT(phi, i - 1, j + 1) + GB_AT(phi, i - 1, j - 1);
    double curv = 0;
    if (fast && mid_range<100>(dx) && mid_range<100>(dy) && mid_range<100>(dxx) && mid_range<100>(dyy) && mid_range<100>(dxy) &&
        !(is_zero(dx) && is_zero(dy))) {
      // The same value: products, root and quotient on the integer pipes but for the six
      // scalings, which balance the two pipes.
      const double px = dx * s.o2dx, py = dy * s.o2dy, pxx = dxx * s.odx2, pyy = dyy * s.ody2, pxy = dxy * s.o2dx * s.o2dy;
      const double x2 = mul_rn(px, px), y2 = mul_rn(py, py);
      const double mag = sqrt_rn(x2 + y2);
      const double od = div_pos(1.0, mul_rn(mul_rn(mag, mag), mag));
      // 2 px py pxy is twice the rounded px py pxy
      const double n = __fma_rn(-2.0, mul_rn(mul_rn(px, py), pxy), mul_rn(x2, pyy)) + mul_rn(y2, pxx);
      curv = negd(mul_rn(n, od));
    } else {
      const Curv g = plain_curvature(c, l, r, b, tp, dxy, s);
      if (g.zero) {
        atomicOr(flag, 2);
        continue;
      }
      curv = g.k;
    }
    // Clamp to [-tol, tol] with IEEE comparisons (tol > 0 finite; a NaN stores nothing)
    const long long cm = mag_bits(curv);
    if (cm <= mag_bits(tol))
      kappa[t] = curv;
    else if (cm <= kInfBits)
      kappa[t] = (int)words(curv).hi >= 0 ? tol : negd(tol);
  }
}

struct AsmArgs {
  int ni, nj;
  Space s;
  double water, air, sigma, one_over_dt, inv_dxdx, inv_dydy;
  double inv_water, inv_air;  // 1/water, 1/air: IEEE quotients taken once on the host
  const double* dtp;          // non-null: the time step is read here (one_over_dt = 1 / *dtp, IEEE)
  double oeh, oev;            // 1 / (1.5 dx), 1 / (1.5 dy): smeared-Heaviside scales
  int fast;                   // densities and cell sizes are in the fast forms' range (mid_range<100>)
};

// 1/rho of a node.  The density takes two values, so the quotient is a select of
// the host's correctly rounded reciprocals (FP64 divides are scarce on this part).
__device__ __forceinline__ double inv_density(double phi, const AsmArgs& a) {
  if (lez(phi)) return a.inv_air;
  if (gtz(phi)) return a.inv_water;
  return 1.0;
}

// 1/rho at a node or at its copied ghost (POISSON_SOLVER.cpp:131-138: the ghost
// layer copies the second interior line).
__device__ __forceinline__ double vnode(const DField& phi, int i, int j, const AsmArgs& a) {
  i = i < 0 ? 1 : (i >= a.ni ? a.ni - 2 : i);
  j = j < 0 ? 1 : (j >= a.nj ? a.nj - 2 : j);
  return inv_density(GB_AT(phi, i, j), a);
}

// vc vn (|pn| + |pc|) / (vc |pn| + vn |pc|); with 1/rho and |phi| in the fast range the
// quotient and half of the products on the integer pipes (the same value).
__device__ __forceinline__ double face_beta(double vc, double vn, double pc, double pn, const AsmArgs& a) {
  const double ac = absd(pc), an = absd(pn);
  if (a.fast && mid_range<300>(pc) && mid_range<300>(pn)) {
    const double sum = an + ac;
    if (!is_zero(sum)) return div_pos(mul_rn(mul_rn(vc, vn), sum), vc * an + vn * ac);
  }
  return plain_beta(vc, vn, ac, an);
}

// Face weights of BuildLinearSystemNodeJumpConditionVaribleCoefficient
// (POISSON_SOLVER.cpp:743-746): one value per face, symmetric in IEEE arithmetic.
__global__ void k_faces(const double* __restrict__ phi_a, double* __restrict__ bx, double* __restrict__ by, AsmArgs a) {
  int ni = a.ni, nj = a.nj;
  DField phi = dfield((double*)phi_a, 2, ni, nj);
  GB_FOR_IJ(i, j, ni + 1, nj) {
    bx[(size_t)j * (ni + 1) + i] = face_beta(vnode(phi, i, j, a), vnode(phi, i - 1, j, a), GB_AT(phi, i, j), GB_AT(phi, i - 1, j), a);
  }
  GB_FOR_IJ(i, j, ni, nj + 1) {
    by[(size_t)j * ni + i] = face_beta(vnode(phi, i, j, a), vnode(phi, i, j - 1, a), GB_AT(phi, i, j), GB_AT(phi, i, j - 1), a);
  }
}

__device__ __forceinline__ double jc_at(const double* kappa, int i, int j, const AsmArgs& a) {
  if (i < 0 || j < 0 || i >= a.ni || j >= a.nj) return 0.0;  // jc_on_solution ghosts stay zero
  return a.sigma * kappa[i + (size_t)j * a.ni];
}

// Jump flux of one arm (POISSON_SOLVER.cpp:881-948) without the derivative-jump
// part, which vanishes because jc_on_derivative is zeroed (PROJECTION_2D.h:501-504).
// Left/bottom and right/top arms follow the same sign rule.  The jump values are
// read only on arms that cross the interface.
__device__ __forceinline__ double arm_flux(double pc, double pn, double jcc, const double* kappa, int in, int jn, double beta, double o2,
                                           const AsmArgs& a) {
  const bool cneg = lez(pc), nneg = lez(pn);
  if (cneg && !nneg && gtz(pn)) {
    double ac = fabs(pc), an = fabs(pn);
    double av = (jcc * an + jc_at(kappa, in, jn, a) * ac) / (ac + an);
    return o2 * av * beta;
  }
  if (!cneg && gtz(pc) && nneg) {
    double ac = fabs(pc), an = fabs(pn);
    double av = (jcc * an + jc_at(kappa, in, jn, a) * ac) / (ac + an);
    return -o2 * av * beta;
  }
  return 0.0;
}

// Diagonal (dx^2 only, POISSON_SOLVER.cpp:872): the face weights of the FULL arms and
// the first cell's Neumann arms (the corner pin).
__global__ void k_diag(const double* __restrict__ bx, const double* __restrict__ by, double* __restrict__ diag, AsmArgs a) {
  int ni = a.ni, nj = a.nj;
  GB_FOR_IJ(i, j, ni, nj) {
    const size_t t = (size_t)j * ni + i;
    double bl = bx[i + (size_t)j * (ni + 1)], br = bx[i + 1 + (size_t)j * (ni + 1)];
    double bb = by[i + (size_t)j * ni], bt = by[i + (size_t)(j + 1) * ni];
    double coef;
    if (i > 0 && i < ni - 1 && j > 0 && j < nj - 1) {
      coef = bl + br + bb + bt;
    } else {
      coef = 0;
      if (i > 0) coef += bl;
      if (i < ni - 1) coef += br;
      if (j > 0) coef += bb;
      if (j < nj - 1) coef += bt;
      if (i == 0 && j == 0) {  // Neumann arms of the first cell (POISSON_SOLVER.cpp:789-806)
        if (i - 1 < 0) coef += bl;
        if (i + 1 > ni - 1) coef += br;
        if (j - 1 < 0) coef += bb;
        if (j + 1 > nj - 1) coef += bt;
      }
    }
    if (is_zero(coef)) coef = 1;
    diag[t] = a.inv_dxdx * coef;
  }
}

// An arm of k_rhs crosses the interface (arm_flux is not zero for it).
__device__ __forceinline__ bool arm_crosses(double pc, double pn) {
  const bool cneg = lez(pc), nneg = lez(pn);
  return cneg ? !nneg && gtz(pn) : nneg && gtz(pc);
}

// k_rhs's value at a node with an arm that crosses the interface (out of line, as plain_mul).
__device__ __noinline__ double rhs_interface(double div, double pc, double pl, double pr, double pb, double pt, const double* kappa,
                                             const double* bx, const double* by, int i, int j, const AsmArgs& a) {
  const int ni = a.ni;
  const double bl = bx[i + (size_t)j * (ni + 1)], br = bx[i + 1 + (size_t)j * (ni + 1)];
  const double bb = by[i + (size_t)j * ni], bt = by[i + (size_t)(j + 1) * ni];
  const double jcc = jc_at(kappa, i, j, a);
  const double FL = arm_flux(pc, pl, jcc, kappa, i - 1, j, bl, a.s.odx2, a);
  const double FR = arm_flux(pc, pr, jcc, kappa, i + 1, j, br, a.s.odx2, a);
  const double FB = arm_flux(pc, pb, jcc, kappa, i, j - 1, bb, a.s.ody2, a);
  const double FT = arm_flux(pc, pt, jcc, kappa, i, j + 1, bt, a.s.ody2, a);
  const double FX = FL + FR, FY = FB + FT;
  return -div - FX - FY;
}

// Right-hand side -div - F_X - F_Y (POISSON_SOLVER.cpp:878-948).  Away from the interface
// the four fluxes are zero and drop out: three FP64 additions and two products a node, the
// third product on the integer pipes.
__global__ void k_rhs(const double* __restrict__ phi_a, const double* __restrict__ kappa, const double* __restrict__ u_a,
                      const double* __restrict__ v_a, const double* __restrict__ bx, const double* __restrict__ by, double* __restrict__ rhs,
                      AsmArgs a) {
  int ni = a.ni, nj = a.nj;
  double one_over_dt = a.one_over_dt;
  if (a.dtp) one_over_dt = mid_range<100>(*a.dtp) && gtz(*a.dtp) ? div_pos(1.0, *a.dtp) : 1.0 / *a.dtp;
  const bool fast = a.fast && mid_range<100>(one_over_dt);
  DField phi = dfield((double*)phi_a, 2, ni, nj);
  DField u = dfield((double*)u_a, 2, ni + 1, nj), v = dfield((double*)v_a, 2, ni, nj + 1);
  GB_FOR_IJ(i, j, ni, nj) {
    const size_t t = (size_t)j * ni + i;
    const double pc = GB_AT(phi, i, j);
    const double pl = GB_AT(phi, i - 1, j), pr = GB_AT(phi, i + 1, j), pb = GB_AT(phi, i, j - 1), pt = GB_AT(phi, i, j + 1);
    const double du = GB_AT(u, i + 1, j) - GB_AT(u, i, j), dv = GB_AT(v, i, j + 1) - GB_AT(v, i, j);
    double div;
    if (fast && mid_range<300>(dv))
      div = (a.s.odx * du + mul_rn(a.s.ody, dv)) * one_over_dt;
    else
      div = plain_div(a.s.odx, du, a.s.ody, dv, one_over_dt);
    if (!(arm_crosses(pc, pl) || arm_crosses(pc, pr) || arm_crosses(pc, pb) || arm_crosses(pc, pt))) {
      rhs[t] = negd(div);
      continue;
    }
    rhs[t] = rhs_interface(div, pc, pl, pr, pb, pt, kappa, bx, by, i, j, a);
  }
}

// CSR_MATRIX::Multiply in the builder's row order (left, right, bottom, top, diagonal).
__global__ void k_apply_exact(const double* __restrict__ bx, const double* __restrict__ by, const double* __restrict__ diag,
                              const double* __restrict__ x, double* __restrict__ y, int ni, int nj, double idx2, double idy2) {
  GB_FOR_IJ(i, j, ni, nj) {
    const size_t t = (size_t)j * ni + i;
    double acc = 0;
    if (i > 0) acc += -bx[i + (size_t)j * (ni + 1)] * idx2 * x[t - 1];
    if (i < ni - 1) acc += -bx[i + 1 + (size_t)j * (ni + 1)] * idx2 * x[t + 1];
    if (j > 0) acc += -by[i + (size_t)j * ni] * idy2 * x[t - ni];
    if (j < nj - 1) acc += -by[i + (size_t)(j + 1) * ni] * idy2 * x[t + ni];
    acc += diag[t] * x[t];
    y[t] = acc;
  }
}

// An interface face's updated velocity (out of line, as plain_mul).
__device__ __noinline__ double velocity_interface(double w, double dp, double dt, double od, double l0, double ln, double jcc, double jcn,
                                                  bool xc, const AsmArgs& a) {
  const double gam = (jcn * fabs(l0) + jcc * fabs(ln)) / (fabs(l0) + fabs(ln));
  const double dh = a.air + (a.water - a.air) * heaviside(0.5 * (l0 + ln), 1.5 * (xc ? a.s.dx : a.s.dy), xc ? a.oeh : a.oev);
  const double odh = 1 / dh;
  if (ltz(l0)) return w - dt * (dp + gam) * odh * od;
  if (gtz(l0)) return w - dt * (dp - gam) * odh * od;
  return w;
}

// UpdateVelocityByPressureGradientVariableDensity (PROJECTION_2D.h:1297-1416):
// same-sign faces use the node density on the + side, interface faces the
// smeared-Heaviside density of the face-averaged phi (eps = 1.5 dx) and the
// |phi|-weighted jump.  Pressure ghosts are zero; wall faces (bc < 0) are skipped.
__global__ void k_velocity_update(const double* __restrict__ phi_a, const double* __restrict__ p_a, const double* __restrict__ kappa,
                                  double* __restrict__ u_a, double* __restrict__ v_a, AsmArgs a, DtArg dt_arg, Scalars* sc) {
  int ni = a.ni, nj = a.nj;
  const double dt = dt_arg.get();
  DField phi = dfield((double*)phi_a, 2, ni, nj), p = dfield((double*)p_a, 1, ni, nj);
  DField u = dfield(u_a, 2, ni + 1, nj), v = dfield(v_a, 2, ni, nj + 1);
  const double odx = a.s.odx, ody = a.s.ody;  // 1 / dx, 1 / dy, taken on the host
  const bool fast = a.fast && mid_range<100>(dt);
  unsigned long long mx = 0, my = 0;  // bits of max |u|, |v| (non-negative doubles order as integers)
  GB_FOR_IJ(i, j, ni, nj) {
    const double l0 = GB_AT(phi, i, j), lw = GB_AT(phi, i - 1, j), ls = GB_AT(phi, i, j - 1);
    const double p0 = GB_AT(p, i, j), dpx = p0 - GB_AT(p, i - 1, j), dpy = p0 - GB_AT(p, i, j - 1);
    double wu = GB_AT(u, i, j), wv = GB_AT(v, i, j);
    const double oor = lez(l0) ? a.inv_air : a.inv_water;  // 1 / rho_ij
    // The x-face's products on the FP64 pipe, the y-face's on the integer pipes (where none
    // can leave the normal range).
    if (prod_ge0(l0, lw))
      wu -= dt * dpx * oor * odx;
    else
      wu = velocity_interface(wu, dpx, dt, odx, l0, lw, jc_at(kappa, i, j, a), jc_at(kappa, i - 1, j, a), true, a);
    if (prod_ge0(l0, ls))
      wv -= fast && mid_range<300>(dpy) ? mul_rn(mul_rn(mul_rn(dt, dpy), oor), ody) : plain_mul4(dt, dpy, oor, ody);
    else
      wv = velocity_interface(wv, dpy, dt, ody, l0, ls, jc_at(kappa, i, j, a), jc_at(kappa, i, j - 1, a), false, a);
    GB_AT(u, i, j) = wu;
    GB_AT(v, i, j) = wv;
    mx = abs_max_bits(wu, mx);
    my = abs_max_bits(wv, my);
  }
  block_max_bits(mx, &sc->maxu_bits);
  block_max_bits(my, &sc->maxv_bits);
}

__global__ void k_copy_interior(const double* __restrict__ src_a, int gs, double* __restrict__ dst_a, int gd, int nI, int nJ) {
  DField s = dfield((double*)src_a, gs, nI, nJ), d = dfield(dst_a, gd, nI, nJ);
  GB_FOR_IJ(i, j, nI, nJ) {
    GB_AT(d, i, j) = GB_AT(s, i, j);
  }
}

// FastSweepingMethodOriginal (LEVELSET_2D.h:281-384): the fixed band |phi| < 2 dx.
__global__ void k_fsm_fixed(const double* __restrict__ phi_a, double* __restrict__ fixed, int ni, int nj, double nb) {
  const DField phi = dfield((double*)phi_a, 2, ni, nj);
  GB_FOR_IJ(i, j, ni, nj) { fixed[(size_t)j * ni + i] = fabs(GB_AT(phi, i, j)) < nb ? 1.0 : 0.0; }
}

// The single-threaded FillGhostCellsContinuousDerivativesFrom (FIELD_STRUCTURE_2D.h:584-639):
// each side innermost layer first.  Thread k extrapolates row k's left and right ghosts and
// column k's top and bottom ghosts (disjoint ghost cells, interior reads only).
__global__ void k_extrapolate_inner_first(double* a, int g, int nI, int nJ) {
  const DField f = dfield(a, g, nI, nJ);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < (nI > nJ ? nI : nJ); k += gridDim.x * blockDim.x) {
    if (k < nJ) {
      for (int i = -1; i >= -g; --i) GB_AT(f, i, k) = 2.0 * GB_AT(f, i + 1, k) - GB_AT(f, i + 2, k);
      for (int i = nI; i <= nI - 1 + g; ++i) GB_AT(f, i, k) = 2.0 * GB_AT(f, i - 1, k) - GB_AT(f, i - 2, k);
    }
    if (k < nI) {
      for (int j = nJ; j <= nJ - 1 + g; ++j) GB_AT(f, k, j) = 2.0 * GB_AT(f, k, j - 1) - GB_AT(f, k, j - 2);
      for (int j = -1; j >= -g; --j) GB_AT(f, k, j) = 2.0 * GB_AT(f, k, j + 1) - GB_AT(f, k, j + 2);
    }
  }
}

// One Gauss-Seidel sweep of LEVELSET_2D::Sweep (LEVELSET_2D.h:507-589) in direction dir
// (0: i+ j+, 1: i- j+, 2: i- j-, 3: i+ j-).  The reference visits rows in order and
// nodes within a row in order; a node reads its two predecessors along i and j (already
// updated) and its two successors (not yet).  Anti-diagonal wavefronts in sweep
// coordinates have the same dependencies, so one block walks them in turn, one barrier
// per wavefront, and produces the reference's values bit for bit.
__global__ void k_fsm_sweep(double* phi_a, const double* __restrict__ fixed, int ni, int nj, double h, int dir) {
  const DField phi = dfield(phi_a, 2, ni, nj);
  const double one_over_two = 1.0 / 2.0, hh = h * h, hh2 = hh * 2.0;
  const bool irev = dir == 1 || dir == 2, jrev = dir == 2 || dir == 3;
  for (int d = 0; d <= ni + nj - 2; ++d) {
    const int lo = d - (nj - 1) > 0 ? d - (nj - 1) : 0, hi = d < ni - 1 ? d : ni - 1;
    for (int a = lo + (int)threadIdx.x; a <= hi; a += blockDim.x) {
      const int i = irev ? ni - 1 - a : a, jj = d - a, j = jrev ? nj - 1 - jj : jj;
      if (fixed[(size_t)j * ni + i] != 0.0) continue;
      double* pc = &GB_AT(phi, i, j);
      const double c = *pc, l = GB_AT(phi, i - 1, j), r = GB_AT(phi, i + 1, j), dn = GB_AT(phi, i, j - 1), up = GB_AT(phi, i, j + 1);
      double av, bv, a1, a2, update;
      if (c > 0) {
        av = l > r ? r : l;
        bv = dn > up ? up : dn;
        if (av <= bv) a1 = av, a2 = bv;
        else a1 = bv, a2 = av;
        update = fabs(a1 - a2) >= h ? a1 + h : one_over_two * (a1 + a2 + sqrt(hh2 - (a1 - a2) * (a1 - a2)));
        *pc = update > c ? c : update;
      } else if (c <= 0) {
        av = l > r ? l : r;
        bv = dn > up ? dn : up;
        if (av <= bv) a1 = av, a2 = bv;
        else a1 = bv, a2 = av;
        update = fabs(a1 - a2) >= h ? a2 - h : one_over_two * (a2 + a1 - sqrt(hh2 - (a2 - a1) * (a2 - a1)));
        *pc = update > c ? update : c;
      }
    }
    __syncthreads();
  }
}

inline dim3 grid2d(int W, int H, dim3 blk) { return dim3((W + blk.x - 1) / blk.x, (H + blk.y - 1) / blk.y); }

LSArgs ls_args(const gb2d_ctx* c, int tile_y) {
  return LSArgs{c->grid.ni, c->grid.nj, c->base.odx, c->base.ody, c->prm.weno_epsilon,
                (float)c->base.odx, (float)c->base.ody, (float)c->prm.weno_epsilon,
                c->prm.weno_epsilon >= 1e-15 && c->prm.weno_epsilon <= 1e8,
                c->prm.weno_epsilon >= 0x1p-100 && c->prm.weno_epsilon <= 0x1p100 &&
                    c->base.dx >= 0x1p-300 && c->base.dx <= 0x1p300,
                0, (c->grid.nj + tile_y - 1) / tile_y};
}

AsmArgs asm_args(const gb2d_ctx* c, double dt) {
  AsmArgs a;
  a.ni = c->grid.ni;
  a.nj = c->grid.nj;
  a.s = c->base;
  a.water = c->prm.water_density;
  a.air = c->prm.air_density;
  a.sigma = c->prm.surface_tension;
  a.one_over_dt = 1.0 / dt;
  a.dtp = c->dt_dev;
  a.inv_dxdx = 1.0 / (c->base.dx * c->base.dx);
  a.inv_dydy = 1.0 / (c->base.dy * c->base.dy);
  a.inv_water = 1.0 / a.water;
  a.inv_air = 1.0 / a.air;
  a.oeh = 1.0 / (1.5 * c->base.dx);
  a.oev = 1.0 / (1.5 * c->base.dy);
  auto mid = [](double x) { return x >= 0x1p-100 && x < 0x1p100; };
  a.fast = mid(a.inv_water) && mid(a.inv_air) && mid(a.s.odx) && mid(a.s.ody);
  return a;
}

// Self-check of div_by<3> / div_by<6> (and, on normal operands, of the functions of
// gb2d_exact_math.cuh) against the IEEE operations: n pseudo-random 64-bit patterns (every exponent, sign, NaN and infinity included) and n more
// with exponents in the range the schemes meet; counts results whose bits differ
// (NaN == NaN).
__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ull;
  x ^= x >> 33;
  return x;
}
__global__ void k_check_div_by(unsigned long long n, unsigned long long seed, unsigned long long* bad) {
  unsigned long long local = 0;
  for (unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; t < 2 * n; t += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long b = mix64(t * 0x9e3779b97f4a7c15ull + seed);
    if (t >= n) b = (b & 0x800fffffffffffffull) | ((unsigned long long)(1023 - 40 + (int)((b >> 52) % 80)) << 52);  // |a| in [2^-40, 2^40)
    const double a = __longlong_as_double((long long)b);
    const double q3 = div_by<3>(a), r3 = a / 3.0, q6 = div_by<6>(a), r6 = a / 6.0;
    const bool ok3 = __double_as_longlong(q3) == __double_as_longlong(r3) || (isnan(q3) && isnan(r3));
    const bool ok6 = __double_as_longlong(q6) == __double_as_longlong(r6) || (isnan(q6) && isnan(r6));
    local += (ok3 ? 0 : 1) + (ok6 ? 0 : 1);
    // exponents in [-300, 300); every eighth significand has a long run of zeros or ones
    auto normal = [](unsigned long long x) {
      if ((x >> 60) == 1) x &= ~0x3ffffffffull;
      if ((x >> 60) == 2) x |= 0xfffffffffull;
      return __longlong_as_double((long long)((x & 0x800fffffffffffffull) | ((1023ull - 300 + (x >> 40) % 600) << 52)));
    };
    const double x = normal(mix64(b + 1)), y = normal(mix64(b + 2)), ax = fabs(x), ay = fabs(y);
    auto differs = [](double u, double v) { return __double_as_longlong(u) != __double_as_longlong(v) ? 1 : 0; };
    local += differs(div_pos(ax, ay), ax / ay) + differs(div_pos(0.3, ay), 0.3 / ay) + differs(mul_rn(x, y), x * y) +
             differs(mul_rn(x, x), x * x) + differs(mul_rn(x, 7.0), x * 7.0) + differs(mul_rn(x, 13.0 / 12.0), x * (13.0 / 12.0)) +
             differs(third_rn<0>(x), x / 3.0) + differs(third_rn<1>(y), y / 6.0) + differs(sqrt_rn(ax), sqrt(ax)) +
             differs(sqrt_rn(ay * ay), sqrt(ay * ay));
  }
  if (local) atomicAdd(bad, local);
}

}  // namespace

unsigned long long check_div_by(unsigned long long n, unsigned long long seed, int* cuda_error) {
  unsigned long long* d = nullptr;
  unsigned long long h = ~0ull;
  cudaError_t e = cudaMalloc(&d, sizeof h);
  if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof h);
  if (e == cudaSuccess) {
    k_check_div_by<<<152 * 8, 256>>>(n, seed, d);
    GB_LAUNCHED(1);
    e = cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost);
  }
  if (d) cudaFree(d);
  *cuda_error = e == cudaSuccess ? 0 : 1;
  return h;
}

void launch_fill_ghost_copy(cudaStream_t s, double* dst, int gd, const double* src, int gs, int nI, int nJ, int g) {
  k_fill_ghost_copy<<<grid_ij(nI + 2 * g, nJ + 2 * g), kThreads, 0, s>>>(dst, gd, src, gs, nI, nJ, g);
  GB_LAUNCHED(1);
}

void launch_extrapolate_ghosts(cudaStream_t s, double* f, int g, int nI, int nJ) {
  int n = nI > nJ ? nI : nJ;
  pdl_launch(s, blocks_for(n, 128), 128, 0, k_extrapolate, f, g, nI, nJ);
  GB_LAUNCHED(1);
}

void launch_weno5_advect(cudaStream_t s, const gb2d_ctx* c, const double* src, double* dst, double dt, int mixed) {
  const unsigned cols = (unsigned)((c->grid.ni + 31) / 32);
  static_assert(kMxX == 32 && kExX == 32, "tile widths");
  LSArgs a = ls_args(c, mixed ? kMxY : kExY);
  for_tile_rows(a.rows + 1, [&](int first, unsigned n) {
    a.row0 = first;
    if (mixed)
      pdl_launch(s, dim3(cols, n), dim3(kMxX, kMxY), 0, k_weno5_advect_mixed, src, dst, c->ua, c->va, a, DtArg{dt, c->dt_dev});
    else
      pdl_launch(s, dim3(cols, n), 2 * kExX * kExY, 0, k_weno5_advect_exact, src, dst, c->ua, c->va, a, DtArg{dt, c->dt_dev});
    GB_LAUNCHED(1);
  });
}

void launch_reinit_sign(cudaStream_t s, const gb2d_ctx* c, const double* phi, double* S) {
  pdl_launch(s, grid_ij(c->grid.ni, c->grid.nj), kThreads, 0, k_reinit_sign, phi, S, c->grid.ni, c->grid.nj, c->base.dx * c->base.dx);
  GB_LAUNCHED(1);
}

void launch_reinit_sweep(cudaStream_t s, const gb2d_ctx* c, const double* src, double* dst, const double* S, double dtau, int mixed,
                         int ring) {
  const int ni = c->grid.ni, nj = c->grid.nj;
  // GB2D_REINIT_UNTILED=1 (read once) selects the per-node mixed kernel, which the tiled one
  // must equal bit for bit.
  static const bool untiled = [] {
    const char* e = getenv("GB2D_REINIT_UNTILED");
    return e && e[0] == '1';
  }();
  LSArgs a = ls_args(c, mixed ? kMxY : kExY);
  if (mixed && untiled) {
    const dim3 blk(32, 8);
    pdl_launch(s, grid2d(ni + 4, nj + 4, blk), blk, 0, k_reinit_sweep_mixed, src, dst, S, a, dtau);
    GB_LAUNCHED(1);
    return;
  }
  const unsigned cols = (unsigned)((ni + 31) / 32);
  if (mixed) {  // one launch, up to 524280 rows: an offset of the tile rows costs it 0.5%
    pdl_launch(s, dim3(cols, a.rows + (ring ? 1 : 0)), dim3(kMxX, kMxY), 0, k_reinit_sweep_tiled, src, dst, S, a, dtau, ring);
    GB_LAUNCHED(1);
    return;
  }
  for_tile_rows(a.rows + (ring ? 1 : 0), [&](int first, unsigned n) {
    a.row0 = first;
    pdl_launch(s, dim3(cols, n), 2 * kExX * kExY, 0, k_reinit_sweep_exact, src, dst, S, a, dtau);
    GB_LAUNCHED(1);
  });
}

void launch_blend(cudaStream_t s, const gb2d_ctx* c, const double* keep, double* phi, double c0, double c1) {
  pdl_launch(s, grid_ij(c->grid.ni, c->grid.nj), kThreads, 0, k_blend, keep, phi, c->grid.ni, c->grid.nj, c0, c1);
  GB_LAUNCHED(1);
}

void launch_eno3(cudaStream_t s, const gb2d_ctx* c, double dt) {
  EnoArgs a;
  a.ni = c->grid.ni;
  a.nj = c->grid.nj;
  a.xs = c->xs;
  a.ys = c->ys;
  const Space* sp[2] = {&c->xs, &c->ys};
  float* out[2] = {a.xs_f, a.ys_f};
  for (int g = 0; g < 2; ++g) {
    const Space& q = *sp[g];
    const double v[8] = {q.odx, q.o2dx, q.odx / 3, q.dx, q.ody, q.o2dy, q.ody / 3, q.dy};
    for (int k = 0; k < 8; ++k) out[g][k] = (float)v[k];
    a.o3[g][0] = q.odx / 3;
    a.o3[g][1] = q.ody / 3;
  }
  auto mid = [](double x) { return x >= 0x1p-30 && x <= 0x1p30; };
  a.fast = mid(c->xs.dx) && mid(c->xs.dy) && mid(c->ys.dx) && mid(c->ys.dy);
  for_tile_rows((c->grid.nj + kEnY) / kEnY, [&](int first, unsigned n) {  // covers ni + 1 and nj + 1 faces
    a.row0 = first;
    const dim3 grd((c->grid.ni + kEnX) / kEnX, n, 2);
    if (c->prm.advection_precision == GB2D_PRECISION_MIXED)
      pdl_launch(s, grd, kEnX * kEnY, 0, k_eno3<true>, c->u, c->v, c->ua, c->va, a, DtArg{dt, c->dt_dev});
    else
      pdl_launch(s, grd, kEnX * kEnY, 0, k_eno3<false>, c->u, c->v, c->ua, c->va, a, DtArg{dt, c->dt_dev});
    GB_LAUNCHED(1);
  });
}

void launch_curvature(cudaStream_t s, const gb2d_ctx* c, const double* phi, double* kappa, int* flag) {
  k_curvature<<<grid_ij(c->grid.ni, c->grid.nj), kThreads, 0, s>>>(phi, kappa, c->grid.ni, c->grid.nj, c->base, flag);
  GB_LAUNCHED(1);
}

void launch_faces(cudaStream_t s, const gb2d_ctx* c, const double* phi, double dt) {
  AsmArgs a = asm_args(c, dt);
  k_faces<<<grid_ij(c->grid.ni + 1, c->grid.nj + 1), kThreads, 0, s>>>(phi, c->bx, c->by, a);
  GB_LAUNCHED(1);
}

// Needs the face weights.
void launch_diag(cudaStream_t s, const gb2d_ctx* c, double dt) {
  AsmArgs a = asm_args(c, dt);
  k_diag<<<grid_ij(c->grid.ni, c->grid.nj), kThreads, 0, s>>>(c->bx, c->by, c->diag, a);
  GB_LAUNCHED(1);
}

// Needs the face weights and the curvature.
void launch_rhs(cudaStream_t s, const gb2d_ctx* c, const double* phi, double dt) {
  AsmArgs a = asm_args(c, dt);
  k_rhs<<<grid_ij(c->grid.ni, c->grid.nj), kThreads, 0, s>>>(phi, c->kappa, c->u, c->v, c->bx, c->by, c->rhs, a);
  GB_LAUNCHED(1);
}

void launch_poisson_apply_exact(cudaStream_t s, const gb2d_ctx* c, const double* x, double* y) {
  double idx2 = 1.0 / (c->base.dx * c->base.dx), idy2 = 1.0 / (c->base.dy * c->base.dy);
  k_apply_exact<<<grid_ij(c->grid.ni, c->grid.nj), kThreads, 0, s>>>(c->bx, c->by, c->diag, x, y, c->grid.ni, c->grid.nj, idx2, idy2);
  GB_LAUNCHED(1);
}

void launch_velocity_update(cudaStream_t s, const gb2d_ctx* c, const double* phi, double dt, Scalars* sc) {
  AsmArgs a = asm_args(c, dt);
  k_velocity_update<<<grid_ij(c->grid.ni, c->grid.nj), kThreads, 0, s>>>(phi, c->p, c->kappa, c->u, c->v, a, DtArg{dt, c->dt_dev}, sc);
  GB_LAUNCHED(1);
}

void launch_fast_sweeping(cudaStream_t s, gb2d_ctx* c, int sweeps) {
  const int ni = c->grid.ni, nj = c->grid.nj, n = ni > nj ? ni : nj;
  double* phi = c->phi_buf[c->phi_cur];
  k_fsm_fixed<<<grid_ij(ni, nj), kThreads, 0, s>>>(phi, c->tmp_a, ni, nj, 2.0 * c->base.dx);
  k_extrapolate_inner_first<<<(n + 127) / 128, 128, 0, s>>>(phi, 2, ni, nj);
  for (int k = 0; k < sweeps; ++k) k_fsm_sweep<<<1, 1024, 0, s>>>(phi, c->tmp_a, ni, nj, c->base.dx, k % 4);
  k_extrapolate_inner_first<<<(n + 127) / 128, 128, 0, s>>>(phi, 2, ni, nj);
  GB_LAUNCHED(3 + sweeps);
}

void launch_copy_interior(cudaStream_t s, const double* src, int gs, double* dst, int gd, int nI, int nJ) {
  k_copy_interior<<<grid_ij(nI, nJ), kThreads, 0, s>>>(src, gs, dst, gd, nI, nJ);
  GB_LAUNCHED(1);
}

}  // namespace gb2d
