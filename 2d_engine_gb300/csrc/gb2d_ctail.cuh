// gb2d_ctail.cuh — the coarse end of the V-cycle as ONE thread-block cluster.
//
// Included by gb2d_solver.cu inside its anonymous namespace (uses Level, Scalars,
// gs_sum, gs_residual, warp_sum, reduce_scratch, publish_rz, kMaxLevels, kCoarseMax).
//
// Every level from the cluster's top level (at most 128^2 cells) down to the dense
// coarse solve runs inside one launch of a cluster of P CTAs, each CTA one SM with 512
// threads: 16 where the part allows it, else 8; fewer, down to a single CTA, on
// hierarchies of too few rows (plan_ctail):
//
//   * distributed levels: the rows of a level are split into P contiguous
//     stripes, one per CTA, nested from level to level (the fine rows of a CTA's
//     coarse rows are its own fine rows).  A CTA works on its stripe and a halo of
//     rows on either side, wide enough that a whole side of smoothing (2 nu half
//     sweeps, each losing one row of exactness at the halo's edge) needs no
//     exchange; halo rows of the right-hand side and of x are pushed into the
//     neighbours' shared memory (distributed shared memory) when a level is left,
//     and one cluster barrier per level makes them visible;
//   * local levels (too few rows for P stripes): the stripes' restricted
//     residuals are pushed to every CTA, which runs these levels and the dense
//     coarse solve redundantly, with block barriers only; every CTA computes
//     identical values (same inputs, same order), and each prolongs from its own.
//
// What bounds it is the chain of dependent half sweeps, a few dozen of them, each on
// a few cells per thread.  So a half sweep does as little as it can: a thread owns
// pairs of neighbouring cells (one of each colour) with their coefficients and x in
// registers; x alone is in shared memory too, split by colour, and an update reads
// three neighbours from there (the fourth is its own) and writes one value.  The
// coefficients are read from global memory at the start of each level's sweeps.
// Clearing the x planes and reading the dense inverse overlap the previous kernel.
//
// <cooperative_groups.h> is included at global scope by the including file.

namespace cgx = cooperative_groups;

constexpr int kClusterMax = 16;
constexpr int kCtThreads = 512;
constexpr int kCtMaxLevels = 10;
constexpr int kCtMinRows = 4;           // rows per CTA on the coarsest distributed level
constexpr int kCtOwnerRows = 256;       // rows of the bottom distributed level at most
// Cell pairs per thread of the usual and of the largest kernel.  FP64: three fill the 128
// registers that a thread of 512 may have (72 bytes of spills; with four 548, with six 2080,
// which cost more than the launches that the cluster replaces: 121 x 132 to 1e-10 2.05 ms
// before the pairs were in registers, 2.38 with the kernel of six, 1.69 with that of three).
constexpr int kCtPairs = 2;
template <typename T>
constexpr int kCtPairsMax = sizeof(T) == 8 ? 3 : 6;
constexpr size_t kCtSmemCap = 220 * 1024;
// Largest top level.  From 64^2 instead, the mixed projection at 1024^2 takes 1.96 ms
// against 1.94 (at 256^2 0.81 against 0.79); a 256^2 level in 16 CTAs would take seven pairs
// a thread with three sweeps a side, more than the largest kernel has.
constexpr int kCtMaxTopCells = 128 * 128;

// Shared-memory offsets are in elements of T.  A plane holds one colour of a level's
// window: element (row - w0) * pairs + pair, w0 the window's first row; x planes have a
// ring of zeros, element (row - w0 + 1) * (pairs + 2) + pair + 1.
template <typename T>
struct CtLevel {
  int nI, nJ, ld;    // ld = nI + 2 (padded global layout)
  int pairs;         // (nI + 1) / 2
  unsigned rpairs;   // 2^32 / pairs, rounded up (pairs > 1): u / pairs as a high product
  int H;             // halo rows of the window (0 on local levels)
  int rcp;           // the residual as the tiled launches form it: dg as 1 / (1/dg), their order
  int x, xplane;     // x: red plane, black plane (xplane elements each)
  int b, xi, plane;  // right-hand side and received halo x: red, black (plane elements each); b -1 on the top level
  const T *cx, *cy, *idg, *dg, *bg;
  T* xg;
};

template <typename T>
struct CtArgs {
  int nlev;   // levels held; level 0 here is hierarchy level 'ctail'
  int ndist;  // levels [0, ndist) are distributed, the rest local
  int kpairs; // cell pairs per thread that the largest window takes
  int res;    // a level's red residuals, own rows: (row - J0) * pairs + pair
  int rg;     // the bottom distributed level's red residuals, all rows
  int bc;     // the coarsest level's right-hand side in cell order
  int zero_n; // elements from 0 to clear: every x, b plane
  int inv;    // dense inverse in shared memory, element (m, row) at m * cells + row (doubles), or -1:
              // rows summed in order by one thread each, as the single-CTA tail does
  int gather; // r.z of all rows summed by the first CTA, as the single-CTA tail sums it
  CtLevel<T> L[kCtMaxLevels];
  short J0[kCtMaxLevels][kClusterMax + 1];  // CTA c owns rows [J0[l][c], J0[l][c+1])
  Scalars* sc;  // set when the top level is the finest: publish r.z and beta
};

// A level's cell pairs in registers: index 0 the red, 1 the black cell of a pair.
template <typename T, int K>
struct CtRegs {
  T b[2][K], idg[2][K], cl[2][K], cr[2][K], y0[2][K], y1[2][K], x[2][K];
  int ad[K];  // element of the pair in the x planes
  int od[K];  // J & 1: which cell of the pair is red
};

// b - A x, every rounding stated.
template <typename T>
__device__ __forceinline__ T ct_residual(T b, T dg, T x, T cxl, T xl, T cxr, T xr, T cyb, T xb, T cyt, T xt) {
  return b - fmad(-cyt, xt, fmad(-cyb, xb, fmad(-cxr, xr, fmad(dg, x, -mulr(cxl, xl)))));
}

// This CTA's view of a level: window rows [w0, w0 + R), own rows [J0, J1).
struct CtWin {
  int J0, J1, w0, R;
};
template <typename T>
__device__ __forceinline__ CtWin ct_win(const CtArgs<T>& a, int l, int c) {
  const CtLevel<T>& L = a.L[l];
  if (l >= a.ndist) return CtWin{0, L.nJ, 0, L.nJ};
  const int J0 = a.J0[l][c], J1 = a.J0[l][c + 1];
  const int w0 = J0 - L.H > 0 ? J0 - L.H : 0, w1 = J1 + L.H < L.nJ ? J1 + L.H : L.nJ;
  return CtWin{J0, J1, w0, w1 - w0};
}
// Window row of pair u.
template <typename T>
__device__ __forceinline__ int ct_row(const CtLevel<T>& L, int u) {
  return L.pairs == 1 ? u : (int)__umulhi((unsigned)u, L.rpairs);
}

// One pair's coefficients: of the red and the black cell 1/dg, the conductances of its
// left, right, lower and upper faces, and the red cell's dg.
template <typename T>
struct CtCoef {
  T idg[2], cl[2], cr[2], y0[2], y1[2], dg;
};
template <typename T>
__device__ __forceinline__ CtCoef<T> ct_coef(const CtLevel<T>& L, const CtWin& w, int u) {
  CtCoef<T> f;
  const int lr = ct_row(L, u), o = (w.w0 + lr) & 1, q = (w.w0 + lr + 1) * L.ld + 2 * (u - lr * L.pairs) + 1;
#pragma unroll
  for (int col = 0; col < 2; ++col) {
    const int p = q + (col == 0 ? o : 1 - o);
    f.idg[col] = L.idg[p];
    f.cl[col] = L.cx[p];
    f.cr[col] = L.cx[p + 1];
    f.y0[col] = L.cy[p];
    f.y1[col] = L.cy[p + L.ld];
  }
  f.dg = L.dg[q + o];
  return f;
}

// Coefficients, right-hand side and places of the pairs that this thread owns (pair tid +
// k kCtThreads).  Beyond the window's pairs they are zero and the place is a ring cell.
template <typename T, int K>
__device__ __forceinline__ void ct_load(const CtLevel<T>& L, const CtWin& w, const T* sm, CtRegs<T, K>& g, T* dg) {
  const int n = w.R * L.pairs;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int u = (int)threadIdx.x + k * kCtThreads;
    CtCoef<T> f = {};
    g.ad[k] = L.pairs + 2;
    g.od[k] = 0;
    g.b[0][k] = g.b[1][k] = (T)0;
    if (u < n) {
      const int lr = ct_row(L, u), m = u - lr * L.pairs, o = (w.w0 + lr) & 1;
      g.ad[k] = (lr + 1) * (L.pairs + 2) + m + 1;
      g.od[k] = o;
      f = ct_coef(L, w, u);
      if (L.b < 0) {
        const int q = (w.w0 + lr + 1) * L.ld + 2 * m + 1;
        g.b[0][k] = __ldcg(L.bg + q + o);  // through L2: the CG kernel's other CTAs write it
        g.b[1][k] = __ldcg(L.bg + q + 1 - o);
      } else {
        g.b[0][k] = sm[L.b + u];
        g.b[1][k] = sm[L.b + L.plane + u];
      }
    }
#pragma unroll
    for (int col = 0; col < 2; ++col) {
      g.idg[col][k] = f.idg[col];
      g.cl[col][k] = f.cl[col];
      g.cr[col][k] = f.cr[col];
      g.y0[col][k] = f.y0[col];
      g.y1[col][k] = f.y1[col];
    }
    if (dg) dg[k] = f.dg;
  }
}

// One colour of a red-black Gauss-Seidel sweep over the window's pairs [lo, hi).  The
// pair's cells are (2m, J), (2m + 1, J); the red one is 2m + (J & 1).  A cell's horizontal
// neighbours are the pair's other cell and the neighbouring pair's cell of the other
// colour; its vertical ones sit at the same pair of rows J -+ 1.  FIRST: x is zero, and
// the update is b / dg.
template <int COLOR, bool FIRST, typename T, int K>
__device__ __forceinline__ void ct_half(T* xp, int xplane, int ps, CtRegs<T, K>& g, int lo, int hi) {
  const T* xo = xp + (COLOR == 0 ? xplane : 0);
  T* xw = xp + (COLOR == 0 ? 0 : xplane);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int u = (int)threadIdx.x + k * kCtThreads;
    if (u < lo || u >= hi) continue;
    const int ad = g.ad[k];
    if (FIRST) {
      xw[ad] = g.x[COLOR][k] = mulr(g.b[COLOR][k], g.idg[COLOR][k]);
      continue;
    }
    const bool right = (g.od[k] != 0) == (COLOR == 0);  // the cell is the pair's right one
    const T own = g.x[1 - COLOR][k], side = xo[right ? ad + 1 : ad - 1], xb = xo[ad - ps], xt = xo[ad + ps];
    const T v = mulr(gs_sum(g.b[COLOR][k], g.cl[COLOR][k], right ? own : side, g.cr[COLOR][k], right ? side : own, g.y0[COLOR][k], xb,
                            g.y1[COLOR][k], xt),
                     g.idg[COLOR][k]);
    g.x[COLOR][k] = v;
    xw[ad] = v;
  }
}
// Barrier of the threads that own the pairs of one level: the whole block, or its first
// four warps (which a block barrier would make wait for the other twelve).
constexpr int kCtFew = 128;
template <bool FEW>
__device__ __forceinline__ void ct_sync() {
  if (FEW)
    asm volatile("bar.sync 1, %0;" ::"n"(kCtFew) : "memory");
  else
    __syncthreads();
}
// 2 nu half sweeps, the first of colour C0, a barrier after each, over rows that
// shrink to the own rows and `last` more on either side: each half sweep needs its
// neighbour rows exact from the one before (FP64 levels are bound by the FP64 pipe, so
// rows that nothing exact reads are left out).
template <int C0, bool FEW, typename T, int K>
__device__ __forceinline__ void ct_smooth(const CtLevel<T>& L, const CtWin& w, T* sm, CtRegs<T, K>& g, int nu, int last) {
  T* xp = sm + L.x;
  const int o0 = (w.J0 - w.w0) * L.pairs, o1 = (w.J1 - w.w0) * L.pairs;
  int e = (last + 2 * nu - 1) * L.pairs;
  for (int s = 0; s < nu; ++s) {
    if (C0 == 0 && s == 0)  // pre-smoothing starts from x = 0
      ct_half<C0, C0 == 0>(xp, L.xplane, L.pairs + 2, g, o0 - e, o1 + e);
    else
      ct_half<C0, false>(xp, L.xplane, L.pairs + 2, g, o0 - e, o1 + e);
    e -= L.pairs;
    ct_sync<FEW>();
    ct_half<1 - C0, false>(xp, L.xplane, L.pairs + 2, g, o0 - e, o1 + e);
    e -= L.pairs;
    ct_sync<FEW>();
  }
}

// Pre-smoothing from x = 0 (the x planes are clear), then the own rows' red residuals
// b - A x; the black ones are zero after the last black half sweep.  On distributed
// levels x of the own rows goes to the CTAs whose windows hold them.
template <int K, bool FEW, typename T>
__device__ __forceinline__ void ct_smooth_down(const CtArgs<T>& a, int l, int c, int P, const CtWin& w, T* sm, CtRegs<T, K>& g, const T* dg,
                                               int nu) {
  const CtLevel<T>& L = a.L[l];
  const int o0 = (w.J0 - w.w0) * L.pairs, o1 = (w.J1 - w.w0) * L.pairs;
#pragma unroll
  for (int k = 0; k < K; ++k) g.x[0][k] = g.x[1][k] = (T)0;
  ct_smooth<0, FEW>(L, w, sm, g, nu, 1);
  const T* xb = sm + L.x + L.xplane;
  const int ps = L.pairs + 2;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int ad = g.ad[k], u = (int)threadIdx.x + k * kCtThreads;
    if (u < o0 || u >= o1) continue;
    const bool right = g.od[k] != 0;
    const T own = g.x[1][k], side = xb[right ? ad + 1 : ad - 1];
    const T xl = right ? own : side, xr = right ? side : own;
    // A pair at an odd row's end may lack its red cell: 1/dg is the padding's zero there.
    const T d = !L.rcp ? dg[k] : g.idg[0][k] == (T)0 ? (T)0 : diag_of(g.idg[0][k]);
    sm[a.res + u - o0] = L.rcp ? gs_residual(g.b[0][k], d, g.x[0][k], g.cl[0][k], xl, g.cr[0][k], xr, g.y0[0][k],
                                             xb[ad - ps], g.y1[0][k], xb[ad + ps])
                               : ct_residual(g.b[0][k], d, g.x[0][k], g.cl[0][k], xl, g.cr[0][k], xr, g.y0[0][k], xb[ad - ps],
                                             g.y1[0][k], xb[ad + ps]);
    if (l < a.ndist) {
      const int J = w.w0 + ct_row(L, u);
      auto push = [&](int d) {
        const int w0 = a.J0[l][d] - L.H > 0 ? a.J0[l][d] - L.H : 0;
        T* dst = cgx::this_cluster().map_shared_rank(sm + L.xi, d) + u + (w.w0 - w0) * L.pairs;
        dst[0] = g.x[0][k];
        dst[L.plane] = g.x[1][k];
      };
      for (int d = c - 1; d >= 0 && a.J0[l][d + 1] + L.H > J; --d) push(d);
      for (int d = c + 1; d < P && a.J0[l][d] - L.H <= J; ++d) push(d);
    }
  }
}

// x (own rows from the x planes, halo rows as received) plus the coarse correction, then
// the post-smoothing (black first).  The top level's own rows go to global memory.
template <int K, bool FEW, typename T>
__device__ __forceinline__ void ct_smooth_up(const CtArgs<T>& a, int l, int c, const CtWin& w, T* sm, CtRegs<T, K>& g, int nu) {
  const CtLevel<T>& L = a.L[l];
  const CtLevel<T>& C = a.L[l + 1];
  const int cw0 = ct_win(a, l + 1, c).w0;
  T* xp = sm + L.x;
  const int o0 = (w.J0 - w.w0) * L.pairs, o1 = (w.J1 - w.w0) * L.pairs, n = w.R * L.pairs;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int ad = g.ad[k], u = (int)threadIdx.x + k * kCtThreads;
    g.x[0][k] = g.x[1][k] = (T)0;
    if (u >= n) continue;
    const int lr = ct_row(L, u), m = u - lr * L.pairs, Jc = (w.w0 + lr) >> 1;
    const T xc = sm[C.x + (((m + Jc) & 1) ? C.xplane : 0) + (Jc - cw0 + 1) * (C.pairs + 2) + (m >> 1) + 1];
    const bool own = u >= o0 && u < o1;
    const T x0 = (own ? xp[ad] : sm[L.xi + u]) + xc, x1 = (own ? xp[ad + L.xplane] : sm[L.xi + L.plane + u]) + xc;
    const bool one = 2 * m + 1 >= L.nI;  // a pair at an odd row's end has one cell, its left one
    g.x[0][k] = one && g.od[k] ? (T)0 : x0;
    g.x[1][k] = one && !g.od[k] ? (T)0 : x1;
    xp[ad] = g.x[0][k];
    xp[ad + L.xplane] = g.x[1][k];
  }
  ct_sync<FEW>();
  ct_smooth<1, FEW>(L, w, sm, g, nu, l == 0 ? 0 : (a.L[l - 1].H + 1) / 2);
  if (l > 0) return;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int u = (int)threadIdx.x + k * kCtThreads;
    if (u < o0 || u >= o1) continue;
    const int lr = ct_row(L, u), m = u - lr * L.pairs;
    T* x = L.xg + (w.w0 + lr + 1) * L.ld + 2 * m + 1;
    x[0] = g.od[k] ? g.x[1][k] : g.x[0][k];
    if (2 * m + 1 < L.nI) x[1] = g.od[k] ? g.x[0][k] : g.x[1][k];
  }
}

template <int K, bool FEW, typename T>
__device__ __forceinline__ void ct_down(const CtArgs<T>& a, int l, int c, int P, T* sm, int nu) {
  const CtWin w = ct_win(a, l, c);
  CtRegs<T, K> g;
  T dg[K];
  ct_load<T, K>(a.L[l], w, sm, g, dg);
  ct_smooth_down<K, FEW>(a, l, c, P, w, sm, g, dg, nu);
}
template <int K, bool FEW, typename T>
__device__ __forceinline__ void ct_up(const CtArgs<T>& a, int l, int c, T* sm, int nu) {
  const CtWin w = ct_win(a, l, c);
  CtRegs<T, K> g;
  ct_load<T, K>(a.L[l], w, sm, g, nullptr);
  ct_smooth_up<K, FEW>(a, l, c, w, sm, g, nu);
}

__device__ __forceinline__ float ct_ainv(double v, float) { return narrow(v); }  // FP32 values, widened
__device__ __forceinline__ double ct_ainv(double v, double) { return v; }

// The dense coarse solve's operands: 16 threads per row, 4 terms each, rows tid / 16 and
// tid / 16 + 32, and the rows' places in the coarsest level's x planes.
template <typename T>
struct CtDense {
  T ai[2][4];
  int zx[2];
};
template <typename T>
__device__ __forceinline__ CtDense<T> ct_dense_load(const CtArgs<T>& a, const double* __restrict__ ainv, T* sm) {
  CtDense<T> d;
  const CtLevel<T>& Z = a.L[a.nlev - 1];
  const int nz = Z.nI * Z.nJ, tid = (int)threadIdx.x;
  if (a.inv >= 0) {
    double* inv = reinterpret_cast<double*>(sm + a.inv);
    for (int u = tid; u < nz * nz; u += kCtThreads) {
      const int r = u / nz, m = u - r * nz;
      inv[m * nz + r] = ainv[u];
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = (tid >> 4) + 32 * h, J = r / Z.nI, I = r - J * Z.nI;
    d.zx[h] = Z.x + (((I + J) & 1) ? Z.xplane : 0) + (J + 1) * (Z.pairs + 2) + (I >> 1) + 1;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int m = (tid & 15) + 16 * q;
      d.ai[h][q] = r < nz && m < nz ? ct_ainv(ainv[r * nz + m], T()) : (T)0;
    }
  }
  return d;
}
// Right-hand side at bc, fixed-order tree sum.
template <typename T>
__device__ __forceinline__ void ct_dense_solve(const CtArgs<T>& a, const CtDense<T>& d, T* sm) {
  const CtLevel<T>& Z = a.L[a.nlev - 1];
  const int nz = Z.nI * Z.nJ, tid = (int)threadIdx.x, part = tid & 15, bc = a.bc;
  if (a.inv >= 0) {
    if (tid < nz) {
      const double* inv = reinterpret_cast<const double*>(sm + a.inv) + tid;
      double acc = 0.0;
      for (int m = 0; m < nz; ++m) acc = __fma_rn(inv[m * nz], (double)sm[bc + m], acc);
      const int J = tid / Z.nI, I = tid - J * Z.nI;
      sm[Z.x + (((I + J) & 1) ? Z.xplane : 0) + (J + 1) * (Z.pairs + 2) + (I >> 1) + 1] = (T)acc;
    }
    __syncthreads();
    return;
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = (tid >> 4) + 32 * h;
    T acc = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (r < nz && part + 16 * q < nz) acc = fmad(d.ai[h][q], sm[bc + part + 16 * q], acc);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (r < nz && part == 0) sm[d.zx[h]] = acc;
  }
  __syncthreads();
}

// A local level's right-hand side from the finer level's red residuals: those of all rows
// of the bottom distributed level, or a local level's.
template <typename T>
__device__ __forceinline__ void ct_restrict_local(const CtArgs<T>& a, int l, T* sm) {
  const CtLevel<T>& F = a.L[l - 1];
  const CtLevel<T>& L = a.L[l];
  const T* rs = sm + (l == a.ndist ? a.rg : a.res);
  for (int u = (int)threadIdx.x; u < L.nI * L.nJ; u += kCtThreads) {
    const int J = ct_row(F, u), I = u - J * F.pairs;  // F.pairs = L.nI
    T acc = 0;
    for (int bb = 0; bb < 2; ++bb)
      if (2 * J + bb < F.nJ) acc += rs[(2 * J + bb) * F.pairs + I];
    const T v = (T)0.25 * acc;
    sm[l == a.nlev - 1 ? a.bc + u : L.b + (((I + J) & 1) ? L.plane : 0) + J * L.pairs + (I >> 1)] = v;
  }
  __syncthreads();
}

// Leaving distributed level l downwards, its residuals complete: the coarse right-hand
// side of the own rows, here and in the windows that hold them, or, from the bottom
// distributed level, the own rows' residuals to every CTA (one warp per CTA).
template <typename T>
__device__ __forceinline__ void ct_hand_down(const CtArgs<T>& a, int l, int c, int P, T* sm) {
  cgx::cluster_group cl = cgx::this_cluster();
  const CtLevel<T>& L = a.L[l];
  const CtWin w = ct_win(a, l, c);
  const int tid = (int)threadIdx.x;
  if (l + 1 < a.ndist) {
    const CtLevel<T>& C = a.L[l + 1];
    const int cJ0 = a.J0[l + 1][c], cJ1 = a.J0[l + 1][c + 1];
    for (int u = tid; u < (cJ1 - cJ0) * C.nI; u += kCtThreads) {
      const int lr = ct_row(L, u), I = u - lr * C.nI, J = cJ0 + lr;  // L.pairs = C.nI
      T acc = 0;
      for (int bb = 0; bb < 2; ++bb)
        if (2 * J + bb < L.nJ) acc += sm[a.res + (2 * J + bb - w.J0) * L.pairs + I];
      const T v = (T)0.25 * acc;
      const int e = C.b + (((I + J) & 1) ? C.plane : 0) + (I >> 1);
      auto put = [&](int d) {
        const int w0 = a.J0[l + 1][d] - C.H > 0 ? a.J0[l + 1][d] - C.H : 0;
        cl.map_shared_rank(sm + e, d)[(J - w0) * C.pairs] = v;
      };
      put(c);
      for (int d = c - 1; d >= 0 && a.J0[l + 1][d + 1] + C.H > J; --d) put(d);
      for (int d = c + 1; d < P && a.J0[l + 1][d] - C.H <= J; ++d) put(d);
    }
  } else {
    const int own = (w.J1 - w.J0) * L.pairs, at = a.rg + w.J0 * L.pairs;
    for (int d = tid >> 5; d < P; d += kCtThreads / 32) {
      T* dst = cl.map_shared_rank(sm + at, d);
      for (int e = tid & 31; e < own; e += 32) dst[e] = sm[a.res + e];
    }
  }
  cl.sync();
}

// r.z when the top level is the finest: a block sum over 1024 strided partials (two per
// thread) in block_sum's order; a warp's sum over no elements is the zero it would add up.
// Valid in the first warp's lane 0.  With a.gather the first CTA sums all rows, from global
// memory, once every CTA's x is there.
template <typename T>
__device__ __forceinline__ double ct_rz(const CtArgs<T>& a, int c, const T* sm) {
  const CtLevel<T>& L = a.L[0];
  CtWin w = ct_win(a, 0, c);
  if (a.gather) {
    cgx::this_cluster().sync();
    if (c > 0) return 0.0;
    w.J0 = 0;
    w.J1 = L.nJ;
  }
  double* scratch = reduce_scratch();
  const int n = (w.J1 - w.J0) * L.nI, tid = (int)threadIdx.x;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    double acc = 0.0;
    if ((tid & ~31) + h * kCtThreads < n) {
      for (int u = tid + h * kCtThreads; u < n; u += 2 * kCtThreads) {
        const int lr = u / L.nI, i = u - lr * L.nI, J = w.J0 + lr;
        const int q = (J + 1) * L.ld + i + 1;
        const T bv = __ldcg(L.bg + q);
        const T xv = a.gather ? __ldcg(L.xg + q) : sm[L.x + (((i + J) & 1) ? L.xplane : 0) + (J - w.w0 + 1) * (L.pairs + 2) + (i >> 1) + 1];
        acc = __fma_rn((double)bv, (double)xv, acc);
      }
      acc = warp_sum(acc);
    }
    if ((tid & 31) == 0) scratch[(tid >> 5) + h * (kCtThreads / 32)] = acc;
  }
  __syncthreads();
  return tid < 32 ? warp_sum(scratch[tid]) : 0.0;
}

// One V-cycle from the top level's right-hand side to its x, both in global memory.
template <int K, typename T>
__device__ __forceinline__ void ct_vcycle(const CtArgs<T>& a, int c, int P, const CtDense<T>& dense, T* sm, int nu) {
  const int nl = a.nlev, nd = a.ndist, tid = (int)threadIdx.x;
  for (int l = 0; l < nl; ++l) {
    if (l >= nd && l > 0) ct_restrict_local(a, l, sm);
    if (l == nl - 1) break;
    const int n = ct_win(a, l, c).R * a.L[l].pairs;
    if (K > 1 && n > kCtThreads)
      ct_down<K, false>(a, l, c, P, sm, nu);
    else if (n > kCtFew)
      ct_down<1, false>(a, l, c, P, sm, nu);
    else if (tid < kCtFew)
      ct_down<1, true>(a, l, c, P, sm, nu);
    __syncthreads();
    if (l < nd) ct_hand_down(a, l, c, P, sm);
  }
  ct_dense_solve(a, dense, sm);
  for (int l = nl - 2; l >= 0; --l) {
    const int n = ct_win(a, l, c).R * a.L[l].pairs;
    if (K > 1 && n > kCtThreads)
      ct_up<K, false>(a, l, c, sm, nu);
    else if (n > kCtFew)
      ct_up<1, false>(a, l, c, sm, nu);
    else if (tid < kCtFew)
      ct_up<1, true>(a, l, c, sm, nu);
    __syncthreads();
  }
}

// The whole tail, up to K pairs per thread.
// Against a cluster of 1024-thread CTAs that staged whole levels in shared memory (ten
// reads and a cluster barrier per half sweep, about 50 barriers): the mixed projection to
// 1e-8 from host arrays 0.88 -> 0.66 ms at 64^2 and 2.77 -> 2.57 ms at 1024^2, about 13 us
// of an iteration's 118; FP64 tails are bound by the FP64 pipe and gain little.  Also
// measured, not kept: the coefficients packed by pairs and staged in shared memory while
// the previous kernel runs, each level's pairs held in registers from the way down to the
// way up (124 registers): 2% faster at 64^2 but 5% slower at 1024^2, where the wider CTAs
// find room only when the previous kernel's blocks have left; 64 and 80 registers a thread
// are no faster than the 96 that it takes.
template <typename T, int K>
__global__ void __launch_bounds__(kCtThreads, 1) k_ctail(const __grid_constant__ CtArgs<T> a, const double* __restrict__ ainv, int nu,
                                                         const int* __restrict__ done) {
  cgx::cluster_group cl = cgx::this_cluster();
  const int P = (int)cl.num_blocks(), c = (int)cl.block_rank(), tid = (int)threadIdx.x;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);
  __shared__ double rz_part[kClusterMax];
  // Before the previous kernel has finished: what it does not write.
  const CtDense<T> dense = ct_dense_load(a, ainv, sm);
  for (int u = tid; u < a.zero_n; u += kCtThreads) sm[u] = (T)0;
  cl.sync();  // every CTA's planes are clear before any remote write
  pdl_enter();
  if (*done) return;  // uniform over the cluster: no CTA writes remotely or reaches a cluster barrier
  ct_vcycle<K>(a, c, P, dense, sm, nu);
  if (a.sc) {
    const double v = ct_rz(a, c, sm);
    if (tid == 0) *cl.map_shared_rank(&rz_part[c], 0) = v;
    cl.sync();
    if (c == 0 && tid == 0) {
      double rz = 0.0;
      for (int o = 0; o < P; ++o) rz += rz_part[o];
      publish_rz(a.sc, rz);
    }
  }
}
