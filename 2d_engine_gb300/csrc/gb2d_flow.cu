// The stages of SolveForRK around the projection (EULERIAN_FLUID_SOLVER_2D.h:1857-1879)
// and the velocity TVD-RK3 blends (:1753-1794): gravity, DetermineDensity, the
// explicit delta-function viscosity (VISCOSITY_2D.h:460-532) and the wall
// conditions, fused into one pass over the two MAC face grids; and the CFL time
// step (:3517-3637).
// Built with --fmad=false, in the reference's association order, like
// gb2d_exact.cu: the results are the reference's FP64 results bit for bit, except
// where the smeared Heaviside's sine (the only libm call) differs in the last ulp.
#include <cmath>

#include "gb2d_internal.cuh"
#include "gb2d_schemes.cuh"

namespace gb2d {

namespace {

// lo + (hi - lo) * H(phi): a smeared density or viscosity.  at0 / at1 are its
// values where H is 0 or 1, formed on the host with the same two operations.
struct Smear {
  double lo, d, at0, at1;
};
Smear make_smear(double lo, double hi) {
  Smear s;
  s.lo = lo;
  s.d = hi - lo;
  s.at0 = lo + s.d * 0.0;
  s.at1 = lo + s.d * 1.0;
  return s;
}

struct SmearF {
  float lo, d, at0, at1;
};

struct FlowArgs {
  int ni, nj;
  int grav, bc;        // add dt * gravity to every face; zero the wall faces' normal velocity
  double gx, gy;       // dt * gravity
  double dt, odx, ody;
  double eps, oe;      // smearing width 1.5 dx (EULERIAN_FLUID_SOLVER_2D.h:347) and its reciprocal
  Smear rho, mu;       // face density and viscosity
  double coef0, coef1; // dt * (1 / rho.at0), dt * (1 / rho.at1)
  double air, water;   // node densities of DetermineDensity
  // Non-null: the time step is read here when the kernel runs, and the dt-derived fields
  // above are formed from it as the host forms them (g_x, g_y: gravity; inv_rho0/1 = 1 / rho.at0/1).
  const double* dtp;
  double g_x, g_y, inv_rho0, inv_rho1;
  // FP32 viscous-flux path
  float odx_f, ody_f, eps_f, oe_f, dt_f, coef0_f, coef1_f;
  SmearF rho_f, mu_f;
  int fast;            // densities, viscosities and cell sizes are in the fast products' range
  int row0;            // the viscous launch's first tile row
};

// FP32 forms for the viscous flux of the mixed path.
__device__ __forceinline__ float heaviside_band_f(float phi, float oe) {
  const float PI_REF = 3.141592f, opi = 1.0f / PI_REF;
  return 0.5f + phi * oe * 0.5f + 0.5f * opi * __sinf(PI_REF * phi * oe);
}
__device__ __forceinline__ float smear_f(float l, const SmearF& s, const FlowArgs& a) {
  if (l < -a.eps_f) return s.at0;
  if (l > a.eps_f) return s.at1;
  return s.lo + s.d * heaviside_band_f(l, a.oe_f);
}

// The dt-dependent fields of FlowArgs, as launch_flow forms them on the host.
__host__ __device__ __forceinline__ void with_time_step(FlowArgs& a, double dt) {
  a.gx = dt * a.g_x;
  a.gy = dt * a.g_y;
  a.dt = dt;
  a.coef0 = dt * a.inv_rho0;
  a.coef1 = dt * a.inv_rho1;
  a.dt_f = (float)dt;
  a.coef0_f = (float)a.coef0;
  a.coef1_f = (float)a.coef1;
}

// Gravity and wall conditions over the (ni+1) x (nj+1) face index space, in place: x-face
// (i, j), i <= ni, j < nj; y-face (i, j), i < ni, j <= nj; node (i, j) for the density.
// density (ghost 2, may be null) receives DetermineDensity (:2162-2180): air where
// phi <= 0, water where phi > 0, unchanged for NaN.
__device__ __forceinline__ void put_density(double* dens_a, const FlowArgs& a, int i, int j, double l) {
  const DField dn = dfield(dens_a, 2, a.ni, a.nj);
  if (lez(l))
    GB_AT(dn, i, j) = a.air;
  else if (gtz(l))
    GB_AT(dn, i, j) = a.water;
}
__global__ void k_flow(const double* __restrict__ phi_a, double* u_a, double* v_a, double* __restrict__ dens_a, FlowArgs a) {
  pdl_enter();
  if (a.dtp) with_time_step(a, *a.dtp);
  const int ni = a.ni, nj = a.nj;
  const DField phi = dfield((double*)phi_a, 2, ni, nj), u = dfield(u_a, 2, ni + 1, nj), v = dfield(v_a, 2, ni, nj + 1);
  GB_FOR_IJ(i, j, ni + 1, nj + 1) {
    if (dens_a && i < ni && j < nj) put_density(dens_a, a, i, j, GB_AT(phi, i, j));
    if (j < nj) {
      double w = GB_AT(u, i, j);
      if (a.grav) w = w + a.gx;
      if (a.bc && (i == 0 || i == ni)) w = 0.0;
      GB_AT(u, i, j) = w;
    }
    if (i < ni) {
      double w = GB_AT(v, i, j);
      if (a.grav) w = w + a.gy;
      if (a.bc && (j == 0 || j == nj)) w = 0.0;
      GB_AT(v, i, j) = w;
    }
  }
}

// ---- the explicit viscosity (ApplyViscosity) with gravity and walls ----
//
// With T the faces after gravity (zero off the face grids, the reference's freshly
// initialised temporaries), node terms and corner terms
//   X(i, j) = mu(phi(i, j)) ox (Tu(i+1, j) - Tu(i, j)),   Y(i, j) = mu(phi(i, j)) oy (Tv(i, j+1) - Tv(i, j)),
//   K(i, j) = mu(phi at the lower left corner) (oy (Tu(i, j) - Tu(i, j-1)) + ox (Tv(i, j) - Tv(i-1, j))),
// the new faces are
//   u = Tu + (2 c ox (X(i, j) - X(i-1, j)) + c oy (K(i, j+1) - K(i, j))),
//   v = Tv + (2 c oy (Y(i, j) - Y(i, j-1)) + c ox (K(i+1, j) - K(i, j))),   c = dt / rho of the face,
// every term with the operations, and their order, of the reference's expression: a term
// that two or four faces share is the same number in each.  A tile forms each term once
// (20 FP64 additions a node instead of 55 operations a face), products on the integer
// pipes.  MIXED (R = float): the terms in FP32 from FP64 differences of the faces before
// gravity (off the grids minus gravity, so that the differences are those of T), the face
// values and the update FP64.
constexpr int kFlX = 32, kFlY = 8;
template <typename R>
struct FlowTile {
  double u[kFlY + 2][kFlX + 2], v[kFlY + 2][kFlX + 2];  // faces (i0 - 1 + x, j0 - 1 + y)
  R p[kFlY + 2][kFlX + 2], mu[kFlY + 2][kFlX + 2];      // phi and mu(phi) at nodes (i0 - 1 + x, j0 - 1 + y)
  R X[kFlY][kFlX + 1], Y[kFlY + 1][kFlX], K[kFlY + 1][kFlX + 1];
};
// dt-derived values, formed once per block.
template <typename R>
struct FlowStep {
  double gx, gy;
  R dt, c0, c1, c0x2, c1x2, c0y2, c1y2, c0x, c1x, c0y, c1y;  // c: outside the band; 2 c ox, 2 c oy, c ox, c oy
  int ok;                                                    // they are in the fast products' range
};
__device__ __noinline__ double smear_band(double l, const Smear& s, double oe) { return s.lo + s.d * heaviside_band(l, oe); }
__device__ __noinline__ double coef_band(double l, const Smear& s, double oe, double dt) { return dt * (1 / (s.lo + s.d * heaviside_band(l, oe))); }
__device__ __forceinline__ double visc_mu(double l, const FlowArgs& a) {
  if (lt_neg(l, a.eps)) return a.mu.at0;
  if (gt_pos(l, a.eps)) return a.mu.at1;
  return smear_band(l, a.mu, a.oe);
}
__device__ __forceinline__ float visc_mu(float l, const FlowArgs& a) { return smear_f(l, a.mu_f, a); }
template <bool FAST>
__device__ __forceinline__ double visc_mul(double x, double y) { return FAST ? mul_rn(x, y) : x * y; }
template <bool FAST>
__device__ __forceinline__ float visc_mul(float x, float y) { return x * y; }
__device__ __forceinline__ double visc_quarter(double s) { return mul_wide(s, 0.25); }
__device__ __forceinline__ float visc_quarter(float s) { return 0.25f * s; }
__device__ __forceinline__ double visc_half(double s) { return mul_wide(s, 0.5); }
__device__ __forceinline__ float visc_half(float s) { return 0.5f * s; }
__device__ __forceinline__ double visc_diff(double x, double y, double) { return x - y; }
__device__ __forceinline__ float visc_diff(double x, double y, float) { return narrow(x - y); }
// 2 c o and c o of a face whose phi averages to l: o = ox (along = true) for 2 c o and the
// other cell size for c o.
__device__ __forceinline__ void visc_coef(double l, bool xface, const FlowArgs& a, const FlowStep<double>& t, double& c2, double& c1) {
  if (lt_neg(l, a.eps)) {
    c2 = xface ? t.c0x2 : t.c0y2;
    c1 = xface ? t.c0y : t.c0x;
  } else if (gt_pos(l, a.eps)) {
    c2 = xface ? t.c1x2 : t.c1y2;
    c1 = xface ? t.c1y : t.c1x;
  } else {
    const double c = coef_band(l, a.rho, a.oe, t.dt);
    c2 = 2.0 * c * (xface ? a.odx : a.ody);
    c1 = c * (xface ? a.ody : a.odx);
  }
}
__device__ __forceinline__ void visc_coef(float l, bool xface, const FlowArgs& a, const FlowStep<float>& t, float& c2, float& c1) {
  const float c = l < -a.eps_f ? t.c0 : l > a.eps_f ? t.c1 : __fdividef(t.dt, a.rho_f.lo + a.rho_f.d * heaviside_band_f(l, a.oe_f));
  c2 = 2.0f * c * (xface ? a.odx_f : a.ody_f);
  c1 = c * (xface ? a.ody_f : a.odx_f);
}

// The tile's terms and new faces, after its staging.  FAST: every product on the integer pipes.
template <typename R, bool FAST>
__device__ __forceinline__ void flow_tile(FlowTile<R>& t, const FlowStep<R>& st, const FlowArgs& a, int i0, int j0, DField uo, DField vo) {
  constexpr int NT = kFlX * kFlY, W = kFlX + 1;
  constexpr bool MIXED = sizeof(R) == 4;
  const int tid = threadIdx.x, tx = tid & (kFlX - 1), ty = tid / kFlX, i = i0 + tx, j = j0 + ty;
  R ox, oy;
  if constexpr (MIXED) {
    ox = a.odx_f;
    oy = a.ody_f;
  } else {
    ox = a.odx;
    oy = a.ody;
  }
  for (int k = tid; k < kFlY * W; k += NT) {  // X of nodes (i0 - 1 + x, j0 + y)
    const int y = k / W, x = k - y * W;
    t.X[y][x] = visc_mul<FAST>(visc_mul<FAST>(t.mu[y + 1][x], ox), visc_diff(t.u[y + 1][x + 1], t.u[y + 1][x], R()));
  }
  for (int k = tid; k < (kFlY + 1) * kFlX; k += NT) {  // Y of nodes (i0 + x, j0 - 1 + y)
    const int y = k / kFlX, x = k - y * kFlX;
    t.Y[y][x] = visc_mul<FAST>(visc_mul<FAST>(t.mu[y][x + 1], oy), visc_diff(t.v[y + 1][x + 1], t.v[y][x + 1], R()));
  }
  for (int k = tid; k < (kFlY + 1) * W; k += NT) {  // K of the lower left corners of nodes (i0 + x, j0 + y)
    const int y = k / W, x = k - y * W;
    const R mu = visc_mu(visc_quarter(t.p[y][x] + t.p[y][x + 1] + t.p[y + 1][x] + t.p[y + 1][x + 1]), a);
    const R du = visc_mul<FAST>(oy, visc_diff(t.u[y + 1][x + 1], t.u[y][x + 1], R()));
    const R dv = visc_mul<FAST>(ox, visc_diff(t.v[y + 1][x + 1], t.v[y + 1][x], R()));
    t.K[y][x] = visc_mul<FAST>(mu, du + dv);
  }
  __syncthreads();
  const R pc = t.p[ty + 1][tx + 1];
  R c2, c1;
  if (i <= a.ni && j < a.nj) {
    visc_coef(visc_half(t.p[ty + 1][tx] + pc), true, a, st, c2, c1);
    const R f = visc_mul<FAST>(c2, t.X[ty][tx + 1] - t.X[ty][tx]) + visc_mul<FAST>(c1, t.K[ty + 1][tx] - t.K[ty][tx]);
    double w = t.u[ty + 1][tx + 1];
    if (MIXED && a.grav) w = w + st.gx;
    w = w + widen(f);
    if (a.bc && (i == 0 || i == a.ni)) w = 0.0;
    GB_AT(uo, i, j) = w;
  }
  if (i < a.ni && j <= a.nj) {
    visc_coef(visc_half(t.p[ty][tx + 1] + pc), false, a, st, c2, c1);
    const R f = visc_mul<FAST>(c2, t.Y[ty + 1][tx] - t.Y[ty][tx]) + visc_mul<FAST>(c1, t.K[ty][tx + 1] - t.K[ty][tx]);
    double w = t.v[ty + 1][tx + 1];
    if (MIXED && a.grav) w = w + st.gy;
    w = w + widen(f);
    if (a.bc && (j == 0 || j == a.nj)) w = 0.0;
    GB_AT(vo, i, j) = w;
  }
}
// Out of line: differences outside the fast products' range.
__device__ __noinline__ void flow_tile_plain(FlowTile<double>& t, const FlowStep<double>& st, const FlowArgs& a, int i0, int j0, DField uo,
                                             DField vo) {
  flow_tile<double, false>(t, st, a, i0, j0, uo, vo);
}

// u_in / v_in to u_out / v_out (other buffers); density as k_flow.  225 -> 83 us at
// 1000 x 750 (FP64), 183 -> 109 us at 2048^2 (mixed).
template <typename R>
__global__ void __launch_bounds__(kFlX* kFlY) k_flow_visc(const double* __restrict__ phi_a, const double* __restrict__ u_in,
                                                          const double* __restrict__ v_in, double* __restrict__ u_out,
                                                          double* __restrict__ v_out, double* __restrict__ dens_a, const FlowArgs a) {
  constexpr int NT = kFlX * kFlY, W = kFlX + 2;
  constexpr bool MIXED = sizeof(R) == 4;
  pdl_enter();
  __shared__ FlowTile<R> t;
  __shared__ FlowStep<R> st;
  const int ni = a.ni, nj = a.nj, tid = threadIdx.x;
  const int i0 = (int)blockIdx.x * kFlX, j0 = (a.row0 + (int)blockIdx.y) * kFlY;
  const DField phi = dfield((double*)phi_a, 2, ni, nj);
  const DField ui = dfield((double*)u_in, 2, ni + 1, nj), vi = dfield((double*)v_in, 2, ni, nj + 1);
  if (tid == 0) {
    FlowArgs b = a;
    if (a.dtp) with_time_step(b, *a.dtp);
    st.gx = b.gx;
    st.gy = b.gy;
    if constexpr (MIXED) {
      st.dt = b.dt_f;
      st.c0 = b.coef0_f;
      st.c1 = b.coef1_f;
    } else {
      st.dt = b.dt;
      st.c0x2 = 2.0 * b.coef0 * a.odx, st.c1x2 = 2.0 * b.coef1 * a.odx;
      st.c0y2 = 2.0 * b.coef0 * a.ody, st.c1y2 = 2.0 * b.coef1 * a.ody;
      st.c0x = b.coef0 * a.odx, st.c1x = b.coef1 * a.odx, st.c0y = b.coef0 * a.ody, st.c1y = b.coef1 * a.ody;
      st.ok = a.fast && mid_range<200>(b.dt) && mid_range<200>(b.coef0) && mid_range<200>(b.coef1);
    }
  }
  __syncthreads();
  bool ok = true;
  for (int k = tid; k < (kFlY + 2) * W; k += NT) {
    const int y = k / W, x = k - y * W, i = i0 - 1 + x, j = j0 - 1 + y;
    const double l = __ldg(&GB_AT(phi, i < ni + 2 ? i : ni + 1, j < nj + 2 ? j : nj + 1));
    R p;
    if constexpr (MIXED)
      p = narrow(l);
    else
      p = l;
    t.p[y][x] = p;
    t.mu[y][x] = visc_mu(p, a);
    // Off the grids T is zero: FP64 tiles hold T, FP32 tiles the faces before gravity.
    double u = MIXED && a.grav ? negd(st.gx) : 0.0, v = MIXED && a.grav ? negd(st.gy) : 0.0;
    if (i >= 0 && i <= ni && j >= 0 && j < nj) {
      u = GB_AT(ui, i, j);
      if (!MIXED && a.grav) u = u + st.gx;
    }
    if (i >= 0 && i < ni && j >= 0 && j <= nj) {
      v = GB_AT(vi, i, j);
      if (!MIXED && a.grav) v = v + st.gy;
    }
    t.u[y][x] = u;
    t.v[y][x] = v;
    if (!MIXED) ok = ok && mid_range<200>(u) && mid_range<200>(v) && mid_range<200>(l);
    if (dens_a && x >= 1 && x <= kFlX && y >= 1 && y <= kFlY && i < ni && j < nj) put_density(dens_a, a, i, j, l);
  }
  const bool fast = __syncthreads_and(MIXED || (ok && st.ok));
  const DField uo = dfield(u_out, 2, ni + 1, nj), vo = dfield(v_out, 2, ni, nj + 1);
  if constexpr (MIXED) {
    flow_tile<R, true>(t, st, a, i0, j0, uo, vo);
  } else {
    if (fast)
      flow_tile<R, true>(t, st, a, i0, j0, uo, vo);
    else
      flow_tile_plain(t, st, a, i0, j0, uo, vo);
  }
}

// Velocity TVD-RK3 blend on every MAC face: w = c0 * keep + c1 * w.
__global__ void k_face_blend(const double* __restrict__ ku_a, double* __restrict__ u_a, const double* __restrict__ kv_a,
                             double* __restrict__ v_a, int ni, int nj, double c0, double c1) {
  const DField ku = dfield((double*)ku_a, 2, ni + 1, nj), u = dfield(u_a, 2, ni + 1, nj);
  const DField kv = dfield((double*)kv_a, 2, ni, nj + 1), v = dfield(v_a, 2, ni, nj + 1);
  GB_FOR_IJ(i, j, ni + 1, nj + 1) {
    if (j < nj) GB_AT(u, i, j) = mul_wide(GB_AT(ku, i, j), c0) + c1 * GB_AT(u, i, j);
    if (i < ni) GB_AT(v, i, j) = mul_wide(GB_AT(kv, i, j), c0) + c1 * GB_AT(v, i, j);
  }
}

// Largest |u|, |v| over the MAC grids and |kappa| over the nodes (CFLOneTimeStep's loops).
__global__ void k_cfl_max(const double* __restrict__ u_a, const double* __restrict__ v_a, const double* __restrict__ kappa,
                          int ni, int nj, Scalars* sc) {
  const DField u = dfield((double*)u_a, 2, ni + 1, nj), v = dfield((double*)v_a, 2, ni, nj + 1);
  unsigned long long mu = 0, mv = 0, mk = 0;
  GB_FOR_IJ(i, j, ni + 1, nj + 1) {
    if (j < nj) mu = abs_max_bits(GB_AT(u, i, j), mu);
    if (i < ni) mv = abs_max_bits(GB_AT(v, i, j), mv);
    if (i < ni && j < nj) mk = abs_max_bits(kappa[i + (size_t)j * ni], mk);
  }
  block_max_bits(mu, &sc->cfl_bits[0]);
  block_max_bits(mv, &sc->cfl_bits[1]);
  block_max_bits(mk, &sc->cfl_bits[2]);
}

struct CflArgs {
  double xs_odx, ys_ody;          // 1/dx of the x-face grid, 1/dy of the y-face grid
  double ody, odx2, ody2, dx, dy; // base grid
  double water_visc, air_visc, water_rho, air_rho, sigma, cfl_number;
};

// The rest of CFLOneTimeStep for air/water (EULERIAN_FLUID_SOLVER_2D.h:3562-3637),
// in the reference's order; one thread.
__global__ void k_cfl_final(CflArgs a, Scalars* sc) {
  const double u_max = __longlong_as_double((long long)sc->cfl_bits[0]);
  const double v_max = __longlong_as_double((long long)sc->cfl_bits[1]);
  const double k_max = __longlong_as_double((long long)sc->cfl_bits[2]);
  const double c_f = (u_max * a.xs_odx + v_max * a.ys_ody);
  const double g_f = sqrt(9.8 * a.ody);  // the constant 9.8, as the reference writes it
  const double rw = a.water_visc / a.water_rho, ra = a.air_visc / a.air_rho;
  const double v_f = (rw < ra ? ra : rw) * (2 * a.odx2 + 2 * a.ody2);
  const double rmin = a.water_rho > a.air_rho ? a.air_rho : a.water_rho;
  const double hmin = a.dy < a.dx ? a.dy : a.dx;
  const double s_f = sqrt(a.sigma * k_max / (rmin * (hmin * hmin)));
  const double CFL = 0.5 * (c_f + v_f + sqrt((c_f + v_f) * (c_f + v_f) + 4 * (g_f * g_f) + 4 * (s_f * s_f)));
  double dt = a.cfl_number / CFL;
  if (CFL == 0) dt = 0;
  sc->cfl[0] = dt;
  sc->cfl[1] = c_f;
  sc->cfl[2] = g_f;
  sc->cfl[3] = v_f;
  sc->cfl[4] = s_f;
}

// The frame's time step: DetermineTimeStep keeps the previous step when the CFL rate is
// zero (SIMULATION_WORLD.h:1201-1204), then the frame's CFL factor.
__global__ void k_frame_dt(Scalars* sc, double cfl) {
  double d = sc->cfl[0];
  if (d == 0) d = sc->dt_frame;
  sc->dt_frame = d * cfl;
}

}  // namespace

void launch_frame_dt(cudaStream_t s, gb2d_ctx* c, double cfl) {
  k_frame_dt<<<1, 1, 0, s>>>(c->sc, cfl);
  GB_LAUNCHED(1);
}

void launch_cfl(cudaStream_t s, gb2d_ctx* c) {
  const int ni = c->grid.ni, nj = c->grid.nj;
  cudaMemsetAsync(c->sc->cfl_bits, 0, sizeof(c->sc->cfl_bits), s);
  k_cfl_max<<<grid_ij(ni + 1, nj + 1), kThreads, 0, s>>>(c->u, c->v, c->kappa, ni, nj, c->sc);
  CflArgs a;
  a.xs_odx = c->xs.odx;
  a.ys_ody = c->ys.ody;
  a.ody = c->base.ody;
  a.odx2 = c->base.odx2;
  a.ody2 = c->base.ody2;
  a.dx = c->base.dx;
  a.dy = c->base.dy;
  a.water_visc = c->flow.water_viscosity;
  a.air_visc = c->flow.air_viscosity;
  a.water_rho = c->prm.water_density;
  a.air_rho = c->prm.air_density;
  a.sigma = c->prm.surface_tension;
  a.cfl_number = c->flow.cfl_number;
  k_cfl_final<<<1, 1, 0, s>>>(a, c->sc);
  GB_LAUNCHED(2);
}

void launch_flow(cudaStream_t s, gb2d_ctx* c, double dt, int grav, int visc, int bc, double* density) {
  const int ni = c->grid.ni, nj = c->grid.nj;
  FlowArgs a;
  a.ni = ni;
  a.nj = nj;
  a.grav = grav;
  a.bc = bc;
  a.g_x = c->flow.gravity_x;
  a.g_y = c->flow.gravity_y;
  a.odx = c->base.odx;
  a.ody = c->base.ody;
  a.eps = 1.5 * c->base.dx;
  a.oe = 1.0 / a.eps;
  a.rho = make_smear(c->prm.air_density, c->prm.water_density);
  a.mu = make_smear(c->flow.air_viscosity, c->flow.water_viscosity);
  a.inv_rho0 = 1 / a.rho.at0;
  a.inv_rho1 = 1 / a.rho.at1;
  a.dtp = c->dt_dev;
  with_time_step(a, dt);
  a.air = c->prm.air_density;
  a.water = c->prm.water_density;
  a.odx_f = (float)a.odx;
  a.ody_f = (float)a.ody;
  a.eps_f = (float)a.eps;
  a.oe_f = (float)a.oe;
  a.rho_f = SmearF{(float)a.rho.lo, (float)a.rho.d, (float)a.rho.at0, (float)a.rho.at1};
  a.mu_f = SmearF{(float)a.mu.lo, (float)a.mu.d, (float)a.mu.at0, (float)a.mu.at1};
  const double* phi = c->phi_buf[c->phi_cur];
  const bool mixed = c->prm.advection_precision == GB2D_PRECISION_MIXED;
  if (visc) {
    auto mid = [](double x) { return x == 0 || (std::fabs(x) >= 0x1p-60 && std::fabs(x) <= 0x1p60); };
    a.fast = mid(a.mu.lo) && mid(a.mu.at0) && mid(a.mu.at1) && mid(a.rho.at0) && mid(a.rho.at1) && mid(a.odx) && mid(a.ody) && a.odx > 0 &&
             a.ody > 0 && mid(c->prm.water_density) && mid(c->prm.air_density);
    const double *u = c->u, *v = c->v;
    for_tile_rows((nj + kFlY) / kFlY, [&](int first, unsigned n) {  // covers ni + 1 and nj + 1 faces
      a.row0 = first;
      const dim3 grd((ni + kFlX) / kFlX, n);
      if (mixed)
        pdl_launch(s, grd, kFlX * kFlY, 0, k_flow_visc<float>, phi, u, v, c->u_alt, c->v_alt, density, a);
      else
        pdl_launch(s, grd, kFlX * kFlY, 0, k_flow_visc<double>, phi, u, v, c->u_alt, c->v_alt, density, a);
      GB_LAUNCHED(1);
    });
    double* t = c->u;
    c->u = c->u_alt;
    c->u_alt = t;
    t = c->v;
    c->v = c->v_alt;
    c->v_alt = t;
  } else {
    a.fast = a.row0 = 0;
    pdl_launch(s, grid_ij(ni + 1, nj + 1), kThreads, 0, k_flow, phi, c->u, c->v, density, a);
    GB_LAUNCHED(1);
  }
}

void launch_face_blend(cudaStream_t s, gb2d_ctx* c, double c0, double c1) {
  const int ni = c->grid.ni, nj = c->grid.nj;
  k_face_blend<<<grid_ij(ni + 1, nj + 1), kThreads, 0, s>>>(c->u_keep, c->u, c->v_keep, c->v, ni, nj, c0, c1);
  GB_LAUNCHED(1);
}

}  // namespace gb2d
