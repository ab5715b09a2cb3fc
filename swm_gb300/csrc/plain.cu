// plain.cu -- FP64 kernels of the drop-in path: the reference's formulas in
// its evaluation order, every product and sum rounded exactly as the FP64 CPU
// restatement rounds it (this translation unit is compiled with -fmad=false).
// Fields are unpadded (Nx, Ny); neighbour indices wrap periodically like the
// reference's cshift index vectors (domain_module.f90:106-115).
//
// The loop nests of a step are grouped by the neighbours they need: what
// depends on the state alone (thickness, vorticity, potential vorticity,
// energy, mass fluxes, wind forcing and the stress of the Laplacian) is one
// kernel at the advance, what needs those of the neighbours (stress
// divergence, tendencies, update) one kernel at the step; biharmonic mixing
// adds two.  Small basins are bound by launches: 14 kernels a step took 17.2
// us on a 257 x 129 linear basin, 9.9 us now.  Large ones are bound by the FP64
// pipe (19 cycles per warp instruction and SM), so sums weighted with powers
// of two are scaled once (exact away from underflow, which is tested), and
// divisors that stay fixed take two operations (divide.cuh): 116 -> 91 us a
// step on 601 x 401 points with quadratic friction.
#include "ctx.h"
#include "divide.cuh"

namespace swm {

#define IDX(i, j) ((size_t)(i) + (size_t)d.nx * (size_t)(j))

__device__ __forceinline__ int ip1(int i, int n) { return i + 1 == n ? 0 : i + 1; }
__device__ __forceinline__ int im1(int i, int n) { return i == 0 ? n - 1 : i - 1; }

// 1 / max(count, 1) for a count of ocean points 0..4: the reference's
// division, taken from its correctly rounded values (1/3 is the constant the
// division by 3 rounds to)
__device__ __forceinline__ double inv_count(int n) { return n >= 4 ? .25 : (n == 3 ? 1. / 3. : (n == 2 ? .5 : 1.)); }

// mask-normalised interpolation weights (calc_lib.f90:253-265, 320-335):
// the mask (0 or 1) times the weight is the weight or +0, as the product
// rounds, taken by a select
__device__ __forceinline__ double mw(int8_t m, double w) { return m ? w : 0.; }
__device__ __forceinline__ double ip2_noland(const double *v, const int8_t *m, size_t k1, size_t k2) {
  double w = inv_count(m[k1] + m[k2]);
  return mw(m[k1], w) * v[k1] + mw(m[k2], w) * v[k2];
}
__device__ __forceinline__ double ip2(const double *v, size_t k1, size_t k2) { return .5 * v[k1] + .5 * v[k2]; }
__device__ __forceinline__ double ip4(const double *v, size_t k1, size_t k2, size_t k3, size_t k4) {
  return .25 * v[k1] + .25 * v[k2] + .25 * v[k3] + .25 * v[k4];
}

// x is of a magnitude in [2^-900, 2^977]: a sum or product this large, scaled
// by a power of two, is the sum or product of its scaled operands, rounding
// included (what an operand loses to underflow when it is scaled first is
// 2^-1075, far below half an ulp of the result)
__device__ __forceinline__ bool scalable(double x) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  return e - 123u <= 1877u;
}
__device__ __forceinline__ bool is_one(double a) { return __double_as_longlong(a) == 0x3ff0000000000000ll; }
__device__ __forceinline__ bool zero2(double a, double b) { return ((__double_as_longlong(a) | __double_as_longlong(b)) << 1) == 0; }

// the mask-weighted means of four and of two values in hand, 0 where the point is land
__device__ __forceinline__ double mean4_noland(double a, double b, double c, double d, int n, int na, int nb, int nc,
                                               int nd) {
  const double s = ((a + b) + c) + d, w = inv_count(n);
  if (n != 3 && scalable(s)) return w * s;
  return mw(na, w) * a + mw(nb, w) * b + mw(nc, w) * c + mw(nd, w) * d;
}
__device__ __forceinline__ double mean2_noland(double a, double b, int n, int na, int nb) {
  const double s = a + b, w = inv_count(n);
  if (scalable(s)) return w * s;
  return mw(na, w) * a + mw(nb, w) * b;
}
// ip2(p) * ip4(m), p1 + p2 and the m in the reference's order
__device__ __forceinline__ double mean2_mean4(double p1, double p2, double a, double b, double c, double d) {
  const double s2 = p1 + p2, s4 = ((a + b) + c) + d, q = s2 * s4;
  if (scalable(s2) && scalable(s4) && scalable(q)) return .125 * q;
  return (.5 * p1 + .5 * p2) * (.25 * a + .25 * b + .25 * c + .25 * d);
}
// a < b; the doubles' order as integers decides, and FP64 only confirms
__device__ __forceinline__ bool less(double a, double b) {
  long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  x ^= (x >> 63) & 0x7fffffffffffffffll;
  y ^= (y >> 63) & 0x7fffffffffffffffll;
  return x < y && a < b;
}
// max(x, 2^-52): FP64 decides only where the high word does not
__device__ __forceinline__ double at_least_eps(double x) {
  const int h = __double2hiint(x);
  return h >= 0x3cc00000 && h < 0x7ff00000 ? x : fmax(x, 2.220446049250313e-16);
}

#define KERNEL_PROLOGUE                               \
  int i = blockIdx.x * blockDim.x + threadIdx.x;      \
  int j = blockIdx.y * blockDim.y + threadIdx.y;      \
  if (i >= d.nx || j >= d.ny) return;                \
  size_t k = IDX(i, j);

// The plain path's fixed divisors per row (plain_prepare): A cos_eta
// (continuity), A cos_u dLambda (zonal pressure gradient), cos_H (vorticity),
// and the vorticity's factors bc / (A cos_H dLambda) for bc = 1 and bc = lbc.
// Quotients by them are the division operator's, bit for bit (divide.cuh).
struct PlainRow {
  FixedDiv e, u, h;
  double z1, zl;
};

__global__ void k_plain_rows(Dev d, PlainRow *rows) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= d.ny) return;
  PlainRow &P = rows[j];
  P.e = fixed_div(d.A * d.cosl[GE][j]);
  P.u = fixed_div(d.A * d.cosl[GU][j] * d.dLambda);
  P.h = fixed_div(d.cosl[GH][j]);
  P.z1 = 1. / (d.A * d.cosl[GH][j] * d.dLambda);
  P.zl = d.lbc / (d.A * d.cosl[GH][j] * d.dLambda);
}

// divisors of the whole grid: dLambda, dTheta, A dTheta, the damping factor of
// u, v, eta where it is the same everywhere, and in the linear modes the
// thickness at the u and v points where that is (its value at ku, kv)
struct PlainConst {
  FixedDiv dL, dT, AdT, impl[3], D[2];
};
__global__ void k_plain_const(Dev d, PlainConst *k, size_t ku, size_t kv) {
  k->D[0] = fixed_div(d.Du[ku]);
  k->D[1] = fixed_div(d.Dv[kv]);
  k->dL = fixed_div(d.dLambda);
  k->dT = fixed_div(d.dTheta);
  k->AdT = fixed_div(d.A * d.dTheta);
  k->impl[0] = fixed_div(d.impl_u[0]);
  k->impl[1] = fixed_div(d.impl_v[0]);
  k->impl[2] = fixed_div(d.impl_e[0]);
}

// the damping factors impl of u, v, eta: 1 / impl per point, and what flags
// says of field f: bit f, a factor outside div_fast's range; bit 3 + f,
// factors that differ
__global__ void k_plain_impl(Dev d, double *r0, double *r1, double *r2, unsigned *flags) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (size_t)d.nx * d.ny) return;
  const double *impl[3] = {d.impl_u, d.impl_v, d.impl_e};
  double *r[3] = {r0, r1, r2};
  unsigned m = 0;
  for (int f = 0; f < 3; f++) {
    const double x = impl[f][k];
    r[f][k] = 1. / x;
    if (!div_rn_range(x)) m |= 1u << f;
    if (__double_as_longlong(x) != __double_as_longlong(impl[f][0])) m |= 8u << f;
  }
  if (m) atomicOr(flags, m);
}

// the thickness at the ocean u and v points in the linear modes, where it does
// not change: 1 / D per point, and as above bits 6, 7 (out of range) and 8, 9
// (not the value at ku, kv)
__global__ void k_plain_depth(Dev d, double *r0, double *r1, size_t ku, size_t kv, unsigned *flags) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (size_t)d.nx * d.ny) return;
  const double *D[2] = {d.Du, d.Dv};
  const int8_t *o[2] = {d.ocean[GU], d.ocean[GV]};
  double *r[2] = {r0, r1};
  const size_t at[2] = {ku, kv};
  unsigned m = 0;
  for (int f = 0; f < 2; f++) {
    const double x = D[f][k];
    r[f][k] = 1. / x;
    if (o[f][k] != 1) continue;
    if (!div_rn_range(x)) m |= 64u << f;
    if (__double_as_longlong(x) != __double_as_longlong(D[f][at[f]])) m |= 256u << f;
  }
  if (m) atomicOr(flags, m);
}

// Lateral-mixing coefficients of _init_p_coefficients (:132-145) and
// lat_mixing_u/v (:84-97).  They depend on the row (cos and tan of the
// latitude) and on two mask bits of the point, so they are formed once per
// row and mask case by the same expressions, in the same order, and the
// step kernels look them up: the values are bit for bit those formed per
// point (this file is compiled without FMA contraction).
constexpr int LATP_N = 14;  // pll: c0, c1[3], c2[3]; plt: c0, c1[3], c2[3]
constexpr int LATUV_N = 10; // lu: c0, c1[2], c2[2]; lv: c0, c1[2], c2[2]

// case of a coefficient that carries mask bit a (with neighbour bit b) in
// the term a * tan / max(a + b, 1): 0 when a = 0, 1 + b otherwise
__device__ __forceinline__ int latp_case(int a, int b) { return a ? 1 + b : 0; }

__global__ void k_latmix_tab_p(Dev d, double Ah, double *tab) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= d.ny) return;
  const double A = d.A, bc = 1.;
  double *T = tab + (size_t)LATP_N * j;
  for (int q = 0; q < 3; q++) {  // mask cases (own bit, other bit): (0, 0), (1, 0), (1, 1)
    const int8_t a = q > 0, b = q > 1;
    {  // pll: c1 carries ovp (a), c2 carries ov (a)
      const int o = a + b;
      const double ot = (double)(o > 1 ? o : 1), tn = d.tanl[GE][j];
      T[1 + q] = Ah / A * (bc / d.dTheta + a * tn / ot);
      T[4 + q] = Ah / A * (-bc / d.dTheta + a * tn / ot);
    }
    {  // plt: c1 carries ou (a), c2 carries oum (a)
      const int o = a + b;
      const double ot = (double)(o > 1 ? o : 1), tn = d.tanl[GH][j];
      T[8 + q] = -Ah / A * (bc / d.dTheta + a * tn / ot);
      T[11 + q] = -Ah / A * (-bc / d.dTheta + a * tn / ot);
    }
  }
  T[0] = -Ah * bc / d.dLambda / A / d.cosl[GE][j];
  T[7] = -Ah * bc / d.dLambda / A / d.cosl[GH][j];
}

__global__ void k_latmix_tab_uv(Dev d, double *tab) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= d.ny) return;
  const double A = d.A, bc = 1.;
  double *T = tab + (size_t)LATUV_N * j;
  for (int q = 0; q < 2; q++) {  // ot = 1, 2
    const double ot = (double)(q + 1);
    const double tu = d.tanl[GU][j], tv = d.tanl[GV][j];
    T[1 + q] = -(bc / A / d.dTheta - 2. * tu / A / ot);
    T[3 + q] = -(-bc / A / d.dTheta - 2. * tu / A / ot);
    T[6 + q] = -(-bc / A / d.dTheta + 2. * tv / A / ot);
    T[8 + q] = -(bc / A / d.dTheta + 2. * tv / A / ot);
  }
  T[0] = -bc / A / d.cosl[GU][j] / d.dLambda;
  T[5] = -bc / A / d.cosl[GV][j] / d.dLambda;
}

// SWM_LateralMixing_compute_p (swm_lateralmixing_module.f90:215-240) at one
// point, without the thickness; T: the row's coefficients from the table of
// this Ah
__device__ __forceinline__ double stress_eta(const Dev &d, const double *T, const double *u, const double *v, int i,
                                             int j) {
  const size_t k = IDX(i, j), kjp = IDX(i, ip1(j, d.ny));
  const int8_t ov = d.ocean[GV][k], ovp = d.ocean[GV][kjp];
  const double c0 = T[0], c1 = T[1 + latp_case(ovp, ov)], c2 = T[4 + latp_case(ov, ovp)];
  return c0 * (u[IDX(ip1(i, d.nx), j)] - u[k]) + c1 * v[kjp] + c2 * v[k];
}
__device__ __forceinline__ double stress_h(const Dev &d, const double *T, const double *u, const double *v, int i,
                                           int j) {
  const size_t k = IDX(i, j), kjm = IDX(i, im1(j, d.ny));
  const int8_t ou = d.ocean[GU][k], oum = d.ocean[GU][kjm];
  const double c0 = T[7], c1 = T[8 + latp_case(ou, oum)], c2 = T[11 + latp_case(oum, ou)];
  return c0 * (v[k] - v[IDX(im1(i, d.nx), j)]) + c1 * u[k] + c2 * u[kjm];
}
// Dp, Dhp null: unit thickness (the biharmonic operator's first pass; 1 x = x)
__global__ void k_latmix_p(Dev d, const double *__restrict__ tab, const double *u, const double *v,
                           const double *Dp, const double *Dhp, double *pll, double *plt) {
  KERNEL_PROLOGUE
  const double *T = tab + (size_t)LATP_N * j;
  if (d.ocean[GE][k] == 1) {
    const double x = stress_eta(d, T, u, v, i, j);
    pll[k] = Dp ? Dp[k] * x : x;
  }
  if (d.ocean[GH][k] == 1) {
    const double x = stress_h(d, T, u, v, i, j);
    plt[k] = Dhp ? Dhp[k] * x : x;
  }
}

// SWM_LateralMixing_compute_uv (:162-186) with lat_mixing_u/v (:84-97) from
// the table at one point, before the division by the thickness
__device__ __forceinline__ double mix_u(const Dev &d, const double *T, const double *pll, const double *plt, int i,
                                        int j) {
  const size_t k = IDX(i, j), kjp = IDX(i, ip1(j, d.ny));
  const int q = d.ocean[GH][k] + d.ocean[GH][kjp] > 1;
  return T[0] * (pll[k] - pll[IDX(im1(i, d.nx), j)]) + T[1 + q] * plt[kjp] + T[3 + q] * plt[k];
}
__device__ __forceinline__ double mix_v(const Dev &d, const double *T, const double *pll, const double *plt, int i,
                                        int j) {
  const size_t k = IDX(i, j), kjm = IDX(i, im1(j, d.ny));
  const int q = d.ocean[GE][k] + d.ocean[GE][kjm] > 1;
  return T[5] * (plt[IDX(ip1(i, d.nx), j)] - plt[k]) + T[6 + q] * pll[k] + T[8 + q] * pll[kjm];
}
// the biharmonic operator's first pass: the thicknesses are 1, and x / 1 = x
__global__ void k_latmix_uv1(Dev d, const double *__restrict__ tab, const double *pll, const double *plt, double *lu,
                             double *lv) {
  KERNEL_PROLOGUE
  const double *T = tab + (size_t)LATUV_N * j;
  if (d.ocean[GU][k] == 1) lu[k] = mix_u(d, T, pll, plt, i, j);
  if (d.ocean[GV][k] == 1) lv[k] = mix_v(d, T, pll, plt, i, j);
}

// what k_plain_diag forms besides the diagnostics
struct DiagJobs {
  int interp;         // the thicknesses on H, u and v points (and D in FULLY_NONLINEAR)
  int pot;            // the potential vorticity (in the linear modes it does not change)
  int forcing;        // reset the forcing and add the wind streams below
  int nwind;
  int merid[2];       // their component
  const double *wind[2];
  const double *tab;  // stress coefficients, or null
  int unit;           // the stress has unit thickness (biharmonic, first pass)
  double *pll, *plt;
};

// SWM_timestep_advance's diagnostics (swm_nonlinear_timestep_module.f90:150-
// 154) and, in FULLY_NONLINEAR, the wind forcing (SWM_forcing_update): all of
// them from the state of the point and its neighbours, in one pass.
//   computeD (:187-217), computeRelVort -> vorticityFromVelocities2D
//   (calc_lib.f90:663-678), computePotVort (:230-257), computeEdens
//   (:259-310; u2/v2 of the reference evaluated in place), computeMassFluxes
//   (:312-326), SWM_forcing_processWindstress (swm_forcing_module.f90:274-324)
__global__ void __launch_bounds__(256) k_plain_diag(Dev d, DiagJobs w) {
  KERNEL_PROLOGUE
  const bool nl = d.mode == SWM_MODE_NONLINEAR;
  const int im = im1(i, d.nx), jm = im1(j, d.ny);
  const size_t ki = IDX(im, j), kj = IDX(i, jm), kij = IDX(im, jm);
  const int8_t *oE = d.ocean[GE], *oU = d.ocean[GU], *oV = d.ocean[GV];
  const int e0 = oE[k] == 1, ou = oU[k] == 1, ov = oV[k] == 1;
  const bool ocean_h = d.ocean[GH][k] == 1;
  const double u = d.u0[k], v = d.v0[k], eta = d.eta0[k];
  double D = 0., Dh, Du, Dv;
  if (w.interp) {
    const int e1 = oE[kij] == 1, e2 = oE[ki] == 1, e3 = oE[kj] == 1;
    auto wet = [&](size_t a) { return nl ? d.eta0[a] + d.Hg[GE][a] : d.D[a]; };
    D = e0 ? (nl ? eta + d.Hg[GE][k] : d.D[k]) : 0.;
    const double D1 = e1 ? wet(kij) : 0., D2 = e2 ? wet(ki) : 0., D3 = e3 ? wet(kj) : 0.;
    Dh = mean4_noland(D, D1, D2, D3, e0 + e1 + e2 + e3, e0, e1, e2, e3);
    Du = mean2_noland(D, D2, e0 + e2, e0, e2);
    Dv = mean2_noland(D, D3, e0 + e3, e0, e3);
    if (nl && e0) d.D[k] = D;
    d.Dh[k] = Dh;
    d.Du[k] = Du;
    d.Dv[k] = Dv;
  } else {
    D = d.D[k];
    Dh = d.Dh[k];
    Du = d.Du[k];
    Dv = d.Dv[k];
  }
  double zeta = 0.;
  if (nl || d.mode == SWM_MODE_LIN_MEAN) {
    const PlainRow &P = d.prow[j];
    double dvdx = 0., dudy = 0.;
    if (oV[ki] + oV[k] != 0)
      dvdx = (d.pdiv ? (ocean_h ? P.z1 : P.zl)
                     : (ocean_h ? 1. : d.lbc) / (d.A * d.cosl[GH][j] * d.dLambda)) * (v - d.v0[ki]);
    if (oU[k] + oU[kj] != 0) {
      double num = d.cosl[GU][j] * u - d.cosl[GU][jm] * d.u0[kj];
      if (!ocean_h) num = d.lbc * num;  // bc = 1 elsewhere
      dudy = d.pdiv ? div_fixed(num, d.pk->AdT) : num / (d.A * d.dTheta);
    }
    zeta = dvdx - (d.pdiv ? div_fixed(dudy, P.h) : dudy / d.cosl[GH][j]);
    d.zeta[k] = zeta;
  }
  if (d.mode != SWM_MODE_NONE) {
    if (w.pot) {
      const double pD = at_least_eps(Dh), fH = d.f[GH][j];
      d.pot[k] = (nl ? fH + zeta : (d.mode == SWM_MODE_LIN_MEAN ? fH + d.zbs[k] : fH)) / pD;
    }
    if (e0) {
      const size_t ku = IDX(ip1(i, d.nx), j), kv = IDX(i, ip1(j, d.ny));
      double E = d.G * eta;
      if (nl) {
        const double ue = d.u0[ku], vn = d.v0[kv];
        const double a = ue * ue, b = u * u, c = vn * vn, f = v * v, su = a + b, sv = c + f, t = su + sv;
        if ((scalable(su) || zero2(ue, u)) && (scalable(sv) || zero2(vn, v)) && scalable(t)) E = .25 * t + E;
        else E = ((.5 * a + .5 * b) + (.5 * c + .5 * f)) * .5 + E;  // halving: the same rounding as / 2
      } else if (d.mode == SWM_MODE_LIN_MEAN) {
        const double a = .5 * (d.u0[ku] * d.ubs[ku]) + .5 * (u * d.ubs[k]);
        const double b = .5 * (d.v0[kv] * d.vbs[kv]) + .5 * (v * d.vbs[k]);
        E = (a + b) + E;
      }
      d.edens[k] = E;
    }
  }
  if (ou) d.mu[k] = Du * u;
  if (ov) d.mv[k] = Dv * v;
  if (w.forcing) {
    double fx = d.Fxc[k], fy = d.Fyc[k];
    for (int q = 0; q < w.nwind; q++) {  // in the reference's stream order
      const double t = w.wind[q][k];
      const double tau = is_one(d.tau_scale) ? t : d.tau_scale * t;
      if (w.merid[q]) fy = ov ? fy + (tau / (d.RHO0 * Dv)) : fy;
      else fx = ou ? fx + (tau / (d.RHO0 * Du)) : fx;
    }
    d.Fe[k] = d.Fec[k];
    d.Fx[k] = fx;
    d.Fy[k] = fy;
  }
  if (w.tab) {
    const double *T = w.tab + (size_t)LATP_N * j;
    if (e0) {
      const double x = stress_eta(d, T, d.u0, d.v0, i, j);
      w.pll[k] = w.unit ? x : D * x;
    }
    if (ocean_h) {
      const double x = stress_h(d, T, d.u0, d.v0, i, j);
      w.plt[k] = w.unit ? x : Dh * x;
    }
  }
}

struct ABCoef {
  double dtc[3];  // dt * c[t], the product the reference forms first (host, the same rounding)
  int tstep;
};

// SWM_timestep_nonlinear (:349-444): stress divergence, tendencies, and
// integrate_AB_vec (time_integration_module.f90:74-112) for the three
// prognostic fields with the FULLY_NONLINEAR thickness clamp (:176-179).
// tuv: the stress divergence's table, or null without mixing.
__global__ void __launch_bounds__(256) k_plain_step(Dev d, const double *__restrict__ tuv, ABCoef ab) {
  KERNEL_PROLOGUE
  const int ip = ip1(i, d.nx), im = im1(i, d.nx), jp = ip1(j, d.ny), jm = im1(j, d.ny);
  const bool mean = d.mode == SWM_MODE_LIN_MEAN;
  const size_t ke = IDX(ip, j), kw = IDX(im, j), kn = IDX(i, jp), ks = IDX(i, jm);
  const PlainRow &P = d.prow[j];
  const PlainConst &K = *d.pk;
  const double *T = tuv + (size_t)LATUV_N * j;
  const double u = d.u0[k], v = d.v0[k];
  double ge, gu, gv;
  // f: 0 by the thickness at the u point, 1 at the v point
  auto by_depth = [&](double x, int f, const double *D) {
    if (d.depth_how[f] == IMPL_SAME) return div_fixed(x, K.D[f]);
    if (d.depth_how[f] == IMPL_FAST) return div_fast(x, D[k], d.rdepth[f][k]);
    return x / D[k];
  };
  if (d.ocean[GE][k] == 1) {  // continuity
    const double *cV = d.cosl[GV];
    auto dL = [&](double x) { return d.pdiv ? div_fixed(x, K.dL) : x / d.dLambda; };
    auto dT = [&](double x) { return d.pdiv ? div_fixed(x, K.dT) : x / d.dTheta; };
    double t = dL(-(d.mu[ke] - d.mu[k])) - dT(d.mv[kn] * cV[jp] - d.mv[k] * cV[j]);
    if (mean) {
      const int8_t *oE = d.ocean[GE];
      int qi = ip1(j % d.nx, d.nx);  // ip1(j): zonal index taken from j in the reference (:360)
      double ea = ip2_noland(d.eta0, oE, IDX(qi, j), IDX(im1(qi, d.nx), j));
      double eb = ip2_noland(d.eta0, oE, k, kw);
      double ec = ip2_noland(d.eta0, oE, kn, IDX(i, im1(jp, d.ny)));
      double ed = ip2_noland(d.eta0, oE, k, ks);
      t = t - dL(ea * d.ubs[ke] - eb * d.ubs[k]) - dT(cV[jp] * ec * d.vbs[kn] - cV[j] * ed * d.vbs[k]);
    }
    ge = (d.pdiv ? div_fixed(t, P.e) : t / (d.A * d.cosl[GE][j])) + d.Fe[k];
    d.Ge[2][k] = ge;
  } else {
    ge = d.Ge[2][k];
  }
  if (d.ocean[GU][k] == 1) {  // zonal momentum
    const size_t a3 = IDX(im, jp);
    double g = mean2_mean4(d.pot[kn], d.pot[k], d.mv[kn], d.mv[kw], d.mv[a3], d.mv[k]);
    if (mean) g = g + ip2(d.zeta, kn, k) * ip4(d.vbs, kn, kw, a3, k);
    const double de = d.edens[k] - d.edens[kw];
    g = g - (d.pdiv ? div_fixed(de, P.u) : de / (d.A * d.cosl[GU][j] * d.dLambda));
    if (d.qbf) {
      double vv = ip4(d.v0, kn, kw, a3, k);
      double q = d.gsq_u[k] * sqrt(u * u + (vv * vv)) * u;
      if (d.barotropic) q = q / d.Hg[GU][k];
      g = g - q;
    }
    if (tuv) {
      const double l = by_depth(mix_u(d, T, d.pll, d.plt, i, j), 0, d.Du);
      d.lmu[k] = l;
      g = g + l;
    }
    gu = g + d.Fx[k];
    d.Gu[2][k] = gu;
  } else {
    gu = d.Gu[2][k];
  }
  if (d.ocean[GV][k] == 1) {  // meridional momentum
    const size_t a4 = IDX(ip, jm);
    double g = -mean2_mean4(d.pot[ke], d.pot[k], d.mu[ke], d.mu[ks], d.mu[k], d.mu[a4]);
    if (mean) g = g - ip2(d.zeta, ke, k) * ip4(d.ubs, ke, ks, k, a4);
    const double de = d.edens[k] - d.edens[ks];
    g = g - (d.pdiv ? div_fixed(de, K.AdT) : de / (d.A * d.dTheta));
    if (d.qbf) {
      double uu = ip4(d.u0, ke, ks, k, a4);
      double q = d.gsq_v[k] * sqrt(v * v + (uu * uu)) * v;
      if (d.barotropic) q = q / d.Hg[GV][k];
      g = g - q;
    }
    if (tuv) {
      const double l = by_depth(mix_v(d, T, d.pll, d.plt, i, j), 1, d.Dv);
      d.lmv[k] = l;
      g = g + l;
    }
    gv = g + d.Fy[k];
    d.Gv[2][k] = gv;
  } else {
    gv = d.Gv[2][k];
  }
  auto sum = [&](double x, double *const *G, double g) {
    for (int t = 0; t < ab.tstep; t++) x = x + ab.dtc[t] * (t == 2 ? g : G[t][k]);
    return x;
  };
  // f: field 0 u, 1 v, 2 eta; x / 1 = x
  auto damp = [&](double x, int f, const double *impl) {
    if (d.impl_how[f] == IMPL_SAME) return is_one(K.impl[f].b) ? x : div_fixed(x, K.impl[f]);
    if (d.impl_how[f] == IMPL_FAST) return div_fast(x, impl[k], d.rimpl[f][k]);
    return x / impl[k];
  };
  double e1 = damp(sum(d.eta0[k], d.Ge, ge), 2, d.impl_e);
  if (d.mode == SWM_MODE_NONLINEAR) {
    const double lim = d.minD - d.Hg[GE][k];
    if (less(e1, lim)) e1 = lim;
  }
  d.eta1[k] = e1;
  d.u1[k] = damp(sum(u, d.Gu, gu), 0, d.impl_u);
  d.v1[k] = damp(sum(v, d.Gv, gv), 1, d.impl_v);
}

// SWM_forcing_update reset (swm_forcing_module.f90:141-149)
__global__ void k_forcing_reset(Dev d) {
  KERNEL_PROLOGUE
  d.Fe[k] = d.Fec[k];
  d.Fx[k] = d.Fxc[k];
  d.Fy[k] = d.Fyc[k];
}

// SWM_forcing_process* for one stream (swm_forcing_module.f90:274-552)
__global__ void k_stream(Dev d, Stream s, double *Fx, double *Fy, double *Fe, double r_iot, double i_iot) {
  KERNEL_PROLOGUE
  const int8_t *oU = d.ocean[GU], *oV = d.ocean[GV], *oE = d.ocean[GE];
  const double *dd = s.d1;
  switch (s.type) {
    case SWM_FRC_WIND: {
      bool z = s.comp == SWM_CMP_ZONAL;
      double *F = z ? Fx : Fy;
      const int8_t *m = z ? oU : oV;
      const double *H = z ? d.Du : d.Dv;
      bool sh = d.barotropic || d.mode == SWM_MODE_NONLINEAR;
      if (m[k] == 1) F[k] = F[k] + (d.tau_scale * dd[k] / (sh ? (d.RHO0 * H[k]) : d.RHO0));
      break;
    }
    case SWM_FRC_OSC: {
      double *F = s.comp == SWM_CMP_ZONAL ? d.Fx : (s.comp == SWM_CMP_MERID ? d.Fy : d.Fe);
      const int8_t *m = s.comp == SWM_CMP_ZONAL ? oU : (s.comp == SWM_CMP_MERID ? oV : oE);
      F[k] = F[k] + (2. * (s.d1[k] * r_iot - s.d2[k] * i_iot)) * m[k];
      break;
    }
    case SWM_FRC_CUSTOM: {
      double *F = s.comp == SWM_CMP_ZONAL ? Fx : (s.comp == SWM_CMP_MERID ? Fy : Fe);
      const int8_t *m = s.comp == SWM_CMP_ZONAL ? oU : (s.comp == SWM_CMP_MERID ? oV : oE);
      if (m[k] == 1) F[k] = F[k] + dd[k];
      break;
    }
    case SWM_FRC_HEAT:
      if (oE[k] == 1) Fe[k] = Fe[k] + dd[k];
      break;
    case SWM_FRC_EMF: {
      double A = d.A;
      const double *He = d.Hg[GE], *Hu = d.Hg[GU], *Hv = d.Hg[GV], *H = d.Hg[GH];
      const double *cu = d.cosl[GU], *cv = d.cosl[GV];
      int nx = d.nx, ny = d.ny;
      auto h2eta = [&](int ii, int jj) {
        return ip4(dd, IDX(ip1(ii, nx), ip1(jj, ny)), IDX(ii, jj), IDX(ii, ip1(jj, ny)), IDX(ip1(ii, nx), jj));
      };
      if (s.comp == SWM_CMP_U2) {
        if (oU[k] != 1) break;
        int im = im1(i, nx);
        Fx[k] = Fx[k] + (-(h2eta(i, j) * He[k] - h2eta(im, j) * He[IDX(im, j)]) / (2 * A * d.dLambda * cu[j] * Hu[k]));
      } else if (s.comp == SWM_CMP_V2) {
        if (oV[k] != 1) break;
        int jm = im1(j, ny);
        Fy[k] = Fy[k] + (-(cu[j] * He[k] * h2eta(i, j) - cu[jm] * He[IDX(i, jm)] * h2eta(i, jm)) /
                         (8 * A * d.dTheta * cv[j] * Hv[k]));
      } else {
        int jp = ip1(j, ny), ip = ip1(i, nx);
        if (oU[k] == 1)
          Fx[k] = Fx[k] + (-(cv[jp] * dd[IDX(i, jp)] * H[IDX(i, jp)] - cv[j] * dd[k] * H[k]) /
                           (2 * A * d.dTheta * cu[j] * Hu[k]));
        if (oV[k] == 1)
          Fy[k] = Fy[k] + (-(dd[IDX(ip, j)] * H[IDX(ip, j)] - dd[k] * H[k]) / (2 * A * d.dLambda * cv[j] * Hv[k]));
      }
      break;
    }
  }
}

__global__ void k_fill(double *p, size_t n, double v) {
  size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) p[k] = v;
}

#undef KERNEL_PROLOGUE

static dim3 blk() { return dim3(32, 8); }
static dim3 grd(const swm_gpu_ctx *c) { return dim3((c->nx + 31) / 32, (c->ny + 7) / 8); }

#define LAUNCH(kern, ...)                                               \
  do {                                                                  \
    kern<<<grd(c), blk(), 0, c->stream>>>(__VA_ARGS__);                 \
    c->launches++;                                                      \
  } while (0)

#define PTRY(x)                          \
  do {                                   \
    int rc_ = (x);                       \
    if (rc_ != SWM_GPU_OK) return rc_;   \
  } while (0)

int plain_fill(swm_gpu_ctx *c, double *p, double value) {
  k_fill<<<(unsigned)((c->n + 255) / 256), 256, 0, c->stream>>>(p, c->n, value);
  c->launches++;
  SWM_CK(cudaGetLastError());
  return SWM_GPU_OK;
}

// the diagnostics alone
int plain_diagnostics(swm_gpu_ctx *c, int64_t itt) {
  const int mode = c->cfg.mode;
  DiagJobs w = {};
  w.interp = mode == SWM_MODE_NONLINEAR || mode == SWM_MODE_NONE || itt == 0;
  w.pot = 1;
  LAUNCH(k_plain_diag, c->dev(), w);
  SWM_CK(cudaGetLastError());
  return SWM_GPU_OK;
}

// Streams in the reference's linked-list order: the head (first namelist
// record) first, then the others newest first (generic_list.f90:87-103
// inserts after the head).
static int plain_streams(swm_gpu_ctx *c, int64_t itt, int constant_part);
static std::vector<int> stream_order(const swm_gpu_ctx *c) {
  const int ns = (int)c->streams.size();
  std::vector<int> order;
  if (ns > 0) order.push_back(0);
  for (int s = ns - 1; s >= 1; s--) order.push_back(s);
  return order;
}

// SWM_forcing_update (:135-170) or the constant part of SWM_forcing_init
// (:124-125)
int plain_forcing_update(swm_gpu_ctx *c, int64_t itt, int constant_part) {
  Dev d = c->dev();
  if (!constant_part) LAUNCH(k_forcing_reset, d);
  return plain_streams(c, itt, constant_part);
}

// the streams' part of it
static int plain_streams(swm_gpu_ctx *c, int64_t itt, int constant_part) {
  Dev d = c->dev();
  for (int q : stream_order(c)) {
    const Stream &s = c->streams[q];
    bool tdf = !s.is_const;
    if (constant_part == (int)tdf) continue;  // process when isTDF != isConstant
    double *Fx = s.is_const ? d.Fxc : d.Fx, *Fy = s.is_const ? d.Fyc : d.Fy, *Fe = s.is_const ? d.Fec : d.Fe;
    double r = 0., im = 0.;
    if (s.type == SWM_FRC_OSC) {
      r = cos(s.omega * (double)itt * c->cfg.dt);
      im = sin(s.omega * (double)itt * c->cfg.dt);
    }
    LAUNCH(k_stream, d, s, Fx, Fy, Fe, r, im);
  }
  SWM_CK(cudaGetLastError());
  return SWM_GPU_OK;
}

// the coefficient table of k_latmix_p for this Ah (formed on first use)
static int latp_table(swm_gpu_ctx *c, double Ah, const double **out) {
  for (int q = 0; q < 2; q++)
    if (c->latp[q] && c->latp_ah[q] == Ah) {
      *out = c->latp[q];
      return SWM_GPU_OK;
    }
  const int q = c->latp[0] ? 1 : 0;
  SWM_REQUIRE(!c->latp[q], "lateral mixing: more than two mixing coefficients");
  SWM_CK(cudaMalloc((void **)&c->latp[q], (size_t)LATP_N * c->ny * sizeof(double)));
  c->latp_ah[q] = Ah;
  k_latmix_tab_p<<<(c->ny + 127) / 128, 128, 0, c->stream>>>(c->dev(), Ah, c->latp[q]);
  c->launches++;
  SWM_CK(cudaGetLastError());
  *out = c->latp[q];
  return SWM_GPU_OK;
}

static int latuv_table(swm_gpu_ctx *c, const double **out) {
  if (!c->latuv) {
    SWM_CK(cudaMalloc((void **)&c->latuv, (size_t)LATUV_N * c->ny * sizeof(double)));
    k_latmix_tab_uv<<<(c->ny + 127) / 128, 128, 0, c->stream>>>(c->dev(), c->latuv);
    c->launches++;
    SWM_CK(cudaGetLastError());
  }
  *out = c->latuv;
  return SWM_GPU_OK;
}

// the coefficient tables the plain step needs, formed before a stream
// capture records steps (they are allocated on first use)
int plain_prepare(swm_gpu_ctx *c) {
  if (!c->pdiv_ready && !(c->impl[0] && c->impl[1] && c->impl[2])) {
    c->pdiv = false;  // no damping factors yet: the division operator
  } else if (!c->pdiv_ready) {
    const size_t n = c->n;
    if (!c->prow) SWM_CK(cudaMalloc((void **)&c->prow, (size_t)c->ny * sizeof(PlainRow)));
    if (!c->pk) SWM_CK(cudaMalloc((void **)&c->pk, sizeof(PlainConst)));
    for (int q = 0; q < 3; q++)
      if (!c->rimpl[q]) SWM_CK(cudaMalloc((void **)&c->rimpl[q], n * sizeof(double)));
    if (!c->pdiv_flags) SWM_CK(cudaMalloc((void **)&c->pdiv_flags, sizeof(unsigned)));
    SWM_CK(cudaMemsetAsync(c->pdiv_flags, 0, sizeof(unsigned), c->stream));
    const Dev d = c->dev();
    k_plain_rows<<<(c->ny + 127) / 128, 128, 0, c->stream>>>(d, c->prow);
    // the thickness stays in the linear modes: divisions by it as by the others
    const bool linear = c->cfg.mode == SWM_MODE_LIN_REST || c->cfg.mode == SWM_MODE_LIN_MEAN;
    size_t at[2] = {0, 0};
    for (int f = 0; f < 2; f++) {
      const std::vector<int8_t> &o = c->hg.ocean[f ? GV : GU];
      while (at[f] + 1 < n && !o[at[f]]) at[f]++;
    }
    k_plain_const<<<1, 1, 0, c->stream>>>(d, c->pk, at[0], at[1]);
    if (linear) {
      for (int f = 0; f < 2; f++)
        if (!c->rdepth[f]) SWM_CK(cudaMalloc((void **)&c->rdepth[f], n * sizeof(double)));
      k_plain_depth<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(d, c->rdepth[0], c->rdepth[1], at[0], at[1],
                                                                     c->pdiv_flags);
      c->launches++;
    }
    k_plain_impl<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(d, c->rimpl[0], c->rimpl[1], c->rimpl[2],
                                                                  c->pdiv_flags);
    c->launches += 3;
    SWM_CK(cudaGetLastError());
    unsigned fl = 0;
    SWM_CK(cudaMemcpyAsync(&fl, c->pdiv_flags, sizeof(fl), cudaMemcpyDeviceToHost, c->stream));
    SWM_CK(cudaStreamSynchronize(c->stream));
    for (int f = 0; f < 3; f++)
      c->impl_how[f] = !((fl >> (3 + f)) & 1) ? IMPL_SAME : ((fl >> f) & 1 ? IMPL_DIVIDE : IMPL_FAST);
    for (int f = 0; f < 2; f++)
      c->depth_how[f] = !linear || ((fl >> (6 + f)) & 1) ? IMPL_DIVIDE : ((fl >> (8 + f)) & 1 ? IMPL_FAST : IMPL_SAME);
    c->pdiv = true;
    c->pdiv_ready = true;
  }
  if (!c->cfg.lateral_mixing) return SWM_GPU_OK;
  const double *t = nullptr;
  PTRY(latuv_table(c, &t));
  if (c->cfg.mixing_kind == SWM_MIX_BIHARMONIC) {
    PTRY(latp_table(c, 1., &t));
    return latp_table(c, -c->cfg.bih, &t);
  }
  return latp_table(c, c->cfg.Ah, &t);
}

// the stress of the state (biharmonic: of the first pass) as k_plain_diag's
// job, for its own kernel too
static int stress_job(swm_gpu_ctx *c, DiagJobs *w) {
  w->unit = c->cfg.mixing_kind == SWM_MIX_BIHARMONIC;
  w->pll = w->unit ? c->bh[0] : c->pll;
  w->plt = w->unit ? c->bh[1] : c->plt;
  return latp_table(c, w->unit ? 1. : c->cfg.Ah, &w->tab);
}

int plain_stress(swm_gpu_ctx *c) {
  if (!c->cfg.lateral_mixing || c->stress_ready) return SWM_GPU_OK;
  DiagJobs w = {};
  PTRY(stress_job(c, &w));
  const Dev d = c->dev();
  LAUNCH(k_latmix_p, d, w.tab, d.u0, d.v0, w.unit ? nullptr : d.D, w.unit ? nullptr : d.Dh, w.pll, w.plt);
  SWM_CK(cudaGetLastError());
  c->stress_ready = true;
  return SWM_GPU_OK;
}

// the drop-in path's SWM_advance after the rotation: diagnostics, forcing,
// and the next step's stress
int plain_advance(swm_gpu_ctx *c, int64_t itt) {
  PTRY(plain_prepare(c));
  const int mode = c->cfg.mode;
  DiagJobs w = {};
  w.interp = mode == SWM_MODE_NONLINEAR || mode == SWM_MODE_NONE || itt == 0;
  w.forcing = 1;
  w.pot = mode == SWM_MODE_NONLINEAR || itt == 0 || !c->pot_ready;
  // up to two wind streams of FULLY_NONLINEAR go with the diagnostics
  // (their stress is divided by the thickness formed there)
  bool others = false;
  for (int q : stream_order(c)) {
    const Stream &s = c->streams[q];
    if (s.is_const) continue;
    if (mode == SWM_MODE_NONLINEAR && s.type == SWM_FRC_WIND && w.nwind < 2) {
      w.merid[w.nwind] = s.comp != SWM_CMP_ZONAL;
      w.wind[w.nwind++] = s.d1;
    } else {
      others = true;
    }
  }
  if (others) w.nwind = 0;
  if (c->cfg.lateral_mixing) PTRY(stress_job(c, &w));
  LAUNCH(k_plain_diag, c->dev(), w);
  SWM_CK(cudaGetLastError());
  c->stress_ready = c->cfg.lateral_mixing != 0;
  c->pot_ready = true;
  return others ? plain_streams(c, itt, 0) : SWM_GPU_OK;
}

// SWM_timestep_step (swm_nonlinear_timestep_module.f90:164-180)
int plain_step(swm_gpu_ctx *c, int64_t itt) {
  PTRY(plain_prepare(c));
  PTRY(plain_stress(c));
  const Dev d = c->dev();
  const double *tuv = nullptr;
  if (c->cfg.lateral_mixing) {
    PTRY(latuv_table(c, &tuv));
    if (c->cfg.mixing_kind == SWM_MIX_BIHARMONIC) {
      // project extension: Laplacian-type operator with unit thickness and
      // Ah = 1, then the thickness-weighted operator with Ah = -bih
      const double *tp = nullptr;
      PTRY(latp_table(c, -c->cfg.bih, &tp));
      LAUNCH(k_latmix_uv1, d, tuv, c->bh[0], c->bh[1], c->bh[2], c->bh[3]);
      LAUNCH(k_latmix_p, d, tp, c->bh[2], c->bh[3], d.D, d.Dh, d.pll, d.plt);
    }
  }
  ABCoef ab;
  ab.tstep = (int)(itt < 3 ? itt : 3);
  const double chi = c->cfg.ab_chi;
  double tab[4][3] = {{0, 0, 0}, {1., 0, 0}, {-0.5 - chi, 1.5 + chi, 0}, {5. / 12., -16. / 12., 23. / 12.}};
  for (int q = 0; q < 3; q++) ab.dtc[q] = c->cfg.dt * tab[ab.tstep][q];
  LAUNCH(k_plain_step, d, tuv, ab);
  SWM_CK(cudaGetLastError());
  c->stress_ready = false;
  return SWM_GPU_OK;
}

}  // namespace swm
