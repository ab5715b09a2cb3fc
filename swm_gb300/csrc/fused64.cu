// fused64.cu -- the FP64 step of the fused path: two kernels (diagnostics and
// stress, then tendencies and update), four with biharmonic mixing.
//
// An FP64 warp instruction holds an SM's pipe for 18 to 19 cycles (8.9 ns), so
// the step is bound by its FP64 operations and not by memory: one operation per
// point of a 1025 x 1025 basin takes 1.9 us, 300 MB of traffic 45 us.  The
// passes therefore form every quantity once per point and hand it on through
// memory, instead of rebuilding it in the halo of a tile: a one-kernel step
// whose tiles of 32 x 8 recompute two halo cells took 615 us there.  Masks are
// selects, metric factors and mask cases per-row tables (of a difference, not
// of its two terms, whose roundings would not cancel), stress and wind are
// added before they are divided by the thickness, and a uniform implicit
// damping factor divides as a fixed divisor (divide.cuh).  131 operations per
// point (biharmonic, counted), three divisions among them.  Multiplying by a
// thickness inverted once from the hardware's seed took 227 us a step, but
// rounds twice.
//
// 1025 x 1025, biharmonic: 615 -> 252 us per step, the FP64 pipe's rate.
//
// Formulas: swm_nonlinear_timestep_module.f90:182-449 (diagnostics and
// tendencies), swm_lateralmixing_module.f90:66-240 (stress), time_integration_
// module.f90:74-112 (Adams-Bashforth), with FMA contraction; results agree
// with the FP64 restatement to rounding.
#include "fused64.h"

namespace swm {

std::vector<double> fused64_rows(const swm_gpu_ctx *c) {
  const HostGrid &g = c->hg;
  const int ny = c->ny;
  const double A = c->cfg.A, dL = g.dLambda, dT = g.dTheta, q1 = 1. / (A * dT);
  const bool bih = c->cfg.mixing_kind == SWM_MIX_BIHARMONIC;
  std::vector<double> rows((size_t)ny * R_NR, 0.);
  for (int j = 0; j < ny; j++) {
    double *r = &rows[(size_t)j * R_NR];
    const int jp = j + 1 == ny ? 0 : j + 1, jm = j == 0 ? ny - 1 : j - 1;
    const double cE = g.cosl[GE][j], cU = g.cosl[GU][j], cV = g.cosl[GV][j], cH = g.cosl[GH][j];
    r[R_FH] = g.f[GH][j] / 8.;
    r[R_ZV] = 1. / (A * cH * dL) / 8.;
    r[R_ZU] = 1. / (A * dT * cH) / 8.;
    r[R_CU] = cU;
    r[R_CUM] = g.cosl[GU][jm];
    r[R_EX] = 1. / (A * cE * dL);
    r[R_EY] = 1. / (A * cE * dT);
    r[R_CV] = cV;
    r[R_CVP] = g.cosl[GV][jp];
    r[R_RU] = 1. / (A * cU * dL);
    for (int pass = 0; pass < 2; pass++) {
      // biharmonic: unit coefficient, then -bih; else the only pass
      const double Ah = bih ? (pass ? -c->cfg.bih : 1.) : c->cfg.Ah;
      double *p = r + pass * R_NP;
      p[R_P0] = -Ah / (dL * A * cE);
      p[R_H0] = -Ah / (dL * A * cH);
      for (int q = 0; q < 3; q++) {
        const double w = (q > 0) / (q > 1 ? 2. : 1.);
        const double tE = g.tanl[GE][j] / A * w, tH = g.tanl[GH][j] / A * w;
        p[R_P1 + q] = Ah * (q1 + tE);
        p[R_P2 + q] = Ah * (-q1 + tE);
        p[R_H1 + q] = -Ah * (q1 + tH);
        p[R_H2 + q] = -Ah * (-q1 + tH);
      }
    }
    r[R_U0] = -1. / (A * cU * dL);
    r[R_V0] = -1. / (A * cV * dL);
    for (int q = 0; q < 2; q++) {
      const double tu = 2. * g.tanl[GU][j] / A / (q + 1), tv = 2. * g.tanl[GV][j] / A / (q + 1);
      r[R_U1 + q] = -(q1 - tu);
      r[R_U2 + q] = q1 + tu;
      r[R_V1 + q] = q1 - tv;
      r[R_V2 + q] = -(q1 + tv);
    }
  }
  return rows;
}

namespace {

// a point and its periodic neighbours
struct At {
  int i, j;
  size_t k, w, e, s, n;  // (i, j), (i-1, j), (i+1, j), (i, j-1), (i, j+1)
  __device__ __forceinline__ At(int i_, int j_, int nx, int ny) : i(i_), j(j_) {
    const size_t r = (size_t)nx * j;
    k = r + i;
    w = i == 0 ? r + nx - 1 : k - 1;
    e = i + 1 == nx ? r : k + 1;
    s = j == 0 ? k + (size_t)nx * (ny - 1) : k - nx;
    n = j + 1 == ny ? (size_t)i : k + nx;
  }
};

__device__ __forceinline__ int mH(unsigned m) { return m & 1; }
__device__ __forceinline__ int mU(unsigned m) { return (m >> 1) & 1; }
__device__ __forceinline__ int mV(unsigned m) { return (m >> 2) & 1; }
__device__ __forceinline__ int mE(unsigned m) { return (m >> 3) & 1; }
__device__ __forceinline__ double inv_count(int n) { return n >= 4 ? .25 : (n == 3 ? 1. / 3. : (n == 2 ? .5 : 1.)); }
// mask case of a stress coefficient with own bit a and other bit b
__device__ __forceinline__ int mcase(int a, int b) { return a ? 1 + b : 0; }

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

// stress of the pair (a, b) at the eta and H points of one cell, per unit
// thickness: T the pass's row factors
__device__ __forceinline__ double stress_eta(const double *T, const At &q, unsigned m, unsigned mn, const double *a,
                                             const double *b) {
  const int ov = mV(m), ovp = mV(mn);
  return T[R_P0] * (a[q.e] - a[q.k]) + T[R_P1 + mcase(ovp, ov)] * b[q.n] + T[R_P2 + mcase(ov, ovp)] * b[q.k];
}
__device__ __forceinline__ double stress_h(const double *T, const At &q, unsigned m, unsigned ms, const double *a,
                                           const double *b) {
  const int ou = mU(m), oum = mU(ms);
  return T[R_H0] * (b[q.k] - b[q.w]) + T[R_H1 + mcase(ou, oum)] * a[q.k] + T[R_H2 + mcase(oum, ou)] * a[q.s];
}
// divergence of the stress at the u and v points
__device__ __forceinline__ double div_u(const double *r, const At &q, unsigned m, unsigned mn, const double *pl,
                                        const double *pt) {
  const int o = mH(m) & mH(mn);
  return r[R_U0] * (pl[q.k] - pl[q.w]) + r[R_U1 + o] * pt[q.n] + r[R_U2 + o] * pt[q.k];
}
__device__ __forceinline__ double div_v(const double *r, const At &q, unsigned m, unsigned ms, const double *pl,
                                        const double *pt) {
  const int o = mE(m) & mE(ms);
  return r[R_V0] * (pt[q.e] - pt[q.k]) + r[R_V1 + o] * pl[q.k] + r[R_V2 + o] * pl[q.s];
}

#define POINT64                                        \
  const int i_ = blockIdx.x * blockDim.x + threadIdx.x; \
  const int j_ = blockIdx.y * blockDim.y + threadIdx.y; \
  if (i_ >= p.nx || j_ >= p.ny) return;                 \
  const At q(i_, j_, p.nx, p.ny);                       \
  const size_t k = q.k;                                 \
  const double *r = p.rows + (size_t)q.j * R_NR;        \
  const unsigned m = p.mc[k];

// mass fluxes, potential vorticity, Bernoulli potential, thicknesses that the
// step divides by and the (first) stress pass
template <int MIX>
__global__ void __launch_bounds__(256) k_f64_diag(P64 p) {
  POINT64
  const size_t ksw = q.i == 0 ? q.s + p.nx - 1 : q.s - 1;
  const unsigned mw = p.mc[q.w], ms = p.mc[q.s], msw = p.mc[ksw], mn = p.mc[q.n];
  const double e = p.e0[k], u = p.u0[k], v = p.v0[k];
  // computeD on the eta points, land left out of the means
  auto wet = [&](size_t a, unsigned mm) {
    const double h = p.He[a];
    return mE(mm) ? (p.nl ? p.e0[a] + h : h) : 0.;
  };
  const double d = wet(k, m), dw = wet(q.w, mw), ds = wet(q.s, ms), dsw = wet(ksw, msw);
  const int a = mE(m), b = mE(mw), c = mE(ms), x = mE(msw);
  const double dwd = d + dw;
  const double Du = dwd * inv_count(a + b), Dv = (d + ds) * inv_count(a + c);
  const double Dh = (dwd + (ds + dsw)) * inv_count(a + b + c + x);
  p.s.mu[k] = mU(m) ? Du * u : 0.;
  p.s.mv[k] = mV(m) ? Dv * v : 0.;
  if (MIX || p.wind_x) p.s.du[k] = Du;
  if (MIX || p.wind_y) p.s.dv[k] = Dv;
  double pot = 0., B = 0.;
  if (p.has_mode) {
    double z = r[R_FH];
    if (p.nl) {
      const double us = p.u0[q.s], vw = p.v0[q.w];
      double dv = r[R_ZV] * (v - vw), du = r[R_ZU] * (r[R_CUM] * us - r[R_CU] * u);
      if (!mH(m)) {
        dv *= p.lbc;
        du *= p.lbc;
      }
      if (mV(m) | mV(mw)) z += dv;
      if (mU(m) | mU(ms)) z += du;
    }
    pot = z / at_least_eps(Dh);
    if (mE(m)) {
      B = p.G * e;
      if (p.nl) {
        const double ue = p.u0[q.e], vn = p.v0[q.n];
        B = .25 * ((ue * ue + u * u) + (vn * vn + v * v)) + B;
      }
    }
  }
  p.s.pot[k] = pot;
  p.s.B[k] = B;
  if (MIX) {
    const double *T = r;
    double pl = 0., pt = 0.;
    if (mE(m)) pl = stress_eta(T, q, m, mn, p.u0, p.v0) * (MIX == 1 ? d : 1.);
    if (mH(m)) pt = stress_h(T, q, m, ms, p.u0, p.v0) * (MIX == 1 ? Dh : 1.);
    p.s.pl[k] = pl;
    p.s.pt[k] = pt;
    if (MIX == 2) p.s.dh[k] = Dh;
  }
}

// biharmonic: divergence of the first pass's stress, unit thickness
__global__ void __launch_bounds__(256) k_f64_bih_uv(P64 p) {
  POINT64
  const unsigned mn = p.mc[q.n], ms = p.mc[q.s];
  p.s.lu[k] = mU(m) ? div_u(r, q, m, mn, p.s.pl, p.s.pt) : 0.;
  p.s.lv[k] = mV(m) ? div_v(r, q, m, ms, p.s.pl, p.s.pt) : 0.;
}

// biharmonic: the second pass's stress, weighted with the thickness
__global__ void __launch_bounds__(256) k_f64_bih_p(P64 p) {
  POINT64
  const unsigned mn = p.mc[q.n], ms = p.mc[q.s];
  const double *T = r + R_NP;
  double pl = 0., pt = 0.;
  if (mE(m)) pl = stress_eta(T, q, m, mn, p.s.lu, p.s.lv) * (p.nl ? p.e0[k] + p.He[k] : p.He[k]);
  if (mH(m)) pt = stress_h(T, q, m, ms, p.s.lu, p.s.lv) * p.s.dh[k];
  p.s.pl[k] = pl;
  p.s.pt[k] = pt;
}

// tendencies, Adams-Bashforth update, implicit damping, thickness clamp
template <int MIX>
__global__ void __launch_bounds__(256) k_f64_step(P64 p) {
  POINT64
  const unsigned mn = p.mc[q.n], ms = p.mc[q.s];
  const size_t knw = q.i == 0 ? q.n + p.nx - 1 : q.n - 1, kse = q.i + 1 == p.nx ? q.s - (p.nx - 1) : q.s + 1;
  const double *mu = p.s.mu, *mv = p.s.mv, *pot = p.s.pot, *B = p.s.B;
  const double e = p.e0[k], u = p.u0[k], v = p.v0[k];
  double ge = 0., gu = 0., gv = 0.;
  if (mE(m)) {
    ge = r[R_EX] * (mu[k] - mu[q.e]) + r[R_EY] * (r[R_CV] * mv[k] - r[R_CVP] * mv[q.n]);
    if (p.has_F) ge += p.Fe[k];
  }
  if (mU(m)) {
    double g = (pot[q.n] + pot[k]) * ((mv[q.n] + mv[q.w]) + (mv[knw] + mv[k])) - r[R_RU] * (B[k] - B[q.w]);
    if (p.qbf) {
      const double vb = .25 * ((p.v0[q.n] + p.v0[q.w]) + (p.v0[knw] + v));
      double f = (p.gsq_uniform ? p.gsq_s[0] : p.gsq[0][k]) * sqrt(u * u + vb * vb) * u;
      if (p.barotropic) f = f / p.Hu[k];
      g -= f;
    }
    if (MIX || p.wind_x) {
      double t = MIX ? div_u(r, q, m, mn, p.s.pl, p.s.pt) : 0.;
      if (p.wind_x) t += p.ts_rho * (p.wind_rows ? p.wx[q.j] : p.wx[k]);
      g += t / p.s.du[k];
    }
    if (p.has_F) g += p.Fx[k];
    gu = g;
  }
  if (mV(m)) {
    double g = -(pot[q.e] + pot[k]) * ((mu[q.e] + mu[q.s]) + (mu[k] + mu[kse])) - p.q1 * (B[k] - B[q.s]);
    if (p.qbf) {
      const double ub = .25 * ((p.u0[q.e] + p.u0[q.s]) + (u + p.u0[kse]));
      double f = (p.gsq_uniform ? p.gsq_s[1] : p.gsq[1][k]) * sqrt(v * v + ub * ub) * v;
      if (p.barotropic) f = f / p.Hv[k];
      g -= f;
    }
    if (MIX || p.wind_y) {
      double t = MIX ? div_v(r, q, m, ms, p.s.pl, p.s.pt) : 0.;
      if (p.wind_y) t += p.ts_rho * (p.wind_rows ? p.wy[q.j] : p.wy[k]);
      g += t / p.s.dv[k];
    }
    if (p.has_F) g += p.Fy[k];
    gv = g;
  }
  p.Ge3[k] = ge;
  p.Gu3[k] = gu;
  p.Gv3[k] = gv;
  // a uniform factor is a fixed divisor: two operations, the division's quotient (x / 1 = x)
  auto next = [&](double x, const double *G1, const double *G2, double g, int f) {
    x += p.ab0 * G1[k] + p.ab1 * G2[k] + p.ab2 * g;
    if (!p.impl_uniform) return x / p.impl[f][k];
    const FixedDiv &d = p.impl_d[f];
    return __double_as_longlong(d.b) == 0x3ff0000000000000ll ? x : div_fixed(x, d);
  };
  double e1 = next(e, p.Ge1, p.Ge2, ge, 2);
  if (p.nl) {
    const double lim = p.minD - p.He[k];
    if (less(e1, lim)) e1 = lim;
  }
  p.e1[k] = e1;
  p.u1[k] = next(u, p.Gu1, p.Gu2, gu, 0);
  p.v1[k] = next(v, p.Gv1, p.Gv2, gv, 1);
}

#undef POINT64

}  // namespace

__global__ void k_f64_divisor(double b, FixedDiv *out) { *out = fixed_div(b); }

int fused64_divisors(swm_gpu_ctx *c, const double *b, int count, FixedDiv *out) {
  FixedDiv *d = nullptr;
  if (cudaMalloc((void **)&d, count * sizeof(FixedDiv)) != cudaSuccess) {
    set_error("fused64: cudaMalloc failed");
    return SWM_GPU_ENOMEM;
  }
  for (int q = 0; q < count; q++) k_f64_divisor<<<1, 1, 0, c->stream>>>(b[q], d + q);
  c->launches += count;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, d, count * sizeof(FixedDiv), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  cudaFree(d);
  SWM_CK(e);
  return SWM_GPU_OK;
}

int fused64_launch(swm_gpu_ctx *c, const P64 &p) {
  const dim3 b(32, 8), g((c->nx + 31) / 32, (c->ny + 7) / 8);
  cudaStream_t st = c->stream;
  if (p.mix == 2) {
    k_f64_diag<2><<<g, b, 0, st>>>(p);
    k_f64_bih_uv<<<g, b, 0, st>>>(p);
    k_f64_bih_p<<<g, b, 0, st>>>(p);
    k_f64_step<2><<<g, b, 0, st>>>(p);
    c->launches += 4;
  } else if (p.mix == 1) {
    k_f64_diag<1><<<g, b, 0, st>>>(p);
    k_f64_step<1><<<g, b, 0, st>>>(p);
    c->launches += 2;
  } else {
    k_f64_diag<0><<<g, b, 0, st>>>(p);
    k_f64_step<0><<<g, b, 0, st>>>(p);
    c->launches += 2;
  }
  SWM_CK(cudaGetLastError());
  return SWM_GPU_OK;
}

}  // namespace swm
