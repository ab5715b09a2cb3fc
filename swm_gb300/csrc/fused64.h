// fused64.h -- parameter block of the FP64 step kernels of the fused path
// (fused64.cu).
#pragma once
#include <vector>
#include "ctx.h"
#include "divide.cuh"

namespace swm {

// per-row factors, formed on the host.  A coefficient that carries mask bits
// is kept for each case: of a stress component, own bit clear, own bit set,
// both set; of a stress divergence, one ocean point or two.
enum {
  R_FH,                           // f / 8 (the potential vorticity is kept divided by 8, the weight
                                  // 1/2 * 1/4 of its product with the mass flux)
  R_ZV, R_ZU,                     // vorticity: 1/(A cosH dL), 1/(A dT cosH), over 8
  R_CU, R_CUM,                    // cosU_j, cosU_{j-1}
  R_EX, R_EY,                     // continuity: 1/(A cosE dL), 1/(A cosE dT)
  R_CV, R_CVP,                    // cosV_j, cosV_{j+1}
  R_RU,                           // 1/(A cosU dL)
  R_P0, R_P1, R_P2 = R_P1 + 3,    // stress at eta points
  R_H0 = R_P2 + 3, R_H1, R_H2 = R_H1 + 3,  // stress at H points
  R_NP = R_H2 + 3 - R_P0,         // one pass's stress factors; the second pass's follow the first's
  R_U0 = R_P0 + 2 * R_NP, R_U1, R_U2 = R_U1 + 2,  // divergence at u points
  R_V0 = R_U2 + 2, R_V1, R_V2 = R_V1 + 2,         // divergence at v points
  R_NR = R_V2 + 2
};
std::vector<double> fused64_rows(const swm_gpu_ctx *c);

// what the passes of a step hand on, one value per point
struct Scratch64 {
  double *mu = nullptr, *mv = nullptr, *pot = nullptr, *B = nullptr;  // mass fluxes, PV / 8, Bernoulli potential
  double *du = nullptr, *dv = nullptr;                     // thickness at u and v points
  double *pl = nullptr, *pt = nullptr;                     // stress
  double *dh = nullptr, *lu = nullptr, *lv = nullptr;      // biharmonic: thickness at H points, first-pass divergence
};

struct P64 {
  int nx, ny, nl, has_mode, mix, qbf, barotropic, has_F, impl_uniform, gsq_uniform, wind_x, wind_y, wind_rows;
  double G, lbc, q1, ts_rho, minD;
  double ab0, ab1, ab2;  // Adams-Bashforth weights times dt
  FixedDiv impl_d[3];  // uniform damping factors
  double gsq_s[2];
  const uint8_t *mc;  // mask code: bit 0 H, 1 u, 2 v, 3 eta
  const double *He, *rows, *Hu, *Hv;
  const double *impl[3], *gsq[2];
  const double *Fx, *Fy, *Fe;
  const double *wx, *wy;
  const double *u0, *v0, *e0;
  double *u1, *v1, *e1;
  const double *Gu1, *Gu2, *Gv1, *Gv2, *Ge1, *Ge2;
  double *Gu3, *Gv3, *Ge3;
  Scratch64 s;
};
// b as fixed divisors
int fused64_divisors(swm_gpu_ctx *c, const double *b, int count, FixedDiv *out);
int fused64_launch(swm_gpu_ctx *c, const P64 &p);

}  // namespace swm
