// sor.cu -- red-black SOR of ElSolv_SOR.f90 on the GPU.
//
// Reference semantics: 5-point masked spherical Laplacian coefficients
// (init_ElSolv_SOR :54-62), colour 1 = i+j even (1-based) then colour 2,
// fixed Chebyshev relaxation schedule from rJacobi = 0.99999178 (binary32
// literal, :175, :206-210), stop on the first iteration whose correction norm
// sqrt(sum res^2) drops below eps (:213-218), max_count = 1000 max(Nx, Ny)
// on a first call and 10 max(Nx, Ny) after it (:166-176).
//
// Layout: the right-hand side, chi and the masks are kept split by colour,
// row by row: cell (i, j) of colour (i + j) % 2 sits at j * W + i / 2 of its
// colour's arrays (W = ceil(Nx / 2)).  The coefficients depend on the row and
// on the masks of the cell's four faces only, so a row keeps its three face
// coefficients and the 16 diagonals its mask cases give, and a cell a byte of
// mask bits: 33 B a point and iteration where one word per coefficient took
// 80.  Each cell's update is the reference's expression in the reference's
// order (this file is compiled without FMA contraction), so chi is bit for
// bit the restatement's when the iteration counts agree; within a colour no
// cell reads another of its own colour (the periodic wrap only pairs land
// cells, which stay fixed).
//
// Division: GB300's FP64 rate is low (an FP64 warp instruction holds an SM's
// pipe for 19 cycles) and a sweep is bound by it, so the division by the
// diagonal is formed from its reciprocal in two words (divide.cuh): 16 FP64
// operations a cell, 19 with the one-word reciprocal.
//
// Control: one cooperative launch runs a batch of iterations, one block per
// SM.  Every block owns an equal, fixed span of cells of each colour (every
// SM gets the same number of FP64 instructions) and publishes, after each
// colour, how far it is; before a colour a block waits only for the blocks
// whose cells are next to its own.  The relaxation schedule depends on the
// iteration number alone.  The stop test is kept off that path: chi
// alternates between two buffers, iteration l's norm is added by one warp of
// every block (all in the same order, so all decide alike) while the others
// run iteration l + 1 into the other buffer, and only iteration l + 2, which
// would overwrite iteration l's chi, waits for the decision.  chi of other
// blocks is read through L2.  Every wait is bounded: a thread that gives up
// sets ctl->failed, which ends the waits of all others.
//
// One iteration, with a launch per colour and one-word reciprocals, and now:
//   201 x 101 points      22.8 us ->   8.3 us  (waits and the FP64 latency chain)
//   1025 x 769            47.0 us ->  32.3 us  (its FP64 instructions take 78 % of that at the pipe's
//                                              rate; the 386 blocks of a colour left a last wave
//                                              half empty)
//   2049 x 2049            186 us ->   140 us  (its FP64 instructions take 95 % of that)
// at 9.75 ns per FP64 warp instruction and SM, measured (19 cycles).  480
// threads of four cells in flight against 992 of one: 15.6 against 17.1 us at
// 513 x 513, the same from 1025 x 769 on.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <string>
#include <vector>
#include "ctx.h"
#include "divide.cuh"

// device control block of a solve
struct SorCtl {
  double relax;      // relaxation factor of the next half-sweep
  double anorm;      // correction norm of the last finished iteration
  double eps;        // stop when the correction norm falls below it
  int l;             // the next iteration (1-based)
  int max_count;
  int done;          // 1: converged (at iteration iters)
  int iters;
  unsigned failed;   // a block gave up at the barrier
};

// one row's coefficients: 1/ax (zonal faces), cos_v / ay at the north and
// south faces, and the diagonal by mask case (bit 0 east, 1 west, 2 north,
// 3 south face open) with its reciprocal
struct SorRow {
  double a, n, s, pad;
  swm::FixedDiv c4[16];
};

struct SorState {
  double *chi = nullptr, *B = nullptr;   // natural layout; chi: calc_lib::chi, kept between
                                         // swm_gpu_nondivergent calls
  double *chi_io = nullptr;              // natural layout: elsolv_sor_gpu_solve's chi
  SorRow *rows = nullptr;
  uint8_t *ms[2] = {};     // mask bits split by colour: 0-3 open faces, 4 ocean (0 on the padding of odd rows)
  double *Bs[2] = {};          // right-hand side split by colour
  double *chis[2][2] = {};     // chi split by colour: [iteration & 1][colour]
  double *partial = nullptr;   // per-block sums of res^2 of the last SOR_PART iterations
  SorCtl *ctl = nullptr;
  unsigned *flags = nullptr;   // per block: half-sweeps of the running batch that it has finished, then
                               // per block: iterations whose sums it has stored
  double *und = nullptr, *vnd = nullptr;  // non-divergent flow
  int W = 0;                   // split row length
  unsigned span = 0;           // cells of a colour per block
  int blocks = 0, threads = 0; // of a batch; the last warp adds the norms
  unsigned parties = 0;        // blocks that wait for one another
  unsigned long long wait_ns = 0;  // a wait that has not ended after this gives up
};

constexpr int SOR_CELL_THREADS = 480;  // most threads of a block that own cells
constexpr int SOR_CELLS = 4;           // cells whose loads a thread has in flight
// kept norms: a block that starts adding iteration l + 3's has decided l + 1,
// for which every block has started l + 2 and so decided l
constexpr int SOR_PART = 4;            // (also the relaxation factors' ring)
constexpr unsigned long long SOR_WAIT_NS = 2000000000ull;  // 2 s

namespace swm {

// init_ElSolv_SOR (:54-62), the coefficients of one row by the reference's
// expressions
__global__ void k_sor_rows(Dev d, SorRow *rows) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, j = t >> 4, q = t & 15;
  if (j >= d.ny) return;
  const int jp = j + 1 == d.ny ? 0 : j + 1;
  const double *cE = d.cosl[GE], *cV = d.cosl[GV];
  const double A = d.A, dL = d.dLambda, dT = d.dTheta;
  const double ax = (A * cE[j] * dL) * (A * cE[j] * dL);
  const double ay = (A * A * cE[j] * (dT * dT));
  const int e = q & 1, w = (q >> 1) & 1, n = (q >> 2) & 1, s = (q >> 3) & 1;
  SorRow &R = rows[j];
  if (q == 0) {
    R.a = 1 / ax;
    R.n = cV[jp] / ay;
    R.s = cV[j] / ay;
  }
  R.c4[q] = fixed_div((-e - w) / ax + (-cV[jp] * n - cV[j] * s) / ay);
}

// natural <-> colour-split layout (join 0: natural -> split, 1: split -> natural)
__global__ void k_sor_split(double *nat, double *s0, double *s1, int nx, int ny, int W, int join) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (size_t)nx * ny) return;
  const int i = (int)(k % nx), j = (int)(k / nx);
  double *sp = ((i + j) & 1) ? s1 : s0;
  const size_t q = (size_t)j * W + (i >> 1);
  if (join) nat[k] = sp[q];
  else sp[q] = nat[k];
}

// set-up: the split mask bits of colour col
__global__ void k_sor_mask(Dev d, uint8_t *__restrict__ ms, int W, int col) {
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (size_t)W * d.ny) return;
  const int j = (int)(q / W), i = 2 * (int)(q % W) + ((col + j) & 1);
  unsigned m = 0;
  if (i < d.nx) {
    const int ip = i + 1 == d.nx ? 0 : i + 1, jp = j + 1 == d.ny ? 0 : j + 1;
    const size_t k = i + (size_t)d.nx * j;
    const int8_t *oU = d.ocean[GU], *oV = d.ocean[GV];
    m = (oU[ip + (size_t)d.nx * j] != 0) | (oU[k] != 0) << 1 | (oV[i + (size_t)d.nx * jp] != 0) << 2 |
        (oV[k] != 0) << 3 | (d.ocean[GE][k] != 0) << 4;
  }
  ms[q] = (uint8_t)m;
}

// Bounded wait: until ready() holds.  False when the wait ran out or another
// thread's did (ctl->failed).
// SLEEP: nanoseconds between looks, for waits that are not urgent.
template <int SLEEP = 0, typename F>
__device__ __forceinline__ bool sor_wait(SorCtl *ctl, unsigned long long limit, F ready) {
  unsigned long long t0 = 0;
  for (unsigned spins = 1;; spins++) {
    if (ready()) return true;
    if (SLEEP) __nanosleep(SLEEP);
    if ((spins & 1023u) == 0) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
      if (t0 == 0) t0 = t;
      if (t - t0 > limit) atomicExch(&ctl->failed, 1u);
      if (*(volatile unsigned *)&ctl->failed) return false;
    }
  }
}

__device__ __forceinline__ unsigned sor_flag(const unsigned *f) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
  return v;
}
// (with the block's writes before the last barrier)
__device__ __forceinline__ void sor_publish(unsigned *f, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(f), "r"(v) : "memory");
}

// Iterations ctl->l .. of the solve, at most niter of them: colour 0 ((i+j)
// even in 0-based indices, the reference's colour 1), then colour 1, until
// the correction norm falls below eps or max_count is reached.  Cooperative
// launch of s.blocks blocks; block b owns cells [b * span, (b + 1) * span) of
// each colour.  FP64-pipe bound.
__global__ void __launch_bounds__(SOR_CELL_THREADS + 32, 1) k_sor_batch(SorState s, int nx, int ny, double rJ,
                                                                        int niter) {
  SorCtl *ctl = s.ctl;
  __shared__ double buf[2][SOR_CELL_THREADS];  // res^2 by thread, of even and odd iterations
  __shared__ double relax[SOR_PART][2];        // factors of the iterations up to decided + 2
  __shared__ volatile int swept;    // the last iteration whose cells are done
  __shared__ volatile int decided;  // the last iteration whose norm is known,
  __shared__ volatile int stop;     // and the one that met the stop test
  __shared__ int go, fail;
  const int l0 = ctl->l, lend = min(l0 + niter - 1, ctl->max_count);
  if (ctl->done || ctl->failed || l0 > lend) return;  // the same in every block: nobody has written yet
  const unsigned W = s.W, ns = W * (unsigned)ny, G = s.parties, blk = blockIdx.x, span = s.span;
  const unsigned q0 = blk * span, q1 = min(q0 + span, ns);
  const unsigned tid = threadIdx.x, T = blockDim.x - 32;  // threads that own cells
  const double eps = ctl->eps;
  double r = ctl->relax;  // the factor of the next half-sweep
  // the schedule of main_ElSolv_SOR (:206-210): after the first colour of the
  // first iteration 1 / (1 - rJ^2 / 2), else 1 / (1 - rJ^2 relax / 4)
  auto schedule = [&](int l) {
    for (int col = 0; col < 2; col++) {
      relax[l % SOR_PART][col] = r;
      r = 1. / (1. - (col == 0 && l == 1 ? .5 * rJ * rJ : .25 * rJ * rJ * r));
    }
  };
  if (tid == T) {
    swept = decided = l0 - 1;
    stop = 0x7fffffff;
    fail = 0;
    schedule(l0);
    schedule(l0 + 1);
  }
  __syncthreads();

  if (tid >= T) {  // the norms and the schedule
    const unsigned lane = tid - T;
    // a total above eps^2 by more than rounding needs no root
    const double far2 = eps * eps * (1. + 1e-12) + 1e-300;
    unsigned *stored = s.flags + G;
    double v = 0.;
    int l = l0;
    bool ok = true, met = false;
    for (; l <= lend && !met; l++) {
      ok = sor_wait(ctl, s.wait_ns, [&]() { return swept >= l; });
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      __threadfence_block();
      // the block's sum, then the blocks', each in a fixed order
      v = 0.;
      for (unsigned k = lane; k < T; k += 32) v += buf[l & 1][k];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      double *part = s.partial + (size_t)(l % SOR_PART) * G;
      if (lane == 0) {
        part[blk] = v;
        sor_publish(stored + blk, (unsigned)(l - l0) + 1u);
        schedule(l + 2);
      }
      __syncwarp();
      for (unsigned b = lane; b < G && ok; b += 32)
        ok = sor_wait<20>(ctl, s.wait_ns, [&]() { return sor_flag(stored + b) >= (unsigned)(l - l0) + 1u; });
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      v = 0.;
      for (unsigned b = lane; b < G; b += 32) v += __ldcg(part + b);
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      met = v < far2 && sqrt(v) < eps;
      if (lane == 0) {
        if (met) stop = l;
        __threadfence_block();
        decided = l;
      }
      __syncwarp();
    }
    if (ok && blk == 0 && lane == 0) {
      ctl->anorm = sqrt(v);
      ctl->relax = relax[l % SOR_PART][0];
      ctl->l = l;
      if (met) {
        ctl->iters = l - 1;
        ctl->done = 1;
      }
    }
    return;
  }

  // blocks whose cells are next to this block's: those of the W + 1 cells
  // before and after the span (rows wrap)
  unsigned first = 0, near = G;  // near blocks, from block `first` on
  if (2 * (W + 1) + 2 * span < ns) {
    first = ((q0 + ns - (W + 1)) % ns) / span;
    near = ((q1 + W) % ns / span + G - first) % G + 1;
  }
  double r2 = 0.;
  unsigned h = 0;  // half-sweeps done
  for (int l = l0; l <= lend; l++) {
    for (int col = 0; col < 2; col++, h++) {
      // the neighbours have finished the half-sweep before this one, and
      // before iteration l overwrites it, iteration l - 2 is known not to be the last
      bool ok = true;
      if (h)
        for (unsigned t = tid; t < near && ok; t += T) {
          const unsigned b = (first + t) % G;
          if (b != blk) ok = sor_wait(ctl, s.wait_ns, [&]() { return sor_flag(s.flags + b) >= h; });
        }
      if (tid == 0 && col == 0) {
        ok = ok && sor_wait(ctl, s.wait_ns, [&]() { return decided >= l - 2; });
        __threadfence_block();
        go = stop > l - 2;
      }
      if (!ok) fail = 1;
      __syncwarp();
      asm volatile("bar.sync 1, %0;" ::"r"(T) : "memory");
      if (fail) return;
      if (col == 0 && !go) return;
      const double rel = relax[l % SOR_PART][col];
      const double *x = s.chis[(l - 1) & 1][col], *Bc = s.Bs[col];
      const double *y = s.chis[(l - 1 + col) & 1][col ^ 1];  // colour 1 reads this iteration's colour 0
      double *xn = s.chis[l & 1][col];
      const uint8_t *ms = s.ms[col];
      for (unsigned qb = q0 + tid; qb < q1; qb += SOR_CELLS * T) {
        unsigned m[SOR_CELLS], jj[SOR_CELLS];
        double xq[SOR_CELLS], b[SOR_CELLS], ve[SOR_CELLS], vw[SOR_CELLS], vn[SOR_CELLS], vs[SOR_CELLS];
#pragma unroll
        for (int u = 0; u < SOR_CELLS; u++) {
          const unsigned q = qb + u * T;
          m[u] = q < q1 ? ms[q] : 0u;
          if (!(m[u] & 16u)) continue;
          const unsigned j = q / W, c = q - j * W, par = (col + j) & 1;
          const int i = 2 * (int)c + (int)par;
          jj[u] = j;
          xq[u] = x[q];
          b[u] = Bc[q];
          if (i > 0 && i + 1 < nx && j > 0 && (int)j + 1 < ny) {
            // the four neighbours are of the other colour
            ve[u] = __ldcg(y + q + par);
            vw[u] = __ldcg(y + q + par - 1);
            vn[u] = __ldcg(y + q + W);
            vs[u] = __ldcg(y + q - W);
          } else {  // the frame: periodic neighbours, of this cell's own colour across an odd wrap
            const int ip = i + 1 == nx ? 0 : i + 1, im = i == 0 ? nx - 1 : i - 1;
            const int jp = (int)j + 1 == ny ? 0 : (int)j + 1, jm = j == 0 ? ny - 1 : (int)j - 1;
            auto at = [&](int a, int bb) {
              const int k = (a + bb) & 1;
              return __ldcg((k == col ? x : y) + (size_t)bb * W + (a >> 1));
            };
            ve[u] = at(ip, (int)j);
            vw[u] = at(im, (int)j);
            vn[u] = at(i, jp);
            vs[u] = at(i, jm);
          }
        }
#pragma unroll
        for (int u = 0; u < SOR_CELLS; u++) {
          if (!(m[u] & 16u)) continue;
          const SorRow &R = s.rows[jj[u]];
          const double ce = m[u] & 1u ? R.a : 0., cw = m[u] & 2u ? R.a : 0.;
          const double cn = m[u] & 4u ? R.n : 0., cs = m[u] & 8u ? R.s : 0.;
          const FixedDiv &D = R.c4[m[u] & 15u];
          const double num = rel * (ce * ve[u] + cw * vw[u] + cn * vn[u] + cs * vs[u] + D.b * xq[u] - b[u]);
          const double res = div_fixed(num, D);
          xn[qb + u * T] = xq[u] - res;
          r2 = r2 + res * res;
        }
      }
      if (col == 1) buf[l & 1][tid] = r2;
      __syncwarp();
      asm volatile("bar.sync 1, %0;" ::"r"(T) : "memory");
      if (tid == 0) {
        sor_publish(s.flags + blk, h + 1);
        if (col == 1) {
          __threadfence_block();
          swept = l;
        }
      }
    }
    r2 = 0.;
  }
}

// computeDivergence (calc_lib.f90:607-622) of (u, v) onto the eta grid:
// pder_zonal(u, u_grid) + pder_meridional(cos_v v, v_grid) / cos_eta, with
// the mask tests of pder_zonal3D / pder_meridional3D (:892-998)
__global__ void k_sor_divergence(Dev d, const double *u, const double *v, double *div) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= d.nx || j >= d.ny) return;
  size_t k = i + (size_t)d.nx * j;
  int ip = i + 1 == d.nx ? 0 : i + 1, jp = j + 1 == d.ny ? 0 : j + 1;
  size_t ki = ip + (size_t)d.nx * j, kj = i + (size_t)d.nx * jp;
  const int8_t *oU = d.ocean[GU], *oV = d.ocean[GV];
  const double bcE = d.ocean[GE][k] == 1 ? 1. : d.lbc;
  const double *cE = d.cosl[GE], *cV = d.cosl[GV];
  double dx = (oU[k] + oU[ki] == 0) ? 0. : bcE / (d.A * cE[j] * d.dLambda) * (u[ki] - u[k]);
  double dy = (oV[kj] + oV[k] == 0) ? 0. : bcE * (cV[jp] * v[kj] - cV[j] * v[k]) / (d.A * d.dTheta);
  div[k] = dx + dy / cE[j];
}

// computeGradient (:638-648) of chi on the eta grid (zonal part onto u,
// meridional onto v) subtracted from (u, v): computeNonDivergentFlowField
// (:548-590), u_nd = u - u_corr, v_nd = v - v_corr
__global__ void k_sor_nondiv(Dev d, const double *chi, const double *u, const double *v, double *u_nd,
                             double *v_nd) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= d.nx || j >= d.ny) return;
  size_t k = i + (size_t)d.nx * j;
  int im = i == 0 ? d.nx - 1 : i - 1, jm = j == 0 ? d.ny - 1 : j - 1;
  size_t ki = im + (size_t)d.nx * j, kj = i + (size_t)d.nx * jm;
  const int8_t *oE = d.ocean[GE];
  const double bcU = d.ocean[GU][k] == 1 ? 1. : d.lbc, bcV = d.ocean[GV][k] == 1 ? 1. : d.lbc;
  double uc = (oE[ki] + oE[k] == 0) ? 0. : bcU / (d.A * d.cosl[GU][j] * d.dLambda) * (chi[k] - chi[ki]);
  double vc = (oE[kj] + oE[k] == 0) ? 0. : bcV * (chi[k] - chi[kj]) / (d.A * d.dTheta);
  u_nd[k] = u[k] - uc;
  v_nd[k] = v[k] - vc;
}

// the pair of k_div_check's sample k: splitmix64 bits; one pair in four
// takes a special significand (all ones, all zeros, or one of them with the
// lowest bits flipped) for a, b or both; one numerator in eight lies
// outside div_rn's range (zeros, subnormal, tiny, huge, infinite, NaN), so
// div_fast's other branches are checked too
__device__ uint64_t mix64(uint64_t z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__device__ double sample_operand(uint64_t r, uint64_t r2, bool special) {
  uint64_t man = r & 0xfffffffffffffull;
  if (special) {
    const uint64_t pat[4] = {0xfffffffffffffull, 0ull, 0xffffffffffff0ull ^ (r2 & 15), r2 & 15};
    man = pat[(r2 >> 8) & 3];
  }
  const uint64_t e = 523 + (r2 >> 16) % 1001;  // binary exponent -500 .. 500
  const uint64_t sign = (r2 >> 40) & 1;
  return __longlong_as_double((long long)((sign << 63) | (e << 52) | man));
}

__global__ void k_div_check(int64_t n, uint64_t seed, unsigned long long *bad) {
  unsigned long long mism = 0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t h = mix64(seed ^ mix64((uint64_t)k));
    const uint64_t r[4] = {mix64(h + 1), mix64(h + 2), mix64(h + 3), mix64(h + 4)};
    const int sp = (int)(h & 15);  // 0, 1, 2: special a, b, both
    double a = sample_operand(r[0], r[1], sp == 0 || sp == 2);
    const double b = sample_operand(r[2], r[3], sp == 1 || sp == 2);
    if (((h >> 4) & 7) == 0) {  // one sample in eight: a numerator outside div_rn's range
      const uint64_t sign = (r[1] >> 41) & 1, man = r[0] & 0xfffffffffffffull;
      const uint64_t lo = 1 + (r[1] >> 16) % 522, hi = 1524 + (r[1] >> 16) % 523;  // exponent fields
      const uint64_t bits[8] = {0, 0, man, lo << 52 | man, hi << 52 | man, 0x7ffull << 52, 0x7ffull << 52,
                                0x7ffull << 52 | 1};  // +-0, subnormal, tiny, huge, inf, inf, NaN
      a = __longlong_as_double((long long)((sign << 63) | bits[(h >> 7) & 7]));
    }
    const double q = __ddiv_rn(a, b), y = __ddiv_rn(1., b), f = div_fast(a, b, y);
    const bool same = __double_as_longlong(f) == __double_as_longlong(q) || (q != q && f != f);
    mism += !same;
    // the two-word reciprocal: this numerator, and the two numerators whose
    // quotients come closest to a midpoint of two doubles
    const FixedDiv D = fixed_div(b);
    double g = div_fixed(a, D);
    mism += !(__double_as_longlong(g) == __double_as_longlong(q) || (q != q && g != g));
    const unsigned long long one = 1ull << 52, B = ((unsigned long long)__double_as_longlong(b) & (one - 1)) | one;
    if (B & 1) {
      unsigned long long x = 1;
      for (int t = 0; t < 54; t++) x = (x & 1) ? (x + B) >> 1 : x >> 1;
      for (int t = 0; t < 2; t++, x = B - x) {
        if (x < one) continue;
        const double w = __longlong_as_double((long long)((1023ull << 52) | (x & (one - 1))));
        mism += __double_as_longlong(div_fixed(w, D)) != __double_as_longlong(__ddiv_rn(w, b));
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) mism += __shfl_down_sync(0xffffffffu, mism, o);
  if ((threadIdx.x & 31) == 0 && mism) atomicAdd(bad, mism);
}

void sor_free(swm_gpu_ctx *c) {
  if (!c->sor) return;
  SorState *s = c->sor;
  for (int col = 0; col < 2; col++) {
    cudaFree(s->Bs[col]);
    cudaFree(s->chis[0][col]);
    cudaFree(s->chis[1][col]);
    cudaFree(s->ms[col]);
  }
  cudaFree(s->rows); cudaFree(s->flags);
  cudaFree(s->chi); cudaFree(s->chi_io); cudaFree(s->B); cudaFree(s->partial); cudaFree(s->ctl);
  cudaFree(s->und); cudaFree(s->vnd);
  delete s;
  c->sor = nullptr;
}

}  // namespace swm

using namespace swm;

extern "C" {

// at most `blocks` blocks with equal spans of cells, of no more threads than
// cells of a colour (and the warp that adds the norms)
static void sor_blocks(SorState *s, size_t ns, int blocks) {
  s->span = (unsigned)std::max<size_t>(32, (ns + blocks - 1) / blocks);
  s->blocks = (int)((ns + s->span - 1) / s->span);
  s->threads = (int)std::min<size_t>(SOR_CELL_THREADS, ((size_t)s->span + 31) / 32 * 32) + 32;
  s->parties = (unsigned)s->blocks;
}

// a whole number from the environment, 0 when unset or not positive
static int sor_env(const char *name) {
  const char *e = getenv(name);
  return e && atoi(e) > 0 ? atoi(e) : 0;
}

int elsolv_sor_gpu_init(swm_gpu_ctx *c) {
  SWM_ON_DEVICE(c ? c->device : -1);
  SWM_REQUIRE(c && c->stage >= 1, "elsolv_sor_gpu_init: call after swm_gpu_domain");
  const size_t n = c->n;
  const int W = (c->nx + 1) / 2;
  const size_t ns = (size_t)W * c->ny;
  SWM_REQUIRE(ns < (1ull << 31), "elsolv_sor_gpu_init: grid too large");
  sor_free(c);
  SorState *s = new SorState();
  c->sor = s;
  s->W = W;
  int sms = 0;
  SWM_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device < 0 ? 0 : c->device));
  // one block per SM, or SWM_GB300_SOR_BLOCKS
  const int want = sor_env("SWM_GB300_SOR_BLOCKS");
  sor_blocks(s, ns, want ? want : sms);
  s->wait_ns = SOR_WAIT_NS;
  SWM_CK(cudaMalloc((void **)&s->rows, (size_t)c->ny * sizeof(SorRow)));
  for (int col = 0; col < 2; col++) {
    SWM_CK(cudaMalloc((void **)&s->Bs[col], ns * 8));
    SWM_CK(cudaMalloc((void **)&s->chis[0][col], ns * 8));
    SWM_CK(cudaMalloc((void **)&s->chis[1][col], ns * 8));
    SWM_CK(cudaMalloc((void **)&s->ms[col], ns));
  }
  SWM_CK(cudaMalloc((void **)&s->chi, n * 8));
  SWM_CK(cudaMalloc((void **)&s->chi_io, n * 8));
  SWM_CK(cudaMalloc((void **)&s->B, n * 8));
  SWM_CK(cudaMalloc((void **)&s->partial, (size_t)SOR_PART * (s->blocks + 1) * 8));
  SWM_CK(cudaMalloc((void **)&s->ctl, sizeof(SorCtl)));
  SWM_CK(cudaMalloc((void **)&s->flags, 2 * (s->blocks + 1) * sizeof(unsigned)));
  SWM_CK(cudaMemsetAsync(s->ctl, 0, sizeof(SorCtl), c->stream));
  SWM_CK(cudaMemsetAsync(s->chi, 0, n * 8, c->stream));  // calc_lib::chi starts at 0
  const Dev d = c->dev();
  k_sor_rows<<<(16 * c->ny + 127) / 128, 128, 0, c->stream>>>(d, s->rows);
  for (int col = 0; col < 2; col++)
    k_sor_mask<<<(unsigned)((ns + 255) / 256), 256, 0, c->stream>>>(d, s->ms[col], W, col);
  c->launches += 3;
  SWM_CK(cudaGetLastError());
  SWM_CK(cudaStreamSynchronize(c->stream));
  return SWM_GPU_OK;
}

}  // extern "C"

// One cooperative launch of niter iterations.  Where fewer blocks fit on the
// GPU at once than there are (a context that is given part of the SMs), the
// launch is refused and half as many blocks take the same cells.
static int sor_batch(swm_gpu_ctx *c, double rJ, int niter) {
  SorState *s = c->sor;
  int nx = c->nx, ny = c->ny;
  void *args[] = {s, &nx, &ny, &rJ, &niter};
  for (;;) {
    SWM_CK(cudaMemsetAsync(s->flags, 0, 2 * s->parties * sizeof(unsigned), c->stream));
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)k_sor_batch, dim3(s->blocks), dim3(s->threads), args,
                                                      0, c->stream);
    if (e != cudaErrorCooperativeLaunchTooLarge || s->blocks == 1) {
      SWM_CK(e);
      c->launches++;
      return SWM_GPU_OK;
    }
    cudaGetLastError();
    sor_blocks(s, (size_t)s->W * c->ny, (s->blocks + 1) / 2);
  }
}

// main_ElSolv_SOR on the device arrays s->B (right-hand side) and chi
// (first guess in, solution out), natural layout; returns
// SWM_GPU_ENOT_CONVERGED after max_count iterations
static int sor_solve_device(swm_gpu_ctx *c, double *chi, double eps, int first_guess, int *iters, double *anorm) {
  SorState *s = c->sor;
  const int mx = c->nx > c->ny ? c->nx : c->ny;
  const int max_count = first_guess ? (int)lround(1000. * mx) : (int)lround(10. * mx);
  const unsigned nb = (unsigned)((c->n + 255) / 256);
  k_sor_split<<<nb, 256, 0, c->stream>>>(s->B, s->Bs[0], s->Bs[1], c->nx, c->ny, s->W, 0);
  for (int b = 0; b < 2; b++)  // both buffers: the sweeps leave land as it is
    k_sor_split<<<nb, 256, 0, c->stream>>>(chi, s->chis[b][0], s->chis[b][1], c->nx, c->ny, s->W, 0);
  c->launches += 3;
  SorCtl ctl = {};
  ctl.relax = 1.;
  ctl.l = 1;
  ctl.max_count = max_count;
  ctl.eps = eps;
  SWM_CK(cudaMemcpyAsync(s->ctl, &ctl, sizeof(SorCtl), cudaMemcpyHostToDevice, c->stream));
  double rJ = (double)(float)9.9999178e-1;  // default-real literal (ElSolv_SOR.f90:175)
  // iterations of a batch: some tens of milliseconds at 4e10 cells a second, or SWM_GB300_SOR_BATCH
  const int want = sor_env("SWM_GB300_SOR_BATCH");
  const int batch = want ? std::min(want, max_count) : (int)std::min(4096., std::max(16., 1e9 / (double)c->n));
  for (int l = 1; l <= max_count; l += batch) {
    const int rc = sor_batch(c, rJ, batch);
    if (rc != SWM_GPU_OK) return rc;
    SWM_CK(cudaMemcpyAsync(&ctl, s->ctl, sizeof(SorCtl), cudaMemcpyDeviceToHost, c->stream));
    SWM_CK(cudaStreamSynchronize(c->stream));
    if (ctl.failed) {
      set_error("elsolv_sor_gpu_solve: a block waited too long for the others");
      return SWM_GPU_EDEVICE;
    }
    if (ctl.done) break;
  }
  const int last = (ctl.done ? ctl.iters : max_count) & 1;  // the buffer of the last iteration
  k_sor_split<<<nb, 256, 0, c->stream>>>(chi, s->chis[last][0], s->chis[last][1], c->nx, c->ny, s->W, 1);
  c->launches++;
  SWM_CK(cudaGetLastError());
  if (anorm) *anorm = ctl.anorm;
  if (ctl.done) {
    if (iters) *iters = ctl.iters;
    return SWM_GPU_OK;
  }
  if (iters) *iters = max_count;
  set_error("elsolv_sor_gpu_solve: not converged after max_count iterations");
  return SWM_GPU_ENOT_CONVERGED;
}

extern "C" {

int elsolv_sor_gpu_solve(swm_gpu_ctx *c, const double *B, double *chi, double eps, int first_guess, int *iters,
                         double *anorm) {
  SWM_ON_DEVICE(c ? c->device : -1);
  SWM_REQUIRE(c && c->sor && B && chi, "elsolv_sor_gpu_solve: call elsolv_sor_gpu_init first");
  SorState *s = c->sor;
  size_t n = c->n;
  SWM_CK(cudaMemcpyAsync(s->B, B, n * 8, cudaMemcpyHostToDevice, c->stream));
  SWM_CK(cudaMemcpyAsync(s->chi_io, chi, n * 8, cudaMemcpyHostToDevice, c->stream));
  int rc = sor_solve_device(c, s->chi_io, eps, first_guess, iters, anorm);
  SWM_CK(cudaMemcpyAsync(chi, s->chi_io, n * 8, cudaMemcpyDeviceToHost, c->stream));
  SWM_CK(cudaStreamSynchronize(c->stream));
  return rc;
}

int swm_gpu_check_sor_wait(swm_gpu_ctx *c, int limit_ms) {
  SWM_ON_DEVICE(c ? c->device : -1);
  SWM_REQUIRE(c && c->sor && limit_ms > 0 && limit_ms <= 1000, "swm_gpu_check_sor_wait: bad arguments");
  SorState *s = c->sor;
  SWM_CK(cudaMemsetAsync(s->chi_io, 0, c->n * 8, c->stream));
  SWM_CK(cudaMemsetAsync(s->B, 0, c->n * 8, c->stream));
  s->parties = (unsigned)s->blocks + 1;  // the last one is no block
  s->wait_ns = 1000000ull * (unsigned)limit_ms;
  const int rc = sor_solve_device(c, s->chi_io, 1e-300, 0, nullptr, nullptr);
  s->parties = (unsigned)s->blocks;
  s->wait_ns = SOR_WAIT_NS;
  return rc;
}

int swm_gpu_check_division(int64_t n, int64_t seed, int64_t *mismatches) {
  SWM_REQUIRE(n >= 0 && mismatches, "swm_gpu_check_division: bad arguments");
  unsigned long long *d = nullptr;
  SWM_CK(cudaMalloc((void **)&d, sizeof(*d)));
  cudaError_t e = cudaMemset(d, 0, sizeof(*d));
  if (e == cudaSuccess) {
    k_div_check<<<4 * 152, 256>>>(n, (uint64_t)seed, d);
    e = cudaGetLastError();
  }
  unsigned long long h = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) {
    set_error(std::string("swm_gpu_check_division: ") + cudaGetErrorString(e));
    return SWM_GPU_ECUDA;
  }
  *mismatches = (int64_t)h;
  return SWM_GPU_OK;
}

// computeNonDivergentFlowField (calc_lib.f90:548-590) of the model's current
// (u, v): divergence, SOR for chi (chi kept on the device between calls as
// the reference keeps calc_lib::chi; first_guess as itt == 1), gradient,
// u_nd = u - grad_lambda chi, v_nd = v - grad_theta chi.  Outputs may be
// NULL.  SOR non-convergence is reported as by elsolv_sor_gpu_solve, with
// the non-divergent flow still formed.
int swm_gpu_nondivergent(swm_gpu_ctx *c, int first_guess, double eps, double *u_nd, double *v_nd, double *chi,
                         int *iters) {
  SWM_ON_DEVICE(c ? c->device : -1);
  SWM_REQUIRE(c && c->stage >= 5 && c->sor, "swm_gpu_nondivergent: call elsolv_sor_gpu_init first");
  SorState *s = c->sor;
  const size_t n = c->n;
  if (!s->und) {
    SWM_CK(cudaMalloc((void **)&s->und, n * 8));
    SWM_CK(cudaMalloc((void **)&s->vnd, n * 8));
  }
  if (c->cfg.path != SWM_PATH_PLAIN_FP64 && c->fused) {
    int rc0 = fused_sync_state(c);
    if (rc0 != SWM_GPU_OK) return rc0;
  }
  Dev d = c->dev();
  dim3 b(32, 8), g((c->nx + 31) / 32, (c->ny + 7) / 8);
  k_sor_divergence<<<g, b, 0, c->stream>>>(d, d.u0, d.v0, s->B);
  c->launches++;
  SWM_CK(cudaGetLastError());
  int rc = sor_solve_device(c, s->chi, eps, first_guess, iters, nullptr);
  if (rc != SWM_GPU_OK && rc != SWM_GPU_ENOT_CONVERGED) return rc;
  k_sor_nondiv<<<g, b, 0, c->stream>>>(d, s->chi, d.u0, d.v0, s->und, s->vnd);
  c->launches++;
  SWM_CK(cudaGetLastError());
  if (u_nd) SWM_CK(cudaMemcpyAsync(u_nd, s->und, n * 8, cudaMemcpyDeviceToHost, c->stream));
  if (v_nd) SWM_CK(cudaMemcpyAsync(v_nd, s->vnd, n * 8, cudaMemcpyDeviceToHost, c->stream));
  if (chi) SWM_CK(cudaMemcpyAsync(chi, s->chi, n * 8, cudaMemcpyDeviceToHost, c->stream));
  SWM_CK(cudaStreamSynchronize(c->stream));
  return rc;
}

}  // extern "C"
