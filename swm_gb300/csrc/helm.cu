// helm.cu -- red-black SOR for the variable-coefficient Helmholtz problem
// div(H^-1 grad psi) - lambda psi = rhs (extension of ElSolv_SOR.f90, whose
// operator is the masked spherical Laplacian with a fixed Chebyshev
// relaxation schedule and an absolute stopping rule).
//
// Same sweep structure as main_ElSolv_SOR (:176-211): colour 0 then colour 1
// of (i + j), each point relaxed with the new values of the other colour.
// Face coefficients are formed on the fly from 1/H (mean of the two cells);
// land cells and the outer frame hold psi = 0.  Stopping: relative residual
// ||rhs - A psi||_2 / ||rhs||_2, checked every CHECK sweeps in FP64.
//
// Two solvers: FP64 sweeps (bit for bit with the FP64 restatement, this file
// is compiled without FMA contraction and the update's fused multiply-adds
// are explicit in both), and mixed precision: FP32 sweeps on
// the correction equation A e = r, with r = rhs - A psi formed in FP64 and
// psi += e accumulated in FP64 (iterative refinement).  An autotuner picks
// the relaxation factor in a given range from short trial solves and the
// thread-block shape of the sweep kernel from timings.
#include <cmath>
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>
#include "ctx.h"

namespace swm {

constexpr int HELM_CHECK = 16;  // sweeps between residual checks
constexpr int HELM_RED = 1024;  // reduction blocks

// One FP32 SOR point update, shared by the global and the tiled kernels so
// both round alike: explicit fused multiply-adds, the diagonal applied as its
// reciprocal (formed once per cell)
__device__ __forceinline__ float sor32_update(float p, float r, float cxw, float cxe, float cys, float cyn, float rcc,
                                              float w, float e, float s, float n, float omega) {
  const float off = fmaf(cyn, n, fmaf(cys, s, fmaf(cxe, e, cxw * w)));
  const float gs = (r - off) * rcc;
  return fmaf(omega, gs - p, p);
}

__device__ __forceinline__ float face32(float a, float b, float rd2) { return (0.5f * (a + b)) * rd2; }


// FP64 coefficients formed once: west and south face coefficients, the
// diagonal and its reciprocal (the sweeps would otherwise be bound by the
// FP64 pipe, which forms them and divides at every point of every sweep)
__global__ void k_h_coeff64(int nx, int ny, const double *__restrict__ h, double rdx2, double rdy2, double lambda,
                            double *cx, double *cy, double *cc, double *rcc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= ny) return;
  const size_t k = (size_t)i + (size_t)nx * j;
  const double hk = h[k];
  const double cxw = i > 0 ? (0.5 * (hk + h[k - 1])) * rdx2 : 0.;
  const double cxe = i < nx - 1 ? (0.5 * (h[k + 1] + hk)) * rdx2 : 0.;
  const double cys = j > 0 ? (0.5 * (hk + h[k - nx])) * rdy2 : 0.;
  const double cyn = j < ny - 1 ? (0.5 * (h[k + nx] + hk)) * rdy2 : 0.;
  cx[k] = cxw;
  cy[k] = cys;
  cc[k] = -(((cxw + cxe) + cys) + cyn) - lambda;
  rcc[k] = 1. / cc[k];
}

// FP64 sweeps run on a colour-split layout: cell (i, j) of colour (i + j) % 2
// sits at j * W + i / 2 of its colour's arrays (W = ceil(nx / 2)) with its
// four face coefficients (0 at the frame), reciprocal diagonal, rhs and mask,
// so a colour pass reads only its own colour's arrays and the other
// colour's psi, contiguous, one thread per cell of the colour
struct Split64 {
  double *c[2][4];  // west, east, south, north face coefficients
  double *rcc[2], *rhs[2], *psi[2];
  uint8_t *mask[2];  // 0 also on the padding of rows with fewer cells
};

__global__ void k_h_split_coeff64(int nx, int ny, int W, const double *__restrict__ cx, const double *__restrict__ cy,
                                  const double *__restrict__ rcc, const int8_t *__restrict__ mask, Split64 s) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (size_t)nx * ny) return;
  const int i = (int)(k % nx), j = (int)(k / nx), col = (i + j) & 1;
  const size_t q = (size_t)j * W + (i >> 1);
  s.c[col][0][q] = cx[k];
  s.c[col][1][q] = i < nx - 1 ? cx[k + 1] : 0.;
  s.c[col][2][q] = cy[k];
  s.c[col][3][q] = j < ny - 1 ? cy[k + nx] : 0.;
  s.rcc[col][q] = rcc[k];
  s.mask[col][q] = mask[k] != 0;
}

// natural <-> colour-split copy of one field (join 0: natural -> split)
__global__ void k_h_split64(int nx, int ny, int W, double *nat, double *s0, double *s1, int join) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (size_t)nx * ny) return;
  const int i = (int)(k % nx), j = (int)(k / nx);
  double *sp = ((i + j) & 1) ? s1 : s0;
  const size_t q = (size_t)j * W + (i >> 1);
  if (join) nat[k] = sp[q];
  else sp[q] = nat[k];
}

// one colour of an FP64 sweep: off = cw w + ce e + cs s + cn n as nested
// fused multiply-adds, psi += omega ((rhs - off) / diag - psi) as one more
// (the arithmetic of orc_helmholtz_sor).  8 FP64 operations and 73 B a cell:
// at 2048^2 a sweep's two colours cannot take less than 67 us in the FP64
// pipe, nor less than 45 us of HBM.  A thread has the loads of H64_CELLS cells
// in flight before it looks at any mask; nothing else hides the time of HBM
// behind the pipe's (90 us a sweep with one cell and its mask first, 72 now).
constexpr int H64_CELLS = 2, H64_T = 128;
struct Colour64 {  // one colour's arrays, and the other colour's psi
  const double *c[4], *rcc, *rhs, *other;
  double *psi;
  const uint8_t *mask;
};
__global__ void __launch_bounds__(H64_T) k_h_sweep64(int nx, int ny, unsigned W, Colour64 s, int col, double omega) {
  const unsigned ns = W * (unsigned)ny, q0 = blockIdx.x * (H64_CELLS * H64_T) + threadIdx.x;
  const double *P = s.other;
  double *X = s.psi;
  double cw[H64_CELLS], ce[H64_CELLS], cs[H64_CELLS], cn[H64_CELLS], w[H64_CELLS], e[H64_CELLS], so[H64_CELLS],
      n[H64_CELLS], b[H64_CELLS], rc[H64_CELLS], x[H64_CELLS];
  bool wet[H64_CELLS];
#pragma unroll
  for (int u = 0; u < H64_CELLS; u++) {
    const unsigned q = q0 + u * H64_T;
    wet[u] = false;
    if (q >= ns) continue;
    const unsigned j = q / W, c = q - j * W, par = (j + (unsigned)col) & 1u;  // column i = 2 c + par
    const unsigned i = 2 * c + par;
    cw[u] = s.c[0][q];
    ce[u] = s.c[1][q];
    cs[u] = s.c[2][q];
    cn[u] = s.c[3][q];
    b[u] = s.rhs[q];
    rc[u] = s.rcc[q];
    x[u] = X[q];
    w[u] = i > 0 ? P[q - 1 + par] : 0.;
    e[u] = i + 1 < (unsigned)nx ? P[q + par] : 0.;
    so[u] = j > 0 ? P[q - W] : 0.;
    n[u] = j + 1 < (unsigned)ny ? P[q + W] : 0.;
    wet[u] = s.mask[q] != 0;
  }
#pragma unroll
  for (int u = 0; u < H64_CELLS; u++) {
    if (!wet[u]) continue;
    const double off = __fma_rn(cw[u], w[u], __fma_rn(ce[u], e[u], __fma_rn(cs[u], so[u], cn[u] * n[u])));
    const double gs = (b[u] - off) * rc[u];
    X[q0 + u * H64_T] = __fma_rn(omega, gs - x[u], x[u]);
  }
}

// the reciprocal diagonals of the tiled sweeps, by the expressions of k_h_sweep32
__global__ void k_h_rcc32(int nx, int ny, const float *__restrict__ h, float rdx2, float rdy2, float lambda,
                            const int8_t *__restrict__ mask, float *rcc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= ny) return;
  const size_t k = (size_t)i + (size_t)nx * j;
  const float hk = h[k];
  const float cxw = i > 0 ? face32(hk, h[k - 1], rdx2) : 0.f;
  const float cxe = i < nx - 1 ? face32(h[k + 1], hk, rdx2) : 0.f;
  const float cys = j > 0 ? face32(hk, h[k - nx], rdy2) : 0.f;
  const float cyn = j < ny - 1 ? face32(h[k + nx], hk, rdy2) : 0.f;
  const float d = 1.f / (-(((cxw + cxe) + cys) + cyn) - lambda);
  // 0 stands for land; an ocean diagonal that overflowed gives NaN, as its update would
  rcc[k] = mask[k] ? (d != 0.f ? d : NAN) : 0.f;
}

// one colour of an FP32 sweep over the whole grid (the arithmetic of k_h_tbr)
__global__ void k_h_sweep32(int nx, int ny, const float *__restrict__ h, const int8_t *__restrict__ mask,
                            const float *__restrict__ rhs, float *psi, float rdx2, float rdy2, float lambda,
                            float omega, int colour) {
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int i = 2 * (blockIdx.x * blockDim.x + threadIdx.x) + ((j + colour) & 1);
  if (i >= nx || j >= ny) return;
  const size_t k = (size_t)i + (size_t)nx * j;
  if (!mask[k]) return;
  const float hk = h[k];
  const float cxw = i > 0 ? face32(hk, h[k - 1], rdx2) : 0.f;
  const float cxe = i < nx - 1 ? face32(h[k + 1], hk, rdx2) : 0.f;
  const float cys = j > 0 ? face32(hk, h[k - nx], rdy2) : 0.f;
  const float cyn = j < ny - 1 ? face32(h[k + nx], hk, rdy2) : 0.f;
  // the tiled kernel forms the next cell's west face as face32(h[k+1], h[k]),
  // this kernel forms this cell's east face the same way: same operand order
  const float rcc = 1.f / (-(((cxw + cxe) + cys) + cyn) - lambda);
  const float w = i > 0 ? psi[k - 1] : 0.f, e = i < nx - 1 ? psi[k + 1] : 0.f;
  const float s = j > 0 ? psi[k - nx] : 0.f, n = j < ny - 1 ? psi[k + nx] : 0.f;
  psi[k] = sor32_update(psi[k], rhs[k], cxw, cxe, cys, cyn, rcc, w, e, s, n, omega);
}

// The update of two cells of a colour at once, in packed FP32x2 instructions
// (each half rounded as sor32_update rounds it; a - b as a + (-1) b, exact)
__device__ __forceinline__ float2 sor32_update2(float2 p, float2 r, float2 cxw, float2 cxe, float2 cys, float2 cyn,
                                                float2 rcc, float2 w, float2 e, float2 s, float2 n, float omega) {
  const float2 neg = make_float2(-1.f, -1.f);
  const float2 off = __ffma2_rn(cyn, n, __ffma2_rn(cys, s, __ffma2_rn(cxe, e, __fmul2_rn(cxw, w))));
  const float2 gs = __fmul2_rn(__ffma2_rn(off, neg, r), rcc);
  return __ffma2_rn(make_float2(omega, omega), __ffma2_rn(p, neg, gs), p);
}

// K red-black sweeps of FP32 SOR on a region of 64 columns by 96 rows (48 rows
// on small grids), of which the interior, 2K cells from its edge, is written.
// A thread owns, for the whole region, four cells a0 b0 a1 b1 of adjacent
// columns in each of TBR_M rows; a0 and a1 (b0 and b1) have one colour and are
// updated together.  Their face coefficients, reciprocal diagonals and rhs are
// kept in registers.  psi is kept in shared memory by column parity, so that a
// pair's neighbours to the north and south are one 64-bit load each; to the
// east and west they are the thread's own registers and one shuffle.  The
// half-warps of warp w of NW own rows w + NW h + 2 NW m (h the half, m < TBR_M),
// which have one parity as NW is even, so a pass is one warp-uniform branch.
// Every neighbour of a cell has the other colour, so a pass reads only what
// the previous passes wrote.  Halo cells are relaxed with the arithmetic of
// the global sweep (same coefficients), so after 2K passes the interior equals
// K global sweeps bit for bit; what the passes leave in cells that no longer
// reach the interior is not used.  Cells outside the grid hold psi = 0 and are
// never relaxed, nor is the region's outer ring (its neighbours lie outside).
//
// What a launch of 4 sweeps of 4096^2 took: 177 us with two columns of a
// thread relaxed one by one, coefficients formed and divided for in each
// launch; as much with packed pairs and four fields read instead, of which
// 105 us before the first pass; 163 us with the next region's fields fetched
// during the passes (k_h_tbr_stream); 149 us with 96 rows instead of 48 (the
// passes and the loads repeat 1.6 cells per written cell, not 2); 136 us with
// faces formed from the reciprocal depth (four fields read, not five).  The
// passes themselves take about 60 us, the four fields and the result 50 us of
// HBM.  80 registers: 24 warps per SM, in one block or two.
constexpr int TBR_M = 2;
constexpr int tbr_rows(int nw) { return 2 * nw * TBR_M; }  // rows of a block of nw warps
struct Region32 {  // what the tiled sweeps read: reciprocal depth, reciprocal diagonal (0 on land)
  int nx, ny;
  float rdx2, rdy2;
  const float *hinv, *rcc;
};

// the cells of one thread: psi, rhs, reciprocal diagonal of (a0, a1) and (b0,
// b1), and their faces
struct TbrCells {
  float2 p[2][TBR_M], f[2][TBR_M], q[2][TBR_M];
  float2 cw[TBR_M], cm[TBR_M], ce[TBR_M];  // (a0 west, a1 west), (a0 east, a1 east), (b0 east, b1 east)
  float2 cs[2][TBR_M], cn[2][TBR_M];
  unsigned relax = 0;  // bit 4m + c: cell c of row m is relaxed

  // row m from the four columns' values; h, hs, hn: reciprocal depth of this
  // row, the row to its south and the row to its north; (gx, gy): the first
  // column's cell in the grid, edge: the region reaches the grid's edge, where
  // faces are 0.  The faces of the ring, which need cells outside the region,
  // are not used.
  __device__ __forceinline__ void set(int m, int ly, int rows, int tx, const Region32 &g, int gx, int gy, bool edge,
                                      const float *pv, const float *fv, const float *h, const float *hs,
                                      const float *hn, const float *d) {
    unsigned mk = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) mk |= d[c] != 0.f ? 1u << c : 0u;
    if (ly == 0 || ly == rows - 1) mk = 0;  // the ring
    if (tx == 0) mk &= ~1u;
    if (tx == 15) mk &= ~8u;
    relax |= mk << (4 * m);
    float x[4], ys[4], yn[4];
    x[0] = face32(h[0], __shfl_up_sync(0xffffffffu, h[3], 1, 16), g.rdx2);
#pragma unroll
    for (int c = 0; c < 4; c++) {
      if (c) x[c] = face32(h[c], h[c - 1], g.rdx2);
      ys[c] = face32(h[c], hs[c], g.rdy2);
      yn[c] = face32(hn[c], h[c], g.rdy2);
    }
    if (edge) {
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if (gx + c <= 0 || gx + c >= g.nx) x[c] = 0.f;
        if (gy <= 0) ys[c] = 0.f;
        if (gy >= g.ny - 1) yn[c] = 0.f;
      }
    }
    const float xe = __shfl_down_sync(0xffffffffu, x[0], 1, 16);  // the next thread's first column (b1's east face)
    cw[m] = make_float2(x[0], x[2]);
    cm[m] = make_float2(x[1], x[3]);
    ce[m] = make_float2(x[2], xe);
#pragma unroll
    for (int c = 0; c < 2; c++) {
      p[c][m] = make_float2(pv[c], pv[c + 2]);
      f[c][m] = make_float2(fv[c], fv[c + 2]);
      q[c][m] = make_float2(d[c], d[c + 2]);
      cs[c][m] = make_float2(ys[c], ys[c + 2]);
      cn[c][m] = make_float2(yn[c], yn[c + 2]);
    }
  }
};

// the passes of one launch; sp: psi of the even / odd region columns, a pair
// per thread; ca: colour of the thread's cells a ((gx + gy) & 1, one in all its rows)
template <int K, int NW>
__device__ __forceinline__ void tbr_passes(TbrCells &t, float2 (*sp)[tbr_rows(NW)][16], int tx, int r0, int ca,
                                           float omega) {
  constexpr int M = TBR_M, RY = tbr_rows(NW);
  auto pass = [&](auto which) {  // 0: cells a, 1: cells b
    constexpr int c = decltype(which)::value;
#pragma unroll
    for (int m = 0; m < M; m++) {
      const int ly = r0 + 2 * NW * m;
      // (the ring rows' loads stay inside the arrays)
      const float2 s = sp[c][m ? ly - 1 : max(ly - 1, 0)][tx], n = sp[c][m == M - 1 ? min(ly + 1, RY - 1) : ly + 1][tx];
      float2 v;
      if (c == 0) {
        const float w = __shfl_up_sync(0xffffffffu, t.p[1][m].y, 1, 16);
        v = sor32_update2(t.p[0][m], t.f[0][m], t.cw[m], t.cm[m], t.cs[0][m], t.cn[0][m], t.q[0][m],
                          make_float2(w, t.p[1][m].x), t.p[1][m], s, n, omega);
      } else {
        const float e = __shfl_down_sync(0xffffffffu, t.p[0][m].x, 1, 16);
        v = sor32_update2(t.p[1][m], t.f[1][m], t.cm[m], t.ce[m], t.cs[1][m], t.cn[1][m], t.q[1][m], t.p[0][m],
                          make_float2(t.p[0][m].y, e), s, n, omega);
      }
      // cells not relaxed (land, outside the grid, the ring) keep their value
      t.p[c][m].x = (t.relax >> (4 * m + c)) & 1 ? v.x : t.p[c][m].x;
      t.p[c][m].y = (t.relax >> (4 * m + c + 2)) & 1 ? v.y : t.p[c][m].y;
      sp[c][ly][tx] = t.p[c][m];
    }
  };
#pragma unroll
  for (int k = 0; k < 2 * K; k++) {
    if (ca == (k & 1)) pass(std::integral_constant<int, 0>{});  // warp-uniform
    else pass(std::integral_constant<int, 1>{});
    __syncthreads();
  }
}

// any grid: a block per region, values read as the thread needs them
template <int K, int NW>
__global__ void __launch_bounds__(32 * NW, 24 / NW) k_h_tbr(Region32 co, const float *__restrict__ rhs, const float *__restrict__ pin,
                                                             float *__restrict__ pout, float omega) {
  const int nx = co.nx, ny = co.ny;
  constexpr int M = TBR_M, W = 2 * K, RY = tbr_rows(NW), TX = 64 - 2 * W, TY = RY - 2 * W;
  __shared__ float2 sp[2][RY][16];
  const int tx = threadIdx.x & 15, r0 = (threadIdx.x >> 5) + NW * ((threadIdx.x >> 4) & 1);
  const int x0 = blockIdx.x * TX - W, y0 = blockIdx.y * TY - W, gx = x0 + 4 * tx;
  TbrCells t;
#pragma unroll
  for (int m = 0; m < M; m++) {
    const int ly = r0 + 2 * NW * m, gy = y0 + ly;
    auto load = [&](const float *a, int g, float *v) {
#pragma unroll
      for (int c = 0; c < 4; c++)
        v[c] = g >= 0 && g < ny && gx + c >= 0 && gx + c < nx ? a[(size_t)(gx + c) + (size_t)nx * g] : 0.f;
    };
    float pv[4], fv[4], h[4], hs[4], hn[4], d[4];
    load(pin, gy, pv);
    load(rhs, gy, fv);
    load(co.hinv, gy, h);
    load(co.hinv, gy - 1, hs);
    load(co.hinv, gy + 1, hn);
    load(co.rcc, gy, d);
    t.set(m, ly, RY, tx, co, gx, gy, true, pv, fv, h, hs, hn, d);
    for (int c = 0; c < 2; c++) sp[c][ly][tx] = t.p[c][m];
  }
  __syncthreads();
  tbr_passes<K, NW>(t, sp, tx, r0, (x0 + y0 + r0) & 1, omega);
#pragma unroll
  for (int m = 0; m < M; m++) {
    const int ly = r0 + 2 * NW * m, gy = y0 + ly;
    if (ly < W || ly >= RY - W || gy >= ny) continue;
    const float v[4] = {t.p[0][m].x, t.p[1][m].x, t.p[0][m].y, t.p[1][m].y};
#pragma unroll
    for (int c = 0; c < 4; c++)
      if (4 * tx + c >= W && 4 * tx + c < 64 - W && gx + c < nx) pout[(size_t)(gx + c) + (size_t)nx * gy] = v[c];
  }
}

// Where rows and regions start at multiples of four columns (nx and 2K are
// multiples of 4): persistent blocks take region after region, and while one
// is relaxed the next one's four fields come into shared memory by
// asynchronous 16-byte copies.  3 sweeps of 4096^2 and rows of odd length
// stay with k_h_tbr, which can start at any column (4095^2: 168 us for 4).
constexpr int TBR_FIELDS = 4;
template <int K, int NW>
__global__ void __launch_bounds__(32 * NW, 24 / NW) k_h_tbr_stream(int nbx, int tiles, Region32 co,
                                                                    const float *__restrict__ rhs,
                                                                    const float *__restrict__ pin,
                                                                    float *__restrict__ pout, float omega) {
  const int nx = co.nx, ny = co.ny;
  constexpr int M = TBR_M, W = 2 * K, RY = tbr_rows(NW), TX = 64 - 2 * W, TY = RY - 2 * W;
  static_assert(W % 4 == 0, "regions start at multiples of four columns");
  extern __shared__ float4 stage[];  // [field][row][16]: psi, rhs, hinv, rcc
  __shared__ float2 sp[2][RY][16];
  const int tx = threadIdx.x & 15, r0 = (threadIdx.x >> 5) + NW * ((threadIdx.x >> 4) & 1);
  const float *src[TBR_FIELDS] = {pin, rhs, co.hinv, co.rcc};
  auto fetch = [&](int tile) {
    const int x0 = (tile % nbx) * TX - W, y0 = (tile / nbx) * TY - W;
    for (int e = threadIdx.x; e < RY * 16; e += 32 * NW) {
      const int ly = e >> 4, gx = x0 + 4 * (e & 15), gy = y0 + ly;
      const bool in = gy >= 0 && gy < ny && gx >= 0 && gx < nx;
      const size_t k = in ? (size_t)gx + (size_t)nx * gy : 0;
#pragma unroll
      for (int f = 0; f < TBR_FIELDS; f++) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(stage + f * RY * 16 + e);
        // outside the grid no byte is read and zeros are written
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src[f] + k), "r"(in ? 16 : 0) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if ((int)blockIdx.x < tiles) fetch(blockIdx.x);
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int x0 = (tile % nbx) * TX - W, y0 = (tile / nbx) * TY - W, gx = x0 + 4 * tx;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const bool edge = x0 <= 0 || y0 <= 0 || x0 + 64 >= nx || y0 + RY >= ny;
    TbrCells t;
#pragma unroll
    for (int m = 0; m < M; m++) {
      const int ly = r0 + 2 * NW * m, e = ly * 16 + tx;
      const float4 a = stage[e], b = stage[RY * 16 + e], c = stage[2 * RY * 16 + e], d = stage[3 * RY * 16 + e],
                   s = stage[2 * RY * 16 + (m ? e - 16 : max(e - 16, tx))],
                   n = stage[2 * RY * 16 + (m == M - 1 ? min(ly + 1, RY - 1) * 16 + tx : e + 16)];
      const float pv[4] = {a.x, a.y, a.z, a.w}, fv[4] = {b.x, b.y, b.z, b.w}, h[4] = {c.x, c.y, c.z, c.w},
                  dv[4] = {d.x, d.y, d.z, d.w}, hs[4] = {s.x, s.y, s.z, s.w}, hn[4] = {n.x, n.y, n.z, n.w};
      t.set(m, ly, RY, tx, co, gx, y0 + ly, edge, pv, fv, h, hs, hn, dv);
      for (int q = 0; q < 2; q++) sp[q][ly][tx] = t.p[q][m];
    }
    __syncthreads();
    if (tile + (int)gridDim.x < tiles) fetch(tile + gridDim.x);
    tbr_passes<K, NW>(t, sp, tx, r0, (x0 + y0 + r0) & 1, omega);
#pragma unroll
    for (int m = 0; m < M; m++) {
      const int ly = r0 + 2 * NW * m, gy = y0 + ly;
      if (ly >= W && ly < RY - W && gy < ny && 4 * tx >= W && 4 * tx < 64 - W && gx < nx)
        *reinterpret_cast<float4 *>(pout + (size_t)gx + (size_t)nx * gy) =
            make_float4(t.p[0][m].x, t.p[1][m].x, t.p[0][m].y, t.p[1][m].y);
    }
  }
}

// out = A psi on ocean cells (0 elsewhere), every product and sum rounded, in
// the order of orc_helmholtz_apply
__global__ void k_h_apply(int nx, int ny, const double *__restrict__ cx, const double *__restrict__ cy,
                          const double *__restrict__ cc, const int8_t *__restrict__ mask,
                          const double *__restrict__ psi, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= ny) return;
  const size_t k = (size_t)i + (size_t)nx * j;
  double a = 0.;
  if (mask[k]) {
    const double cxe = i < nx - 1 ? cx[k + 1] : 0., cyn = j < ny - 1 ? cy[k + nx] : 0.;
    const double w = i > 0 ? psi[k - 1] : 0., e = i < nx - 1 ? psi[k + 1] : 0.;
    const double s = j > 0 ? psi[k - nx] : 0., nn = j < ny - 1 ? psi[k + nx] : 0.;
    a = cx[k] * w + cxe * e + cy[k] * s + cyn * nn + cc[k] * psi[k];
  }
  out[k] = -(0. - a);
}

// x in FP64: a normal number's or zero's bits are moved by integer operations
// (a conversion instruction takes the FP64 pipe's time)
__device__ __forceinline__ double widen(double x) { return x; }
__device__ __forceinline__ double widen(float x) {
  const unsigned b = __float_as_uint(x), e = (b >> 23) & 255u;
  if (e - 1u < 254u) return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))), (int)(b << 29));
  if ((b << 1) == 0) return __hiloint2double((int)b, 0);
  return (double)x;
}

// r = rhs - A psi on ocean cells (0 elsewhere; r may be null) for an FP64 or
// FP32 iterate, and per-block sums of r^2.  FP64-pipe bound: a thread walks
// RES_ROWS rows of a column, so that a row's values are converted once, the
// diagonal is read and not added up, and products are fused: 7 FP64
// operations a cell.  4096^2: 684 us (FP32 iterate) and 554 us (FP64) with 20
// and 16 operations, 339 and 234 us now; the coefficients, mask, right-hand
// side and iterate, 33 to 41 B a cell, take about 110 us of HBM.
constexpr int RES_X = 128, RES_ROWS = 32;
template <typename T>
__global__ void __launch_bounds__(RES_X) k_h_resid(int nx, int ny, int rows, const double *__restrict__ cx,
                                                   const double *__restrict__ cy, const double *__restrict__ cc,
                                                   const int8_t *__restrict__ mask, const T *__restrict__ rhs,
                                                   const T *__restrict__ psi, double *r, double *partial) {
  __shared__ double red[RES_X / 32];
  const int i = blockIdx.x * RES_X + threadIdx.x, j0 = blockIdx.y * rows, j1 = min(j0 + rows, ny);
  double acc = 0.;
  if (i < nx) {
    size_t k = (size_t)i + (size_t)nx * j0;
    double s = j0 > 0 ? widen(psi[k - nx]) : 0., p = widen(psi[k]), cys = cy[k];
#pragma unroll 2
    for (int j = j0; j < j1; j++, k += nx) {
      const bool top = j == ny - 1;
      const double n = top ? 0. : widen(psi[k + nx]), cyn = top ? 0. : cy[k + nx];
      double rr = 0.;
      if (mask[k]) {
        const double w = i > 0 ? widen(psi[k - 1]) : 0., e = i < nx - 1 ? widen(psi[k + 1]) : 0.;
        const double cxe = i < nx - 1 ? cx[k + 1] : 0.;
        const double off = __fma_rn(cx[k], w, __fma_rn(cxe, e, __fma_rn(cys, s, cyn * n)));
        rr = widen(rhs[k]) - __fma_rn(cc[k], p, off);
        acc = __fma_rn(rr, rr, acc);
      }
      if (r) r[k] = rr;
      s = p;
      p = n;
      cys = cyn;
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = red[0];
    for (int w = 1; w < RES_X / 32; w++) t += red[w];
    partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = t;
  }
}

__global__ void k_h_sumsq(const double *x, const int8_t *mask, size_t n, double *partial) {
  __shared__ double red[256];
  double acc = 0.;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
    if (mask[k]) acc += x[k] * x[k];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

__global__ void k_h_final(const double *partial, int nb, double *out) {
  __shared__ double red[256];
  double a = 0.;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) a += partial[b];
  red[threadIdx.x] = a;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0];
}

__global__ void k_h_to32(const double *r, float *r32, float *e32, size_t n, double inv_scale) {
  size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) {
    r32[k] = (float)(r[k] * inv_scale);
    e32[k] = 0.f;
  }
}

__global__ void k_h_axpy(double *psi, const float *e32, size_t n, double scale) {
  size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) psi[k] = psi[k] + scale * (double)e32[k];
}

}  // namespace swm

struct swm_helm {
  int device = -1;  // the CUDA device the solver was created on
  double *cx = nullptr, *cy = nullptr, *cc = nullptr, *rcc = nullptr;  // FP64 coefficients
  swm::Split64 s64 = {};  // the FP64 sweeps' colour-split arrays (first FP64 solve)
  bool has_s64 = false;
  int W = 0;              // cells of a colour-split row
  int nx = 0, ny = 0;
  size_t n = 0;
  double dx = 0, dy = 0, lambda = 0;
  cudaStream_t stream = nullptr;
  double *hinv = nullptr, *psi = nullptr, *rhs = nullptr, *r = nullptr, *partial = nullptr, *out = nullptr;
  double *host = nullptr;  // pinned, 1 double
  float *rcc32 = nullptr;  // reciprocal diagonals of the tiled FP32 sweeps
  float *hinv32 = nullptr, *e32 = nullptr, *r32 = nullptr, *e32b = nullptr;  // e32b: ping-pong of e32
  int tbk = 4;  // sweeps per temporally blocked FP32 launch
  int sms = 0;
  int tb_blocks[2][2] = {};  // resident blocks of the streamed launches: 2 and 4 sweeps, 12 and 24 warps (0: not asked yet)
  int8_t *mask = nullptr;
  dim3 blk = dim3(64, 4);
  int64_t launches = 0;
};

namespace {
using namespace swm;

#define HTRY(x)                          \
  do {                                   \
    int rc_ = (x);                       \
    if (rc_ != SWM_GPU_OK) return rc_;   \
  } while (0)

dim3 sweep_grid(const swm_helm *h, dim3 b) {
  return dim3((unsigned)(((h->nx + 1) / 2 + b.x - 1) / b.x), (unsigned)((h->ny + b.y - 1) / b.y));
}

void sweep64(swm_helm *h, double omega) {
  const unsigned per = H64_CELLS * H64_T, g = (unsigned)(((size_t)h->W * h->ny + per - 1) / per);
  const Split64 &s = h->s64;
  for (int colour = 0; colour < 2; colour++) {
    const Colour64 a = {{s.c[colour][0], s.c[colour][1], s.c[colour][2], s.c[colour][3]}, s.rcc[colour], s.rhs[colour],
                        s.psi[colour ^ 1], s.psi[colour], s.mask[colour]};
    k_h_sweep64<<<g, H64_T, 0, h->stream>>>(h->nx, h->ny, h->W, a, colour, omega);
  }
  h->launches += 2;
}

// the colour-split arrays of the FP64 sweeps, set up at the first FP64 solve
int split64_setup(swm_helm *h) {
  if (h->has_s64) return SWM_GPU_OK;
  h->W = (h->nx + 1) / 2;
  const size_t ns = (size_t)h->W * h->ny;
  Split64 &s = h->s64;
  for (int col = 0; col < 2; col++) {
    for (int f = 0; f < 4; f++) SWM_CK(cudaMalloc((void **)&s.c[col][f], ns * 8));
    SWM_CK(cudaMalloc((void **)&s.rcc[col], ns * 8));
    SWM_CK(cudaMalloc((void **)&s.rhs[col], ns * 8));
    SWM_CK(cudaMalloc((void **)&s.psi[col], ns * 8));
    SWM_CK(cudaMalloc((void **)&s.mask[col], ns));
    SWM_CK(cudaMemsetAsync(s.mask[col], 0, ns, h->stream));
  }
  h->has_s64 = true;
  const unsigned nb = (unsigned)((h->n + 255) / 256);
  k_h_split_coeff64<<<nb, 256, 0, h->stream>>>(h->nx, h->ny, h->W, h->cx, h->cy, h->rcc, h->mask, s);
  h->launches++;
  SWM_CK(cudaGetLastError());
  return SWM_GPU_OK;
}

// one field between the natural layout and the FP64 sweeps' split layout
void split64_field(swm_helm *h, double *nat, double *const *sp, int join) {
  const unsigned nb = (unsigned)((h->n + 255) / 256);
  k_h_split64<<<nb, 256, 0, h->stream>>>(h->nx, h->ny, h->W, nat, sp[0], sp[1], join);
  h->launches++;
}

void sweep32(swm_helm *h, float omega, dim3 b) {
  const dim3 g = sweep_grid(h, b);
  const float rdx2 = (float)(1. / (h->dx * h->dx)), rdy2 = (float)(1. / (h->dy * h->dy)), lam = (float)h->lambda;
  for (int colour = 0; colour < 2; colour++)
    k_h_sweep32<<<g, b, 0, h->stream>>>(h->nx, h->ny, h->hinv32, h->mask, h->r32, h->e32, rdx2, rdy2, lam, omega,
                                        colour);
  h->launches += 2;
}

template <int K, int NW>
int launch_tb32(swm_helm *h, float omega) {
  constexpr int TX = 64 - 4 * K, TY = tbr_rows(NW) - 4 * K;
  const dim3 g((h->nx + TX - 1) / TX, (h->ny + TY - 1) / TY), b(32 * NW);
  const Region32 co = {h->nx, h->ny, (float)(1. / (h->dx * h->dx)), (float)(1. / (h->dy * h->dy)), h->hinv32, h->rcc32};
  if constexpr (K % 2 == 0) {
    if (h->nx % 4 == 0) {
      constexpr int bytes = TBR_FIELDS * tbr_rows(NW) * 16 * (int)sizeof(float4);
      int &blocks = h->tb_blocks[K / 2 - 1][NW == 24];
      if (blocks == 0) {
        int per_sm = 0;
        SWM_CK(cudaFuncSetAttribute(k_h_tbr_stream<K, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        SWM_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_h_tbr_stream<K, NW>, 32 * NW, bytes));
        blocks = std::max(1, per_sm) * h->sms;
      }
      const int tiles = (int)(g.x * g.y);
      k_h_tbr_stream<K, NW><<<std::min(tiles, blocks), b, bytes, h->stream>>>((int)g.x, tiles, co, h->r32, h->e32,
                                                                              h->e32b, omega);
      SWM_CK(cudaGetLastError());
      return SWM_GPU_OK;
    }
  }
  k_h_tbr<K, NW><<<g, b, 0, h->stream>>>(co, h->r32, h->e32, h->e32b, omega);
  SWM_CK(cudaGetLastError());
  return SWM_GPU_OK;
}

// Blocks of 24 warps where every SM gets one of their regions, else blocks of
// 12 with half the rows: 256^2 5.9 against 7.8 us, 768^2 (160 tall regions)
// and above faster with 24.
template <int K>
int launch_tb32(swm_helm *h, float omega) {
  const int nx = (h->nx + 63 - 4 * K) / (64 - 4 * K), ny = (h->ny + 95 - 4 * K) / (96 - 4 * K);
  return (int64_t)nx * ny >= h->sms ? launch_tb32<K, 24>(h, omega) : launch_tb32<K, 12>(h, omega);
}

// whole temporally blocked launches in n sweeps (none when tbk is 0: global
// sweeps only)
int tb_part(const swm_helm *h, int n) { return h->tbk > 0 ? n - n % h->tbk : 0; }

// n FP32 sweeps (a multiple of h->tbk) on A e = r32, ping-ponging e32/e32b;
// the result ends in h->e32
int sweeps_tb32(swm_helm *h, float omega, int n) {
  for (int s = 0; s < n && h->tbk > 0; s += h->tbk) {
    if (h->tbk == 4) HTRY(launch_tb32<4>(h, omega));
    else if (h->tbk == 3) HTRY(launch_tb32<3>(h, omega));
    else if (h->tbk == 2) HTRY(launch_tb32<2>(h, omega));
    else HTRY(launch_tb32<1>(h, omega));
    std::swap(h->e32, h->e32b);
    h->launches++;
  }
  return SWM_GPU_OK;
}

// rows of a column that a thread of k_h_resid walks: RES_ROWS, fewer where
// that leaves the chip without eight blocks per SM (a row is a serial step of
// 2 to 3 us; 256^2, FP32: 90 us with 32 rows, 9 with 2)
int resid_rows(const swm_helm *h) {
  int rows = RES_ROWS;
  while (rows > 2 && (int64_t)((h->nx + RES_X - 1) / RES_X) * ((h->ny + rows - 1) / rows) < 8 * h->sms) rows /= 2;
  return rows;
}
dim3 resid_grid(const swm_helm *h) {
  const int rows = resid_rows(h);
  return dim3((h->nx + RES_X - 1) / RES_X, (h->ny + rows - 1) / rows);
}

// ||rhs - A psi||^2 (FP64 accumulation); r written when wanted
template <typename T>
int resid2(swm_helm *h, const T *rhs, const T *psi, double *r, double *out) {
  const dim3 g = resid_grid(h);
  k_h_resid<T><<<g, RES_X, 0, h->stream>>>(h->nx, h->ny, resid_rows(h), h->cx, h->cy, h->cc, h->mask, rhs, psi, r, h->partial);
  k_h_final<<<1, 256, 0, h->stream>>>(h->partial, (int)(g.x * g.y), h->out);
  h->launches += 2;
  SWM_CK(cudaGetLastError());
  SWM_CK(cudaMemcpyAsync(h->host, h->out, 8, cudaMemcpyDeviceToHost, h->stream));
  SWM_CK(cudaStreamSynchronize(h->stream));
  *out = h->host[0];
  return SWM_GPU_OK;
}

int rhs_norm(swm_helm *h, double *bn) {
  k_h_sumsq<<<HELM_RED, 256, 0, h->stream>>>(h->rhs, h->mask, h->n, h->partial);
  k_h_final<<<1, 256, 0, h->stream>>>(h->partial, HELM_RED, h->out);
  h->launches += 2;
  SWM_CK(cudaGetLastError());
  SWM_CK(cudaMemcpyAsync(h->host, h->out, 8, cudaMemcpyDeviceToHost, h->stream));
  SWM_CK(cudaStreamSynchronize(h->stream));
  *bn = std::sqrt(h->host[0]);
  return SWM_GPU_OK;
}

// FP32 sweeps on A e = r32 from e = 0 until ||r32 - A e|| <= tol ||r32||,
// until binary32 rounding stops the progress (a check that gains less than
// STALL over the previous one), or max_sweeps; returns the sweeps done and
// the reached relative residual
constexpr double STALL = 0.7;
int inner32(swm_helm *h, float omega, double tol, int max_sweeps, int *sweeps, double *rel) {
  double rn2 = 0.;
  // ||r32||: residual of e = 0
  HTRY(resid2<float>(h, h->r32, h->e32, nullptr, &rn2));
  const double rn = std::sqrt(rn2);
  int s = 0, checks = 0;
  double rr = 1., prev = 1.;
  while (s < max_sweeps) {
    // 2 * HELM_CHECK sweeps between checks of the correction equation
    int blk = std::min(2 * HELM_CHECK, max_sweeps - s);
    const int tb = tb_part(h, blk);
    HTRY(sweeps_tb32(h, omega, tb));
    for (int q = tb; q < blk; q++) sweep32(h, omega, h->blk);
    s += blk;
    double e2 = 0.;
    HTRY(resid2<float>(h, h->r32, h->e32, nullptr, &e2));
    rr = rn > 0 ? std::sqrt(e2) / rn : 0.;
    if (rr <= tol || (++checks >= 2 && rr > STALL * prev)) break;
    prev = rr;
  }
  *sweeps = s;
  *rel = rr;
  return SWM_GPU_OK;
}

void helm_free(swm_helm *h) {
  if (!h) return;
  if (h->stream) cudaStreamSynchronize(h->stream);
  cudaFree(h->hinv); cudaFree(h->psi); cudaFree(h->rhs); cudaFree(h->r); cudaFree(h->partial); cudaFree(h->out);
  cudaFreeHost(h->host);
  cudaFree(h->hinv32); cudaFree(h->e32); cudaFree(h->r32); cudaFree(h->mask); cudaFree(h->e32b);
  cudaFree(h->rcc32);
  cudaFree(h->cx); cudaFree(h->cy); cudaFree(h->cc); cudaFree(h->rcc);
  for (int col = 0; col < 2; col++) {
    for (int f = 0; f < 4; f++) cudaFree(h->s64.c[col][f]);
    cudaFree(h->s64.rcc[col]); cudaFree(h->s64.rhs[col]); cudaFree(h->s64.psi[col]); cudaFree(h->s64.mask[col]);
  }
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

}  // namespace

extern "C" {

int swm_helm_create(int nx, int ny, double dx, double dy, double lambda, const double *H, const int8_t *ocean,
                    swm_helm **out) {
  SWM_REQUIRE(nx >= 3 && ny >= 3 && dx > 0 && dy > 0 && H && ocean && out, "swm_helm_create: bad arguments");
  *out = nullptr;
  swm_helm *h = new swm_helm();
  if (cudaGetDevice(&h->device) != cudaSuccess) h->device = -1;
  h->nx = nx; h->ny = ny; h->n = (size_t)nx * ny; h->dx = dx; h->dy = dy; h->lambda = lambda;
  const size_t n = h->n;
  std::vector<double> hinv(n);
  std::vector<float> hinv32(n);
  for (size_t k = 0; k < n; k++) {
    if (!(H[k] > 0.)) {
      helm_free(h);
      set_error("swm_helm_create: depth must be positive everywhere (land is given by the ocean mask)");
      return SWM_GPU_EINVAL;
    }
    hinv[k] = 1. / H[k];
    hinv32[k] = (float)hinv[k];
  }
  if (cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, h->device) != cudaSuccess) h->sms = 1;
  const dim3 rg = resid_grid(h);
  bool ok = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) == cudaSuccess &&
            cudaMalloc((void **)&h->hinv, n * 8) == cudaSuccess && cudaMalloc((void **)&h->psi, n * 8) == cudaSuccess &&
            cudaMalloc((void **)&h->rhs, n * 8) == cudaSuccess && cudaMalloc((void **)&h->r, n * 8) == cudaSuccess &&
            cudaMalloc((void **)&h->partial, std::max<size_t>(HELM_RED, (size_t)rg.x * rg.y) * 8) == cudaSuccess &&
            cudaMalloc((void **)&h->out, 8) == cudaSuccess && cudaMallocHost((void **)&h->host, 8) == cudaSuccess &&
            cudaMalloc((void **)&h->hinv32, n * 4) == cudaSuccess && cudaMalloc((void **)&h->e32, n * 4) == cudaSuccess &&
            cudaMalloc((void **)&h->r32, n * 4) == cudaSuccess && cudaMalloc((void **)&h->mask, n) == cudaSuccess &&
            cudaMalloc((void **)&h->e32b, n * 4) == cudaSuccess &&
            cudaMalloc((void **)&h->rcc32, n * 4) == cudaSuccess &&
            cudaMalloc((void **)&h->cx, n * 8) == cudaSuccess && cudaMalloc((void **)&h->cy, n * 8) == cudaSuccess &&
            cudaMalloc((void **)&h->cc, n * 8) == cudaSuccess && cudaMalloc((void **)&h->rcc, n * 8) == cudaSuccess;
  if (!ok) {
    helm_free(h);
    set_error("swm_helm_create: device allocation failed");
    return SWM_GPU_ENOMEM;
  }
  SWM_CK(cudaMemcpyAsync(h->hinv, hinv.data(), n * 8, cudaMemcpyHostToDevice, h->stream));
  SWM_CK(cudaMemcpyAsync(h->hinv32, hinv32.data(), n * 4, cudaMemcpyHostToDevice, h->stream));
  SWM_CK(cudaMemcpyAsync(h->mask, ocean, n, cudaMemcpyHostToDevice, h->stream));
  dim3 b(32, 8), g((nx + 31) / 32, (ny + 7) / 8);
  k_h_coeff64<<<g, b, 0, h->stream>>>(nx, ny, h->hinv, 1. / (dx * dx), 1. / (dy * dy), lambda, h->cx, h->cy, h->cc, h->rcc);
  k_h_rcc32<<<g, b, 0, h->stream>>>(nx, ny, h->hinv32, (float)(1. / (dx * dx)), (float)(1. / (dy * dy)),
                                    (float)lambda, h->mask, h->rcc32);
  h->launches += 2;
  SWM_CK(cudaGetLastError());
  SWM_CK(cudaStreamSynchronize(h->stream));
  *out = h;
  return SWM_GPU_OK;
}

int swm_helm_destroy(swm_helm *h) {
  SWM_ON_DEVICE(h ? h->device : -1);
  helm_free(h);
  return SWM_GPU_OK;
}

void *swm_helm_stream(swm_helm *h) { return h ? (void *)h->stream : nullptr; }
int64_t swm_helm_launch_count(swm_helm *h) { return h ? h->launches : -1; }

// out = A psi (ocean cells; 0 elsewhere), FP64
int swm_helm_apply(swm_helm *h, const double *psi, double *out) {
  SWM_ON_DEVICE(h ? h->device : -1);
  SWM_REQUIRE(h && psi && out, "swm_helm_apply: bad arguments");
  SWM_CK(cudaMemcpyAsync(h->psi, psi, h->n * 8, cudaMemcpyHostToDevice, h->stream));
  const dim3 b(32, 8), g((h->nx + 31) / 32, (h->ny + 7) / 8);
  k_h_apply<<<g, b, 0, h->stream>>>(h->nx, h->ny, h->cx, h->cy, h->cc, h->mask, h->psi, h->r);
  h->launches++;
  SWM_CK(cudaGetLastError());
  SWM_CK(cudaMemcpyAsync(out, h->r, h->n * 8, cudaMemcpyDeviceToHost, h->stream));
  SWM_CK(cudaStreamSynchronize(h->stream));
  return SWM_GPU_OK;
}

// FP64 red-black SOR from psi (in/out) to ||rhs - A psi|| < rtol ||rhs||
// (checked every 16 sweeps) or max_sweeps.
int swm_helm_solve_fp64(swm_helm *h, const double *rhs, double *psi, double omega, double rtol, int max_sweeps,
                        int *sweeps, double *relres) {
  SWM_ON_DEVICE(h ? h->device : -1);
  SWM_REQUIRE(h && rhs && psi && max_sweeps > 0, "swm_helm_solve_fp64: bad arguments");
  SWM_CK(cudaMemcpyAsync(h->rhs, rhs, h->n * 8, cudaMemcpyHostToDevice, h->stream));
  SWM_CK(cudaMemcpyAsync(h->psi, psi, h->n * 8, cudaMemcpyHostToDevice, h->stream));
  double bn;
  HTRY(rhs_norm(h, &bn));
  HTRY(split64_setup(h));
  split64_field(h, h->rhs, h->s64.rhs, 0);
  split64_field(h, h->psi, h->s64.psi, 0);
  int s = 0;
  double rel = 1.;
  while (s < max_sweeps) {
    int blk = std::min(HELM_CHECK, max_sweeps - s);
    for (int q = 0; q < blk; q++) sweep64(h, omega);
    s += blk;
    split64_field(h, h->psi, h->s64.psi, 1);  // the residual reads the natural layout
    double r2;
    HTRY(resid2<double>(h, h->rhs, h->psi, nullptr, &r2));
    rel = bn > 0 ? std::sqrt(r2) / bn : std::sqrt(r2);
    if (rel < rtol) break;
  }
  SWM_CK(cudaMemcpyAsync(psi, h->psi, h->n * 8, cudaMemcpyDeviceToHost, h->stream));
  SWM_CK(cudaStreamSynchronize(h->stream));
  if (sweeps) *sweeps = s;
  if (relres) *relres = rel;
  if (rel < rtol) return SWM_GPU_OK;
  set_error("swm_helm_solve_fp64: relative residual above rtol after max_sweeps");
  return SWM_GPU_ENOT_CONVERGED;
}

// Mixed precision: residual r = rhs - A psi in FP64, FP32 SOR sweeps on
// A e = r / ||r|| until its residual falls by inner_tol, psi += ||r|| e in
// FP64; repeated until the FP64 relative residual is below rtol.
int swm_helm_solve_mixed(swm_helm *h, const double *rhs, double *psi, double omega, double rtol, double inner_tol,
                         int max_sweeps, int *sweeps, int *outer, double *relres) {
  SWM_ON_DEVICE(h ? h->device : -1);
  SWM_REQUIRE(h && rhs && psi && max_sweeps > 0 && inner_tol > 0, "swm_helm_solve_mixed: bad arguments");
  SWM_CK(cudaMemcpyAsync(h->rhs, rhs, h->n * 8, cudaMemcpyHostToDevice, h->stream));
  SWM_CK(cudaMemcpyAsync(h->psi, psi, h->n * 8, cudaMemcpyHostToDevice, h->stream));
  double bn;
  HTRY(rhs_norm(h, &bn));
  const unsigned nb = (unsigned)((h->n + 255) / 256);
  int s = 0, o = 0;
  double rel = 1.;
  for (;;) {
    double r2;
    HTRY(resid2<double>(h, h->rhs, h->psi, h->r, &r2));
    const double rn = std::sqrt(r2);
    rel = bn > 0 ? rn / bn : rn;
    if (rel < rtol || s >= max_sweeps || rn == 0.) break;
    k_h_to32<<<nb, 256, 0, h->stream>>>(h->r, h->r32, h->e32, h->n, 1. / rn);
    int si = 0;
    double ri;
    HTRY(inner32(h, (float)omega, inner_tol, max_sweeps - s, &si, &ri));
    k_h_axpy<<<nb, 256, 0, h->stream>>>(h->psi, h->e32, h->n, rn);
    h->launches += 2;
    s += si;
    o++;
  }
  SWM_CK(cudaGetLastError());
  SWM_CK(cudaMemcpyAsync(psi, h->psi, h->n * 8, cudaMemcpyDeviceToHost, h->stream));
  SWM_CK(cudaStreamSynchronize(h->stream));
  if (sweeps) *sweeps = s;
  if (outer) *outer = o;
  if (relres) *relres = rel;
  if (rel < rtol) return SWM_GPU_OK;
  set_error("swm_helm_solve_mixed: relative residual above rtol after max_sweeps");
  return SWM_GPU_ENOT_CONVERGED;
}

// Autotuner: the sweep kernel's block shape by timing FP32 sweeps, then the
// relaxation factor in [omega_lo, omega_hi] (ngrid values) as the one whose
// trial solve of trial_sweeps FP32 sweeps on A e = rhs / ||rhs|| from e = 0
// reaches the smallest residual.
int swm_helm_autotune(swm_helm *h, const double *rhs, double omega_lo, double omega_hi, int ngrid,
                      int trial_sweeps, double *omega, int *block_x, int *block_y) {
  SWM_ON_DEVICE(h ? h->device : -1);
  SWM_REQUIRE(h && rhs && ngrid >= 1 && trial_sweeps > 0 && omega_lo > 0 && omega_hi < 2 && omega_lo <= omega_hi,
              "swm_helm_autotune: bad arguments");
  SWM_CK(cudaMemcpyAsync(h->rhs, rhs, h->n * 8, cudaMemcpyHostToDevice, h->stream));
  double bn;
  HTRY(rhs_norm(h, &bn));
  const unsigned nb = (unsigned)((h->n + 255) / 256);
  k_h_to32<<<nb, 256, 0, h->stream>>>(h->rhs, h->r32, h->e32, h->n, bn > 0 ? 1. / bn : 1.);
  h->launches++;
  // block shape
  const dim3 shapes[4] = {dim3(32, 8), dim3(64, 4), dim3(128, 2), dim3(256, 1)};
  cudaEvent_t a, b;
  int best_k = 4;
  SWM_CK(cudaEventCreate(&a));
  SWM_CK(cudaEventCreate(&b));
  float tbest = 1e30f;
  for (const dim3 &shp : shapes) {
    sweep32(h, 1.f, shp);
    SWM_CK(cudaEventRecord(a, h->stream));
    for (int q = 0; q < 4; q++) sweep32(h, 1.f, shp);
    SWM_CK(cudaEventRecord(b, h->stream));
    SWM_CK(cudaEventSynchronize(b));
    float ms;
    SWM_CK(cudaEventElapsedTime(&ms, a, b));
    if (ms < tbest) { tbest = ms; h->blk = shp; }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  // sweeps per temporally blocked launch (SWM_GB300_HELM_K overrides; 0:
  // global sweeps only)
  const char *ek = getenv("SWM_GB300_HELM_K");
  if (ek && atoi(ek) >= 0 && atoi(ek) <= 4 && ek[0] >= '0' && ek[0] <= '9') {
    h->tbk = atoi(ek);
  } else {
    SWM_CK(cudaEventCreate(&a));
    SWM_CK(cudaEventCreate(&b));
    float kbest = 1e30f;
    for (int kk : {1, 2, 3, 4}) {
      h->tbk = kk;
      HTRY(sweeps_tb32(h, 1.f, 4));
      SWM_CK(cudaEventRecord(a, h->stream));
      HTRY(sweeps_tb32(h, 1.f, 8));
      SWM_CK(cudaEventRecord(b, h->stream));
      SWM_CK(cudaEventSynchronize(b));
      float ms;
      SWM_CK(cudaEventElapsedTime(&ms, a, b));
      if (ms < kbest) { kbest = ms; best_k = kk; }
    }
    h->tbk = best_k;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
  }
  // relaxation factor
  double best = omega_lo, rbest = 1e300;
  for (int q = 0; q < ngrid; q++) {
    const double om = ngrid == 1 ? omega_lo : omega_lo + (omega_hi - omega_lo) * q / (ngrid - 1);
    k_h_to32<<<nb, 256, 0, h->stream>>>(h->rhs, h->r32, h->e32, h->n, bn > 0 ? 1. / bn : 1.);
    h->launches++;
    const int tb = tb_part(h, trial_sweeps);
    HTRY(sweeps_tb32(h, (float)om, tb));
    for (int s = tb; s < trial_sweeps; s++) sweep32(h, (float)om, h->blk);
    double e2;
    HTRY(resid2<float>(h, h->r32, h->e32, nullptr, &e2));
    if (e2 < rbest) { rbest = e2; best = om; }
  }
  if (omega) *omega = best;
  if (block_x) *block_x = (int)h->blk.x;
  if (block_y) *block_y = (int)h->blk.y;
  return SWM_GPU_OK;
}

}  // extern "C"
