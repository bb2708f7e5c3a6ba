// ttfld_krylov.cu -- preconditioned conjugate gradients on the FLD system.
//
//  * ttfld_solve_with_hypre: the IRAD=2 path's SOLVE_WITH_HYPRE
//    (pphypre.f:1-111).  Its system is FILLHYPREMATRIX / FILLHYPREVECTORS
//    (pphypre.f:115-334): SOLVE_WITH_SOR's 7-point matrix (ppsor.f:202-272)
//    with the i = 1 rows made identity rows (pphypre.f:281-294), the west
//    coupling of the i = 2 rows removed (pphypre.f:298-300) and b zero on the
//    same boundary rows (pphypre.f:137-205).  hypre solves it by PCG from
//    x = 1 (pphypre.f:136) to a relative residual of 1e-6 in at most 50
//    iterations (pphypre.f:45-55), preconditioned by one SMG cycle.  Here
//    the same PCG runs on the device with a radial line preconditioner.
//  * TTFLD_SOLVER_PCG: SOLVE_WITH_SOR's own system solved by the same PCG,
//    stopped like the mixed solver on ||b - A x||_1 / ||b||_1 <= tol.
//
// Symmetric form.  Row n of the matrix is (EVAL7 + EVAL8 EVAL_1_6) x_n -
// EVAL8 sum_m EVALm x_m, and each EVALm is a face coefficient shared by the
// two cells of the face divided by the metric factor of cell n
// (ppenergy.f:995-1013).  Multiplied by W_n = V_n / |EVAL8_n| with
// V = surxb dxa dya surzb dza, the rows form a symmetric matrix (the
// identity rows are decoupled and get W = V).  PCG runs on
// S = Sigma sym(W A) Sigma, Sigma = diag(1 / sqrt(W_n A_nn)), which has a
// unit diagonal; sym() is the symmetric part, which differs from W A only
// where the two cells of a face were given different face coefficients (the
// phi seam of the periodic halo).  An FP64 defect correction on the rows as
// they are (r = b - A x, x += Sigma e) removes that difference and the FP32
// rounding of the inner iteration:
//
//   loop: r = b - A x (FP64); stop test; solve S e = Sigma W r by FP32 PCG
//         to a relative reduction of its preconditioned residual norm; x += Sigma e.
//
// Preconditioner.  The radial couplings dominate by two to three orders of
// magnitude (the shell is thin in r), so the preconditioner is built on the
// exact solve of the tridiagonal radial line of a (j,k) column, factored
// once per solve (Thomas algorithm, FP32 pivots): TTFLD_SOLVER_PCG applies
// it to every column (block Jacobi); SOLVE_WITH_HYPRE, whose caller bounds
// the iterations at hypre's 50, applies one symmetric red-black line
// Gauss-Seidel sweep (half the iterations, three times the cost of one).
//
// Layout.  The FP32 inner arrays are line-major, q = (i-1)*NY*NZ +
// (k-1)*NY + (j-1): in a line solve of block Jacobi one thread walks one
// column and the threads of a warp touch 32 consecutive columns of the same
// radius (coalesced), line Gauss-Seidel copies tiles of 32 such columns to
// shared memory; in the operator pass the phi and theta neighbours are at q
// +- 1 and q +- NY.  The inner iteration is one persistent cooperative
// kernel with two grid barriers per iteration (after s = S p for alpha,
// after the line solve for beta).
#include <math.h>
#include <stdlib.h>

#include "ttfld_internal.cuh"

namespace ttfld {
namespace {

// one block per SM: 256 threads with up to 255 registers for the batched line
// passes, or 768 in groups for the line Gauss-Seidel tiles
constexpr int kJacobiThreads = 256, kGsThreads = 768;
extern __shared__ __align__(128) float tile_sh[];
constexpr int kPcgStall = 25;      // iterations without a new minimum of r.z end an inner run
constexpr double kInnerReduce = 1e-4;  // relative reduction of sqrt(r.z) asked of one inner run
constexpr int kMaxGsSweeps = 32;       // symmetric line Gauss-Seidel sweeps per preconditioner application

struct Kry {
  int nx, ny, nz;
  long long n, ncol;
  // couplings of S to the +i, +j (periodic) and +k neighbour, and the
  // reciprocal pivots of the radial line factorisation (line-major, FP32)
  float *cr, *cp, *ct, *g;
  float *e, *r, *z, *s, *p[2];
  double *sig, *wgt;  // Sigma_n and W_n (cell order, FP64)
};

struct KryWork {
  Kry k;
  void* mem;
  float* tiles;  // line tiles in global memory (lines too long for shared memory)
};

// The rows of the system being solved: SOR_A..G, with the hypre changes.
struct Row {
  double a, b, c, d, e, f, g;
};
// hypre's grid has only its extents (pphypre.f:404-413, no periodicity), so
// the j-1 entry of rows j = 1 and the j+1 entry of rows j = NY reach outside
// it and are dropped.  With poles (SOLVE_WITH_SOR's system only): the theta
// neighbour across either edge is the cell itself (the mirror the pole
// shifts keep), so rows 1 and NZ-1 take that coupling into their diagonal,
// and row NZ, which the SOR does not solve (ppsor.f:39-43) and the pole
// shift overwrites, is a decoupled identity row.  Both keep the symmetric
// form: the couplings between rows 1 and 2, NZ-2 and NZ-1 are unchanged.
__device__ __forceinline__ Row row_of(const Dev& d, size_t t, int i, int j, int k, bool hypre) {
  Row r{d.SA[t], d.SB[t], d.SC[t], d.SD[t], d.SE[t], d.SF[t], d.SG[t]};
  if (hypre) {
    if (i == 1) r = Row{1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // pphypre.f:281-294
    else if (i == 2) r.b = 0.0;                               // pphypre.f:298-300
    if (j == 1) r.d = 0.0;
    if (j == d.ny) r.e = 0.0;
  } else if (d.poles) {
    if (k == d.nz) return Row{1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (k == 1) { r.a += r.f; r.f = 0.0; }
    if (k == d.nz - 1) { r.a += r.g; r.g = 0.0; }
  }
  return r;
}

// b of the hypre system (pphypre.f:137-205): zero at i >= upperbnd, i = 1,
// i = NX, k = 1 and k = NZ; with poles, of SOLVE_WITH_SOR's system zero on
// the identity row NZ.
__device__ __forceinline__ double b_of(const Dev& d, const double* b, size_t t, int i, int j, int k, bool hypre) {
  if (hypre && (i >= PA(UB, j, k) || i == 1 || i == d.nx || k == 1 || k == d.nz)) return 0.0;
  if (!hypre && d.poles && k == d.nz) return 0.0;
  return b[t];
}

// W_n and Sigma_n (cell order).  A coupled row needs EVAL8 < 0.
__global__ void __launch_bounds__(kThreads) kry_weights_kernel(Dev d, Kry kr, int hypre) {
  const unsigned int n = (unsigned int)ncell(d);
  for (unsigned int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    int i, j, k;
    cell_ijk(d, t, i, j, k);
    const Row r = row_of(d, t, i, j, k, hypre != 0);
    const bool decoupled = r.b == 0.0 && r.c == 0.0 && r.d == 0.0 && r.e == 0.0 && r.f == 0.0 && r.g == 0.0;
    const double v = mul_rn(mul_rn(mul_rn(mul_rn(G(surxb, i), G(dxa, i)), G(dya, j)), G(surzb, k)), G(dza, k));
    const double e8 = d.E8[t];
    const double w = decoupled ? v : div_rn(v, -e8);
    const double dd = mul_rn(w, r.a);
    bool ok = (decoupled || e8 < 0.0) && dd > 0.0 && isfinite(dd);
    kr.wgt[t] = ok ? w : 0.0;
    kr.sig[t] = ok ? div_rn(1.0, sqrt_rn(dd)) : 0.0;  // any positive scaling serves; it is used consistently
    if (!ok) atomicExch(&d.sol->bad_weights, 1);
  }
}

// The kernels between the cell order (radius fastest) and the line-major
// order (phi fastest) work in strips of kStripCols neighbouring columns of
// one theta row, walked in cell order, with the line-major side going through
// shared memory, so that both sides are coalesced.  (A warp that writes its 32
// radii straight to the line-major arrays writes 32 sectors of 32 bytes for 4
// bytes each: 140 us an anchor at 100x256x128.)  Strips are cut along the
// radius into pieces of the same length (StripCut), so that few of them still
// fill the SMs and a piece fits in shared memory.
constexpr int kStripCols = 32;
struct StripCut {
  unsigned int pieces;  // strips times pieces of a strip
  unsigned int per;     // pieces of a strip
  FastDiv by_len;       // radii of a piece (the last may have fewer)
};
struct Strip {
  int j0, k, cols;        // columns j0 .. j0 + cols - 1 (from 1) of theta row k
  int i0, ni;             // radii i0 + 1 .. i0 + ni
  unsigned int t0;        // first cell
};
__device__ __forceinline__ Strip strip_of(const Dev& d, const StripCut& cut, unsigned int m) {
  const unsigned int across = ((unsigned int)d.ny + kStripCols - 1) / kStripCols, strip = m / cut.per;
  Strip p;
  p.k = (int)(strip / across) + 1;
  p.j0 = (int)(strip % across) * kStripCols + 1;
  p.cols = d.ny - p.j0 + 1 < kStripCols ? d.ny - p.j0 + 1 : kStripCols;
  p.i0 = (int)((m % cut.per) * cut.by_len.d);
  p.ni = d.nx - p.i0 < (int)cut.by_len.d ? d.nx - p.i0 : (int)cut.by_len.d;
  p.t0 = (unsigned int)cidx(d, p.i0 + 1, p.j0, p.k);
  return p;
}
constexpr int kStripPitch = kStripCols + 1;
// Line-major index of a piece's radius i (from 0) in its column `lane`.
__device__ __forceinline__ size_t strip_line(const Kry& kr, const Strip& p, int i, int lane) {
  return (size_t)(p.i0 + i) * kr.ncol + (size_t)(p.k - 1) * kr.ny + (size_t)(p.j0 - 1 + lane);
}
// Write the staged values of a piece, stage[i * kStripPitch + column], to a
// line-major array.
__device__ __forceinline__ void strip_out(const Kry& kr, const Strip& p, const float* stage, float* to) {
  const int lane = threadIdx.x & 31;
  if (lane < p.cols)
    for (int i = threadIdx.x >> 5; i < p.ni; i += blockDim.x >> 5)
      to[strip_line(kr, p, i, lane)] = stage[i * kStripPitch + lane];
}

// Couplings of S (the symmetric part of Sigma W A Sigma) to the +i, +j, +k
// neighbours, written line-major; stage holds three pieces.
__global__ void __launch_bounds__(kThreads) kry_couplings_kernel(Dev d, Kry kr, int hypre, StripCut cut) {
  extern __shared__ float stage[];
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const bool h = hypre != 0;
  const int one = (int)cut.by_len.d * kStripPitch;
  for (unsigned int m = blockIdx.x; m < cut.pieces; m += gridDim.x) {
    const Strip p = strip_of(d, cut, m);
    for (unsigned int u = threadIdx.x; u < cut.by_len.d * p.cols; u += blockDim.x) {
      unsigned int iu;
      const int col = (int)div_rem(cut.by_len, u, iu), i = p.i0 + (int)iu + 1, j = p.j0 + col, k = p.k;
      if ((int)iu >= p.ni) continue;
      const size_t t = p.t0 + (unsigned int)(nx * col) + iu;
      const Row r = row_of(d, t, i, j, k, h);
      const double wn = kr.wgt[t], sn = kr.sig[t];
      float cr = 0.f, cp = 0.f, ct = 0.f;
      if (i < nx) {
        const size_t q = t + 1;
        const Row rm = row_of(d, q, i + 1, j, k, h);
        cr = f32_rn(mul_rn(mul_rn(0.5 * (mul_rn(wn, r.c) + mul_rn(kr.wgt[q], rm.b)), sn), kr.sig[q]));
      }
      {
        const int jp = j == ny ? 1 : j + 1;
        const size_t q = cidx(d, i, jp, k);
        const Row rm = row_of(d, q, i, jp, k, h);
        cp = f32_rn(mul_rn(mul_rn(0.5 * (mul_rn(wn, r.e) + mul_rn(kr.wgt[q], rm.d)), sn), kr.sig[q]));
      }
      if (k < nz) {
        const size_t q = cidx(d, i, j, k + 1);
        const Row rm = row_of(d, q, i, j, k + 1, h);
        ct = f32_rn(mul_rn(mul_rn(0.5 * (mul_rn(wn, r.g) + mul_rn(kr.wgt[q], rm.f)), sn), kr.sig[q]));
      }
      const int o = (int)iu * kStripPitch + col;
      stage[o] = cr;
      stage[one + o] = cp;
      stage[2 * one + o] = ct;
    }
    __syncthreads();
    strip_out(kr, p, stage, kr.cr);
    strip_out(kr, p, stage + one, kr.cp);
    strip_out(kr, p, stage + 2 * one, kr.ct);
    __syncthreads();
  }
}

// Reciprocal pivots of every radial line (diagonal 1, off-diagonal cr):
// u_1 = 1, u_i = 1 - cr_{i-1}^2 / u_{i-1}; g = 1/u.  One thread per column;
// FP32 (the factorisation only preconditions).
__global__ void __launch_bounds__(32) kry_factor_kernel(Kry kr, SolverDev* sol) {
  constexpr int U = 16;  // loads in flight: the recurrence waits one memory latency per 16 radii
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= kr.ncol) return;
  float g = 1.f, cprev = 0.f;
  for (int i0 = 0; i0 < kr.nx; i0 += U) {
    float cc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) cc[u] = i0 + u < kr.nx ? kr.cr[(size_t)(i0 + u) * kr.ncol + c] : 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i0 + u >= kr.nx) break;
      const float piv = fmaf(-cprev * cprev, g, 1.f);
      if (!(piv > 0.f)) atomicExch(&sol->bad_weights, 1);
      g = 1.f / piv;
      kr.g[(size_t)(i0 + u) * kr.ncol + c] = g;
      cprev = cc[u];
    }
  }
}

// FP64 anchor: r = b - A x, its L1 norm, the scaled right-hand side
// Sigma W r of the inner system (FP32, line-major) and, with L2, its
// squared 2-norm; with WITH_B also ||b||_1 and ||Sigma W b||_2^2 (b does not
// change during a solve).  The last block writes the totals to
// sol->true_l1, sol->scratch[0], sol->rhsnorm, sol->scratch[1].  The
// residual is a chain of FP64 fused multiply-adds: GB300's FP64 pipe, not
// HBM, bounds this kernel.
template <bool L2, bool WITH_B>
__global__ void __launch_bounds__(kThreads) kry_anchor_kernel(Dev d, Kry kr, const double* __restrict__ x,
                                                              const double* __restrict__ b, int hypre,
                                                              double* partials, int nbmax, StripCut cut) {
  extern __shared__ float stage[];
  __shared__ double sh[32];
  __shared__ bool last;
  const int nx = d.nx, ny = d.ny;
  const size_t sj = (size_t)(nx + 4), sk = (size_t)(nx + 4) * (ny + 4);
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (unsigned int m = blockIdx.x; m < cut.pieces; m += gridDim.x) {
    const Strip p = strip_of(d, cut, m);
    for (unsigned int u = threadIdx.x; u < cut.by_len.d * p.cols; u += blockDim.x) {
      unsigned int iu;
      const int col = (int)div_rem(cut.by_len, u, iu), i = p.i0 + (int)iu + 1, j = p.j0 + col, k = p.k;
      if ((int)iu >= p.ni) continue;
      const size_t t = p.t0 + (unsigned int)(nx * col) + iu;
      const Row r = row_of(d, t, i, j, k, hypre != 0);
      const size_t q = hidx(d, i, j, k);
      const size_t qjm = (j == 1) ? hidx(d, i, ny, k) : q - sj;
      const size_t qjp = (j == ny) ? hidx(d, i, 1, k) : q + sj;
      const double bb = b_of(d, b, t, i, j, k, hypre != 0);
      // a zero coupling contributes nothing, whatever the ghost it points at holds
      double ax = r.a * x[q];
      ax = fma(r.b, r.b != 0.0 ? x[q - 1] : 0.0, ax);
      ax = fma(r.c, r.c != 0.0 ? x[q + 1] : 0.0, ax);
      ax = fma(r.d, r.d != 0.0 ? x[qjm] : 0.0, ax);
      ax = fma(r.e, r.e != 0.0 ? x[qjp] : 0.0, ax);
      ax = fma(r.f, r.f != 0.0 ? x[q - sk] : 0.0, ax);
      ax = fma(r.g, r.g != 0.0 ? x[q + sk] : 0.0, ax);
      const double rr = bb - ax;
      const double sw = mul_rn(kr.sig[t], kr.wgt[t]);
      const double rs = mul_rn(sw, rr);
      s[0] += fabs(rr);
      if (L2) s[1] = fma(rs, rs, s[1]);
      if (WITH_B) {
        const double bs = mul_rn(sw, bb);
        s[2] += fabs(hypre ? bb : b[t]);  // RHSNORM over every row (ppsor.f:33)
        s[3] = fma(bs, bs, s[3]);
      }
      stage[(int)iu * kStripPitch + col] = f32_rn(rs);
    }
    __syncthreads();
    strip_out(kr, p, stage, kr.r);
    if ((threadIdx.x & 31) < p.cols)
      for (int i = threadIdx.x >> 5; i < p.ni; i += blockDim.x >> 5)
        kr.e[strip_line(kr, p, i, threadIdx.x & 31)] = 0.f;
    __syncthreads();
  }
  for (int m = 0; m < 4; ++m) {
    const double v = block_sum(s[m], sh);
    if (threadIdx.x == 0) partials[m * nbmax + blockIdx.x] = v;
  }
  if (threadIdx.x == 0) {
    __threadfence();
    last = (atomicAdd(&d.sol->ticket2, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (last) {
    __threadfence();
    double tot[4];
    for (int m = 0; m < 4; ++m) tot[m] = block_sum_array(partials + m * nbmax, gridDim.x, sh);
    if (threadIdx.x == 0) {
      d.sol->true_l1 = tot[0];
      if (L2) d.sol->scratch[0] = tot[1];
      if (WITH_B) {
        d.sol->rhsnorm = tot[2];
        d.sol->scratch[1] = tot[3];
      }
      d.sol->ticket2 = 0;
    }
  }
}

// x += Sigma e (x a halo array, e line-major).
__global__ void __launch_bounds__(kThreads) kry_update_kernel(Dev d, Kry kr, double* x, StripCut cut) {
  extern __shared__ float stage[];
  const int nx = d.nx, lane = threadIdx.x & 31;
  for (unsigned int m = blockIdx.x; m < cut.pieces; m += gridDim.x) {
    const Strip p = strip_of(d, cut, m);
    __syncthreads();
    if (lane < p.cols)
      for (int i = threadIdx.x >> 5; i < p.ni; i += blockDim.x >> 5)
        stage[i * kStripPitch + lane] = kr.e[strip_line(kr, p, i, lane)];
    __syncthreads();
    for (unsigned int u = threadIdx.x; u < cut.by_len.d * p.cols; u += blockDim.x) {
      unsigned int iu;
      const int col = (int)div_rem(cut.by_len, u, iu);
      if ((int)iu >= p.ni) continue;
      const float e = stage[(int)iu * kStripPitch + col];
      x[hidx(d, p.i0 + (int)iu + 1, p.j0 + col, p.k)] +=
          mul_rn(kr.sig[p.t0 + (unsigned int)(nx * col) + iu], f64_of_f32(e));
    }
  }
}

// Column m of colour C (0: (j+k) even, 1: odd) in the red-black order of
// the columns; NY is even, so each theta row holds NY/2 of each colour.
__device__ __forceinline__ long long col_of(long long m, int C, int ny) {
  const long long half = ny >> 1;
  const long long k0 = m / half;
  const long long jj = m - k0 * half;
  return k0 * ny + 2 * jj + ((k0 + C) & 1);
}

// One radial line of block Jacobi for column c, by one thread.  With UPDATE,
// first r -= alpha s along the line.  Then z = T^-1 r by the factored
// tridiagonal T (forward: y_i = r_i - cr_{i-1} g_{i-1} y_{i-1}; backward:
// z_i = (y_i - cr_i z_{i+1}) g_i).  Returns this line's share of r.z, which is
// sum y_i^2 g_i.  y waits in shared memory (SHARED: `y`, one value per radius
// and thread), so that the backward pass reads two arrays and not four; where
// NX is too long for that it waits in z.  The loads of kLineBatch radii are
// issued before any of their stores (the compiler may not move a load above a
// store it cannot prove independent, and a warp stalls at the first use of a
// pending load), so a pass waits one memory latency per batch, not per radius.
constexpr int kLineBatch = 16;
template <bool UPDATE, bool SHARED>
__device__ __forceinline__ float line_pass(const Kry& k, unsigned int c0, float alpha, float* y) {
  constexpr int U = kLineBatch;
  // 32-bit offsets (a context holds fewer than 2^31 cells per array)
  const unsigned int ncol = (unsigned int)k.ncol;
  const int nx = k.nx;
  float yprev = 0.f, lprev = 0.f, dot = 0.f;
  for (int i0 = 0; i0 < nx; i0 += U) {
    const unsigned int qb = c0 + (unsigned int)i0 * ncol;
    float rr[U], cc[U], gg[U], ss[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i0 + u < nx) {
        const unsigned int q = qb + (unsigned int)u * ncol;
        rr[u] = k.r[q];
        cc[u] = k.cr[q];
        gg[u] = k.g[q];
        if (UPDATE) ss[u] = k.s[q];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i0 + u < nx) {
        const unsigned int q = qb + (unsigned int)u * ncol;
        float ri = rr[u];
        if (UPDATE) {
          ri = fmaf(-alpha, ss[u], ri);
          k.r[q] = ri;
        }
        const float v = fmaf(-lprev, yprev, ri);
        if (SHARED) y[(i0 + u) * kJacobiThreads] = v;
        else k.z[q] = v;
        dot = fmaf(v * gg[u], v, dot);
        lprev = cc[u] * gg[u];
        yprev = v;
      }
    }
  }
  float znext = 0.f;
  for (int i1 = nx - 1; i1 >= 0; i1 -= U) {
    const unsigned int qb = c0 + (unsigned int)i1 * ncol;
    float yy[U], cc[U], gg[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i1 - u >= 0) {
        const unsigned int q = qb - (unsigned int)u * ncol;
        yy[u] = SHARED ? y[(i1 - u) * kJacobiThreads] : k.z[q];
        cc[u] = k.cr[q];
        gg[u] = k.g[q];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i1 - u >= 0) {
        const unsigned int q = qb - (unsigned int)u * ncol;
        const float zi = fmaf(-cc[u], znext, yy[u]) * gg[u];
        k.z[q] = zi;
        znext = zi;
      }
    }
  }
  return dot;
}

// Line Gauss-Seidel in tiles of kTileCols radial lines, a tile by a group of threads:
// the group copies the lines to shared memory together (cp.async, everything
// in flight at once), forms the right-hand sides there, and one lane per line
// runs the recurrences on shared memory (forward y_i = b_i - cr_{i-1} g_{i-1}
// y_{i-1}, backward z_i = (y_i - cr_i z_{i+1}) g_i).  What bounded a pass with
// one thread per line on global memory was the memory latency per batch of
// radii, with seven warps (32,768 columns) or one (the 4,096 of a colour of
// 8,192) per SM.  A tile holds b (r), cr, g and s, each nx x kTileCols.
// (Block Jacobi, whose tiles are many, is faster with one thread per line: two
// tiles in flight per group take 205 KB of shared memory, and what L1 is left
// then holds too few copies in flight, 27-44 us a pass at 100x256x128.)
constexpr int kTileCols = 32;
__device__ __forceinline__ void group_sync(int group, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(threads) : "memory");
}
__device__ __forceinline__ void copy_async4(float* to, const float* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned int)__cvta_generic_to_shared(to)), "l"(from)
               : "memory");
}
// The threads of a group, and its tile (from value `at` on, in shared memory if
// SHARED, else in `global`).
struct Group {
  int id, threads, tid;
  unsigned int at;
  float* global;
};

// The recurrences of one lane's line; NB: z takes its share of r.z with the
// residual in the fourth array, else r.z = sum y_i^2 g_i.  Shared memory is
// read in batches of R radii before the batch's first write (the compiler
// cannot tell the arrays apart itself, and would wait for each read).
// Not inlined: among the other passes' live registers the recurrences were
// scheduled read by read, 60 clocks a radius instead of 12.
template <bool NB, bool SHARED>
__device__ __noinline__ float solve_line(int nx, unsigned int ncol, float* z, float* global, unsigned int at, int lane,
                                         bool valid, unsigned int c0) {
  constexpr int R = 8;
  float* tile = SHARED ? tile_sh + at : global + at;
  float *sb = tile + lane, *sc = sb + nx * kTileCols, *sg = sc + nx * kTileCols, *sr = sg + nx * kTileCols;
  float dot = 0.f, yprev = 0.f, lprev = 0.f;
  int i = 0;
  for (; i + R <= nx; i += R) {
    float bb[R], cc[R], gg[R];
#pragma unroll
    for (int u = 0; u < R; ++u) {
      bb[u] = sb[(i + u) * kTileCols];
      cc[u] = sc[(i + u) * kTileCols];
      gg[u] = sg[(i + u) * kTileCols];
    }
#pragma unroll
    for (int u = 0; u < R; ++u) {
      bb[u] = fmaf(-lprev, yprev, bb[u]);
      if (!NB) dot = fmaf(bb[u] * gg[u], bb[u], dot);
      lprev = cc[u] * gg[u];
      yprev = bb[u];
    }
#pragma unroll
    for (int u = 0; u < R; ++u) sb[(i + u) * kTileCols] = bb[u];
  }
  for (; i < nx; ++i) {
    const float g = sg[i * kTileCols], y = fmaf(-lprev, yprev, sb[i * kTileCols]);
    sb[i * kTileCols] = y;
    if (!NB) dot = fmaf(y * g, y, dot);
    lprev = sc[i * kTileCols] * g;
    yprev = y;
  }
  float znext = 0.f;
  for (i = nx - 1; i >= R - 1; i -= R) {
    float bb[R], cc[R], gg[R], rr[R];
#pragma unroll
    for (int u = 0; u < R; ++u) {
      bb[u] = sb[(i - u) * kTileCols];
      cc[u] = sc[(i - u) * kTileCols];
      gg[u] = sg[(i - u) * kTileCols];
      if (NB) rr[u] = sr[(i - u) * kTileCols];
    }
#pragma unroll
    for (int u = 0; u < R; ++u) {
      znext = fmaf(-cc[u], znext, bb[u]) * gg[u];
      if (NB) dot = fmaf(rr[u], znext, dot);
      if (valid) z[(unsigned int)(i - u) * ncol + c0] = znext;
    }
  }
  for (; i >= 0; --i) {
    znext = fmaf(-sc[i * kTileCols], znext, sb[i * kTileCols]) * sg[i * kTileCols];
    if (NB) dot = fmaf(sr[i * kTileCols], znext, dot);
    if (valid) z[(unsigned int)i * ncol + c0] = znext;
  }
  return valid ? dot : 0.f;
}

// One tile of lines of one colour (line `col` of this lane).  NB: the couplings
// to the four phi/theta neighbour columns, which all have the other colour,
// times their z are taken off the right-hand side (the red-black line
// Gauss-Seidel step).  Returns this thread's share of r.z.
template <bool UPDATE, bool NB, bool SHARED>
__device__ __forceinline__ float colour_lines(const Kry& k, const Group& g, long long col, bool valid, float alpha) {
  constexpr int U = 4;
  const int W = g.threads >> 5, nx = k.nx, lane = threadIdx.x & 31, warp = g.tid >> 5;
  // 32-bit offsets (a context holds fewer than 2^31 cells per array)
  const unsigned int ncol = (unsigned int)k.ncol, c0 = (unsigned int)(valid ? col : 0);
  float* tile = SHARED ? tile_sh + g.at : g.global + g.at;
  float *sb = tile + lane, *sc = sb + nx * kTileCols, *sg = sc + nx * kTileCols, *sr = sg + nx * kTileCols;
  unsigned int cjp = c0, cjm = c0, ckp = c0, ckm = c0;
  bool hkm = false;
  if (NB) {  // theta neighbours outside the grid read column c0 with a zero coupling
    const unsigned int ny = (unsigned int)k.ny, k0 = c0 / ny, j0 = c0 - k0 * ny;
    cjp = j0 == ny - 1 ? c0 - (ny - 1) : c0 + 1;
    cjm = j0 == 0 ? c0 + (ny - 1) : c0 - 1;
    hkm = k0 > 0;
    if ((int)k0 + 1 < k.nz) ckp = c0 + ny;
    if (hkm) ckm = c0 - ny;
  }
  group_sync(g.id, g.threads);  // the tile before this one is solved
  // each thread copies the values that it alone reads back
  for (int i = warp; i < nx; i += W) {
    const unsigned int q = (unsigned int)i * ncol + c0;
    const int o = i * kTileCols;
    if (SHARED) {
      copy_async4(sb + o, k.r + q);
      if (UPDATE) copy_async4(sr + o, k.s + q);
      copy_async4(sc + o, k.cr + q);
      copy_async4(sg + o, k.g + q);
    } else {
      sb[o] = k.r[q];
      if (UPDATE) sr[o] = k.s[q];
      sc[o] = k.cr[q];
      sg[o] = k.g[q];
    }
  }
  bool waited = false;
  for (int i0 = warp; i0 < nx; i0 += W * U) {
    float nb[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + W * u;
      nb[u] = 0.f;
      if (NB && i < nx) {
        const unsigned int o = (unsigned int)i * ncol;
        const float ctm = hkm ? k.ct[o + ckm] : 0.f;
        nb[u] = fmaf(k.cp[o + c0], k.z[o + cjp],
                fmaf(k.cp[o + cjm], k.z[o + cjm], fmaf(k.ct[o + c0], k.z[o + ckp], ctm * k.z[o + ckm])));
      }
    }
    if (!waited) asm volatile("cp.async.wait_all;" ::: "memory");
    waited = true;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + W * u, o = i * kTileCols;
      if (i < nx) {
        float ri = sb[o];
        if (UPDATE) {
          ri = fmaf(-alpha, sr[o], ri);
          if (valid) k.r[(unsigned int)i * ncol + c0] = ri;
        }
        if (NB) sr[o] = ri;
        sb[o] = NB ? ri - nb[u] : ri;
      }
    }
  }
  group_sync(g.id, g.threads);
  return g.tid < 32 ? solve_line<NB, SHARED>(nx, ncol, k.z, g.global, g.at, lane, valid, c0) : 0.f;
}

__device__ __forceinline__ float4 ldf4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void stf4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float4 axpy4(float a, float4 x, float4 y) {
  return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}
__device__ __forceinline__ float4 fma4(float4 a, float4 b, float4 c) {
  return make_float4(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y), fmaf(a.z, b.z, c.z), fmaf(a.w, b.w, c.w));
}
__device__ __forceinline__ float4 keep4(bool on, float4 v) { return on ? v : make_float4(0.f, 0.f, 0.f, 0.f); }

// The operator pass on four cells q..q+3 of one phi row (NY a multiple of
// four, q a multiple of four): e += alpha_prev p_old (the previous
// iteration's update of e, deferred to here so that the line pass reads
// fewer arrays), p_new = z + beta p_old, s = S p_new; returns p_new . s.
// Every load is issued before the first arithmetic (neighbours that do not
// exist are read at q and their couplings zeroed), so the quad waits one
// memory latency.
__device__ __forceinline__ float op_quad(const Kry& k, const float* po, float* pn, float beta, float alpha_prev,
                                         long long q) {
  const long long ncol = k.ncol;
  const int ny = k.ny;
  const long long il = q / ncol;
  const long long cc = q - il * ncol;
  const int j0 = (int)(cc % ny);
  const long long k0 = cc / ny;
  const bool hn = il + 1 < k.nx, hs = il > 0, ht = k0 + 1 < k.nz, hb = k0 > 0;
  const long long qn = hn ? q + ncol : q, qs = hs ? q - ncol : q;
  const long long qt = ht ? q + ny : q, qb = hb ? q - ny : q;
  const long long qm = j0 == 0 ? q + ny - 1 : q - 1;   // phi neighbours (periodic)
  const long long qp = j0 + 4 == ny ? q + 4 - ny : q + 4;
  const float4 zc = ldf4(k.z + q), oc = ldf4(po + q), ec = ldf4(k.e + q);
  const float4 zn = ldf4(k.z + qn), on = ldf4(po + qn), zs = ldf4(k.z + qs), os = ldf4(po + qs);
  const float4 zt = ldf4(k.z + qt), ot = ldf4(po + qt), zb = ldf4(k.z + qb), ob = ldf4(po + qb);
  const float4 crn = ldf4(k.cr + q), crs = ldf4(k.cr + qs), ctt = ldf4(k.ct + q), ctb = ldf4(k.ct + qb);
  const float4 cp = ldf4(k.cp + q);
  const float zm = k.z[qm], om = po[qm], zp = k.z[qp], op = po[qp], cl = k.cp[qm];
  stf4(k.e + q, axpy4(alpha_prev, oc, ec));
  const float4 pc = axpy4(beta, oc, zc);
  float4 sv = pc;
  sv = fma4(keep4(hn, crn), axpy4(beta, on, zn), sv);
  sv = fma4(keep4(hs, crs), axpy4(beta, os, zs), sv);
  sv = fma4(keep4(ht, ctt), axpy4(beta, ot, zt), sv);
  sv = fma4(keep4(hb, ctb), axpy4(beta, ob, zb), sv);
  const float pl = fmaf(beta, om, zm), pr = fmaf(beta, op, zp);
  sv.x = fmaf(cp.x, pc.y, fmaf(cl, pl, sv.x));
  sv.y = fmaf(cp.y, pc.z, fmaf(cp.x, pc.x, sv.y));
  sv.z = fmaf(cp.z, pc.w, fmaf(cp.y, pc.y, sv.z));
  sv.w = fmaf(cp.w, pr, fmaf(cp.z, pc.z, sv.w));
  stf4(pn + q, pc);
  stf4(k.s + q, sv);
  return fmaf(pc.x, sv.x, fmaf(pc.y, sv.y, fmaf(pc.z, sv.z, pc.w * sv.w)));
}

// The same for one cell (NY not a multiple of four).
__device__ __forceinline__ float op_one(const Kry& k, const float* po, float* pn, float beta, float alpha_prev,
                                        long long q) {
  const long long ncol = k.ncol;
  const int ny = k.ny;
  const long long il = q / ncol;
  const long long cc = q - il * ncol;
  const int j0 = (int)(cc % ny);
  const long long k0 = cc / ny;
  const bool hn = il + 1 < k.nx, hs = il > 0, ht = k0 + 1 < k.nz, hb = k0 > 0;
  const long long qn = hn ? q + ncol : q, qs = hs ? q - ncol : q;
  const long long qt = ht ? q + ny : q, qb = hb ? q - ny : q;
  const long long qm = j0 == 0 ? q + ny - 1 : q - 1;
  const long long qp = j0 == ny - 1 ? q - (ny - 1) : q + 1;
  const float zc = k.z[q], oc = po[q], ec = k.e[q];
  const float zn = k.z[qn], on = po[qn], zs = k.z[qs], os = po[qs], zt = k.z[qt], ot = po[qt];
  const float zb = k.z[qb], ob = po[qb], zm = k.z[qm], om = po[qm], zp = k.z[qp], op = po[qp];
  const float crn = k.cr[q], crs = k.cr[qs], ctt = k.ct[q], ctb = k.ct[qb], cpp = k.cp[q], cpm = k.cp[qm];
  k.e[q] = fmaf(alpha_prev, oc, ec);
  const float pc = fmaf(beta, oc, zc);
  float sv = pc;
  sv = fmaf(hn ? crn : 0.f, fmaf(beta, on, zn), sv);
  sv = fmaf(hs ? crs : 0.f, fmaf(beta, os, zs), sv);
  sv = fmaf(ht ? ctt : 0.f, fmaf(beta, ot, zt), sv);
  sv = fmaf(hb ? ctb : 0.f, fmaf(beta, ob, zb), sv);
  sv = fmaf(cpp, fmaf(beta, op, zp), sv);
  sv = fmaf(cpm, fmaf(beta, om, zm), sv);
  pn[q] = pc;
  k.s[q] = sv;
  return pc * sv;
}

// z = M^-1 r for the preconditioner M, with UPDATE first r -= alpha s.
// SGS: `sweeps` symmetric red-black line Gauss-Seidel sweeps from z = 0
// (red lines, then black lines against the new red z, red against the new
// black, ...: 2 sweeps + 1 colour passes, a grid barrier between passes; two
// symmetric sweeps in a row share their middle red pass), a symmetric
// preconditioner; otherwise the radial line solve of every column (block
// Jacobi).  acc gains this thread's share of r.z (from each colour's last
// pass).  False if a barrier gave up.
template <bool UPDATE, bool SGS, bool SHARED>
__device__ __forceinline__ bool precondition(const Kry& k, SolverDev* sol, unsigned int nb, float alpha, float& acc,
                                             int sweeps, unsigned long long& passed, const Group& g) {
  if (!SGS) {  // the warps of all blocks take groups of 32 neighbouring columns in turn
    const long long stride = (long long)(blockDim.x >> 5) * nb * 32;
    for (long long c = ((long long)(threadIdx.x >> 5) * nb + blockIdx.x) * 32 + (threadIdx.x & 31); c < k.ncol; c += stride)
      acc += line_pass<UPDATE, SHARED>(k, (unsigned int)c, alpha, tile_sh + threadIdx.x);
    return true;
  }
  // tiles are dealt to the blocks first, then to the groups of a block
  const int groups = (int)blockDim.x / g.threads, lane = threadIdx.x & 31;
  const long long first = (long long)g.id * nb + blockIdx.x, step = (long long)groups * nb;
  const long long half = k.ncol >> 1;
  for (long long m0 = first * kTileCols; m0 < half; m0 += step * kTileCols)
    (void)colour_lines<UPDATE, false, SHARED>(k, g, col_of(m0 + lane, 0, k.ny), m0 + lane < half, alpha);
  if (!grid_sync(sol, nb, passed)) return false;
  float ab = 0.f;  // r.z of the black lines' first pass (their last with one sweep)
  for (long long m0 = first * kTileCols; m0 < half; m0 += step * kTileCols)
    ab += colour_lines<UPDATE, true, SHARED>(k, g, col_of(m0 + lane, 1, k.ny), m0 + lane < half, alpha);
  if (sweeps == 1) acc += ab;
#pragma unroll 1
  for (int p = 2; p <= 2 * sweeps; ++p) {
    if (!grid_sync(sol, nb, passed)) return false;
    float ap = 0.f;
    for (long long m0 = first * kTileCols; m0 < half; m0 += step * kTileCols)
      ap += colour_lines<false, true, SHARED>(k, g, col_of(m0 + lane, p & 1, k.ny), m0 + lane < half, 0.f);
    if (p >= 2 * sweeps - 1) acc += ap;  // the last pass of its colour
  }
  return true;
}

// The FP32 PCG iteration on S e = r from e = 0 (r, e set by the anchor).
// Line phases: tiles of 32 columns, dealt to the groups of threads of all
// blocks.  Operator phase: p_new = z + beta p (p read from
// p[cur], written to p[1-cur], so that neighbours read the old values),
// s = S p_new, and the previous iteration's e += alpha p.  Every block forms
// alpha and beta from all block partials in the same fixed order, so all
// blocks take the same decisions.  The run ends when sqrt(r.z / r0.z0) <=
// stop_ratio, after kPcgStall iterations without a new minimum of r.z (the
// FP32 floor), on a non-positive p.s, or after maxit iterations; the last
// iteration's e update is then applied.  maxit = 0 only computes r0.z0
// (sol->scratch[2]).
template <bool SGS, bool SHARED>
__global__ void __launch_bounds__(SGS ? kGsThreads : kJacobiThreads, 1) pcg32_persistent(Kry k, SolverDev* sol, double* partials,
                                                                   int maxit, double stop_ratio, int sweeps,
                                                                   float* tiles, int groups) {
  __shared__ double sh[33];
  const unsigned int nb = gridDim.x;
  const int it0 = sol->iter;
  unsigned long long passed = 0;  // grid barriers this block has passed
  const long long n = k.n;
  const int ny = k.ny;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nth = (long long)gridDim.x * blockDim.x;
  Group g;
  g.threads = (int)blockDim.x / groups;
  g.id = (int)threadIdx.x / g.threads;
  g.tid = (int)threadIdx.x - g.id * g.threads;
  const unsigned int len = 4u * (unsigned int)k.nx * kTileCols;
  g.at = (unsigned int)g.id * len;
  g.global = SHARED ? nullptr : tiles + (size_t)blockIdx.x * groups * len;

  // z0 = T^-1 r0, gamma0 = r0.z0.  Per-thread partial sums (a few hundred
  // terms) are FP32 -- GB300's FP64 pipe is narrow -- and widened to FP64
  // for the block and grid sums.
  float acc = 0.f;
  if (!precondition<false, SGS, SHARED>(k, sol, nb, 0.f, acc, sweeps, passed, g)) return;
  double gamma;
  if (!grid_sum(sol, nb, passed, (double)acc, partials, sh, gamma)) return;
  const double gamma0 = gamma;
  if (blockIdx.x == 0 && threadIdx.x == 0) sol->scratch[2] = gamma0;
  if (maxit <= 0 || !(gamma0 > 0.0) || !isfinite(gamma0)) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && !isfinite(gamma0)) sol->nonfinite = 1;
    return;
  }
  const double stop2 = stop_ratio * stop_ratio * gamma0;
  double gmin = gamma0;
  int since_min = 0;
  float beta = 0.f, alpha_prev = 0.f;
  int cur = 0;
  bool pending = false;  // e += alpha_prev p[cur] still to be applied
  for (int it = 1; it <= maxit; ++it) {
    const float* po = cur ? k.p[1] : k.p[0];
    float* pn = cur ? k.p[0] : k.p[1];
    // operator phase
    acc = 0.f;
    const float ap = pending ? alpha_prev : 0.f;
    if ((ny & 3) == 0) {
      for (long long g = tid; g < (n >> 2); g += nth) acc += op_quad(k, po, pn, beta, ap, g << 2);
    } else {
      for (long long q = tid; q < n; q += nth) acc += op_one(k, po, pn, beta, ap, q);
    }
    pending = false;
    double ps;
    if (!grid_sum(sol, nb, passed, (double)acc, partials, sh, ps)) return;
    if (!(ps > 0.0) || !isfinite(ps)) {  // breakdown: S p_new not positive (rounding)
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        sol->stalled = 1;
        if (!isfinite(ps)) sol->nonfinite = 1;
      }
      break;
    }
    const float alpha = (float)(gamma / ps);
    // line phase: r -= alpha s, z = M^-1 r, r.z
    acc = 0.f;
    if (!precondition<true, SGS, SHARED>(k, sol, nb, alpha, acc, sweeps, passed, g)) return;
    alpha_prev = alpha;
    pending = true;
    cur = 1 - cur;  // p[cur] is now this iteration's p
    double gnew;
    if (!grid_sum(sol, nb, passed, (double)acc, partials, sh, gnew)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) sol->iter = it0 + it;
    if (!isfinite(gnew)) {
      if (blockIdx.x == 0 && threadIdx.x == 0) sol->nonfinite = 1;
      break;
    }
    if (gnew < gmin) {
      gmin = gnew;
      since_min = 0;
    } else if (++since_min >= kPcgStall) {
      if (blockIdx.x == 0 && threadIdx.x == 0) sol->stalled = 1;
      break;
    }
    if (!(gnew > stop2)) {
      if (blockIdx.x == 0 && threadIdx.x == 0) sol->done = 1;
      break;
    }
    beta = (float)(gnew / gamma);
    gamma = gnew;
  }
  if (pending) {
    const float* pl = cur ? k.p[1] : k.p[0];
    for (long long q = tid; q < n; q += nth) k.e[q] = fmaf(alpha_prev, pl[q], k.e[q]);
  }
}

int grid_cells(long long n) {
  int nb = grid_for(n);
  return nb > 1024 ? 1024 : nb;
}

KryWork* kry_work(ttfld_ctx* c) {
  if (c->krylov) return (KryWork*)c->krylov;
  const Dev& d = c->d;
  KryWork* w = (KryWork*)calloc(1, sizeof(KryWork));
  if (!w) return nullptr;
  Kry& k = w->k;
  k.nx = d.nx; k.ny = d.ny; k.nz = d.nz;
  k.n = (long long)ncell(d);
  k.ncol = (long long)d.ny * d.nz;
  const size_t n = (size_t)k.n;
  const size_t bytes = n * (10 * sizeof(float) + 2 * sizeof(double));
  if (cudaMalloc(&w->mem, bytes) != cudaSuccess) {
    free(w);
    return nullptr;
  }
  double* dp = (double*)w->mem;
  k.sig = dp; dp += n;
  k.wgt = dp; dp += n;
  float* fp = (float*)dp;
  float** arrs[] = {&k.cr, &k.cp, &k.ct, &k.g, &k.e, &k.r, &k.z, &k.s, &k.p[0], &k.p[1]};
  for (float** a : arrs) { *a = fp; fp += n; }
  c->krylov = w;
  return w;
}

int poll_sol(ttfld_ctx* c) {
  TT_CHECK(cudaMemcpyAsync(c->host_sol, c->sol, sizeof(SolverDev), cudaMemcpyDeviceToHost, c->stream));
  TT_CHECK(cudaStreamSynchronize(c->stream));
  if (c->host_sol->bar_timeout) {
    fprintf(stderr, "ttfld: a grid barrier of the PCG kernel timed out\n");
    return TTFLD_E_CUDA;
  }
  return 0;
}

// Launch shape of the PCG kernel, one block per SM.  Line Gauss-Seidel: a
// colour has few tiles, and what they wait for is the reads of their
// neighbours, so a block has as many groups as it has tiles, up to three and
// to what fits in shared memory; a line too long for that (NX > 440) keeps its
// tile in global memory.  Block Jacobi: the forward results of a line wait in
// shared memory up to kJacobiShared, beyond which L1 would get too small for
// the loads in flight.
constexpr size_t kJacobiShared = 168 * 1024;
struct PcgShape {
  int blocks, threads, groups;
  size_t smem;
  bool shared;
};
const void* pcg_kernel(bool gs, bool shared) {
  if (shared) return gs ? (const void*)pcg32_persistent<true, true> : (const void*)pcg32_persistent<false, true>;
  return gs ? (const void*)pcg32_persistent<true, false> : (const void*)pcg32_persistent<false, false>;
}
PcgShape pcg_shape(const Kry& k, bool gs) {
  int dev = 0, sms = 0, coop = 0, room = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&room, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  PcgShape p{0, gs ? kGsThreads : kJacobiThreads, 1, 0, false};
  if (!coop || sms <= 0) return p;
  if (gs) {
    const size_t tile = (size_t)4 * k.nx * kTileCols * sizeof(float);
    const int fit = (int)(((size_t)room - 1024) / tile);
    p.shared = fit > 0;
    if (p.shared) {
      const long long tiles = (k.ncol / 2 + kTileCols - 1) / kTileCols, per = (tiles + sms - 1) / sms;
      p.groups = per < 3 ? (int)per : 3;
      if (p.groups > fit) p.groups = fit;
      p.smem = (size_t)p.groups * tile;
    }
  } else {
    const size_t y = (size_t)k.nx * kJacobiThreads * sizeof(float);
    p.shared = y <= kJacobiShared;
    p.smem = p.shared ? y : 0;
  }
  const void* kern = pcg_kernel(gs, p.shared);
  int per_sm = 0;
  if (smem_room(kern) < p.smem ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, p.threads, p.smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return p;
  }
  const long long need = (k.n + 255) / 256;
  p.blocks = (int)(need < sms ? need : sms);
  if (p.blocks > kMaxPartials) p.blocks = kMaxPartials;
  return p;
}

// One inner run; returns its iterations in *its.
// gs: 0 block-Jacobi radial lines, m >= 1 m symmetric line Gauss-Seidel sweeps.
int launch_inner(ttfld_ctx* c, KryWork* w, int maxit, double stop_ratio, int gs, int* its) {
  const PcgShape shape = pcg_shape(w->k, gs > 0);
  if (shape.blocks > 0 && gs > 0 && !shape.shared && !w->tiles)
    TT_CHECK(cudaMalloc((void**)&w->tiles, (size_t)shape.blocks * 4 * w->k.nx * kTileCols * sizeof(float)));
  if (shape.blocks <= 0) {
    fprintf(stderr, "ttfld: the PCG solver needs cooperative launch\n");
    return TTFLD_E_UNSUPPORTED;
  }
  TT_CHECK(cudaMemsetAsync(w->k.p[0], 0, (size_t)w->k.n * sizeof(float), c->stream));
  TT_CHECK(cudaMemsetAsync(&c->sol->iter, 0, sizeof(int), c->stream));
  TT_CHECK(cudaMemsetAsync(&c->sol->done, 0, sizeof(int), c->stream));
  TT_CHECK(cudaMemsetAsync(&c->sol->stalled, 0, sizeof(int), c->stream));
  Kry k = w->k;
  SolverDev* sol = c->sol;
  double* partials = c->partials;
  int sweeps = gs > 0 ? gs : 1;
  float* tiles = w->tiles;
  int groups = shape.groups;
  void* args[] = {&k, &sol, &partials, &maxit, &stop_ratio, &sweeps, &tiles, &groups};
  const void* kern = pcg_kernel(gs > 0, shape.shared);
  TT_CHECK(cudaMemsetAsync(&sol->arrivals, 0, sizeof(unsigned long long), c->stream));  // grid barrier
  TT_CHECK(cudaLaunchCooperativeKernel(kern, dim3(shape.blocks), dim3(shape.threads), args, shape.smem, c->stream));
  count_launches(1);
  int rc = poll_sol(c);
  if (rc) return rc;
  if (c->host_sol->nonfinite) return TTFLD_E_NONFINITE;
  *its = c->host_sol->iter;
  return 0;
}

// The pieces of a grid's strips, the blocks that walk them, and the shared
// memory of `arrays` staged pieces.  Strips are cut until there are two pieces
// per SM, but to no less than 16 radii (two lines of an FP64 array), and in any
// case to what 200 KB hold.  Uncut, 96 strips leave a third of the SMs without a
// block and the others with one: at 180x64x48 the couplings took 101 us, an
// anchor 57 and an update 39, cut 31, 34 and 14 (a PCG solve 1117 -> 976 us; 883
// -> 839 at 100x64x70, 960 -> 883 at 98x70x52).  Seven pieces per SM instead of
// two: 1014 us at 180x64x48, and 2-3 % slower than uncut at 64x96x100 and
// 30x200x100, where the pieces were then 16 radii.
constexpr int kStripPieces = 304, kStripBlocks = 1024;
struct StripShape {
  StripCut cut;
  int blocks;
  size_t smem;
};
StripShape strip_shape(const Kry& k, const void* kernel, int arrays) {
  StripShape s;
  const unsigned int strips = (unsigned int)k.nz * (((unsigned int)k.ny + kStripCols - 1) / kStripCols);
  const unsigned int nx = (unsigned int)k.nx, want = (kStripPieces + strips - 1) / strips;
  const size_t radius = (size_t)arrays * kStripPitch * sizeof(float);
  unsigned int len = (nx + want - 1) / want;
  if (len < 16) len = nx < 16 ? nx : 16;
  if (len * radius > 200 * 1024) len = (unsigned int)(200 * 1024 / radius);
  if (len * radius > 48 * 1024 && smem_room(kernel) < len * radius) len = (unsigned int)(48 * 1024 / radius);
  s.cut.per = (nx + len - 1) / len;
  s.cut.pieces = strips * s.cut.per;
  s.cut.by_len = fast_div((int)len);
  s.blocks = s.cut.pieces < kStripBlocks ? (int)s.cut.pieces : kStripBlocks;
  s.smem = len * radius;
  return s;
}

template <bool L2, bool WITH_B>
int launch_anchor(ttfld_ctx* c, KryWork* w, const double* x, const double* b, int h) {
  const StripShape s = strip_shape(w->k, (const void*)kry_anchor_kernel<L2, WITH_B>, 1);
  kry_anchor_kernel<L2, WITH_B><<<s.blocks, kThreads, s.smem, c->stream>>>(c->d, w->k, x, b, h, c->partials, 1024,
                                                                           s.cut);
  count_launches(1);
  TT_CHECK_LAUNCH();
  return 0;
}

int anchor(ttfld_ctx* c, KryWork* w, const double* x, const double* b, bool hypre, bool l2, bool with_b) {
  const int h = hypre ? 1 : 0;
  const int rc = l2 ? (with_b ? launch_anchor<true, true>(c, w, x, b, h) : launch_anchor<true, false>(c, w, x, b, h))
                    : (with_b ? launch_anchor<false, true>(c, w, x, b, h) : launch_anchor<false, false>(c, w, x, b, h));
  return rc ? rc : poll_sol(c);
}

// Factor the system (weights, couplings, line pivots).
int prepare(ttfld_ctx* c, KryWork* w, bool hypre) {
  const int nb = grid_cells(w->k.n);
  TT_CHECK(cudaMemsetAsync(&c->sol->bad_weights, 0, sizeof(int), c->stream));
  kry_weights_kernel<<<nb, kThreads, 0, c->stream>>>(c->d, w->k, hypre ? 1 : 0);
  const StripShape s = strip_shape(w->k, (const void*)kry_couplings_kernel, 3);
  kry_couplings_kernel<<<s.blocks, kThreads, s.smem, c->stream>>>(c->d, w->k, hypre ? 1 : 0, s.cut);
  kry_factor_kernel<<<(unsigned int)((w->k.ncol + 31) / 32), 32, 0, c->stream>>>(w->k, c->sol);
  count_launches(3);
  TT_CHECK_LAUNCH();
  return 0;
}

// PCG with FP64 defect correction on x (halo array, holding the initial
// iterate).  l2 = false: stop on ||b - A x||_1 / ||b||_1 <= tol (the SOR
// system's rule); l2 = true: on ||Sigma W (b - A x)||_2 / ||Sigma W b||_2 <=
// tol (the hypre system's PCG rule on the symmetric form).  budget bounds
// the PCG iterations.  With guess_test, the initial iterate is kept only if
// its preconditioned residual norm r.z is below that of the zero iterate.
int pcg_core(ttfld_ctx* c, double* x, const double* b, bool hypre, double tol, long long budget, bool l2, int gs,
             int guess_test, int* fallback, ttfld_solve_stats* st) {
  KryWork* w = kry_work(c);
  if (!w) return TTFLD_E_CUDA;
  TT_CHECK(cudaMemsetAsync(c->sol, 0, sizeof(SolverDev), c->stream));
  int rc = prepare(c, w, hypre);
  if (rc) return rc;
  if (fallback) *fallback = 0;
  if ((rc = anchor(c, w, x, b, hypre, l2, true))) return rc;
  if (c->host_sol->bad_weights) {
    fprintf(stderr, "ttfld: PCG needs EVAL8 < 0 on every coupled row (the symmetrising weight)\n");
    return TTFLD_E_UNSUPPORTED;
  }
  if (guess_test) {
    int its = 0;
    if ((rc = launch_inner(c, w, 0, 0.0, gs, &its))) return rc;
    const double g_guess = c->host_sol->scratch[2];
    // the zero iterate: r = b
    double* zero_x = c->guess_tmp;
    if (!zero_x) {
      TT_CHECK(cudaMalloc((void**)&c->guess_tmp, nhalo(c->d) * 8));
      zero_x = c->guess_tmp;
    }
    TT_CHECK(cudaMemsetAsync(zero_x, 0, nhalo(c->d) * 8, c->stream));
    if ((rc = anchor(c, w, zero_x, b, hypre, l2, false)) || (rc = launch_inner(c, w, 0, 0.0, gs, &its))) return rc;
    const double g_zero = c->host_sol->scratch[2];
    if (!(g_guess < g_zero)) {
      TT_CHECK(cudaMemsetAsync(x, 0, nhalo(c->d) * 8, c->stream));
      if (fallback) *fallback = 1;
      // the anchor of the zero iterate is current
    } else if ((rc = anchor(c, w, x, b, hypre, l2, false))) {
      return rc;
    }
  }
  long long total = 0;
  int anchors = 0, status = TTFLD_OK, slow = 0, stalls = 0;
  double prev = INFINITY, ratio = INFINITY;
  for (;;) {
    const SolverDev& h = *c->host_sol;
    ratio = l2 ? (h.scratch[1] > 0.0 ? sqrt(h.scratch[0] / h.scratch[1]) : 0.0)
               : (h.rhsnorm > 0.0 ? h.true_l1 / h.rhsnorm : 0.0);
    if (!isfinite(ratio)) return TTFLD_E_NONFINITE;
    if (!(ratio > tol)) break;
    if (total >= budget) { status = TTFLD_MAXITER; break; }
    // an anchor that does not halve the residual twice in a row: the
    // symmetric part is too far from the rows (or FP32 cannot resolve them)
    if (ratio > 0.5 * prev) {
      if (++slow >= 2) { status = TTFLD_MAXITER; break; }
    } else {
      slow = 0;
    }
    prev = ratio;
    double target = 0.3 * tol / ratio;
    if (target < kInnerReduce) target = kInnerReduce;
    long long left = budget - total;
    int its = 0;
    if ((rc = launch_inner(c, w, (int)(left < 1000000 ? left : 1000000), target, gs, &its))) return rc;
    total += its;
    ++anchors;
    if (c->host_sol->stalled) ++stalls;
    const StripShape up = strip_shape(w->k, (const void*)kry_update_kernel, 1);
    kry_update_kernel<<<up.blocks, kThreads, up.smem, c->stream>>>(c->d, w->k, x, up.cut);
    count_launches(1);
    TT_CHECK_LAUNCH();
    if ((rc = anchor(c, w, x, b, hypre, l2, false))) return rc;
  }
  // SOLVE_WITH_SOR leaves the phi halo of DELTA_ER refreshed (PLANETSHIFT(8)
  // after the last colour); SOLVE_WITH_HYPRE writes the interior only and its
  // caller shifts (ppenergy.f:353-356)
  if (!hypre && ((rc = halo_shift(c, x)) || (rc = pole_shift(c, x)))) return rc;
  if (st) {
    st->sor_iter = (int)total;
    st->corrections = anchors;
    // rnorm / rhsnorm is the stopping measure (L1, or the scaled 2-norm)
    st->rhsnorm = l2 ? sqrt(c->host_sol->scratch[1]) : c->host_sol->rhsnorm;
    st->rnorm = l2 ? sqrt(c->host_sol->scratch[0]) : c->host_sol->true_l1;
    st->true_resid_l1 = c->host_sol->true_l1;
    st->status = status;
    st->stalls = stalls;
  }
  return status;
}

}  // namespace

int solve_pcg(ttfld_ctx* c, double* x, const double* b, ttfld_solve_stats* st, int guess_test, int* fallback) {
  const long long budget = c->opts.max_sweeps > 0 ? c->opts.max_sweeps : (long long)c->d.itmax;
  return pcg_core(c, x, b, false, c->opts.tol, budget, false, 0, guess_test, fallback, st);
}

void krylov_free(ttfld_ctx* c) {
  KryWork* w = (KryWork*)c->krylov;
  if (!w) return;
  if (w->mem) cudaFree(w->mem);
  if (w->tiles) cudaFree(w->tiles);
  free(w);
  c->krylov = nullptr;
}

}  // namespace ttfld

extern "C" {

int ttfld_solve_with_hypre(ttfld_ctx* c, double tol, int maxit, ttfld_solve_stats* st) {
  using namespace ttfld;
  if (!c) return TTFLD_E_ARGS;
  if (c->d.poles) return TTFLD_E_UNSUPPORTED;  // hypre's pole graph (pphypre.f:458-540) is not built
  if (!(tol > 0.0)) tol = 1e-6;  // pphypre.f:45
  if (maxit <= 0) maxit = 50;    // pphypre.f:54-55
  TT_CHECK(cudaSetDevice(c->device));
  ttfld_solve_stats local{};
  if (!st) st = &local;
  int rc = fill_sor_matrix(c, false);  // the 7-point rows; b is taken from RHS_ER as it is
  if (rc) return rc;
  Dev d = c->d;
  double* x = d.DELTA_ER;
  // hypre's PCG is preconditioned by a multigrid cycle, which keeps its
  // iteration count nearly independent of the grid; the line Gauss-Seidel
  // preconditioner here needs more iterations on finer (phi, theta) grids.
  // Its strength is the number m of symmetric sweeps per application: a
  // solve that reaches the iteration cap before tol is run again from
  // x = 1 with m raised from the rate that solve showed (iterations scale
  // about as m^-1/2), and the context keeps m for its later solves.
  int m = c->hypre_gs > 0 ? c->hypre_gs : 1;
  TT_CHECK(cudaEventRecord(c->ev0, c->stream));
  for (;;) {
    // x = 1 in the interior (pphypre.f:136); the halo is left as it is, as
    // SOLVE_WITH_HYPRE only writes delta_ER(1:NX,1:NY,1:NZ) (pphypre.f:84-92)
    launch_box(c->stream, box(1, d.nx, 1, d.ny, 1, d.nz), [=] __device__(int i, int j, int k) { x[hidx(d, i, j, k)] = 1.0; });
    TT_CHECK_LAUNCH();
    rc = pcg_core(c, x, d.RHS, true, tol, maxit, true, m, 0, nullptr, st);
    if (rc != TTFLD_MAXITER || m >= kMaxGsSweeps) break;
    const double ratio = st->rhsnorm > 0.0 ? st->rnorm / st->rhsnorm : 1.0;
    double grow = 4.0;
    if (ratio > 0.0 && ratio < 1.0) {
      const double need = maxit * log(tol) / log(ratio);  // iterations at this m, at this rate
      const double f = need / (0.8 * maxit);
      grow = f * f;
    }
    int m2 = (int)ceil(m * (grow < 2.0 ? 2.0 : grow));
    m = m2 < kMaxGsSweeps ? m2 : kMaxGsSweeps;
  }
  c->hypre_gs = m;
  st->gs_sweeps = m;
  TT_CHECK(cudaEventRecord(c->ev1, c->stream));
  TT_CHECK(cudaEventSynchronize(c->ev1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, c->ev0, c->ev1);
  st->solve_ms = ms;
  c->last_solve_ms = ms;
  return rc;
}

}  // extern "C"
