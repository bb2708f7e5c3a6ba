// ttfld_raddif.cu -- the IRAD=1 radiation step: RADDIF (pprad.f:1-38) with
// DIFFEL (pprad.f:40-72), SOLVMAT (ppmat.f:1-186) and RADIATIVEBOUND
// (ppbou.f:2049-2299).
//
// RADDIF sets ER = arad T^4, forms the diffusion couplings AX..CZ from DIFF's
// face coefficients, B = c_v rho / (dt 4 arad T^3) - sum of the couplings and
// RHS = ER c_v rho / (dt 4 arad T^3), solves B ER + sum(couplings * ER_nb) =
// RHS for ER by red-black SOR on ER itself, and returns T = (ER/arad)^(1/4).
// SOLVMAT's stopping rule is the L2 ratio ||XS|| / ||RHS|| <= EPSMAT after at
// least ITMIN = 5 iterations (ppmat.f:152-178); after each colour
// RADIATIVEBOUND resets the bottom (T and ER at i <= 1 from the gradient D_T)
// and the top (ER at i >= upperbnd), copies the theta ghosts and shifts the
// phi halo.  Every kernel keeps the reference's operation order (the library
// is built with --fmad=false), so the iterates equal the reference loop's
// except where pow() enters (the IBDRAD = 9 top and the final T), and beside a
// column whose UPPERBND is 1, for whose faces the reference forms no limiter.
#include <math.h>

#include "ttfld_sweep64.cuh"

namespace ttfld {
int asm_diff(ttfld_ctx* c, int energy_iter);

namespace {

struct RadWork {
  double *ax, *cx, *ay, *cy, *az, *cz, *b, *rhs, *xs;
  double *volxb, *volyb, *volzb;  // (1:NX), (1:NY), (1:NZ)
};

__global__ void __launch_bounds__(kThreads) er_from_t_kernel(Dev d) {
  const long long n = (long long)nhalo(d);
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
    d.ER[q] = TT_ARAD * p4(d.T[q]);
}

__global__ void __launch_bounds__(kThreads) t_from_er_kernel(Dev d) {
  const long long n = (long long)nhalo(d);
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
    d.T[q] = pow(d.ER[q] / TT_ARAD, 0.25);
}

// DIFFEL (pprad.f:56-66) and B, RHS (pprad.f:21-29); SURYA = 1 (ppinit.f:1367).
__global__ void __launch_bounds__(kThreads) diffel_kernel(Dev d, RadWork w) {
  const unsigned int n = (unsigned int)ncell(d);
  for (unsigned int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    int i, j, k;
    cell_ijk(d, t, i, j, k);
    const double vx = w.volxb[i - 1], vy = w.volyb[j - 1], vz = w.volzb[k - 1];
    const double ax = div_rn(-FA(DIFRX, i, j, k) * G(surxa, i), vx);
    const double cx = div_rn(-FA(DIFRX, i + 1, j, k) * G(surxa, i + 1), vx);
    const double ay = div_rn(div_rn(div_rn(-FA(DIFRY, i, j, k), vy), G(geoxg, i)), G(geozg, k));
    const double cy = div_rn(div_rn(div_rn(-FA(DIFRY, i, j + 1, k), vy), G(geoxg, i)), G(geozg, k));
    const double az = div_rn(div_rn(-FA(DIFRZ, i, j, k) * G(surza, k), vz), G(geoxh, i));
    const double cz = div_rn(div_rn(-FA(DIFRZ, i, j, k + 1) * G(surza, k + 1), vz), G(geoxh, i));
    const double tt = HA(T, i, j, k);
    const double t3 = mul_rn(mul_rn(mul_rn(4.0 * TT_ARAD, tt), tt), tt);
    const double wt = div_rn(mul_rn(div_rn(1.0, d.delt) * HA(CV, i, j, k), HA(RH, i, j, k)), t3);
    w.ax[t] = ax; w.cx[t] = cx; w.ay[t] = ay; w.cy[t] = cy; w.az[t] = az; w.cz[t] = cz;
    w.b[t] = wt - ax - cx - ay - cy - az - cz;
    w.rhs[t] = div_rn(mul_rn(div_rn(HA(ER, i, j, k), d.delt) * HA(CV, i, j, k), HA(RH, i, j, k)), t3);
  }
}

// One colour of SOLVMAT (ppmat.f:66-82, 110-121): XS = B ER - RHS + the
// couplings (left to right), ER -= OM * XS / B.
template <int PARITY>
__global__ void __launch_bounds__(kThreads) solvmat_colour_kernel(Dev d, RadWork w, double om) {
  if (solver_done(d)) return;
  const int nx = d.nx, ny = d.ny;
  const unsigned int n = d.by_nxh.d * (unsigned int)ny * d.nz;
  const size_t sj = (size_t)(nx + 4), sk = (size_t)(nx + 4) * (ny + 4);
  for (unsigned int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    unsigned int h, j0;
    const int k = (int)div_rem(d.by_ny, div_rem(d.by_nxh, t, h), j0) + 1, j = (int)j0 + 1;
    const int i = 2 - ((j + k + PARITY) & 1) + 2 * (int)h;
    if (i > nx) continue;
    const size_t c = cidx(d, i, j, k);
    const size_t q = hidx(d, i, j, k);
    double* er = d.ER;
    const double bc = w.b[c], e = er[q];
    const double x = mul_rn(bc, e) - w.rhs[c] + mul_rn(w.ax[c], er[q - 1]) + mul_rn(w.cx[c], er[q + 1]) +
                     mul_rn(w.ay[c], er[q - sj]) + mul_rn(w.cy[c], er[q + sj]) + mul_rn(w.az[c], er[q - sk]) +
                     mul_rn(w.cz[c], er[q + sk]);
    w.xs[c] = x;
    er[q] = e - div_rn(om * x, bc);
  }
}

// RADIATIVEBOUND's bottom of one column (ppbou.f:2127-2139): T and ER at
// i <= 1 from the gradient D_T.
__device__ __forceinline__ void radbound_bottom(const Dev& d, int j, int k, double d_t, double tinit_bottom) {
  if (d.bcxmin == 6) HA(T, 1, j, k) = tinit_bottom;
  HA(T, 0, j, k) = HA(T, 1, j, k) - d_t * (G(xxb, 1) - G(xxb, 0));
  HA(T, -1, j, k) = HA(T, 1, j, k) - d_t * (G(xxb, 1) - G(xxb, -1));
  HA(ER, 1, j, k) = TT_ARAD * p4(HA(T, 1, j, k));
  HA(ER, 0, j, k) = TT_ARAD * p4(HA(T, 0, j, k));
  HA(ER, -1, j, k) = TT_ARAD * p4(HA(T, -1, j, k));
}

// Its top of one interior column (ppbou.f:2145-2236): ER at i >= upperbnd.
// Sets sol->nonfinite = 2 (read as an error) if upperbnd >= NX+1, where the
// reference stops (:2238-2240).
__device__ __forceinline__ void radbound_top(const Dev& d, int j, int k) {
  const int ub = PA(UB, j, k);
  if (!(ub < d.nx + 1)) {
    atomicExch(&d.sol->nonfinite, 2);
    return;
  }
  double tj = 0.0;
  switch (d.ibdrad) {
    case 4: tj = d.tirr; break;
    case 7: tj = HA(T, ub - 1, j, k); break;
    default:  // 9
      if (d.iii <= 1) tj = HA(T, ub - 1, j, k);
      else
        tj = pow(HA(ER, ub, j, k) / TT_ARAD +
                     HA(SI, ub - 1, j, k) / (4.0 * TT_SBCONST * HA(RH, ub - 1, j, k) * HA(XKAPP, ub - 1, j, k)),
                 0.25);
  }
  const double e = TT_ARAD * p4(tj);
  for (int i = ub; i <= d.nx + 2; ++i) HA(ER, i, j, k) = e;
}

// RADIATIVEBOUND, part 1: the bottom on (j,k) in -1..N+2, the top on the
// interior columns.
__global__ void __launch_bounds__(kThreads) radbound_xkernel(Dev d, double d_t, double tinit_bottom) {
  if (solver_done(d)) return;  // applied once more after the stop it would move the IBDRAD = 9 top
  const int ny = d.ny, nz = d.nz;
  const long long n = (long long)(ny + 4) * (nz + 4);
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(t % (ny + 4)) - 1, k = (int)(t / (ny + 4)) - 1;
    radbound_bottom(d, j, k, d_t, tinit_bottom);
    if (j >= 1 && j <= ny && k >= 1 && k <= nz) radbound_top(d, j, k);
  }
}

// PLANETSHIFT(6) and, with poles, the pole shifts of E_R that follow it
// everywhere in RADDIF (ppmat.f:39-49, 87-97, 126-136; ppbou.f:2280-2290).
static int er_shift(ttfld_ctx* c) {
  int rc = halo_shift(c, c->d.ER);
  return rc ? rc : pole_shift(c, c->d.ER);
}

// RADIATIVEBOUND, part 2 (ppbou.f:2256-2271): theta ghosts from k = 1, NZ.
__global__ void __launch_bounds__(kThreads) radbound_zkernel(Dev d) {
  if (solver_done(d)) return;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const long long n = (long long)(nx + 4) * (ny + 4);
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t % (nx + 4)) - 1, j = (int)(t / (nx + 4)) - 1;
    HA(ER, i, j, -1) = HA(ER, i, j, 1);
    HA(ER, i, j, 0) = HA(ER, i, j, 1);
    HA(ER, i, j, nz + 1) = HA(ER, i, j, nz);
    HA(ER, i, j, nz + 2) = HA(ER, i, j, nz);
  }
}

// sqrt(sum a^2) over the cells, fixed order; the last block applies the
// stopping rule when `stop` (ratio against sol->rhsnorm, ITMIN = 5).
__global__ void __launch_bounds__(kThreads) l2_kernel(Dev d, const double* a, double* partials, int stop, int itmax,
                                                      double eps) {
  __shared__ double sh[32];
  __shared__ bool last;
  if (stop && solver_done(d)) return;
  const long long n = (long long)ncell(d);
  double acc = 0.0;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    acc += mul_rn(a[t], a[t]);
  const double s = block_sum(acc, sh);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = s;
    __threadfence();
    last = (atomicAdd(&d.sol->ticket2, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (last) {
    __threadfence();
    const double tot = block_sum_array(partials, gridDim.x, sh);
    if (threadIdx.x == 0) {
      const double nrm = sqrt(tot);
      SolverDev* sol = d.sol;
      if (!stop) {
        sol->rhsnorm = nrm;
      } else {
        const int it = sol->iter + 1;
        sol->iter = it;
        sol->rnorm = nrm;
        sol->ratio = nrm / sol->rhsnorm;
        if (!isfinite(nrm)) { sol->nonfinite = 1; sol->done = 1; }
        else if (it == itmax) { sol->maxit = 1; sol->done = 1; }
        else if (!(sol->ratio > eps) && it >= 5) sol->done = 1;
      }
      sol->ticket2 = 0;
    }
  }
}

int cell_blocks(const Dev& d) {
  const int nb = grid_for((long long)ncell(d));
  return nb > kMaxPartials ? kMaxPartials : nb;
}

// With poles the theta ghosts come from the pole shifts instead
// (ppbou.f:2256-2271 run only without poles; :2280-2290).
int radiativebound(ttfld_ctx* c, double d_t, double tinit_bottom) {
  const Dev& d = c->d;
  radbound_xkernel<<<grid_for((long long)(d.ny + 4) * (d.nz + 4)), kThreads, 0, c->stream>>>(d, d_t, tinit_bottom);
  count_launches(1);
  if (!d.poles) {
    radbound_zkernel<<<grid_for((long long)(d.nx + 4) * (d.ny + 4)), kThreads, 0, c->stream>>>(d);
    count_launches(1);
  }
  TT_CHECK_LAUNCH();
  return er_shift(c);
}

// SOLVMAT's colours with RADIATIVEBOUND after each, for the persistent FP64
// sweeps, without poles.  Every boundary application that leaves a value as
// it is, is left out: T(1) never changes, so ER(1) = arad T(1)^4, which it
// starts from, is simply not overwritten, ER at i <= 0 is set once, and the
// top (but for IBDRAD = 9 with III > 1, whose top moves on with every
// application) is set once and not overwritten.  An application writes cells
// of both colours, which the neighbouring columns read in the colour before it
// (ER at i >= UPPERBND of a column lies beside interior cells of another where
// UPPERBND differs, and beside the top itself); so a block writes them once its
// neighbours have finished that colour, and they begin the next once it has
// written them (boundary_step): one exchange more per solve, or per colour
// where the top moves (4.6 us a colour with a fixed top, 12.2 with a moving one,
// whose decisions are waited for too, at 40x64x32).  The theta ghosts are
// copies of the cell next to them, so after the first colour the cell itself
// is read in their place, the phi neighbours by wrapping j.  The ghosts
// themselves are filled after the last sweep (radbound_ghost_bottom, radbound_ghost_theta).
struct RadRows {
  typedef double Word;
  typedef double Kept;
  static constexpr int kWords = 8, kThreads = 1024;
  static constexpr bool kStrided = true, kBoundary = true;
  Dev d;
  RadWork w;
  double om, d_t, tinit_bottom;
  long long rows;
  int ny, moving_top;
  FastDiv by_items;
  __device__ double norm(double sum) const { return sqrt(sum); }
  template <int COL>
  __device__ __forceinline__ unsigned int cell(unsigned int row, unsigned int h, unsigned int& j0,
                                               unsigned int& k0) const {
    k0 = div_rem(d.by_ny, row, j0);
    return 2 * h + ((j0 + k0 + COL + 1) & 1);
  }
  // The corner ghosts (j and k outside) keep what the theta copies of the
  // second colour's RADIATIVEBOUND find in the phi ghosts: the wrapped
  // values from before that colour.
  template <int COL>
  __device__ void before(unsigned int r0, unsigned int r1) const {
    if (COL == 0) return;
    const unsigned int nyu = (unsigned int)d.ny, last = nyu * (unsigned int)(d.nz - 1);
    if (r0 >= nyu && r1 <= last) return;  // no row of the planes k = 1, NZ
    for (int m = 0; m < 8; ++m) {
      const int k = m < 4 ? 1 : d.nz;
      const int j = (m & 3) == 0 ? 1 : (m & 3) == 1 ? 2 : (m & 3) == 2 ? d.ny - 1 : d.ny;
      const unsigned int row = (unsigned int)(k - 1) * nyu + (unsigned int)(j - 1);
      if (row < r0 || row >= r1) continue;
      const int jg = j <= 2 ? d.ny + j : j - d.ny;
      for (int i = 2 + (int)threadIdx.x; i <= d.nx + 2; i += (int)blockDim.x) {
        const double e = HA(ER, i, j, k);
        HA(ER, i, jg, k == 1 ? 0 : d.nz + 1) = e;
        HA(ER, i, jg, k == 1 ? -1 : d.nz + 2) = e;
      }
    }
    __syncthreads();
  }
  __device__ bool boundary(bool first) const { return first || moving_top; }
  __device__ void write_boundary(unsigned int r0, unsigned int r1, bool first) const {
    for (unsigned int r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
      unsigned int j0;
      const int k = (int)div_rem(d.by_ny, r, j0) + 1, j = (int)j0 + 1;
      // (a top that begins at i <= 1 starts from the bottom's value each time)
      if (first || PA(UB, j, k) <= 1) radbound_bottom(d, j, k, d_t, tinit_bottom);
      radbound_top(d, j, k);
    }
  }
  template <int COL>
  __device__ __forceinline__ void fetch(unsigned int row, unsigned int h, double* to, unsigned int T, uint64_t pol) const {
    unsigned int j0, k0;
    const unsigned int i0 = cell<COL>(row, h, j0, k0);
    if ((int)i0 >= d.nx) return;
    const size_t c = i0 + (size_t)d.nx * row;
    copy_async(to, w.b + c, pol);
    copy_async(to + T, w.rhs + c, pol);
    copy_async(to + 2 * T, w.ax + c, pol);
    copy_async(to + 3 * T, w.cx + c, pol);
    copy_async(to + 4 * T, w.ay + c, pol);
    copy_async(to + 5 * T, w.cy + c, pol);
    copy_async(to + 6 * T, w.az + c, pol);
    copy_async(to + 7 * T, w.cz + c, pol);
  }
  template <int COL>
  __device__ __forceinline__ double update(unsigned int row, unsigned int h, const double* c, unsigned int T,
                                           bool first, double* kept) const {
    unsigned int j0, k0;
    const unsigned int i0 = cell<COL>(row, h, j0, k0);
    const int nx = d.nx, i = (int)i0 + 1;
    if (i > nx) return 0.0;
    const size_t sj = (size_t)(nx + 4), sk = sj * (size_t)(ny + 4);
    const size_t q = (i0 + 2) + sj * (j0 + 2) + sk * (k0 + 2);
    const size_t qjm = j0 == 0 ? q + sj * (size_t)(ny - 1) : q - sj;
    const size_t qjp = (int)j0 == ny - 1 ? q - sj * (size_t)(ny - 1) : q + sj;
    double* er = d.ER;
    const double e = er[q], b = c[0];
    const double ekm = !first && k0 == 0 ? e : er[q - sk];
    const double ekp = !first && (int)k0 == d.nz - 1 ? e : er[q + sk];
    const double x = mul_rn(b, e) - c[T] + mul_rn(c[2 * T], er[q - 1]) + mul_rn(c[3 * T], er[q + 1]) +
                     mul_rn(c[4 * T], er[qjm]) + mul_rn(c[5 * T], er[qjp]) + mul_rn(c[6 * T], ekm) +
                     mul_rn(c[7 * T], ekp);
    const int ub = PA(UB, (int)j0 + 1, (int)k0 + 1);
    // i = 1 and i > upperbnd (at upperbnd only a moving top reads it) keep
    // their boundary values
    if (i != 1 && (i < ub || (moving_top && i == ub) || ub > nx)) er[q] = e - div_rn(om * x, b);
    if (kept) *kept = e;
    return mul_rn(x, x);
  }
  __device__ __forceinline__ void restore(unsigned int row, unsigned int h, double kept) const {
    unsigned int j0, k0;
    const unsigned int i0 = cell<0>(row, h, j0, k0);
    if ((int)i0 < d.nx) HA(ER, (int)i0 + 1, (int)j0 + 1, (int)k0 + 1) = kept;
  }
};

// The ghosts RADIATIVEBOUND leaves after SOLVMAT's last colour: the bottom of
// the ghost columns, then the theta copies of every column but the corner
// ghosts' cells above i = 1 (RadRows::before).
__global__ void __launch_bounds__(kThreads) radbound_ghost_bottom(Dev d, double d_t, double tinit_bottom) {
  const int n = (d.ny + 4) * (d.nz + 4);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int j = t % (d.ny + 4) - 1, k = t / (d.ny + 4) - 1;
    if (j < 1 || j > d.ny || k < 1 || k > d.nz) radbound_bottom(d, j, k, d_t, tinit_bottom);
  }
}
__global__ void __launch_bounds__(kThreads) radbound_ghost_theta(Dev d) {
  const int nx = d.nx, ny = d.ny, nz = d.nz, n = (nx + 4) * (ny + 4);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int i = t % (nx + 4) - 1, j = t / (nx + 4) - 1;
    if ((j < 1 || j > ny) && i >= 2) continue;
    HA(ER, i, j, -1) = HA(ER, i, j, 1);
    HA(ER, i, j, 0) = HA(ER, i, j, 1);
    HA(ER, i, j, nz + 1) = HA(ER, i, j, nz);
    HA(ER, i, j, nz + 2) = HA(ER, i, j, nz);
  }
}

// SOLVMAT in one launch (no poles); 1 where that is not possible.
int solvmat_persistent(ttfld_ctx* c, const RadWork& w, double d_t, double tinit_bottom) {
  const Dev& d = c->d;
  if (d.poles) return 1;
  RadRows s;
  s.d = d;
  s.w = w;
  s.om = d.sorparam;
  s.d_t = d_t;
  s.tinit_bottom = tinit_bottom;
  s.rows = (long long)d.ny * d.nz;
  s.ny = d.ny;
  s.moving_top = d.ibdrad == 9 && d.iii > 1;
  s.by_items = d.by_nxh;
  // a moving top is not kept: its decisions are waited for
  const int rc = launch_sweeps64_persistent(s, c->stream, c->sol, c->partials, c->flags64, c->staging,
                                            s.moving_top ? 0 : c->staging_bytes, d.itmax, 5, d.itmax, d.epsmat, c);
  if (rc) return rc;
  radbound_ghost_bottom<<<grid_for((long long)(d.ny + 4) * (d.nz + 4)), kThreads, 0, c->stream>>>(d, d_t, tinit_bottom);
  radbound_ghost_theta<<<grid_for((long long)(d.nx + 4) * (d.ny + 4)), kThreads, 0, c->stream>>>(d);
  count_launches(2);
  TT_CHECK_LAUNCH();
  return er_shift(c);
}

}  // namespace
}  // namespace ttfld

extern "C" int ttfld_raddif(ttfld_ctx* c, const ttfld_raddif_params* p, ttfld_solve_stats* st) {
  using namespace ttfld;
  if (!c || !p || !p->volxb || !p->volyb || !p->volzb) return TTFLD_E_ARGS;
  const Dev& d = c->d;
  if (d.nz == 1) return TTFLD_E_UNSUPPORTED;
  if (!(d.ibdrad == 4 || d.ibdrad == 7 || d.ibdrad == 9) || p->modver > 5)
    return TTFLD_E_UNSUPPORTED;
  TT_CHECK(cudaSetDevice(c->device));
  ttfld_solve_stats local{};
  if (!st) st = &local;
  RadWork w{};
  const size_t n = ncell(d);
  const size_t bytes = (9 * n + (size_t)d.nx + d.ny + d.nz) * sizeof(double);
  // kept with the context: from the stream's pool it was mapped and unmapped
  // again on every call
  if (!c->rad_mem) TT_CHECK(cudaMalloc(&c->rad_mem, bytes));
  double* q = (double*)c->rad_mem;
  double** arrs[] = {&w.ax, &w.cx, &w.ay, &w.cy, &w.az, &w.cz, &w.b, &w.rhs, &w.xs};
  for (double** a : arrs) { *a = q; q += n; }
  w.volxb = q; q += d.nx;
  w.volyb = q; q += d.ny;
  w.volzb = q;
  int rc = 0;
  TT_CHECK(cudaMemcpyAsync(w.volxb, p->volxb, d.nx * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  TT_CHECK(cudaMemcpyAsync(w.volyb, p->volyb, d.ny * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  TT_CHECK(cudaMemcpyAsync(w.volzb, p->volzb, d.nz * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  TT_CHECK(cudaEventRecord(c->ev0, c->stream));
  er_from_t_kernel<<<grid_for((long long)nhalo(d)), kThreads, 0, c->stream>>>(d);
  count_launches(1);
  TT_CHECK_LAUNCH();
  rc = asm_diff(c, p->energy_iter);
  if (!rc) {
    diffel_kernel<<<grid_for((long long)n), kThreads, 0, c->stream>>>(d, w);
    count_launches(1);
    TT_CHECK_LAUNCH();
    TT_CHECK(cudaMemsetAsync(c->sol, 0, sizeof(SolverDev), c->stream));
    const int nb = cell_blocks(d);
    l2_kernel<<<nb, kThreads, 0, c->stream>>>(d, w.rhs, c->partials, 0, d.itmax, d.epsmat);
    count_launches(1);
    rc = er_shift(c);
  }
  // one launch for the whole loop, or (with poles) iterations in chunks
  // between polls of the stopping flag
  bool queued = false;
  if (!rc) {
    rc = solvmat_persistent(c, w, p->d_t, p->tinit_bottom);
    queued = rc == 0;
    if (rc == 1) rc = 0;
  }
  const int sweeps_nb = grid_for((long long)((d.nx + 1) / 2) * d.ny * d.nz);
  int chunk = 8;
  while (!rc) {
    for (int s = 0; s < chunk && !rc && !queued; ++s) {
      solvmat_colour_kernel<0><<<sweeps_nb, kThreads, 0, c->stream>>>(d, w, d.sorparam);
      count_launches(1);
      if ((rc = radiativebound(c, p->d_t, p->tinit_bottom)) || (rc = er_shift(c))) break;
      solvmat_colour_kernel<1><<<sweeps_nb, kThreads, 0, c->stream>>>(d, w, d.sorparam);
      count_launches(1);
      if ((rc = radiativebound(c, p->d_t, p->tinit_bottom)) || (rc = er_shift(c))) break;
      l2_kernel<<<cell_blocks(d), kThreads, 0, c->stream>>>(d, w.xs, c->partials, 1, d.itmax, d.epsmat);
      count_launches(1);
      TT_CHECK_LAUNCH();
    }
    if (rc) break;
    TT_CHECK(cudaMemcpyAsync(c->host_sol, c->sol, sizeof(SolverDev), cudaMemcpyDeviceToHost, c->stream));
    TT_CHECK(cudaStreamSynchronize(c->stream));
    if (c->host_sol->bar_timeout) {
      fprintf(stderr, "ttfld: a wait of the persistent FP64 sweeps timed out\n");
      rc = TTFLD_E_CUDA;
      break;
    }
    if (c->host_sol->nonfinite == 2) { rc = TTFLD_E_UNSUPPORTED; break; }
    if (c->host_sol->done) break;
    if (queued) { rc = TTFLD_E_INTERNAL; break; }  // the rule fires at ITMAX at the latest
    if (chunk < 64) chunk *= 2;
  }
  // the colour kernels, bounds and norms queued after the stop return at
  // once or leave ER unchanged (the bounds re-apply the same values)
  if (!rc) {
    t_from_er_kernel<<<grid_for((long long)nhalo(d)), kThreads, 0, c->stream>>>(d);
    count_launches(1);
    TT_CHECK_LAUNCH();
  }
  TT_CHECK(cudaEventRecord(c->ev1, c->stream));
  TT_CHECK(cudaStreamSynchronize(c->stream));
  if (rc) return rc;
  float ms = 0.f;
  cudaEventElapsedTime(&ms, c->ev0, c->ev1);
  const SolverDev& h = *c->host_sol;
  st->sor_iter = h.iter;
  st->rnorm = h.rnorm;
  st->rhsnorm = h.rhsnorm;
  st->solve_ms = ms;
  st->status = h.nonfinite ? TTFLD_E_NONFINITE : (h.maxit ? TTFLD_MAXITER : TTFLD_OK);
  if (h.maxit) printf("Max iteration reached in SOR matrix solver %8d %8d %12.6e %12.6e %12.6e %12.6e %12.6e\n", d.iii,
                      h.iter, h.ratio, h.rnorm, h.rhsnorm, d.epsmat, d.sorparam);
  return st->status;
}
