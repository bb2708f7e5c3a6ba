// ttfld_sweep64.cuh -- FP64 red-black sweeps with the reference's stopping
// rule after every sweep, any number of them in one cooperative launch.
//
// One launch per colour leaves the chip idle between the launches, and a
// grid of a few hundred thousand cells is a few microseconds of work per
// colour: the waves of blocks, their partial sums and the launch gaps cost
// several times that.  Here one block per SM owns a contiguous run of (j,k)
// rows for all sweeps, and after each colour waits only for the blocks that
// own rows within one theta plane of its own (wait_flags).  Every block adds
// all blocks' shares of a sweep's norm in the same fixed order and takes the
// same stop decision -- one colour later: it begins the next sweep, keeping
// the values that its first colour replaces, and reads the shares, by then
// there, before the second; if the rule says stop it puts those values back.
// (Where the values cannot be kept, the decision is waited for.)  A block adds
// up its own share behind its flag, which its neighbours wait for: 5.75 -> 5.48
// ms for the exact SOR at 64x128x64 against adding it up before.  The cells'
// updates and their operands are those of one launch per colour, so the
// iterate is the same bit for bit; only the order in which the norm is
// summed differs.  Where boundary values are written behind a colour, that
// takes a wait of its own (boundary_step).
//
// What does not change during a solve (the coefficients and b) each thread
// copies for its next item into its own slots of shared memory (cp.async)
// before it updates the present one, across the colours too, so that these
// reads, eight of the 16 values of a cell, wait for nothing.  Where a block's
// share of them fits in shared memory (RESIDENT: 227 KB a block, 540,000
// cells in all) it is copied once for all sweeps.  Beyond L2 most of their
// lines are marked to be evicted first (l2_keep), so that the iterate stays:
// 52.2 -> 50.0 ms for the scaled SOR and 5.06 -> 4.75 ms for DIFFUSION at
// 100x256x128, 11.9 -> 11.3 ms for DIFFUSION at 160x256x192.
//
// Where a system's items are every other cell of its arrays (kStrided), each
// colour's pass reads the lines of both colours.  Not RESIDENT, the first
// sweep therefore stores what each thread has fetched for its items, in the
// order in which it will want it, and later sweeps fetch from that copy, half
// the bytes: DIFFUSION 4.72 -> 4.46 ms at 100x256x128 and 11.3 -> 10.4 at
// 160x256x192, the exact SOR 58.9 -> 56.5 ms at 100x256x100, RADDIF 25.2 ->
// 24.2 there.  (The FP64 pipe is then busy two thirds of the time.)
//
// A system is a struct with
//   rows, by_items          (j,k) rows, and the items of a colour in a row
//   kWords, Word            its coefficients of an item, as kWords of Word
//   fetch<COL>(row, h, to)  queues their copies to to[0], to[T], to[2 T], ...
//                           (T threads)
//   update<COL>(row, h, w, T, first, kept)  updates item h of a row with them,
//                           returns its share of the norm; first: no colour
//                           has run yet; kept: where the old value (Kept) goes
//   restore(row, h, kept)   puts a value of the first colour back
//   kStrided                the items of a colour are not contiguous in memory
//   before<COL>(r0, r1)     a block's own work ahead of a colour (all its threads),
//                           on values that no update reads
//   boundary(first)         whether boundary values of the rows are written
//                           behind the colour (the same for all blocks)
//   write_boundary(r0, r1, first)  the block's share of them (all its threads).
//                           Its neighbours read these values in the colour, so
//                           it is called once they have finished it
//   kBoundary               there may be such values
//   norm(sum)               the norm from the sum of the shares
#pragma once
#include "ttfld_internal.cuh"

namespace ttfld {

// The norm of sweep sw from every block's share and the reference's rule on
// it, by one warp of every block: 0 go on, 1 stop, 2 a block has given up
// (every lane gets it).  Block 0 records the sweep.
template <class Sys>
__device__ __forceinline__ int gather_norm(const Sys& s, const Partial* gather, int nb, int sw, int it0, int itmin,
                                           int itmax, double eps, double rhsnorm, SolverDev* sol) {
  const int lane = threadIdx.x & 31;
  double tot;
  if (!gather_sum(gather, nb, sw, sol, tot)) return 2;
  tot = s.norm(tot);
  const double ratio = tot / rhsnorm;
  const int it = it0 + sw;
  const bool fin = isfinite(tot), out = it == itmax, met = !(ratio > eps) && it >= itmin;
  const int stop = !fin || out || met ? 1 : 0;
  if (lane == 0 && blockIdx.x == 0) {
    sol->iter = it;
    sol->rnorm = tot;
    sol->ratio = ratio;
    if (!fin && sol->nonfinite == 0) sol->nonfinite = 1;
    else if (out) sol->maxit = 1;
    if (stop) sol->done = 1;
  }
  return stop;
}

// A block's share of the norm of sweep sw, from its warps' sums, by one warp.
__device__ __forceinline__ void put_share(const double* sh, int nw, Partial* gather, int b, int sw) {
  const int lane = threadIdx.x & 31;
  const double part = warp_sum_all(lane < nw ? sh[lane] : 0.0);
  if (lane == 0) put_partial(gather, b, sw, part);
}

// Put back the first colour's values from before the present sweep.
template <class Sys>
__device__ __forceinline__ void undo_colour(const Sys& s, unsigned int r0, unsigned int n,
                                            const typename Sys::Kept* mine) {
  for (unsigned int u = threadIdx.x; u < n; u += blockDim.x) {
    unsigned int h;
    const unsigned int r = r0 + div_rem(s.by_items, u, h);
    s.restore(r, h, mine[u]);
  }
}

// The copy that later sweeps fetch from: word q of item u of a block at
// at[COL][q * n + u] (null: none, or not yet written).
template <class Word>
struct SweepCopy {
  const Word* now;   // of this colour
  const Word* next;  // of the colour that follows
  Word* store;       // written in the first sweep
};

// Queue the copies of item u of a block's n.
template <int COL, class Sys>
__device__ __forceinline__ void fetch_item(const Sys& s, unsigned int r0, unsigned int n, unsigned int u,
                                           const typename Sys::Word* copy, typename Sys::Word* to, unsigned int T,
                                           uint64_t pol) {
  if (Sys::kStrided && copy) {
#pragma unroll
    for (int q = 0; q < Sys::kWords; ++q) copy_async(to + q * T, copy + (size_t)q * n + u, pol);
    return;
  }
  unsigned int h;
  const unsigned int r = r0 + div_rem(s.by_items, u, h);
  s.template fetch<COL>(r, h, to, T, pol);
}

// The items of one colour of a block's rows.  Not RESIDENT: the thread's
// next item (of this colour, or its first of the other) is fetched before
// the present one is updated.  mine: where to keep the values replaced.
template <int COL, bool RESIDENT, class Sys>
__device__ __forceinline__ double sweep_colour(const Sys& s, unsigned int r0, unsigned int n, bool first,
                                               typename Sys::Word* slots, int& stage, typename Sys::Kept* mine,
                                               uint64_t pol, const SweepCopy<typename Sys::Word>& copy) {
  double acc = 0.0;
  const unsigned int T = blockDim.x;
  for (unsigned int u = threadIdx.x; u < n; u += T) {
    unsigned int h;
    const unsigned int r = r0 + div_rem(s.by_items, u, h);
    if (RESIDENT) {
      acc += s.template update<COL>(r, h, slots + (size_t)COL * Sys::kWords * n + u, n, first, mine ? mine + u : nullptr);
      continue;
    }
    const typename Sys::Word* now = slots + (size_t)stage * Sys::kWords * T + threadIdx.x;
    stage ^= 1;
    typename Sys::Word* next = slots + (size_t)stage * Sys::kWords * T + threadIdx.x;
    if (u + T < n) fetch_item<COL>(s, r0, n, u + T, copy.now, next, T, pol);
    else fetch_item<1 - COL>(s, r0, n, threadIdx.x, copy.next, next, T, pol);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    if (Sys::kStrided && copy.store) {
#pragma unroll
      for (int q = 0; q < Sys::kWords; ++q) copy.store[(size_t)q * n + u] = now[q * T];
    }
    acc += s.template update<COL>(r, h, now, T, first, mine ? mine + u : nullptr);
  }
  return acc;
}

// The boundary values behind a colour, if any, as a step of its own between
// two flags: the first says that this block has read what its neighbours will
// write, the caller's next one that its own values are there.  False if the
// wait gave up.
template <class Sys>
__device__ __forceinline__ bool boundary_step(const Sys& s, unsigned int r0, unsigned int r1, bool first,
                                              unsigned int* flags, int lo, int hi, unsigned int& half,
                                              SolverDev* sol) {
  if (!Sys::kBoundary || !s.boundary(first)) return true;
  publish_flag(flags + (size_t)blockIdx.x * kFlagStride, ++half);
  if (!wait_flags(flags, lo, hi, half, sol)) return false;
  s.write_boundary(r0, r1, first);
  return true;
}

template <class Sys, bool RESIDENT>
__global__ void __launch_bounds__(Sys::kThreads, 1)
    sweeps64_persistent(Sys s, SolverDev* sol, Partial* gather, unsigned int* flags, typename Sys::Kept* keep,
                        int nsweeps, int itmin, int itmax, double eps, uint64_t pol,
                        typename Sys::Word* copy) {
  __shared__ double sh[32];
  __shared__ int stop_sh, ok_sh;
  if (threadIdx.x == 0) {  // read after block barriers only
    stop_sh = 0;
    ok_sh = 1;
  }
  const int nb = (int)gridDim.x, b = (int)blockIdx.x;
  if (*(volatile int*)&sol->done) return;  // set before the launch, so the same for every block
  const long long rows = s.rows;
  const unsigned int r0 = (unsigned int)(rows * b / nb), r1 = (unsigned int)(rows * (b + 1) / nb);
  const long long ny = s.ny;
  const int lo = owner_block(r0 > ny ? r0 - ny : 0, rows, nb);
  const int hi = owner_block(r1 - 1 + ny < rows ? r1 - 1 + ny : rows - 1, rows, nb);
  const unsigned int n = (r1 - r0) * s.by_items.d;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const double rhsnorm = sol->rhsnorm;
  const int it0 = sol->iter;
  extern __shared__ __align__(16) unsigned char slots_raw[];
  typename Sys::Word* slots = reinterpret_cast<typename Sys::Word*>(slots_raw);
  int stage = 0;
  if (RESIDENT) {  // each thread copies what it will read itself
    for (unsigned int u = threadIdx.x; u < n; u += blockDim.x) {
      unsigned int h;
      const unsigned int r = r0 + div_rem(s.by_items, u, h);
      s.template fetch<0>(r, h, slots + u, n, pol);
      s.template fetch<1>(r, h, slots + (size_t)Sys::kWords * n + u, n, pol);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (threadIdx.x < n) {
    unsigned int h;
    const unsigned int r = r0 + div_rem(s.by_items, threadIdx.x, h);
    s.template fetch<0>(r, h, slots + threadIdx.x, blockDim.x, pol);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  typedef SweepCopy<typename Sys::Word> Copy;
  typename Sys::Word* copy0 = copy ? copy + (size_t)r0 * s.by_items.d * 2 * Sys::kWords : nullptr;
  typename Sys::Word* copy1 = copy ? copy0 + (size_t)Sys::kWords * n : nullptr;
  typename Sys::Kept* mine = keep ? keep + (size_t)r0 * s.by_items.d : nullptr;
  unsigned int* own = flags + (size_t)b * kFlagStride;
  unsigned int half = 0;  // half-sweeps (and boundary steps) this block has finished
  int stop = 0;
  for (int sw = 1; sw <= nsweeps && !stop; ++sw) {
    if (sw > 1) {
      if (!wait_flags(flags, lo, hi, half, sol)) break;  // its block barrier also orders sh
      if (mine && warp == 0) put_share(sh, nw, gather, b, sw - 1);
    }
    s.template before<0>(r0, r1);
    double acc = sweep_colour<0, RESIDENT>(s, r0, n, sw == 1, slots, stage, sw > 1 ? mine : nullptr, pol,
                                            sw > 1 ? Copy{copy0, copy1, nullptr} : Copy{nullptr, nullptr, copy0});
    if (!boundary_step(s, r0, r1, sw == 1, flags, lo, hi, half, sol)) break;
    publish_flag(own, ++half);
    // the first warp waits for the neighbours, the last takes the last
    // sweep's rule, and with it whether this sweep begins at all
    if (warp == 0 && !poll_flags(flags, lo, hi, half, sol) && lane == 0) ok_sh = 0;
    if (warp == nw - 1 && mine && sw > 1) {
      const int r = gather_norm(s, gather, nb, sw - 1, it0, itmin, itmax, eps, rhsnorm, sol);
      if (lane == 0) stop_sh = r;
    }
    __syncthreads();
    stop = stop_sh;
    if (stop || !ok_sh) {
      if (stop == 1) undo_colour(s, r0, n, mine);
      break;
    }
    s.template before<1>(r0, r1);
    acc += sweep_colour<1, RESIDENT>(s, r0, n, false, slots, stage, nullptr, pol,
                                      sw > 1 ? Copy{copy1, copy0, nullptr} : Copy{nullptr, copy0, copy1});
    if (!boundary_step(s, r0, r1, false, flags, lo, hi, half, sol)) break;
    publish_flag(own, ++half);
    // behind the flag, that the neighbours wait for; where the decision comes
    // a colour later the block's share is put at the next sweep's start
    acc = warp_sum_all(acc);
    if (lane == 0) sh[warp] = acc;
    if (!mine || sw == nsweeps) {
      __syncthreads();
      if (warp == 0) put_share(sh, nw, gather, b, sw);
      if (warp == nw - 1) {
        const int r = gather_norm(s, gather, nb, sw, it0, itmin, itmax, eps, rhsnorm, sol);
        if (lane == 0) stop_sh = r;
      }
      __syncthreads();
      stop = stop_sh;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The context's copy of a system's coefficients, 64 bytes a cell, allocated by
// the first solve that wants it; null where there is no room.
inline void* sweep_copy(ttfld_ctx* c, size_t bytes) {
  if (c->sweep_copy_bytes < bytes) {
    if (c->sweep_copy) cudaFree(c->sweep_copy);
    c->sweep_copy = nullptr;
    c->sweep_copy_bytes = 0;
    if (cudaMalloc(&c->sweep_copy, bytes) != cudaSuccess) {
      cudaGetLastError();
      c->sweep_copy = nullptr;
      return nullptr;
    }
    c->sweep_copy_bytes = bytes;
  }
  return c->sweep_copy;
}

// Queue nsweeps sweeps of a system (fewer if the rule fires).  1 where the
// launch is not possible (no cooperative launch, or fewer SMs to be had than
// blocks): the caller runs one launch per colour instead.  owner: the context
// that holds the copy of the coefficients (null: none is made).
template <class Sys>
int launch_sweeps64_persistent(const Sys& s, cudaStream_t st, SolverDev* sol, double* partials, unsigned int* flags,
                               void* kept, size_t kept_bytes, int nsweeps, int itmin, int itmax, double eps,
                               ttfld_ctx* owner) {
  int dev = 0, sms = 0, coop = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!coop || sms <= 0 || nsweeps <= 0) return 1;
  if (sms > kMaxLocalBlocks) sms = kMaxLocalBlocks;
  // one block per SM, but no block of less than two warps' items
  const long long items = (long long)s.rows * s.by_items.d;
  long long nb = (items + 63) / 64;
  if (nb > sms) nb = sms;
  if (nb > s.rows) nb = s.rows;
  // threads for the fewest rounds over a block's items, evenly filled
  const long long most = (s.rows + nb - 1) / nb * s.by_items.d;
  const long long rounds = (most + Sys::kThreads - 1) / Sys::kThreads;
  const int threads = (int)(((most + rounds - 1) / rounds + 31) / 32 * 32);
  int room = 0;
  cudaDeviceGetAttribute(&room, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t item = 2 * (size_t)Sys::kWords * sizeof(typename Sys::Word);  // both colours, or both stages
  const bool resident = item * (size_t)most + 1024 <= (size_t)room;
  const size_t smem = item * (size_t)(resident ? most : threads);
  const void* kernel = resident ? (const void*)sweeps64_persistent<Sys, true> : (const void*)sweeps64_persistent<Sys, false>;
  if (smem_room(kernel) < smem) return 1;
  TT_CHECK(cudaMemsetAsync(flags, 0, (size_t)nb * kFlagStride * sizeof(unsigned int), st));
  Partial* gather = (Partial*)partials;  // two a block
  TT_CHECK(cudaMemsetAsync(gather, 0, (size_t)nb * 2 * sizeof(Partial), st));
  Sys sys = s;
  typename Sys::Kept* keep =
      (size_t)items * sizeof(typename Sys::Kept) <= kept_bytes ? (typename Sys::Kept*)kept : nullptr;
  const double word = 2.0 * (double)items * sizeof(typename Sys::Word);  // an array of both colours
  uint64_t pol = resident ? l2_policy(0.0, st) : l2_keep(word, Sys::kWords * word, st).coef;  // resident: read once
  if (!pol) return TTFLD_E_CUDA;
  // the first sweep's stores cost about what half a sweep's reads do
  typename Sys::Word* copy = nullptr;
  if (Sys::kStrided && !resident && owner && nsweeps >= 4)
    copy = (typename Sys::Word*)sweep_copy(owner, (size_t)(Sys::kWords * word));
  void* args[] = {&sys, &sol, &gather, &flags, &keep, &nsweeps, &itmin, &itmax, &eps, &pol, &copy};
  const cudaError_t e =
      cudaLaunchCooperativeKernel(kernel, dim3((unsigned int)nb), dim3(threads), args, smem, st);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return 1;
  }
  TT_CHECK(e);
  count_launches(1);
  return 0;
}

// SOLVE_WITH_SOR's rows in the reference's layout and operand order
// (ppsor.f:59-136): the coefficients and b in cell order, x a halo array
// whose phi direction is read by wrapping j.  With poles the theta
// neighbours across the edges are the cell itself (x_km, x_kp).  The
// products and the quotient run on the integer pipes, the sums on the FP64
// pipe (ttfld_fp64.cuh); omega times the residual too (5.48 -> 5.16 ms for the
// exact SOR at 64x128x64, 4.43 -> 4.36 for DIFFUSION at 100x256x128; RADDIF at
// 40x64x32, which waits for its chain, is 1 % faster with the FP64 product).
struct SorRows {
  typedef double Word;
  typedef double Kept;
  static constexpr int kWords = 8, kThreads = 1024;
  static constexpr bool kStrided = true, kBoundary = false;
  const double *a, *xm, *xp, *jm, *jp, *km, *kp, *b;
  double* x;
  double omega;
  long long rows;  // ny times the theta rows that are swept
  int nx, ny, nz, poles;
  FastDiv by_items, by_ny;
  template <int COL>
  __device__ void before(unsigned int, unsigned int) const {}
  __device__ bool boundary(bool) const { return false; }
  __device__ void write_boundary(unsigned int, unsigned int, bool) const {}
  __device__ double norm(double sum) const { return sum; }
  // radial index (from 0) of item h of a row: i + j + k, all from 1, has COL's parity
  template <int COL>
  __device__ __forceinline__ unsigned int cell(unsigned int row, unsigned int h, unsigned int& j0,
                                               unsigned int& k0) const {
    k0 = div_rem(by_ny, row, j0);
    return 2 * h + ((j0 + k0 + COL + 1) & 1);
  }
  template <int COL>
  __device__ __forceinline__ void fetch(unsigned int row, unsigned int h, double* to, unsigned int T, uint64_t pol) const {
    unsigned int j0, k0;
    const unsigned int i0 = cell<COL>(row, h, j0, k0);
    if ((int)i0 >= nx) return;
    const size_t c = i0 + (size_t)nx * row;
    copy_async(to, a + c, pol);
    copy_async(to + T, xm + c, pol);
    copy_async(to + 2 * T, xp + c, pol);
    copy_async(to + 3 * T, jm + c, pol);
    copy_async(to + 4 * T, jp + c, pol);
    copy_async(to + 5 * T, km + c, pol);
    copy_async(to + 6 * T, kp + c, pol);
    copy_async(to + 7 * T, b + c, pol);
  }
  template <int COL>
  __device__ __forceinline__ double update(unsigned int row, unsigned int h, const double* w, unsigned int T, bool,
                                           double* kept) const {
    unsigned int j0, k0;
    const unsigned int i0 = cell<COL>(row, h, j0, k0);
    if ((int)i0 >= nx) return 0.0;
    const size_t sj = (size_t)(nx + 4), sk = sj * (size_t)(ny + 4);
    const size_t q = (i0 + 2) + sj * (j0 + 2) + sk * (k0 + 2);
    const size_t qjm = j0 == 0 ? q + sj * (size_t)(ny - 1) : q - sj;
    const size_t qjp = (int)j0 == ny - 1 ? q - sj * (size_t)(ny - 1) : q + sj;
    const double xc = x[q], ac = w[0];
    const double xkm = poles && k0 == 0 ? xc : x[q - sk];
    const double xkp = poles && (int)k0 == nz - 2 ? xc : x[q + sk];
    const double resid = mul_rn(ac, xc) + mul_rn(w[T], x[q - 1]) + mul_rn(w[2 * T], x[q + 1]) +
                         mul_rn(w[3 * T], x[qjm]) + mul_rn(w[4 * T], x[qjp]) + mul_rn(w[5 * T], xkm) +
                         mul_rn(w[6 * T], xkp) - w[7 * T];
    x[q] = xc - div_rn(mul_rn(omega, resid), ac);
    if (kept) *kept = xc;
    return fabs(resid);
  }
  __device__ __forceinline__ void restore(unsigned int row, unsigned int h, double kept) const {
    unsigned int j0, k0;
    const unsigned int i0 = cell<0>(row, h, j0, k0);
    if ((int)i0 < nx) x[(i0 + 2) + (size_t)(nx + 4) * ((j0 + 2) + (size_t)(ny + 4) * (k0 + 2))] = kept;
  }
};

inline SorRows sor_rows(const double* const coef[7], const double* b, double* x, int nx, int ny, int nz, int zmax,
                        int poles, double omega) {
  SorRows s;
  s.a = coef[0]; s.xm = coef[1]; s.xp = coef[2]; s.jm = coef[3]; s.jp = coef[4]; s.km = coef[5]; s.kp = coef[6];
  s.b = b;
  s.x = x;
  s.omega = omega;
  s.rows = (long long)ny * zmax;
  s.nx = nx; s.ny = ny; s.nz = nz; s.poles = poles;
  s.by_items = fast_div((nx + 1) / 2);
  s.by_ny = fast_div(ny);
  return s;
}

}  // namespace ttfld
