// fb_thermdiff.cu -- thermal diffusion of the energy equation: SubStep0
// (src/SourceEuler.c:722-762) with ComputeEntropyDiffusion (:1740-1789),
// ComputeRadiativeDiffusion (:1791-1876) and the implicit solver
// SORsolver_RadiativeDiffusion (:1878-2052).
//
// Per substep, after the controller has set dt and before the sound speed:
//  1. k_td_fields: per cell the entropy logarithm log((gamma-1) e /
//     Sigma^gamma) (0 where the argument is not positive) and the
//     temperature (gamma-1) e / Sigma;
//  2. explicit radiative diffusion: k_td_coefficient, the flux-limited (Kley
//     1989) diffusion coefficient K per cell of rings 0..nr-2 (ring nr-1
//     reads ring nr-2's, as the reference copies it), from the opacity of
//     the current state;
//  3. k_td_apply: the entropy and radiative sources of rings 1..nr-2 and
//     the explicit update energy += EntropyDiff dt, then += RadiativeDiff dt
//     (two roundings, as the reference adds them one after the other);
//  4. implicit radiative diffusion: the opacity of the (explicitly updated)
//     state, k_td_fields again for the temperature, k_td_coefficient (chi per
//     cell), k_sor_coef (the coefficients a..f of rings 1..nr-2 and each CTA's part
//     of the initial residual norm), then the solver.
//
// The solve is one persistent kernel: k_sor_cluster, one thread-block cluster,
// on grids that it holds, else k_sor_solve with a CTA on every SM.  An iteration is the reference's two chessboard passes: pass 1
// updates the cells (i, j) of rings 1..nr-2 with i + j odd, pass 2 those
// with i + j even.  A cell's five-point stencil reaches only cells of the
// other colour (with an even NSEC the azimuthal wrap keeps that true), so
// the cells of one pass are independent and updating them in parallel gives
// exactly the reference's sequential sweep.  Between the passes and after
// the second the CTAs meet at a barrier (the cluster's own, or an atomic arrival
// counter on which every wait is bounded: one that runs out sets
// FB_ERR_TIMEOUT in the control block and the kernel returns).  The
// residual norm sum(|resid|) of an iteration is summed per CTA and the
// partial sums, double-buffered by iteration parity, are added by every CTA
// in the same fixed order, so every CTA takes the same convergence decision
// (norm < epsilonSOR x initial norm).  The norm's order of summation differs
// from the reference's sequential one by rounding only, which can move the
// decision only for a norm within ~1e-16 relative of the threshold.
// On convergence Energy = Sigma T / (gamma-1) on rings 0..nr-1; after
// MAXITS iterations without it the energy is left as it was, as the
// reference leaves it.  omegaSOR and niterbuf then evolve as SubStep0 has
// them evolve.
#include <math.h>
#include <cooperative_groups.h>
#include "fb_dev.cuh"

#define TD_BS 256

// ---------------------------------------------------------------- fields
// entropy logarithm (ComputeEntropyDiffusion's TempInt) and temperature
// (ComputeRadiativeDiffusion's and the solver's TempInt), rings 0..nr-1
__global__ void __launch_bounds__(TD_BS) k_td_fields(KP k, int want_s, int want_t)
{
  fb_grid_dependency();
  const size_t n = (size_t)k.nr * k.ns;
  for (size_t l = (size_t)blockIdx.x * TD_BS + threadIdx.x; l < n; l += (size_t)gridDim.x * TD_BS) {
    const double energy = k.e[l], dens = k.rho[l];
    if (want_s) {
      const double buf = (k.gamma - 1.0) * energy / pow(dens, k.gamma);
      double s = 0.0;
      if (buf > 0.0) s = log(buf);
      k.td_s[l] = s;
    }
    if (want_t) k.td_t[l] = (k.gamma - 1.0) * energy / dens;
  }
}

// Flux limiter lambda(R) of Kley (1989) as the reference writes it
static __device__ __forceinline__ double td_lambda(double Rl)
{
  if (Rl <= 2.0) return 2. / (3. + sqrt(9.0 + 10.0 * Rl * Rl));
  return 10. / (10. * Rl + 9.0 + sqrt(180. * Rl + 81.));
}

// R of the flux limiter at cell (i, j) of the temperature field t
static __device__ __forceinline__ double td_rl(const KP &k, const double *t, int i, int j, size_t l)
{
  const int ns = k.ns;
  const size_t lip = l + ns, ljp = (j == ns - 1) ? (size_t)i * ns : l + 1;
  const double a = k.invdiffrmed[i + 1] * (t[lip] - t[l]);
  const double b = k.invrmed[i] * k.invdphi * (t[ljp] - t[l]);
  const double gradT = sqrt(a * a + b * b);
  return (8.0 * sqrt(k.gamma * t[l]) * k.p15[i] / k.rho[l] / k.opacity[l]) * (gradT / t[l]);
}

// K (explicit, :1826-1838) or chi (implicit, :1921-1933) of rings 0..nr-2
__global__ void __launch_bounds__(TD_BS) k_td_coefficient(KP k, int implicit)
{
  fb_grid_dependency();
  const int ns = k.ns;
  const size_t n = (size_t)(k.nr - 1) * ns;
  for (size_t l = (size_t)blockIdx.x * TD_BS + threadIdx.x; l < n; l += (size_t)gridDim.x * TD_BS) {
    const int i = (int)(l / ns), j = (int)(l - (size_t)i * ns);
    const double *t = k.td_t;
    const double lambda = td_lambda(td_rl(k, t, i, j, l));
    const double dens = k.rho[l], opacity = k.opacity[l];
    if (!implicit)
      k.td_k[l] = 32.0 * k.sigma_sb * lambda * sqrt(k.gamma) * pow(t[l], 3.5) * k.p15[i] / dens / opacity;
    else
      k.td_k[l] = 64.0 * k.sigma_sb * lambda * k.gamma * (k.gamma - 1.0) * pow(t[l], 4.0) * pow(k.rmed[i], 3.0) *
                  pow(dens, -2.0) / opacity;
  }
}

// the coefficient at cell l of ring i, ring nr-1 reading ring nr-2's
static __device__ __forceinline__ double td_coef(const KP &k, int i, size_t l)
{
  return (i == k.nr - 1) ? k.td_k[l - k.ns] : k.td_k[l];
}

// Explicit thermal diffusion: EntropyDiff (:1770-1788) and RadiativeDiff
// (:1845-1874) of rings 1..nr-2 (the other rings' sources stay zero, as the
// reference never writes them), then SubStep0's update of rings 0..nr-1
// (:737-746).  Each cell reads only the entropy and temperature fields and
// K, none of which this kernel writes, so the update is made in place.
__global__ void __launch_bounds__(TD_BS) k_td_apply(KP k)
{
  fb_grid_dependency();
  const int ns = k.ns, nr = k.nr;
  const double dt = k.ctl->dt;
  const size_t n = (size_t)nr * ns;
  for (size_t l = (size_t)blockIdx.x * TD_BS + threadIdx.x; l < n; l += (size_t)gridDim.x * TD_BS) {
    const int i = (int)(l / ns), j = (int)(l - (size_t)i * ns);
    double energy = k.e[l];
    if (i >= 1 && i <= nr - 2) {
      const size_t lip = l + ns, lim = l - ns;
      const size_t ljp = (j == ns - 1) ? (size_t)i * ns : l + 1;
      const size_t ljm = (j == 0) ? (size_t)i * ns + ns - 1 : l - 1;
      const double irm = k.invrmed[i];
      if (k.ent_diff) {
        const double *t = k.td_s;
        const double laplacien =
            k.invdiffrsup[i] * irm *
                (k.rsup[i] * k.invdiffrmed[i + 1] * (t[lip] - t[l]) - k.rinf[i] * k.invdiffrmed[i] * (t[l] - t[lim])) +
            irm * irm * k.invdphi * k.invdphi * (t[ljp] + t[ljm] - 2.0 * t[l]);
        const double ed = energy * k.diffusivity * laplacien;
        k.td_ent[l] = ed;
        energy += ed * dt;
      }
      if (k.rad_diff == 1) {
        const double *t = k.td_t;
        const double kl = k.td_k[l], kip = td_coef(k, i + 1, lip), kim = k.td_k[lim];
        const double kjp = k.td_k[ljp], kjm = k.td_k[ljm];
        const double rm = k.rmed[i], rmp = k.rmed[i + 1], rmm = k.rmed[i - 1];
        const double KRsup = ((rmp - k.rsup[i]) * kl + (k.rsup[i] - rm) * kip) / (rmp - rm);
        const double KRinf = ((rm - k.rinf[i]) * kim + (k.rinf[i] - rmm) * kl) / (rm - rmm);
        const double KPhisup = 0.5 * (kl + kjp);
        const double KPhiinf = 0.5 * (kl + kjm);
        const double divF =
            k.invdiffrsup[i] * irm *
                (k.rsup[i] * KRsup * k.invdiffrmed[i + 1] * (t[lip] - t[l]) -
                 k.rinf[i] * KRinf * k.invdiffrmed[i] * (t[l] - t[lim])) +
            irm * irm * k.invdphi * k.invdphi * (KPhisup * (t[ljp] - t[l]) - KPhiinf * (t[l] - t[ljm]));
        const double rd = 2.0 * sqrt(k.gamma * t[l]) * k.p15[i] * divF;
        k.td_rad[l] = rd;
        energy += rd * dt;
      }
    }
    k.e[l] = energy;
  }
}

// ------------------------------------------------------------------ solver
#define SOR_BS 512  // threads per CTA of k_sor_solve

// Sum over the CTA in a fixed order (warp trees, then the warps' sums)
static __device__ double td_block_sum(double v, double *sh)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sh[0] = v;
  }
  __syncthreads();
  const double r = sh[0];
  __syncthreads();
  return r;
}

// Sum of the n partial sums p[0..n) in a fixed order (every CTA that calls
// it gets the same value); the partials come from other CTAs: read past L1
static __device__ double td_partials_sum(const double *p, int n, double *sh)
{
  double v = 0.0;
  for (int q = threadIdx.x; q < n; q += blockDim.x) v += __ldcg(p + q);
  return td_block_sum(v, sh);
}

// the five-point residual of the solver's equation at cell l
// (SourceEuler.c:1993, 2012) with the temperatures read past L1
static __device__ __forceinline__ double sor_resid(const KP &k, const double *t, int i, int j, size_t l)
{
  const int ns = k.ns;
  const size_t lip = l + ns, lim = l - ns;
  const size_t ljp = (j == ns - 1) ? (size_t)i * ns : l + 1;
  const size_t ljm = (j == 0) ? (size_t)i * ns + ns - 1 : l - 1;
  return k.sor_c[0][l] * __ldcg(t + lip) + k.sor_c[1][l] * __ldcg(t + lim) + k.sor_c[2][l] * __ldcg(t + ljp) +
         k.sor_c[3][l] * __ldcg(t + ljm) + k.sor_c[4][l] * __ldcg(t + l) - k.sor_c[5][l];
}

// The coefficients a..f of the cells of rings 1..nr-2 (SourceEuler.c:
// 1941-1966) from chi and the temperature, and this CTA's part of the
// initial residual norm (:1977-1991), stored at sor_part[2 G + CTA].  The
// CTA resets the solver's barrier counter first (no barrier is active now).
__global__ void __launch_bounds__(TD_BS) k_sor_coef(KP k)
{
  fb_grid_dependency();
  __shared__ double sh[32];
  const int ns = k.ns, nr = k.nr, G = gridDim.x;
  if (blockIdx.x == 0 && threadIdx.x == 0) k.sor_bar[0] = 0u;
  const double dt = k.ctl->dt;
  const double *chi = k.td_k, *t = k.td_t;
  const size_t n0 = (size_t)ns, n1 = (size_t)(nr - 1) * ns;
  double acc = 0.0;
  for (size_t l = n0 + (size_t)blockIdx.x * TD_BS + threadIdx.x; l < n1; l += (size_t)G * TD_BS) {
    const int i = (int)(l / ns), j = (int)(l - (size_t)i * ns);
    const size_t lip = l + ns, lim = l - ns;
    const size_t ljp = (j == ns - 1) ? (size_t)i * ns : l + 1;
    const size_t ljm = (j == 0) ? (size_t)i * ns + ns - 1 : l - 1;
    const double cl = chi[l], cip = td_coef(k, i + 1, lip), cim = chi[lim];
    const double rm = k.rmed[i], rmp = k.rmed[i + 1], rmm = k.rmed[i - 1];
    const double chiRsup = ((rmp - k.rsup[i]) * cl + (k.rsup[i] - rm) * cip) / (rmp - rm);
    const double chiRinf = ((rm - k.rinf[i]) * cim + (k.rinf[i] - rmm) * cl) / (rm - rmm);
    const double chiPhisup = 0.5 * (cl + chi[ljp]);
    const double chiPhiinf = 0.5 * (cl + chi[ljm]);
    const double irm = k.invrmed[i];
    const double a = -dt * k.rsup[i] * k.invdiffrsup[i] * chiRsup * irm * k.invdiffrmed[i + 1];
    const double b = -dt * k.rinf[i] * k.invdiffrsup[i] * chiRinf * irm * k.invdiffrmed[i];
    const double c = -dt * chiPhisup * irm * irm * k.invdphi * k.invdphi;
    const double d = -dt * chiPhiinf * irm * irm * k.invdphi * k.invdphi;
    const double e = 1.0 - a - b - c - d;
    const double f = t[l];
    k.sor_c[0][l] = a;
    k.sor_c[1][l] = b;
    k.sor_c[2][l] = c;
    k.sor_c[3][l] = d;
    k.sor_c[4][l] = e;
    k.sor_c[5][l] = f;
    const double resid = a * t[lip] + b * t[lim] + c * t[ljp] + d * t[ljm] + e * t[l] - f;
    acc += fabs(resid);
  }
  acc = td_block_sum(acc, sh);
  if (threadIdx.x == 0) k.sor_part[2 * G + blockIdx.x] = acc;
}

#define SOR_WAIT_LIMIT (1 << 21)  // polls of the arrival counter (each an L2 round trip: about 1.5 s)

// Grid barrier of the solver's CTAs: everyone adds one to the arrival counter
// (reset by k_sor_coef) and waits, a bounded number of polls, until it has
// reached `goal`, the CTAs times the barriers so far.  Returns false (for the
// whole CTA) if the wait ran out.
static __device__ bool sor_barrier(unsigned int *bar, unsigned int &goal, int *flag)
{
  goal += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    int ok = 0;
    for (int it = 0; it < SOR_WAIT_LIMIT; it++) {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if (v >= goal) { ok = 1; break; }
    }
    __threadfence();
    *flag = ok;
  }
  __syncthreads();
  return *flag != 0;
}

// SubStep0's omegaSOR and niterbuf after a solve of niter iterations
// (:751-759); MAXITS + 1 when it did not converge
static __device__ void sor_statics(fb_ctl *c, int niter)
{
  const double best = c->sor_omega;
  double w = c->sor_omega;
  if (!(niter < c->sor_niterbuf)) {
    w *= 0.9999;
    if ((w >= 2.0) || (w <= 1.0)) w = best;
  }
  c->sor_omega = w;
  c->sor_niterbuf = niter;
  c->sor_iters = niter;
}

__global__ void __launch_bounds__(SOR_BS) k_sor_solve(KP k, int gcoef)
{
  __shared__ double sh[32];
  __shared__ int flag;
  const int ns = k.ns, nr = k.nr, G = gridDim.x, half = ns / 2;
  unsigned int gen = 0;
  const double omega = k.ctl->sor_omega;
  const double init = td_partials_sum(k.sor_part + 2 * gcoef, gcoef, sh);
  double *t = k.td_t;
  const size_t ncol = (size_t)(nr - 2) * half;
  int n, converged = 0;
  for (n = 1; n <= FB_SOR_MAXITS; n++) {
    double acc = 0.0;
    for (int pass = 0; pass < 2; pass++) {
      // pass 1: the cells with i + j odd (jchess starts at 0 on ring 1),
      // pass 2: i + j even
      for (size_t c = (size_t)blockIdx.x * SOR_BS + threadIdx.x; c < ncol; c += (size_t)G * SOR_BS) {
        const int i = 1 + (int)(c / half), jj = (int)(c - (size_t)(i - 1) * half);
        const int j = 2 * jj + (pass == 0 ? ((i - 1) & 1) : (i & 1));
        const size_t l = (size_t)i * ns + j;
        const double resid = sor_resid(k, t, i, j, l);
        acc += fabs(resid);
        __stcg(t + l, __ldcg(t + l) - omega * resid / k.sor_c[4][l]);
      }
      if (pass == 0 && !sor_barrier(k.sor_bar, gen, &flag)) goto timeout;
    }
    acc = td_block_sum(acc, sh);
    if (threadIdx.x == 0) k.sor_part[(n & 1) * G + blockIdx.x] = acc;
    if (!sor_barrier(k.sor_bar, gen, &flag)) goto timeout;
    if (td_partials_sum(k.sor_part + (n & 1) * G, G, sh) < FB_SOR_EPS * init) {
      converged = 1;
      break;
    }
  }
  if (converged) {  // Energy from the solved temperature (:2031-2036)
    const size_t nc = (size_t)nr * ns;
    for (size_t l = (size_t)blockIdx.x * SOR_BS + threadIdx.x; l < nc; l += (size_t)G * SOR_BS)
      k.e[l] = k.rho[l] * __ldcg(t + l) / (k.gamma - 1.0);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) sor_statics(k.ctl, n);
  return;
timeout:
  if (threadIdx.x == 0) {
    k.ctl->status = FB_ERR_TIMEOUT;
    k.ctl->done = 1;
  }
}

// ------------------------------------------------------- solver in a cluster
// The same iteration by one thread-block cluster, for grids that fit its
// shared memory.  A red-black pass is a few dozen FP64 operations a cell on
// data that never change owner, so what the solve costs is its two grid
// barriers an iteration (about 3 us each over 296 CTAs through global
// atomics); a cluster's hardware barrier takes a fraction of that.  CTA
// `rank` holds the temperatures of its block of rings in shared memory, the two
// colours apart (all four neighbours of a cell are of the other colour, at the
// same or the next index, so no access conflicts), with one halo ring on each
// side; who updates a ring next to another CTA's block also stores it into that
// CTA's halo.  A thread keeps the coefficients of its M cells per colour (with
// the reciprocal of e) in registers: grids of more than three cells per colour
// and thread go to k_sor_solve (reread from the caches, the coefficients cost
// more than the barrier saves: 192 x 576 2357 us a substep against 1846).
// Measured, us per substep of an adiabatic disc (before / grid-wide kernel
// below / this one): 8 x 16 1833 / 1357 / 523, 64 x 192 2332 / 1741 / 573, 128 x
// 384 2106 / 1803 / 823; 192 x 576 2401 / 1846 / -, 512 x 1536 3775 / 3632 / -.
#define SORC_MAX 16  // CTAs of the largest cluster
#define SORC_BS 512
#define SORC_M 3     // most cells per colour and thread

static __device__ __forceinline__ double sorc_update(double a, double b, double c, double d, double e, double f,
                                                     double re, double omega, double tip, double tim, double tjp,
                                                     double tjm, double t, double &acc)
{
  const double resid = a * tip + b * tim + c * tjp + d * tjm + e * t - f;
  acc += fabs(resid);
  return t - fb_quot(omega * resid, e, re);
}

template <int M>
__global__ void __launch_bounds__(SORC_BS) k_sor_cluster(KP k, int G)
{
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ double sorc_t[];  // [colour][row -1 .. rows][half]
  __shared__ double sh[32];
  __shared__ double part[2][SORC_MAX];
  const int ns = k.ns, nr = k.nr, half = ns / 2, T = blockDim.x, tid = threadIdx.x;
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int rows = (nr - 2 + C - 1) / C;             // rings per CTA (the last may hold fewer, or none)
  const int ra = 1 + rank * rows, rn = max(0, min(rows, nr - 1 - ra));
  const size_t plane = (size_t)(rows + 2) * half;
  // cell (ring i, azimuth j) of this CTA's block and halo: colour (i + j) & 1
  auto at = [&](double *base, int col, int lr, int jj) -> double & { return base[(size_t)col * plane + (size_t)(lr + 1) * half + jj]; };
  if (rn > 0)
    for (int c = tid; c < (rn + 2) * ns; c += T) {
      const int lr = c / ns - 1, j = c - (lr + 1) * ns, i = ra + lr;
      at(sorc_t, (i + j) & 1, lr, j >> 1) = k.td_t[(size_t)i * ns + j];
    }
  double *below = (rank > 0 && rn > 0) ? cl.map_shared_rank(sorc_t, rank - 1) : nullptr;
  double *above = (ra + rn < nr - 1) ? cl.map_shared_rank(sorc_t, rank + 1) : nullptr;
  const int ncell = rn * half;  // of each colour
  const double omega = k.ctl->sor_omega;
  const double init = td_partials_sum(k.sor_part + 2 * G, G, sh);
  // own cells c = tid + m T of each colour: row c / half, azimuth index c % half
  double ca[2][M], cb[2][M], cc[2][M], cd[2][M], ce[2][M], cf[2][M],
      cr[2][M];
#pragma unroll
  for (int pass = 0; pass < 2; pass++)
#pragma unroll
    for (int m = 0; m < M; m++) {
      const int c = tid + m * T;
      if (c >= ncell) continue;
      const int lr = c / half, jj = c - lr * half, i = ra + lr, j = 2 * jj + ((pass == 0) ? ((i - 1) & 1) : (i & 1));
      const size_t l = (size_t)i * ns + j;
      ca[pass][m] = k.sor_c[0][l];
      cb[pass][m] = k.sor_c[1][l];
      cc[pass][m] = k.sor_c[2][l];
      cd[pass][m] = k.sor_c[3][l];
      ce[pass][m] = k.sor_c[4][l];
      cf[pass][m] = k.sor_c[5][l];
      cr[pass][m] = fb_rcp(ce[pass][m]);
    }
  // where the cells sit in a colour's plane, and their azimuthal neighbours
  int off[M], offp[M], offm[M];
  bool first[M], lastr[M], odd[M];  // in the block's first / last ring; j odd in pass 0
#pragma unroll
  for (int m = 0; m < M; m++) {
    const int c = tid + m * T, lr = c / half, jj = c - lr * half;
    off[m] = c + half;  // row lr + 1
    offp[m] = (jj + 1 == half) ? off[m] + 1 - half : off[m] + 1;
    offm[m] = (jj == 0) ? off[m] + half - 1 : off[m] - 1;
    first[m] = (lr == 0);
    lastr[m] = (lr == rn - 1);
    odd[m] = ((ra + lr - 1) & 1) != 0;
  }
  cl.sync();
  int n, converged = 0;
  for (n = 1; n <= FB_SOR_MAXITS; n++) {
    double acc = 0.0;
#pragma unroll
    for (int pass = 0; pass < 2; pass++) {
      const int col = (pass == 0) ? 1 : 0;  // pass 1 of the reference: i + j odd
      double *own = sorc_t + (size_t)col * plane;
      const double *oth = sorc_t + (size_t)(col ^ 1) * plane;
      // the cell at o, its neighbours at the next (op) and the previous (om)
      // index: an odd j's are jj and jj + 1, an even j's jj - 1 and jj
      auto cell = [&](int o, int op, int om, bool od, bool fst, bool lst, double a, double b, double cx, double d,
                      double e, double f, double re) {
        const double t = sorc_update(a, b, cx, d, e, f, re, omega, oth[o + half], oth[o - half], oth[od ? op : o],
                                     oth[od ? o : om], own[o], acc);
        own[o] = t;
        if (fst && below) below[(size_t)col * plane + o + (size_t)rows * half] = t;  // a block below another is full
        if (lst && above) above[(size_t)col * plane + o - (size_t)rn * half] = t;
      };
#pragma unroll
      for (int m = 0; m < M; m++)
        if (tid + m * T < ncell)
          cell(off[m], offp[m], offm[m], odd[m] != (pass == 1), first[m], lastr[m], ca[pass][m], cb[pass][m],
               cc[pass][m], cd[pass][m], ce[pass][m], cf[pass][m], cr[pass][m]);
      if (pass == 0) cl.sync();
    }
    acc = td_block_sum(acc, sh);
    if (tid < C) *cl.map_shared_rank(&part[n & 1][rank], tid) = acc;  // to every CTA
    cl.sync();
    double sum = 0.0;
    for (int q = 0; q < C; q++) sum += part[n & 1][q];
    if (sum < FB_SOR_EPS * init) {
      converged = 1;
      break;
    }
  }
  if (converged) {  // Energy from the solved temperature (:2031-2036)
    for (int c = tid; c < rn * ns; c += T) {
      const int lr = c / ns, j = c - lr * ns, i = ra + lr;
      const size_t l = (size_t)i * ns + j;
      k.e[l] = k.rho[l] * at(sorc_t, (i + j) & 1, lr, j >> 1) / (k.gamma - 1.0);
    }
    if (rank == 0)
      for (int c = tid; c < 2 * ns; c += T) {  // the rings the solver leaves alone
        const size_t l = (c < ns) ? (size_t)c : (size_t)(nr - 1) * ns + (c - ns);
        k.e[l] = k.rho[l] * k.td_t[l] / (k.gamma - 1.0);
      }
  }
  if (rank == 0 && tid == 0) sor_statics(k.ctl, n);
  cl.sync();  // no CTA leaves while another may still store into its halo
}

// ------------------------------------------------------------------ launch
static int td_grid(const KP &k)
{
  const size_t n = (size_t)k.nr * k.ns;
  const size_t g = (n + TD_BS - 1) / TD_BS;
  return (int)(g < 4096 ? g : 4096);
}

// CTAs of k_sor_coef (the size of the partial sums' arrays): two per SM
int fb_sor_grid(void)
{
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return 2 * sms;
}

// CTAs of the grid-wide solver: one per SM (all resident together; the launch
// is cooperative too), fewer where a pass has fewer cells than they have
// threads: the barrier costs by the CTA.
static int sor_solve_grid(const KP &k)
{
  const long ncol = (long)(k.nr - 2) * (k.ns / 2), g = (ncol + SOR_BS - 1) / SOR_BS, sms = k.sor_grid / 2;
  return (int)(g < 1 ? 1 : g < sms ? g : sms);
}

static size_t sorc_smem(int nr, int ns, int C)
{
  return (size_t)2 * ((nr - 2 + C - 1) / C + 2) * (ns / 2) * sizeof(double);
}

// cells per colour and thread of a cluster of C CTAs
static int sorc_m(const KP &k, int C)
{
  const int rows = (k.nr - 2 + C - 1) / C;
  return (rows * (k.ns / 2) + SORC_BS - 1) / SORC_BS;
}

static cudaLaunchConfig_t sorc_config(const KP &k, int C, cudaLaunchAttribute *at, cudaStream_t s)
{
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = C;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(SORC_BS);
  cfg.dynamicSmemBytes = sorc_smem(k.nr, k.ns, C);
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// CTAs of the cluster that solves this grid, 0 where the grid-wide kernel
// does: the largest cluster the device schedules, 16 (which functions must opt
// into) or 8, that holds the grid.  Its colours' planes need an even nsec; a
// parameter file with an odd one is refused, overrides of its fields are not.
static int sorc_size(const KP &k)
{
  if (k.nr < 4 || (k.ns & 1)) return 0;
  const void *fns[SORC_M] = {(const void *)k_sor_cluster<1>, (const void *)k_sor_cluster<2>,
                             (const void *)k_sor_cluster<3>};
  for (int C = SORC_MAX; C >= 8; C /= 2) {
    const int m = sorc_m(k, C);
    if (m > SORC_M) continue;
    const void *fn = fns[m - 1];
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg = sorc_config(k, C, at, 0);
    int nc = 0;
    if (fb_allow_max_dynamic_smem(fn) != FB_OK ||
        (C > 8 && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
        cudaOccupancyMaxActiveClusters(&nc, fn, &cfg) != cudaSuccess || nc < 1) {
      cudaGetLastError();
      continue;
    }
    return C;
  }
  return 0;
}

int fb_launch_substep0(const KP &k, cudaStream_t s)
{
  int n = 0;
  const int g = td_grid(k);
  if (k.ent_diff || k.rad_diff == 1) {  // explicit sources and update (:737-746)
    fb_launch(k_td_fields, g, TD_BS, 0, s, k, k.ent_diff, k.rad_diff == 1 ? 1 : 0);
    n++;
    if (k.rad_diff == 1) {  // the opacity of this state was computed before the CFL kernel
      fb_launch(k_td_coefficient, g, TD_BS, 0, s, k, 0);
      n++;
    }
    fb_launch(k_td_apply, g, TD_BS, 0, s, k);
    n++;
  }
  if (k.rad_diff == 2) {  // implicit radiative diffusion (:749-760)
    n += fb_launch_opacity_now(k, s);
    fb_launch(k_td_fields, g, TD_BS, 0, s, k, 0, 1);
    fb_launch(k_td_coefficient, g, TD_BS, 0, s, k, 1);
    fb_launch(k_sor_coef, k.sor_grid, TD_BS, 0, s, k);
    cudaLaunchAttribute at[1];
    const int C = sorc_size(k);
    if (C > 0) {
      const cudaLaunchConfig_t cfg = sorc_config(k, C, at, s);
      switch (sorc_m(k, C)) {
        case 1: cudaLaunchKernelEx(&cfg, k_sor_cluster<1>, k, k.sor_grid); break;
        case 2: cudaLaunchKernelEx(&cfg, k_sor_cluster<2>, k, k.sor_grid); break;
        default: cudaLaunchKernelEx(&cfg, k_sor_cluster<3>, k, k.sor_grid); break;
      }
    } else {
      cudaLaunchConfig_t cfg = {};
      cfg.stream = s;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      at[0].id = cudaLaunchAttributeCooperative;
      at[0].val.cooperative = 1;
      cfg.gridDim = dim3(sor_solve_grid(k));
      cfg.blockDim = dim3(SOR_BS);
      cudaLaunchKernelEx(&cfg, k_sor_solve, k, k.sor_grid);
    }
    n += 4;
  }
  return n;
}

// The explicit radiative diffusion's time-step limit invdt6 of every cell
// of rings 1..nr-1 (SourceEuler.c:1413-1424), into the RadiativeDiff
// scratch field (free until SubStep0) for the CFL kernel that follows.  The
// Temperature field of the reference is (gamma-1) e / Sigma of the current
// state on rings 0..nr-1 and zero on ring nr, which it never writes; the
// opacity is the one computed for this state just before.
__global__ void __launch_bounds__(TD_BS) k_td_cfl(KP k)
{
  fb_grid_dependency();
  const int ns = k.ns, nr = k.nr;
  const size_t n0 = (size_t)ns, n1 = (size_t)nr * ns;
  for (size_t l = n0 + (size_t)blockIdx.x * TD_BS + threadIdx.x; l < n1; l += (size_t)gridDim.x * TD_BS) {
    const int i = (int)(l / ns), j = (int)(l - (size_t)i * ns);
    const size_t ljp = (j == ns - 1) ? (size_t)i * ns : l + 1;
    const double dens = k.rho[l];
    const double T = (k.gamma - 1.0) * k.e[l] / dens;
    const double Tip = (i + 1 <= nr - 1) ? (k.gamma - 1.0) * k.e[l + ns] / k.rho[l + ns] : 0.0;
    const double Tjp = (k.gamma - 1.0) * k.e[ljp] / k.rho[ljp];
    const double opacity = k.opacity[l];
    const double a = k.invdiffrmed[i + 1] * (Tip - T), b = k.invrmed[i] * k.invdphi * (Tjp - T);
    const double gradT = sqrt(a * a + b * b);
    const double Rl = (8.0 * sqrt(k.gamma * T) * k.p15[i] / dens / opacity) * gradT / T;
    const double lambda = td_lambda(Rl);
    const double chicoeff = 64.0 * lambda * k.sigma_sb * k.gamma * (k.gamma - 1.0) * pow(T, 4.0) / opacity /
                            (dens * dens) * pow(k.rmed[i], 3.0);
    k.td_rad[l] = chicoeff * 4.0 / k.mindx2[i];
  }
}

int fb_launch_td_cfl(const KP &k, cudaStream_t s)
{
  fb_launch(k_td_cfl, td_grid(k), TD_BS, 0, s, k);
  return 1;
}
