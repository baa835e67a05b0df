// fb_source.cu -- the source terms of one gas substep in one pass:
// FillForcesArrays (src/Pframeforce.c:44-129), SubStep1 (src/SourceEuler.c:
// 765-1009), the velocity kicks of self-gravity (src/sgupdate.c),
// ComputeViscousTerms and UpdateVelocitiesWithViscosity (src/Viscosity.c:
// 159-378) and SubStep2 (src/SourceEuler.c:1012-1116).
//
// The expressions and their operand order are the reference's, term for term
// (the parity build's results do not depend on how the pass is cut up).
#include <cuda_runtime.h>
#include <math.h>
#include "fb_dev.cuh"

// A CTA owns a tile of SRC_CO azimuths and 5 fewer rings than it holds rows: a
// lane per column, SRC_R consecutive rings per warp, with a halo of three
// columns and rings before the tile and two after it, as far as the stencils
// of the five steps reach.  Every cell of the tile goes through a step at the
// same time; a neighbouring column's value comes by a warp shuffle, a
// neighbouring ring's from the thread's own registers or, across warps,
// through a row in shared memory, one barrier per step.  So every field is
// read once and only the final velocities and energy are written.
//
// What bounds it: FP64 issue and the latency of each step's chain (divisions,
// roots); the five kernels it replaces, one cell a thread, spent their time on
// 4-5 passes over memory and on launches.  Isothermal 768x2304: 126 us in
// launches of their own -> 70 (280.6 -> 246.7 a substep), 333x1001 with energy
// 116.9 -> 107.9 a substep, 128x384 51.5 -> 47.3, 48x144 45.3 -> 41.9.  A
// version that marched down a column lost on small grids (48x144: 54 a
// substep): a ring's chain of some 4,800 cycles is then serial.
#define SRC_MAXW 16  // warps per CTA
#define SRC_LEFT 3
#define SRC_CO 27    // 32 - SRC_LEFT - 2
#define SRC_HALO 5   // rows of the CTA's tile that are halo: three below, two above

// per-ring table rows: fb_source_table's, then those that each CTA fills in
enum { T_RINF, T_RSUP, T_RMED, T_INVRMED, T_INVDIFFRMED, T_INVDIFFRSUP, T_INVRINF, T_INVDXTHETA, T_C0, T_C1, T_P15,
       T_CS, T_TORQUE, T_NU, T_N };
static_assert(T_TORQUE == FB_SRC_TAB, "the rows of fb_source_table");

int fb_source_tiles(int ns) { return (ns + SRC_CO - 1) / SRC_CO; }

void fb_source_table(const fb_geom *g, const double *invdxtheta, const double *p15, const double *cs_ring, double *out)
{
  const int nr = g->nr;
  for (int i = 0; i < nr; i++) {
    double *t = out + (size_t)i * FB_SRC_TAB;
    t[T_RINF] = g->rinf[i];
    t[T_RSUP] = g->rsup[i];
    t[T_RMED] = g->rmed[i];
    t[T_INVRMED] = g->invrmed[i];
    t[T_INVDIFFRMED] = g->invdiffrmed[i];
    t[T_INVDIFFRSUP] = g->invdiffrsup[i];
    t[T_INVRINF] = g->invrinf[i];
    t[T_INVDXTHETA] = invdxtheta[i];
    t[T_C0] = (i > 0) ? g->rinf[i] - g->rmed[i - 1] : 0.0;  // sgupdate.c's weights of the two cell-centred accelerations
    t[T_C1] = g->rmed[i] - g->rinf[i];
    t[T_P15] = p15[i];
    t[T_CS] = cs_ring[i];
  }
}

// SMs of the current device
static int fb_sms(void)
{
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    cudaGetLastError();
  return sms > 0 ? sms : 1;
}

struct SrcPlanets {
  int np;
  double m[FB_MAX_PLANETS], x[FB_MAX_PLANETS], y[FB_MAX_PLANETS], s2[FB_MAX_PLANETS], invd3[FB_MAX_PLANETS];
  double ind_x, ind_y;
};

static __device__ __forceinline__ double up1(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }    // column j-1's
static __device__ __forceinline__ double dn1(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }  // column j+1's

// Quotients by d = rho(l) + rho(neighbour): pressure gradient a / d, viscosity
// a / (0.5 d) and artificial viscosity a / d share the reciprocal of d (2 r is
// the correctly rounded reciprocal of 0.5 d), so that a quotient whose
// numerator comes late in the chain costs three dependent operations.
// fb_quot is exact with the parity build's fb_rcp.

// ENERGY: energy equation (else the pressure is rho cs^2 of the ring's sound
// speed); PART: the grids the particles read are written too; SG: with
// self-gravity the potential and SubStep1 have run beside the convolution
// (k_potential, k_substep1: they do not need its result) and left vri and vti;
// this pass starts from them with the kicks.  R rings per warp.
template <bool ENERGY, bool PART, bool SG, int R>
__global__ void __launch_bounds__(SRC_MAXW * 32, 2) k_sources(KP k, int ntiles)
{
  fb_grid_dependency();
  __shared__ SrcPlanets pl;
  __shared__ double tab[SRC_MAXW * R][T_N];
  // rows handed to the warp above (top: a warp's last ring) or below
  // (bottom: its first ring)
  __shared__ double s_rho[SRC_MAXW][32], s_p[SRC_MAXW][32], s_pot[SRC_MAXW][32], s_vt[SRC_MAXW][32];
  __shared__ double s_ar[SG ? SRC_MAXW : 1][32], s_ip[PART ? SRC_MAXW : 1][32];
  __shared__ double s_vti[SRC_MAXW][32], s_vri[SRC_MAXW][32], s_trp[SRC_MAXW][32];
  const fb_ctl *c = k.ctl;
  const int ns = k.ns, nr = k.nr;
  const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x, rows = nw * R - SRC_HALO;
  const int i0 = blockIdx.y * rows, i1 = min(nr, i0 + rows);
  const int rb = i0 - 3;                              // ring of the CTA's first row
  const int m = lane - SRC_LEFT;                      // tile column
  const bool col = (m >= 0) && (m < SRC_CO) && (tile * SRC_CO + m < ns);
  int j = (tile * SRC_CO + m) % ns;
  if (j < 0) j += ns;
  // every global load first
  double rho[R], en[R], vr[R], vt[R], pot[R], ip[R], ar[R], at[R];
#pragma unroll
  for (int q = 0; q < R; q++) {
    const int r = rb + w * R + q;
    rho[q] = en[q] = vr[q] = vt[q] = pot[q] = ip[q] = ar[q] = at[q] = 0.0;
    if (r >= 0 && r < nr) {
      const size_t l = (size_t)r * ns + j;
      rho[q] = k.rho[l];
      if (ENERGY) en[q] = k.e[l];
      vr[q] = SG ? k.vri[l] : k.vr[l];
      vt[q] = SG ? k.vti[l] : k.vt[l];
      if (!SG && k.lsa) {  // k_potential has left both
        pot[q] = k.pot[l];
        if (PART) ip[q] = k.indpot[l];
      }
      if (SG) {
        ar[q] = k.sg_accr[l];
        at[q] = k.sg_acct[l];
      }
    }
  }
  const double ca = SG ? 0.0 : k.cosaz[j], sa = SG ? 0.0 : k.sinaz[j];
  const double dt = c->dt, om = omf(k), domega = k.corot ? c->domega : 0.0;
  // the last substep of a DT leaves the derived fields (fb_download_derived)
  const bool keep = c->done || c->status || c->substeps >= k.cap;
  const bool snap = !SG && c->crash_snap_now;  // the first crash's state (WriteDiskPolar ..., 999)
  const bool visc = (k.visc_mode != 0);
  const size_t dgrid = PART ? dust_grid_write(k) : 0;
  {
    const int np = SG ? 0 : c->np;
    if ((int)threadIdx.x < np) {
      const int p = threadIdx.x;
      pl.m[p] = c->pot_m[p];
      pl.x[p] = c->pot_x[p];
      pl.y[p] = c->pot_y[p];
      pl.s2[p] = c->pot_smooth2[p];
      pl.invd3[p] = c->pot_invd3[p];
    }
    if (threadIdx.x == 0) {
      pl.np = np;
      pl.ind_x = c->ind_x;
      pl.ind_y = c->ind_y;
    }
    for (int t = threadIdx.x; t < nw * R; t += blockDim.x) {
      const int r = rb + t;
      if (r < 0 || r >= nr) continue;
      const double *g = k.src_tab + (size_t)r * FB_SRC_TAB;
#pragma unroll
      for (int f = 0; f < FB_SRC_TAB; f++) tab[t][f] = g[f];
      tab[t][T_TORQUE] = k.supp_torque[r];
      // FViscosity(Rmed[r]) (Viscosity.c:23-69)
      tab[t][T_NU] = (k.visc_mode == 1) ? k.alpha * k.gcs[r] * k.gcs[r] * g[T_P15] : k.nu_const;
    }
  }
  const size_t ncell = (size_t)nr * ns;
  if (blockIdx.y == 0 && w == 0 && col) {  // ring nr: SubStep2's copies leave zeros there (nothing reads it before)
    const size_t l = ncell + j;
    k.vr[l] = 0.0;
    k.vt[l] = 0.0;
    if (ENERGY) k.e[l] = 0.0;
  }
  __syncthreads();
  // ---- pressure and potential
  const bool use_ind = (!k.discard_gas_it) && (fabs(k.pmax - k.pmin - 2. * M_PI) < 0.01);
  double P[R];
#pragma unroll
  for (int q = 0; q < R; q++) {
    const int t = w * R + q, r = rb + t;
    P[q] = 0.0;
    if (SG || r < 0 || r >= nr) continue;
    // CorrectVtheta (SideEuler.c:1133-1147): the frame's angular velocity has
    // just changed by domega (k_planets).  Particles have read the corrected
    // state before this pass: k_correct_vtheta ran then.
    if (!PART && k.corot) vt[q] -= domega * tab[t][T_RMED];
    P[q] = ENERGY ? (k.gamma - 1.0) * en[q] : rho[q] * tab[t][T_CS] * tab[t][T_CS];
    if (!k.lsa) {
      const double x = tab[t][T_RMED] * ca, y = tab[t][T_RMED] * sa;
      double sum = 0.0;
      for (int p = 0; p < pl.np; p++) {
        const double dx = x - pl.x[p], dy = y - pl.y[p];
        const double distancesmooth = sqrt(dx * dx + dy * dy + pl.s2[p]);
        double pp = -FB_G * pl.m[p] / distancesmooth;
        if (k.indirect_term) {
          const double ind = FB_G * pl.m[p] * pl.invd3[p] * (x * pl.x[p] + y * pl.y[p]);
          pp += ind;
          if (PART && k.dust_feel_planets) ip[q] = ind;  // Pframeforce.c:102-103 assigns, last planet wins
        }
        sum += pp;
      }
      double ps = -FB_G * 1.0 * tab[t][T_INVRMED];  // 1.0 / Rmed[r], correctly rounded on the host
      if (use_ind) {
        ps -= pl.ind_x * x + pl.ind_y * y;
        if (PART && k.dust_feel_disk) ip[q] -= pl.ind_x * x + pl.ind_y * y;
      }
      pot[q] = sum + ps;
    }
    if ((keep || PART || snap) && col && r >= i0 && r < i1) {
      const size_t l = (size_t)r * ns + j;
      if (keep) {
        k.pres[l] = P[q];
        if (!k.lsa) k.pot[l] = pot[q];
      }
      if (PART && !k.lsa) k.indpot[l] = ip[q];  // IndPotential (Pframeforce.c:55-121)
      if (snap) {
        k.crash_snap[l] = rho[q];
        k.crash_snap[ncell + l] = vr[q];
        k.crash_snap[2 * ncell + l] = vt[q];
        if (ENERGY) k.crash_snap[3 * ncell + l] = en[q];
      }
    }
  }
  s_rho[w][lane] = rho[R - 1];
  if (SG) {
    s_ar[w][lane] = ar[R - 1];
  } else {
    s_p[w][lane] = P[R - 1];
    s_pot[w][lane] = pot[R - 1];
    s_vt[w][lane] = vt[R - 1];
    if (PART) s_ip[w][lane] = ip[R - 1];
  }
  __syncthreads();
  // ---- SubStep1 (SourceEuler.c:765-1009) and the kicks (sgupdate.c)
  const int wb = (w > 0) ? w - 1 : 0, wa = (w < nw - 1) ? w + 1 : w;  // the first and last rows are halo
  double rhob = s_rho[wb][lane], rhomb = s_rho[wb][max(lane - 1, 0)];  // the ring below the warp's first
  double Pb = 0.0, potb = 0.0, vtb = 0.0, vtbp = 0.0, arb = 0.0, ipb = 0.0;
  if (SG) {
    arb = s_ar[wb][lane];
  } else {
    Pb = s_p[wb][lane];
    potb = s_pot[wb][lane];
    vtb = s_vt[wb][lane];
    vtbp = s_vt[wb][min(lane + 1, 31)];
    if (PART) ipb = s_ip[wb][lane];
  }
  const double rho_below = rhob, rhom_below = rhomb;
  double vri[R], vti[R], dr[R], rdr[R], dm[R], rdm[R], rhom[R];
#pragma unroll
  for (int q = 0; q < R; q++) {
    const int t = w * R + q, r = rb + t;
    const double *T = tab[t];
    rhom[q] = up1(rho[q]);
    vri[q] = vti[q] = 0.0;
    dr[q] = rho[q] + rhob;
    rdr[q] = fb_rcp(dr[q]);
    dm[q] = rho[q] + rhom[q];
    rdm[q] = fb_rcp(dm[q]);
    const bool in = (r >= 0 && r < nr), mine = PART && col && r >= i0 && r < i1;
    const size_t l = (size_t)r * ns + j;
    double vtp = 0.0;
    if (SG) {
      const double atm = up1(at[q]);
      if (in) {
        vri[q] = vr[q];
        if (r >= 1) {
          const double radsgacc = (T[T_C0] * ar[q] + T[T_C1] * arb) * T[T_INVDIFFRMED];
          vri[q] = vri[q] + dt * radsgacc;
          if (mine) k.rsga[l] = radsgacc;
        }
        const double azisgacc = 0.5 * (at[q] + atm);
        vti[q] = vt[q] + dt * azisgacc;
        if (mine) k.asga[l] = azisgacc;
      }
    } else {
      vtp = dn1(vt[q]);
      const double Pm = up1(P[q]), potm = up1(pot[q]);
      const double ipm = PART ? up1(ip[q]) : 0.0;
      if (in) {
        if (r >= 1) {
          const double idrm = T[T_INVDIFFRMED];
          const double gradp = fb_quot((P[q] - Pb) * 2.0, dr[q], rdr[q]) * idrm;
          const double gradphi = (pot[q] - potb) * idrm;
          double vt2 = vt[q] + vtp + vtb + vtbp;
          vt2 = vt2 / 4.0 + T[T_RINF] * om;
          vt2 = vt2 * vt2;
          vri[q] = vr[q] + dt * (-gradp - gradphi + vt2 * T[T_INVRINF]);
          if (mine) {  // RadGradP, RadIndAcc (SourceEuler.c:875-877)
            k.rgp[l + dgrid] = (P[q] - Pb) * idrm;
            k.rind[l + dgrid] = -(ip[q] - ipb) * idrm;
          }
        }
        const double idx = T[T_INVDXTHETA];
        const double gradp = fb_quot((P[q] - Pm) * 2.0, dm[q], rdm[q]) * idx;
        const double gradphi = (pot[q] - potm) * idx;
        vti[q] = vt[q] - dt * (gradp + gradphi);
        vti[q] += dt * T[T_TORQUE];
        if (mine) {  // AziGradP, AziIndAcc (SourceEuler.c:944-951)
          k.agp[l + dgrid] = (P[q] - Pm) * idx;
          k.aind[l + dgrid] = -(ip[q] - ipm) * idx;
        }
      }
    }
    rhob = rho[q];
    Pb = P[q];
    potb = pot[q];
    vtb = vt[q];
    vtbp = vtp;
    arb = ar[q];
    ipb = ip[q];
  }
  if (visc) {
    s_vti[w][lane] = vti[R - 1];
    s_vri[w][lane] = vri[0];
    __syncthreads();
    // ---- ComputeViscousTerms (Viscosity.c:159-303)
    const double vri_above = (w < nw - 1) ? s_vri[wa][lane] : 0.0;
    double vtib = s_vti[wb][lane];
    double trr[R], tpp[R], trp[R];
    rhob = rho_below;
    rhomb = rhom_below;
    const double invdphi = k.invdphi, onethird = 1.0 / 3.0;
#pragma unroll
    for (int q = 0; q < R; q++) {
      const int t = w * R + q, r = rb + t;
      const double *T = tab[t];
      const double vrim = up1(vri[q]), vtip = dn1(vti[q]);
      trr[q] = tpp[q] = trp[q] = 0.0;
      if (r >= 0 && r < nr) {
        const double nu = T[T_NU], irm = T[T_INVRMED], idrs = T[T_INVDIFFRSUP];
        const double vrip = (q + 1 < R) ? vri[(q + 1 < R) ? q + 1 : q] : vri_above;
        double div = (vrip * T[T_RSUP] - vri[q] * T[T_RINF]) * idrs * irm;
        div += (vtip - vti[q]) * invdphi * irm;
        const double Drr = (vrip - vri[q]) * idrs;
        const double Dpp = (vtip - vti[q]) * invdphi * irm + 0.5 * (vrip + vri[q]) * irm;
        trr[q] = 2.0 * rho[q] * nu * (Drr - onethird * div);
        tpp[q] = 2.0 * rho[q] * nu * (Dpp - onethird * div);
        if (r >= 1 && t >= 1) {
          const double Drp = 0.5 * (T[T_RINF] * (vti[q] * irm - vtib * tab[t - 1][T_INVRMED]) * T[T_INVDIFFRMED] +
                                    (vri[q] - vrim) * invdphi * T[T_INVRINF]);
          trp[q] = 2.0 * 0.25 * (rho[q] + rhob + rhom[q] + rhomb) * nu * Drp;
        }
        if (!ENERGY && keep && col && r >= i0 && r < i1) k.divv[(size_t)r * ns + j] = div;
      }
      rhob = rho[q];
      rhomb = rhom[q];
      vtib = vti[q];
    }
    s_p[w][lane] = trr[R - 1];  // the pressure's and potential's rows are done with
    s_pot[w][lane] = tpp[R - 1];
    s_trp[w][lane] = trp[0];
    __syncthreads();
    // ---- UpdateVelocitiesWithViscosity (Viscosity.c:305-378)
    const double trp_above = s_trp[wa][lane];
    double trrb = s_p[wb][lane], tppb = s_pot[wb][lane];
#pragma unroll
    for (int q = 0; q < R; q++) {
      const int t = w * R + q, r = rb + t;
      const double *T = tab[t];
      const double trpp = dn1(trp[q]), tppm = up1(tpp[q]);
      if (r >= 1 && r < nr && t >= 1) {
        const double trpip = (q + 1 < R) ? trp[(q + 1 < R) ? q + 1 : q] : trp_above;
        if (r < nr - 1)
          vti[q] = vti[q] +
                   fb_quot(dt * T[T_INVRMED] *
                               ((T[T_RSUP] * trpip - T[T_RINF] * trp[q]) * T[T_INVDIFFRSUP] + (tpp[q] - tppm) * invdphi +
                                0.5 * (trp[q] + trpip)),
                           0.5 * dm[q], 2.0 * rdm[q]);
        vri[q] = vri[q] +
                 fb_quot(dt * T[T_INVRINF] *
                             ((T[T_RMED] * trr[q] - tab[t - 1][T_RMED] * trrb) * T[T_INVDIFFRMED] +
                              (trpp - trp[q]) * invdphi - 0.5 * (tpp[q] + tppb)),
                         0.5 * dr[q], 2.0 * rdr[q]);
      }
      trrb = trr[q];
      tppb = tpp[q];
    }
  }
  s_vti[w][lane] = vri[R - 1];  // both rows are done with (or unused without viscosity)
  s_vri[w][lane] = vri[0];
  __syncthreads();
  // ---- SubStep2 (SourceEuler.c:1012-1116)
  const double vri_above = (w < nw - 1) ? s_vri[wa][lane] : 0.0;
  double vrib = s_vti[wb][lane];
  rhob = rho_below;
#pragma unroll
  for (int q = 0; q < R; q++) {
    const int t = w * R + q, r = rb + t;
    const double *T = tab[t];
    const double vtp = dn1(vti[q]);
    const double vrip = (q + 1 < R) ? vri[(q + 1 < R) ? q + 1 : q] : vri_above;
    const double dvr = vrip - vri[q], dvb = vri[q] - vrib, dvt = vtp - vti[q];
    const double qr = (dvr < 0.0) ? FB_CVNR * FB_CVNR * rho[q] * dvr * dvr : 0.0;
    const double qrb = (r >= 1 && dvb < 0.0) ? FB_CVNR * FB_CVNR * rhob * dvb * dvb : 0.0;
    const double qt = (dvt < 0.0) ? FB_CVNR * FB_CVNR * rho[q] * dvt * dvt : 0.0;
    const double qtm = up1(qt);
    if (r >= i0 && r < i1) {
      const size_t l = (size_t)r * ns + j;
      const double vrn = (r >= 1) ? vri[q] - fb_quot(dt * 2.0, dr[q], rdr[q]) * (qr - qrb) * T[T_INVDIFFRMED] : 0.0;
      const double vtn = vti[q] - fb_quot(dt * 2.0, dm[q], rdm[q]) * (qt - qtm) * T[T_INVDXTHETA];
      if (col) {
        k.vr_mid[l] = vrn;
        k.vt_mid[l] = vtn;
        if (ENERGY) k.e_mid[l] = en[q] - dt * qr * dvr * T[T_INVDIFFRSUP] - dt * qt * dvt * T[T_INVDXTHETA];
      }
      if (ENERGY && k.beta_cooling) {
        // SubStep3's ring mean of vtheta (SourceEuler.c:1196-1203): this
        // tile's part, summed in a fixed order
        double v = col ? vtn + T[T_RMED] * om : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) k.vt_part[(size_t)r * ntiles + tile] = v;
      }
    }
    vrib = vri[q];
    rhob = rho[q];
  }
}

template <bool ENERGY, bool PART, bool SG>
static void launch_sources(const KP &k, cudaStream_t s)
{
  // two rings per warp, except where one per warp still fits the GPU at once:
  // the fewer rows then only shorten every thread's chain
  const int ntiles = fb_source_tiles(k.ns), rows1 = SRC_MAXW - SRC_HALO, rows2 = 2 * SRC_MAXW - SRC_HALO;
  const int g1 = (k.nr + rows1 - 1) / rows1, g2 = (k.nr + rows2 - 1) / rows2;
  if ((long)ntiles * g1 <= 2L * fb_sms())
    fb_launch(k_sources<ENERGY, PART, SG, 1>, dim3(ntiles, g1), SRC_MAXW * 32, 0, s, k, ntiles);
  else
    fb_launch(k_sources<ENERGY, PART, SG, 2>, dim3(ntiles, g2), SRC_MAXW * 32, 0, s, k, ntiles);
}

void fb_launch_sources(const KP &k, cudaStream_t s)
{
  const bool part = k.particles != 0, sg = k.self_gravity != 0;
  if (k.energy) {
    if (part)
      sg ? launch_sources<true, true, true>(k, s) : launch_sources<true, true, false>(k, s);
    else
      sg ? launch_sources<true, false, true>(k, s) : launch_sources<true, false, false>(k, s);
  } else {
    if (part)
      sg ? launch_sources<false, true, true>(k, s) : launch_sources<false, true, false>(k, s);
    else
      sg ? launch_sources<false, false, true>(k, s) : launch_sources<false, false, false>(k, s);
  }
}
