// fp64_path.cu -- the FP64 drop-in path (LB3DC_FP64).
//
// Stage-by-stage kernels whose arithmetic is, expression for expression,
// the FP64 restatement of the reference (the oracle): the same operation
// order, no FMA contraction (this file is compiled with --fmad=false) and
// the deterministic exp/tanh of detmath.h, so that the device reproduces
// the host restatement bit for bit.  The 1e-12-after-1000-steps parity
// target is below the chaotic amplification of a single rounding
// difference, which is why bit identity is the design goal here.
//
// Layout in HBM (structure of arrays, site index x fastest):
//   f, g   : [nc][19][nsites]  pre-stream state / post-stream populations
//   rho    : [nc][nsites]      post-stream densities
//   psi    : [nc][nsites]      1 - exp(-rho), evaluated once per site
//   mom    : [nc][3][nsites]   post-stream momenta (the reference's u_*)
//   da, db : [3][nsites]       advected dipole flux / dipoles (ternary)
//   rock   : [nsites] uint8
// Lees-Edwards x-halo planes (binary): [nc][19][nz][ny] pre-stream, and
// [nc][nz][ny] densities after streaming.

#include <cstdio>

#include "common.cuh"
#include "detmath.h"
#include "fp64_path.h"
#include "inflow.cuh"
#include "le_common.cuh"

namespace lb3d {
namespace fp64 {

using lb3d_detmath::det_exp;
using lb3d_detmath::det_tanh;

__device__ __forceinline__ double get_psi(double rho) { return 1.0 - det_exp(-rho); }

__device__ __forceinline__ void site_xyz(long long i, int nx, int ny, int &x, int &y, int &z) {
  long long t = i / nx;
  x = (int)(i - t * nx);
  z = (int)(t / ny);
  y = (int)(t - (long long)z * ny);
}

// Site offsets of the -1, 0, +1 neighbours along each axis with the periodic
// wrap applied once, as byte offsets of a double array: a kernel adds three of
// them per neighbour and reads every field at that one 32-bit offset (lattices
// of more than 2^29 sites, where they would overflow, take 370 GB binary and 580
// GB ternary; lb3dc_create refuses them).  Ternary 128^3: dipole pass 113 -> 92
// us (with four CTAs per SM), surfactant stream 126 -> 106 us (with three),
// collide pass 453 -> 438 us; its pulls keep their 64-bit addresses, with which
// the compiler does not hoist them into spills.
struct Nb {
  unsigned x[3], y[3], z[3];
  __device__ __forceinline__ Nb(int px, int py, int pz, int nx, int ny, int nz) {
    const unsigned row = 8u * nx, pl = row * ny;
    x[0] = 8u * (px == 0 ? nx - 1 : px - 1), x[1] = 8u * px, x[2] = 8u * (px == nx - 1 ? 0 : px + 1);
    y[0] = row * (py == 0 ? ny - 1 : py - 1), y[1] = row * py, y[2] = row * (py == ny - 1 ? 0 : py + 1);
    z[0] = pl * (pz == 0 ? nz - 1 : pz - 1), z[1] = pl * pz, z[2] = pl * (pz == nz - 1 ? 0 : pz + 1);
  }
  // of the neighbour at +c_q (SGN 1) or the upstream site at -c_q (SGN -1)
  template <int SGN>
  __device__ __forceinline__ unsigned at(int q) const {
    return x[1 + SGN * cx(q)] + y[1 + SGN * cy(q)] + z[1 + SGN * cz(q)];
  }
};
// A plain load: with programmatic dependent launch most of what it reads is
// written by the kernel just before, which may still run when this one starts.
__device__ __forceinline__ double ld(const double *p, unsigned byte) {
  return *reinterpret_cast<const double *>(reinterpret_cast<const char *>(p) + byte);
}

// src: populations [NC][19][nsites], or (COMPACT) the boundary planes
// [2][NC][19][nz][ny] of x = nx - 1 and x = 0.  Writes the halo planes and,
// when rlo is given, their densities and psi (for the force stencil).  Threads
// [0, ny nz) build the bottom halo sites, the next ny nz the top ones, whose
// clipping rule reads the adjusted bottom site: a top thread builds it only
// when the rule applies.  A few thousand threads with a long FP64 chain each:
// one side a thread in 64-thread blocks 16-17 us, both sides a thread in
// 128-thread blocks 20 and 24 us (97x66x63 sites).
template <int NC, bool COMPACT>
__global__ void __launch_bounds__(64) k_le_halo(DevParams P, LEStep S, const double *src,
                          double *__restrict__ hlo, double *__restrict__ hhi,
                          double *__restrict__ rlo, double *__restrict__ rhi,
                          double *__restrict__ plo, double *__restrict__ phi) {
  const int nx = P.nx, ny = P.ny, nz = P.nz, NPi = ny * nz;
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_wait_previous();
  pdl_launch_next();
  if (u >= 2 * NPi) return;
  const bool top = u >= NPi;
  const int t = top ? u - NPi : u;
  const int y = t % ny, z = t / ny;
  const long long N = P.nsites, NP = NPi;
  const double f = S.lefrac;
  auto at = [&](int c, int q, bool low, int zz) {
    const int zw = (zz % nz + nz) % nz;
    if (COMPACT) return src[((low ? 0 : NC * 19) + c * 19 + q) * NP + y + ny * zw];
    return src[(c * 19 + q) * N + sidx(low ? nx - 1 : 0, y, zw, nx, ny)];
  };
  double hb[NC][19];
  auto bottom = [&]() {
    for (int c = 0; c < NC; ++c)
      for (int q = 0; q < 19; ++q)
        hb[c][q] = (1.0 - f) * at(c, q, true, z + S.eoff) + f * at(c, q, true, z + S.eoff + 1);
    le_adjust<NC>(P, hb, hb, S.shear_u, -1.0);
  };
  auto put = [&](const double h[NC][19], double *hp, double *rp, double *pp) {
    if (hp)
      for (int c = 0; c < NC; ++c)
        for (int q = 0; q < 19; ++q) hp[(c * 19 + q) * NP + t] = h[c][q];
    if (rp)
      for (int c = 0; c < NC; ++c) {
        double a = 0.0;
#pragma unroll
        for (int q = 0; q < 19; ++q) a = a + h[c][q] * (double)gw(q);
        rp[c * NP + t] = a;
        pp[c * NP + t] = get_psi(a);
      }
  };
  if (!top) {
    bottom();
    put(hb, hlo, rlo, plo);
    return;
  }
  double ht[NC][19], df[NC][19];
  for (int c = 0; c < NC; ++c)
    for (int q = 0; q < 19; ++q)
      ht[c][q] = f * at(c, q, false, z - S.eoff - 1) + (1.0 - f) * at(c, q, false, z - S.eoff);
  const bool neg = le_adjust_df<NC>(P, ht, S.shear_u, +1.0, df);
  if (neg) bottom();
  le_adjust_apply<NC>(ht, hb, df, neg);
  put(ht, hhi, rhi, phi);
}

// ---------------------------------------------------------------------------
// Advection: pull streaming with half-way bounce-back, the advected dipole
// flux and the post-stream moments (code/lb3d_advection.F90:54-151,
// code/lb3d_bc_bounce.F90:53-90, code/lb3d_analysis.F90:64-102).
// ---------------------------------------------------------------------------
// A thread streams one component (components are independent here; the
// advected dipole flux uses the surfactant only), c0 + blockIdx.y, which keeps
// one component's 19 pulls live; FLUX compiles the dipole flux, accumulated
// for the surfactant.  STORE writes the post-stream populations to fout: the
// moments pass of the pulling step (k_collide with PULL) writes the moments
// only, and under Lees-Edwards the populations of the x boundary planes
// ([2][NC][19][nz][ny], x = nx - 1 and x = 0) to fout for the stage-8 halo.
template <int NC, bool LE, bool FLUX, bool ROCK, bool STORE = true>
__global__ void __launch_bounds__(256, FLUX ? 3 : 2) k_stream(DevParams P, const double *fin,
                                                double *__restrict__ fout, double *__restrict__ rho,
                                                double *__restrict__ psi, double *__restrict__ mom,
                                                double *__restrict__ da,
                                                const double *db,
                                                const uint8_t *__restrict__ rock,
                                                const double *hlo,
                                                const double *hhi, int c0) {
  const int c = c0 + blockIdx.y;
  const long long N = P.nsites;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  int x, y, z;
  site_xyz(i, nx, ny, x, y, z);
  // without rock every site is fluid and the pulls do not wait on rock loads
  const bool fluid = !ROCK || rock[i] == 0;
  const long long NP = (long long)ny * nz;

  const Nb nb(x, y, z, nx, ny, nz);
  // upstream site of each moving direction (32-bit: the FP64 path bounds a
  // lattice at 2^31 sites); negative values mark the LE halo planes
  int up[18];
  bool upf[18];
#pragma unroll
  for (int q = 0; q < 18; ++q) {
    int xu = x - cx(q), yu = wrap(y - cy(q), ny), zu = wrap(z - cz(q), nz);
    if (LE && xu < 0) {
      up[q] = -1 - (yu + ny * zu);  // bottom halo
      upf[q] = true;
    } else if (LE && xu >= nx) {
      up[q] = -1 - (int)NP - (yu + ny * zu);  // top halo
      upf[q] = true;
    } else {
      up[q] = (int)sidx(wrap(xu, nx), yu, zu, nx, ny);
      upf[q] = !ROCK || rock[up[q]] == 0;
    }
  }
  // address of the pulled population: selected, not loaded under a branch, so
  // that the pulls overlap
  auto pulled = [&](int q) -> const double * {
    const double *src = fin + (c * 19 + q) * N + up[q];
    if (LE && up[q] < 0) {
      const long long h = -1 - (long long)up[q];
      src = h < NP ? hlo + (c * 19 + q) * NP + h : hhi + (c * 19 + q) * NP + (h - NP);
    }
    return src;
  };

  pdl_wait_previous();  // from here on, data of earlier kernels
  pdl_launch_next();
  double d0 = 0.0, d1 = 0.0, d2 = 0.0;
  {
    double n[19];
#pragma unroll
    for (int q = 0; q < 18; ++q) {
      if constexpr (!ROCK && !LE) {
        n[q] = ld(fin + (c * 19 + q) * N, nb.at<-1>(q));
      } else {
        const double *src = pulled(q);
        if (!upf[q]) src = fin + (c * 19 + bounce(q)) * N + i;
        if (!fluid) src = fin + (c * 19 + q) * N + i;
        n[q] = *src;
      }
    }
    n[REST] = fin[(c * 19 + REST) * N + i];
    if (LE && !STORE) {
      const long long t = y + (long long)ny * z;
#pragma unroll
      for (int q = 0; q < 19; ++q) {
        if (x == nx - 1) fout[(c * 19 + q) * NP + t] = n[q];
        if (x == 0) fout[((NC + c) * 19 + q) * NP + t] = n[q];
      }
    }
    if (FLUX && c == 2) {
      // advected dipole flux: bounce-back terms first (lb3d_bc_bounce_back_hw
      // runs before lb3d_advection_step), then the pulls, then the rest
      // population (code/lb3d_advection.F90:137-148).
      if (fluid) {
        if (ROCK) {
#pragma unroll
          for (int s = 0; s < 18; ++s) {
            long long ja = sidx(wrap(x + cx(s), nx), wrap(y + cy(s), ny), wrap(z + cz(s), nz), nx, ny);
            if (rock[ja] != 0) {
              double ng = fin[(2 * 19 + s) * N + i] * (double)gw(s);
              d0 = d0 + ng * db[ja];
              d1 = d1 + ng * db[N + ja];
              d2 = d2 + ng * db[2 * N + ja];
            }
          }
        }
#pragma unroll
        for (int q = 0; q < 18; ++q) {
          if (upf[q]) {
            const unsigned j = nb.at<-1>(q);
            double ng = n[q] * (double)gw(q);
            d0 = d0 + ng * ld(db, j);
            d1 = d1 + ng * ld(db + N, j);
            d2 = d2 + ng * ld(db + 2 * N, j);
          }
        }
      }
      double ng = n[REST] * (double)gw(REST);
      d0 = d0 + ng * db[i];
      d1 = d1 + ng * db[N + i];
      d2 = d2 + ng * db[2 * N + i];
    }
    double r = 0.0, u0 = 0.0, u1 = 0.0, u2 = 0.0;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
      if (STORE) fout[(c * 19 + q) * N + i] = n[q];
      r = r + n[q] * (double)gw(q);
    }
    rho[c * N + i] = r;
    psi[c * N + i] = get_psi(r);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
      double ng = n[q] * (double)gw(q);
      u0 = u0 + ng * (double)cx(q);
      u1 = u1 + ng * (double)cy(q);
      u2 = u2 + ng * (double)cz(q);
    }
    mom[(c * 3 + 0) * N + i] = u0;
    mom[(c * 3 + 1) * N + i] = u1;
    mom[(c * 3 + 2) * N + i] = u2;
  }
  if (FLUX && c == 2) {
    da[i] = d0;
    da[N + i] = d1;
    da[2 * N + i] = d2;
  }
}

// ---------------------------------------------------------------------------
// Zou-He flux boundaries, code/lb3d_invasion.F90:2143-2457 (one rank: both
// z planes are boundary planes).  One thread per site of the z = 1 and
// z = nz planes; per component (surfactant, red, blue) the populations
// entering the lattice are closed from the known ones and the inflow uz
// (divided by the density for inv_type < 0), in the expression order of
// the reference; the surfactant's advected dipole flux is recomputed from
// its new populations and the dipoles of the upstream sites (periodic
// images across the planes, as the stage-6 halo holds them).  Densities
// and velocities keep their advection values, as in the reference.
// F(i) is the reference's 1-based direction i.
// ---------------------------------------------------------------------------
template <int NC>
__global__ void k_zouhe_flux(DevParams P, double *__restrict__ g, double *__restrict__ da,
                             const double *__restrict__ db, const uint8_t *__restrict__ rock) {
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  const long long N = P.nsites;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 2 * nx * ny) return;
  const bool bottom = t < nx * ny;
  const int xy = bottom ? t : t - nx * ny;
  const int x = xy % nx, y = xy / nx, z = bottom ? 0 : nz - 1;
  const long long i = sidx(x, y, z, nx, ny);
  if (rock[i] != 0) return;
  const int order[3] = {2, 0, 1};  // surfactant, red, blue
  for (int k = 0; k < 3; ++k) {
    const int c = order[k];
    if (c >= NC) continue;
    double F[19];
    for (int q = 0; q < 19; ++q) F[q] = g[(c * 19 + q) * N + i] * (double)gw(q);
    zouhe_flux_site(F, P.zh_uz[c], bottom, P.inv_type);
    for (int q = 0; q < 19; ++q) g[(c * 19 + q) * N + i] = F[q] / (double)gw(q);
    if (NC == 3 && c == 2) {
      double d0 = 0.0, d1 = 0.0, d2 = 0.0;
      for (int q = 0; q < 19; ++q) {
        const long long j =
            sidx(wrap(x - cx(q), nx), wrap(y - cy(q), ny), wrap(z - cz(q), nz), nx, ny);
        const double ng = g[(2 * 19 + q) * N + i] * (double)gw(q);
        d0 = d0 + ng * db[j];
        d1 = d1 + ng * db[N + j];
        d2 = d2 + ng * db[2 * N + j];
      }
      da[i] = d0;
      da[N + i] = d1;
      da[2 * N + i] = d2;
    }
  }
}

// Zou-He density boundaries, lbe_invade_zouandhe
// (code/lb3d_invasion.F90:1459-1796): the red and blue populations of the
// fluid sites of z = 0 take the densities fr, fb, those of z = nz - 1 the
// densities pr, pb, through the five-population density closure of the
// non-SINGLEFLUID build (Shan-Chen terms zero).  The velocity closure the
// reference runs first writes only populations that this closure
// overwrites, and reads none of them.  F(i) is the reference's 1-based
// direction i; the blue F(13) at z = 0 divides by amass_r as the reference
// writes it (:1567).
__global__ void k_zouhe_density(DevParams P, double *__restrict__ g, const uint8_t *__restrict__ rock,
                                double fr, double fb, double pr, double pb) {
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  const long long N = P.nsites;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 2 * nx * ny) return;
  const bool bottom = t < nx * ny;
  const int xy = bottom ? t : t - nx * ny;
  const int x = xy % nx, y = xy / nx, z = bottom ? 0 : nz - 1;
  const long long i = sidx(x, y, z, nx, ny);
  if (rock[i] != 0) return;
  const double rho_c[2] = {bottom ? fr : pr, bottom ? fb : pb};
  for (int c = 0; c < 2; ++c) {
    double F[19];
    for (int q = 0; q < 19; ++q) F[q] = g[(c * 19 + q) * N + i] * (double)gw(q);
    zouhe_density_site(F, rho_c[c], P.amass[c], bottom ? P.amass[0] : P.amass[c], P.tau[c], bottom);
    for (int q = 0; q < 19; ++q) g[(c * 19 + q) * N + i] = F[q] / (double)gw(q);
  }
}

// ---------------------------------------------------------------------------
// Recolouring inflow of binary mixtures, lbe_invade_binary
// (code/lb3d_invasion.F90:1257-1358): on the post-stream populations, the
// bottom planes z = 0, 1 become red = a * (n_r + n_b), blue = b * (n_r + n_b)
// with (a, b) = (mr, mb), then the top planes z = nz - 2, nz - 1 with
// (a, b) = (mb, mr); rock sites are left alone.  One thread per (x, y)
// column runs the four planes in that order, so lattices with nz < 4, whose
// bottom and top planes coincide, are recoloured as the reference does.
// ---------------------------------------------------------------------------
__global__ void k_recolour(DevParams P, double *__restrict__ g, const uint8_t *__restrict__ rock,
                           double mr, double mb) {
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  const long long N = P.nsites;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nx * ny) return;
  const int x = t % nx, y = t / nx;
  const int zs[4] = {0, 1, nz - 2, nz - 1};
  for (int k = 0; k < 4; ++k) {
    const long long i = sidx(x, y, zs[k], nx, ny);
    if (rock[i] != 0) continue;
    const double a = k < 2 ? mr : mb, b = k < 2 ? mb : mr;
    for (int q = 0; q < 19; ++q) {
      const double pop = g[q * N + i] + g[(19 + q) * N + i];
      g[q * N + i] = a * pop;
      g[(19 + q) * N + i] = b * pop;
    }
  }
}

// c . v of a lattice direction, the products and sums in axis order.  Terms of
// a zero component are left out here and in the sums over directions below:
// adding +-0 changes no finite value, and the compiler may not drop a product
// with 0 by itself.  24 of the 54 components of the moving directions are zero;
// ternary 128^3, a step: 0.830 -> 0.792 ms.  A product of 0 and a number that is
// not finite, which such a term would have added as NaN, belongs to one that
// leaves the sums below without a finite result, too: only then are they formed
// again with every term.
__device__ __forceinline__ double cdot(const int c[3], const double v[3]) {
  double r = 0.0;
  bool any = false;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (c[k]) {
      const double t = v[k] * (double)c[k];
      r = any ? r + t : t;
      any = true;
    }
  return r;
}

__device__ __forceinline__ bool finite_sum(const double a[3]) { return isfinite((a[0] + a[1]) + a[2]); }

// The field of k_dipole with the terms of zero components.
__device__ __forceinline__ void dipole_field_all(const DevParams &P, int x, int y, int z, long long i,
                                                 const double *rho, const double *da, double sgn, double h[3]) {
  const long long N = P.nsites;
  double h_c[3] = {0.0, 0.0, 0.0};
  double h_s[3] = {da[i], da[N + i], da[2 * N + i]};
#pragma unroll 1
  for (int q = 0; q < 18; ++q) {
    const long long j = sidx(wrap(x + cx(q), P.nx), wrap(y + cy(q), P.ny), wrap(z + cz(q), P.nz), P.nx, P.ny);
    const double pas[3] = {da[j], da[N + j], da[2 * N + j]};
    const double hc_m = -(sgn * ((0.0 + rho[N + j]) - (0.0 + rho[j])) * (double)gw(q));
    const double c[3] = {(double)cx(q), (double)cy(q), (double)cz(q)};
    for (int k = 0; k < 3; ++k) h_c[k] = h_c[k] + hc_m * c[k];
    const double hs_dot = 2.0 * ((c[0] * pas[0] + c[1] * pas[1]) + c[2] * pas[2]);
    for (int k = 0; k < 3; ++k) h_s[k] = h_s[k] + (pas[k] - c[k] * hs_dot) * (double)gw(q);
  }
  for (int k = 0; k < 3; ++k) h[k] = h_c[k] + h_s[k];
}

// ---------------------------------------------------------------------------
// Dipole relaxation, code/lb3d_collision.F90:296-403 (ternary, periodic).
// Reads rho and da of the 18 neighbours; writes db in place (no neighbour
// reads db in this pass).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256, 4) k_dipole(DevParams P, const double *rho,
                                                const double *da,
                                                double *__restrict__ db) {
  const long long N = P.nsites;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  int x, y, z;
  site_xyz(i, nx, ny, x, y, z);
  const Nb nb(x, y, z, nx, ny, nz);
  const double *rho_b = rho + N, *da1 = da + N, *da2 = da + 2 * N;
  pdl_wait_previous();
  pdl_launch_next();
  double h_c[3] = {0.0, 0.0, 0.0};
  double h_s[3] = {da[i], da[N + i], da[2 * N + i]};
  double sN_tmp = fmaxf_(rho[2 * N + i], CLIP_RHO_S);
  double sd_tmp[3];
  for (int k = 0; k < 3; ++k) sd_tmp[k] = h_s[k] / sN_tmp;
  const double sgn = (P.g_bs >= 0.0) ? 1.0 : -1.0;
#pragma unroll
  for (int q = 0; q < 18; ++q) {
    const unsigned j = nb.at<1>(q);
    double psi_r = 0.0 + ld(rho, j);
    double psi_b = 0.0 + ld(rho_b, j);
    double pas[3] = {ld(da, j), ld(da1, j), ld(da2, j)};
    double hc_m = -(sgn * (psi_b - psi_r) * (double)gw(q));
    const int c[3] = {cx(q), cy(q), cz(q)};
    for (int k = 0; k < 3; ++k)
      if (c[k]) h_c[k] = h_c[k] + hc_m * (double)c[k];
    double hs_dot = 2.0 * cdot(c, pas);
    for (int k = 0; k < 3; ++k)
      h_s[k] = h_s[k] + (c[k] ? pas[k] - (double)c[k] * hs_dot : pas[k]) * (double)gw(q);
  }
  double h[3];
  for (int k = 0; k < 3; ++k) h[k] = h_c[k] + h_s[k];
  double h_m = P.beta * sqrt((h[0] * h[0] + h[1] * h[1]) + h[2] * h[2]);
  if (!isfinite(h_m)) {
    dipole_field_all(P, x, y, z, i, rho, da, sgn, h);
    h_m = P.beta * sqrt((h[0] * h[0] + h[1] * h[1]) + h[2] * h[2]);
  }
  double sd_eq[3];
  const double third = 1.0 / 3.0;
  for (int k = 0; k < 3; ++k) sd_eq[k] = (third * P.beta) * h[k];
  if (h_m > 10.0e-3) {
    double exh = 1.0 / det_tanh(h_m);
    double sd_mag = exh - 1.0 / h_m;
    for (int k = 0; k < 3; ++k) sd_eq[k] = ((P.beta * h[k]) / h_m) * sd_mag;
  }
  for (int k = 0; k < 3; ++k) sd_eq[k] = sd_eq[k] * P.d_0;
  for (int k = 0; k < 3; ++k) db[k * N + i] = P.omega_d * sd_eq[k] + (1.0 - P.omega_d) * sd_tmp[k];
}

// ---------------------------------------------------------------------------
// Shan-Chen forces (code/lb3d_force_shanchen.F90:127-330).  LE selects the
// Lees-Edwards neighbourhood: x-halo sites from the halo planes (never
// rock), and rock neighbours reached through the y/z halo without their
// rock colour (the Lees-Edwards y/z swaps do not copy it, :1079-1308).
// ---------------------------------------------------------------------------
// ROCK false: no site is rock.
template <bool LE, bool ROCK>
__device__ __forceinline__ void sc_force_binary(const DevParams &P, int x, int y, int z, long long i,
                                                const double *rho, const double *psi,
                                                const uint8_t *__restrict__ rock,
                                                const double *plo, const double *phi, double *fr,
                                                double *fb) {
  const long long N = P.nsites;
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  const long long NP = (long long)ny * nz;
  double f_br[3] = {0, 0, 0}, f_rb[3] = {0, 0, 0}, f_wr[3] = {0, 0, 0}, f_wb[3] = {0, 0, 0};
  // psi of the neighbour in direction q; rk: it is rock
  auto neighbour = [&](int q, double &psi_r, double &psi_b, bool &rk) {
    int xn = x + cx(q), yn = y + cy(q), zn = z + cz(q);
    rk = false;
    if (LE && (xn < 0 || xn >= nx)) {
      long long h = wrap(yn, ny) + (long long)ny * wrap(zn, nz);
      const double *pp = (xn < 0) ? plo : phi;
      psi_r = pp[h];
      psi_b = pp[NP + h];
    } else {
      long long j = sidx(wrap(xn, nx), wrap(yn, ny), wrap(zn, nz), nx, ny);
      if (ROCK && rock[j] != 0) {
        rk = true;
        bool through_halo = (yn < 0 || yn >= ny || zn < 0 || zn >= nz || xn < 0 || xn >= nx);
        double rcr = (LE && through_halo) ? 0.0 : P.rc_r;
        double rcb = (LE && through_halo) ? 0.0 : P.rc_b;
        // rock sites hold no populations, so their density is 0 and their
        // psi is that of the rock colour alone (evaluated once on the host
        // by the same detmath routine: the same bits)
        const double rj = rho[j], bj = rho[N + j];
        const bool coloured = !(LE && through_halo);
        psi_r = (coloured && rj == 0.0) ? P.psi_rc[0] : get_psi(rj + rcr);
        psi_b = (coloured && bj == 0.0) ? P.psi_rc[1] : get_psi(bj + rcb);
      } else {
        psi_r = psi[j];
        psi_b = psi[N + j];
      }
    }
  };
#pragma unroll
  for (int q = 0; q < 18; ++q) {
    const int c[3] = {cx(q), cy(q), cz(q)};
    double psi_r, psi_b;
    bool rk;
    neighbour(q, psi_r, psi_b, rk);
    double green_r = psi_b * (double)gw(q);
    double green_b = psi_r * (double)gw(q);
    if (rk) {
      for (int k = 0; k < 3; ++k) {
        if (c[k] == 0) continue;
        f_wb[k] = f_wb[k] + green_r * (double)c[k];
        f_wr[k] = f_wr[k] + green_b * (double)c[k];
      }
    } else {
      for (int k = 0; k < 3; ++k) {
        if (c[k] == 0) continue;
        f_rb[k] = f_rb[k] + green_r * (double)c[k];
        f_br[k] = f_br[k] + green_b * (double)c[k];
      }
    }
  }
  const double pb = psi[N + i], prr = psi[i];
  auto forces = [&]() {
    for (int k = 0; k < 3; ++k) {
      double br = -(P.g_br * f_br[k]);
      double rb = -(P.g_br * f_rb[k]);
      double wr = -(P.g_wr * f_wr[k]);
      double wb = -(P.g_wb * f_wb[k]);
      fb[k] = (br + ((wb / P.tau[1]) * P.tau_wb)) * pb;
      fr[k] = (rb + ((wr / P.tau[0]) * P.tau_wr)) * prr;
    }
  };
  forces();
  if (finite_sum(fb) && finite_sum(fr)) return;
  // with the terms of zero components
  for (int k = 0; k < 3; ++k) f_br[k] = f_rb[k] = f_wr[k] = f_wb[k] = 0.0;
#pragma unroll 1
  for (int q = 0; q < 18; ++q) {
    const double c[3] = {(double)cx(q), (double)cy(q), (double)cz(q)}, g = (double)gw(q);
    double psi_r, psi_b;
    bool rk;
    neighbour(q, psi_r, psi_b, rk);
    const double green_r = psi_b * g, green_b = psi_r * g;
    for (int k = 0; k < 3; ++k) {
      if (rk) {
        f_wb[k] = f_wb[k] + green_r * c[k];
        f_wr[k] = f_wr[k] + green_b * c[k];
      } else {
        f_rb[k] = f_rb[k] + green_r * c[k];
        f_br[k] = f_br[k] + green_b * c[k];
      }
    }
  }
  forces();
}

// The sums over the directions of sc_force_ternary.
struct TernarySums {
  double br[3] = {0, 0, 0}, rb[3] = {0, 0, 0}, cs[3] = {0, 0, 0}, sc[3] = {0, 0, 0}, ss[3] = {0, 0, 0};
};

// With the terms of zero components.
__device__ __forceinline__ void ternary_sums_all(const DevParams &P, int x, int y, int z, const double *psi,
                                                 const double *db, const double dbx[3], TernarySums &f) {
  const long long N = P.nsites;
  f = TernarySums();
#pragma unroll 1
  for (int q = 0; q < 18; ++q) {
    const long long j = sidx(wrap(x + cx(q), P.nx), wrap(y + cy(q), P.ny), wrap(z + cz(q), P.nz), P.nx, P.ny);
    const double c[3] = {(double)cx(q), (double)cy(q), (double)cz(q)}, g = (double)gw(q);
    const double psi_r = psi[j], psi_b = psi[N + j], pss = psi[2 * N + j];
    const double green_r = psi_b * g, green_b = psi_r * g;
    const double dd[3] = {db[j] * pss, db[N + j] * pss, db[2 * N + j] * pss};
    const double d_dotc = (dd[0] * c[0] + dd[1] * c[1]) + dd[2] * c[2];
    const double di_dotc = (dbx[0] * c[0] + dbx[1] * c[1]) + dbx[2] * c[2];
    const double greenc_s = (psi_b - psi_r) * g, green_ss = 8.0 * g;
    const double di_dot_d = (dd[0] * dbx[0] + dd[1] * dbx[1]) + dd[2] * dbx[2];
    for (int k = 0; k < 3; ++k) {
      f.rb[k] = f.rb[k] + green_r * c[k];
      f.br[k] = f.br[k] + green_b * c[k];
      f.cs[k] = f.cs[k] + (dd[k] - (2.0 * d_dotc) * c[k]) * g;
      f.sc[k] = f.sc[k] + greenc_s * (dbx[k] - (2.0 * di_dotc) * c[k]);
      f.ss[k] = f.ss[k] + green_ss * (((di_dot_d - (2.0 * di_dotc) * d_dotc) * c[k] + dd[k] * di_dotc) +
                                      d_dotc * dbx[k]);
    }
  }
}

__device__ __forceinline__ void sc_force_ternary(const DevParams &P, int x, int y, int z, long long i,
                                                 const double *psi, const double *db, double *fr,
                                                 double *fb, double *fs) {
  const long long N = P.nsites;
  const double *psi_b_ = psi + N, *psi_s_ = psi + 2 * N, *db1 = db + N, *db2 = db + 2 * N;
  TernarySums f;
  const double dbx[3] = {db[i], db[N + i], db[2 * N + i]};
  const Nb nb(x, y, z, P.nx, P.ny, P.nz);
#pragma unroll
  for (int q = 0; q < 18; ++q) {
    const unsigned j = nb.at<1>(q);
    const int c[3] = {cx(q), cy(q), cz(q)};
    const double g = (double)gw(q);
    double psi_r = ld(psi, j);
    double psi_b = ld(psi_b_, j);
    double green_r = psi_b * g;
    double green_b = psi_r * g;
    for (int k = 0; k < 3; ++k) {
      if (c[k] == 0) continue;
      f.rb[k] = f.rb[k] + green_r * (double)c[k];
      f.br[k] = f.br[k] + green_b * (double)c[k];
    }
    double pss = ld(psi_s_, j);
    double dd[3] = {ld(db, j) * pss, ld(db1, j) * pss, ld(db2, j) * pss};
    double d_dotc = cdot(c, dd);
    for (int k = 0; k < 3; ++k)
      f.cs[k] = f.cs[k] + (c[k] ? dd[k] - (2.0 * d_dotc) * (double)c[k] : dd[k]) * g;
    double di_dotc = cdot(c, dbx);
    double greenc_s = (psi_b - psi_r) * g;
    for (int k = 0; k < 3; ++k)
      f.sc[k] = f.sc[k] + greenc_s * (c[k] ? dbx[k] - (2.0 * di_dotc) * (double)c[k] : dbx[k]);
    double di_dot_d = (dd[0] * dbx[0] + dd[1] * dbx[1]) + dd[2] * dbx[2];
    double green_ss = 8.0 * g;
    const double along = di_dot_d - (2.0 * di_dotc) * d_dotc;
    for (int k = 0; k < 3; ++k) {
      const double t = dd[k] * di_dotc;
      f.ss[k] = f.ss[k] + green_ss * ((c[k] ? along * (double)c[k] + t : t) + d_dotc * dbx[k]);
    }
  }
  const double pb = psi[N + i], prr = psi[i], ps = psi[2 * N + i];
  auto forces = [&]() {
    for (int k = 0; k < 3; ++k) {
      double br = -(P.g_br * f.br[k]);
      double rb = -(P.g_br * f.rb[k]);
      double sc = (2.0 * P.g_bs) * f.sc[k];
      double cs = -((2.0 * P.g_bs) * f.cs[k]);
      double ss = -(P.g_ss * f.ss[k]);
      fb[k] = (br + cs) * pb;
      fr[k] = (rb - cs) * prr;
      fs[k] = (sc + ss) * ps;
    }
  };
  forces();
  if (!(finite_sum(fb) && finite_sum(fr) && finite_sum(fs))) {
    ternary_sums_all(P, x, y, z, psi, db, dbx, f);
    forces();
  }
}

template <int NC, bool LE, bool ROCK>
__device__ __forceinline__ void sc_forces(const DevParams &P, int x, int y, int z, long long i,
                                          const double *rho, const double *psi, const double *db,
                                          const uint8_t *rock, const double *plo,
                                          const double *phi, double F[NC][3]) {
  for (int c = 0; c < NC; ++c) F[c][0] = F[c][1] = F[c][2] = 0.0;
  if (rock[i] != 0) return;
  if (NC == 2)
    sc_force_binary<LE, ROCK>(P, x, y, z, i, rho, psi, rock, plo, phi, F[0], F[1]);
  else
    sc_force_ternary(P, x, y, z, i, psi, db, F[0], F[1], F[NC - 1]);
}

// ---------------------------------------------------------------------------
// Forces + BGK, code/lb3d_collision.F90:151-289.  With PULL (lattices without
// inflow boundaries) g is the pre-stream state and each
// post-stream population is pulled from it as k_stream pulls it
// (code/lb3d_advection.F90:109-151, bounce-back from a rock upstream site,
// rock sites unmoved): the moments pass before (k_stream without STORE)
// wrote rho, psi and the momenta, and the post-stream populations never go
// to HBM.  The values are those k_stream would have stored, so f comes out
// the same bit for bit.  Occupancy (measured): the pulling variants run 2
// CTAs of 256 threads per SM, the binary one with rock 3 (faster despite
// its spills: 8.4 against 9.2 ms per step on a 256^3 porous lattice, where
// the ternary one at 3 ran 15 % slower), the staged binary ones 4.
// ---------------------------------------------------------------------------
template <int NC, bool LE, bool PULL = false, bool ROCK = true>
__global__ void __launch_bounds__(256, (PULL && ROCK && NC == 2) ? 3 : ((PULL || NC == 3) ? 2 : 4)) k_collide(DevParams P, const double *__restrict__ g,
                                                 double *__restrict__ f,
                                                 const double *rho,
                                                 const double *psi,
                                                 const double *mom,
                                                 const double *db,
                                                 const uint8_t *__restrict__ rock,
                                                 const double *plo,
                                                 const double *phi,
                                                 const double *__restrict__ hlo = nullptr,
                                                 const double *__restrict__ hhi = nullptr) {
  const long long N = P.nsites;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  int x, y, z;
  site_xyz(i, P.nx, P.ny, x, y, z);
  double F[NC][3];
  pdl_wait_previous();
  pdl_launch_next();
  sc_forces<NC, LE, ROCK>(P, x, y, z, i, rho, psi, db, rock, plo, phi, F);
  double r[NC];
  for (int c = 0; c < NC; ++c) r[c] = rho[c * N + i];
  if (applyforce(P, x + 1, y + 1, z + 1)) {
    for (int c = 0; c < NC; ++c) {
      double mass = P.amass[c] * r[c];
      F[c][2] = F[c][2] + mass * P.g_accn;
      F[c][1] = F[c][1] + mass * P.g_accn_y;
      F[c][0] = F[c][0] + mass * P.g_accn_x;
    }
  }
  double pt[3];
  for (int k = 0; k < 3; ++k) pt[k] = (P.amass[0] * P.omega[0]) * mom[k * N + i];
  for (int c = 1; c < NC; ++c)
    for (int k = 0; k < 3; ++k) pt[k] = pt[k] + (P.amass[c] * P.omega[c]) * mom[(c * 3 + k) * N + i];
  double rho_tilde = (P.amass[0] * r[0]) * P.omega[0];
  for (int c = 1; c < NC; ++c) rho_tilde = rho_tilde + (P.amass[c] * r[c]) * P.omega[c];
  double rt = fmaxf_(rho_tilde, CLIP_RHO);
  double ut[3];
  for (int k = 0; k < 3; ++k) ut[k] = pt[k] / rt;
  auto bgk = [&](int c) {
    double pon = 1.0 / fmaxf_(r[c], CLIP_RHO);
    double du[3];
    for (int k = 0; k < 3; ++k) du[k] = ((P.tau[c] * pon) * F[c][k]) / P.amass[c];
    double b[19];
    boltz2(ut[0], ut[1], ut[2], du[0], du[1], du[2], b);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
      double nq;
      if (q == REST || (ROCK && rock[i] != 0)) {
        nq = g[(c * 19 + q) * N + i];
      } else {
        const int yu = wrap(y - cy(q), P.ny), zu = wrap(z - cz(q), P.nz), xu = x - cx(q);
        const long long j = sidx(wrap(xu, P.nx), yu, zu, P.nx, P.ny);
        // the address is selected, not the load: a branch around each load would
        // keep the 19 pulls from overlapping (172 us against 81 for the sheared
        // 97x66x63 lattice)
        const double *src = g + (c * 19 + q) * N + j;
        bool bounced = ROCK && rock[j] != 0;
        if (LE) {
          // across the sheared boundary: the stage-6 halo planes, never rock
          const long long NP = (long long)P.ny * P.nz, t = (c * 19 + q) * NP + yu + (long long)P.ny * zu;
          if (xu < 0) src = hlo + t, bounced = false;
          if (xu >= P.nx) src = hhi + t, bounced = false;
        }
        if (ROCK && bounced) src = g + (c * 19 + bounce(q)) * N + i;
        nq = *src;
      }
      double eq = r[c] * b[q];
      f[(c * 19 + q) * N + i] = nq - P.omega[c] * (nq - eq);
    }
  };
  // unrolled over the components where the pulls fill the loop (keeps r and
  // F in registers)
  if constexpr (PULL) {
#pragma unroll
    for (int c = 0; c < NC; ++c) bgk(c);
  } else {
    for (int c = 0; c < NC; ++c) {
      double pon = 1.0 / fmaxf_(r[c], CLIP_RHO);
      double du[3];
      for (int k = 0; k < 3; ++k) du[k] = ((P.tau[c] * pon) * F[c][k]) / P.amass[c];
      double b[19];
      boltz2(ut[0], ut[1], ut[2], du[0], du[1], du[2], b);
#pragma unroll
      for (int q = 0; q < 19; ++q) {
        double nq = g[(c * 19 + q) * N + i];
        double eq = r[c] * b[q];
        f[(c * 19 + q) * N + i] = nq - P.omega[c] * (nq - eq);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Science dumps (code/lb3d_io_dump_data.F90:922-1460).  The XDR dump path
// gathers the lattice into a fresh arena with a plain periodic halo
// (code/lb3d_io.F90:387-442, code/lb3d_mpi.F90:783-859), so the dump-time
// forces always use the periodic neighbourhood.
// ---------------------------------------------------------------------------
template <int NC>
__global__ void k_dump(DevParams P, int field, const double *__restrict__ f,
                       const double *__restrict__ rho, const double *__restrict__ psi,
                       const double *__restrict__ db, const uint8_t *__restrict__ rock,
                       double *__restrict__ out) {
  const long long N = P.nsites;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  int x, y, z;
  site_xyz(i, P.nx, P.ny, x, y, z);
  const bool fluid = rock[i] == 0;
  auto sumg = [&](int c, int dir) {
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
      double cc = dir == 0 ? (double)cx(q) : dir == 1 ? (double)cy(q) : dir == 2 ? (double)cz(q) : 1.0;
      acc = acc + (f[(c * 19 + q) * N + i] * (double)gw(q)) * cc;
    }
    return acc;
  };
  switch (field) {
    case 0:  // od
      out[i] = fluid ? P.amass[0] * sumg(0, 3) : 0.0;
      break;
    case 1:  // wd
      out[i] = fluid ? P.amass[1] * sumg(1, 3) : 0.0;
      break;
    case 2:  // sur
      out[i] = (NC == 3) ? P.amass[NC - 1] * sumg(NC - 1, 3) : 0.0;
      break;
    case 3:  // dir
      for (int k = 0; k < 3; ++k) out[3 * i + k] = (NC == 3) ? db[k * N + i] : 0.0;
      break;
    case 4: {  // vel
      if (fluid) {
        double v = 0.0, den = 0.0;
        for (int c = 0; c < NC; ++c) {
          double term = (sumg(c, 2) * P.amass[c]) * P.omega[c];
          v = (c == 0) ? term : v + term;
          double dterm = (sumg(c, 3) * P.amass[c]) * P.omega[c];
          den = (c == 0) ? dterm : den + dterm;
        }
        v = v / fmaxf_(10.0e-9, den);
        if (in_accn_box(P, x + 1, y + 1, z + 1)) v = v - P.g_accn / 2.0;
        out[i] = v;
      } else {
        out[i] = 0.0;
      }
      break;
    }
    case 5: {  // arr
      double F[NC][3];
      sc_forces<NC, false, true>(P, x, y, z, i, rho, psi, db, rock, nullptr, nullptr, F);
      double den = 0.0;
      for (int c = 0; c < NC; ++c) {
        double t = sumg(c, 3) * P.amass[c];
        den = (c == 0) ? t : den + t;
      }
      float dd = (float)den;
      float denf = (1.0e-8f < dd) ? dd : 1.0e-8f;
      for (int k = 0; k < 3; ++k) {
        double v = 0.0;
        for (int c = 0; c < NC; ++c) {
          double m = sumg(c, k) * P.amass[c];
          double corr = ((F[c][k] / 2.0) * sumg(c, 3)) * P.amass[c];
          v = (c == 0) ? (m - corr) : ((v + m) - corr);
        }
        out[3 * i + k] = v / (double)denf;
      }
      if (in_accn_box(P, x + 1, y + 1, z + 1) && fluid) {
        out[3 * i + 0] = out[3 * i + 0] - P.g_accn_x / 2.0;
        out[3 * i + 1] = out[3 * i + 1] - P.g_accn_y / 2.0;
        out[3 * i + 2] = out[3 * i + 2] - P.g_accn / 2.0;
      }
      break;
    }
    case 6:  // rock
      out[i] = fluid ? 0.0 : 1.0;
      break;
  }
}

// Moments of the current state (used by downloads after a collision: the
// reference's rho/u fields then still hold the post-stream moments, which
// the stream kernel stored; this kernel is for states loaded by upload).
template <int NC>
__global__ void k_moments(DevParams P, const double *__restrict__ f, double *__restrict__ rho,
                          double *__restrict__ psi, double *__restrict__ mom) {
  const long long N = P.nsites;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  for (int c = 0; c < NC; ++c) {
    double r = 0.0, u0 = 0.0, u1 = 0.0, u2 = 0.0;
#pragma unroll
    for (int q = 0; q < 19; ++q) r = r + f[(c * 19 + q) * N + i] * (double)gw(q);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
      double ng = f[(c * 19 + q) * N + i] * (double)gw(q);
      u0 = u0 + ng * (double)cx(q);
      u1 = u1 + ng * (double)cy(q);
      u2 = u2 + ng * (double)cz(q);
    }
    rho[c * N + i] = r;
    psi[c * N + i] = get_psi(r);
    mom[(c * 3 + 0) * N + i] = u0;
    mom[(c * 3 + 1) * N + i] = u1;
    mom[(c * 3 + 2) * N + i] = u2;
  }
}

__global__ void k_detmath(int fn, const double *x, double *y, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double v = x[i];
  y[i] = fn == 0 ? det_exp(v) : fn == 1 ? lb3d_detmath::det_expm1(v) : det_tanh(v);
}

static inline unsigned grid_for(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

}  // namespace fp64

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
using namespace fp64;


// A kernel launch; pdl: the kernel may start while the one launched before it
// on the stream, one of those below, drains.  Each kernel waits for the
// previous grid first and lets the next one launch after that, so only
// neighbours overlap: the populations that k_collide pulls were complete before
// it could start and stay read-only loads (as plain loads, which may not pass
// the stores before them, they took the step of ternary 128^3 from 0.76 to 1.35
// ms); every field of an earlier kernel of the step is a plain load.  A step, before ->
// after: ternary 16^3 24.3 -> 19.8 us, 32^3 27.1 -> 26.0, binary 64^3 59.2 ->
// 57.3, sheared 97x66x63 155 -> 144, ternary 128^3 758 -> 753.
template <typename... K, typename... A>
static cudaError_t launch(void (*k)(K...), dim3 grid, int block, cudaStream_t st, bool pdl, A... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, static_cast<K>(a)...);
}

cudaError_t fp64_le_halo(const DevParams &P, const LEStep &S, const double *src, bool compact, double *hlo,
                         double *hhi, double *rlo, double *rhi, double *plo, double *phi,
                         cudaStream_t st, bool pdl) {
  const unsigned g = grid_for(2LL * P.ny * P.nz, 64);
  if (P.nc != 2) return cudaErrorInvalidValue;
  return launch(compact ? k_le_halo<2, true> : k_le_halo<2, false>, dim3(g), 64, st, pdl, P, S, src, hlo, hhi, rlo,
                rhi, plo, phi);
}

// Threads per block of the site kernels, on both sides of each line (a step, 64
// / 128 / 256 threads).  Small lattices take small blocks, which spread their
// sites over more SMs, the smallest 128, whose neighbours share more of an L1:
// ternary 16^3 15.6 / 15.1 / 16.4 us, 25^3 18.6 / 18.2 / 19.6, 32^3 21.1 / 22.2 /
// 24.8, 64^3 110 / 109 / 110; binary 64^3 52.7 / 53.1 / 55.0.  Large ones: ternary
// 68^3 136 / 134 / 134, 96^3 355 / 348 / 345, 128^3 821 / 797 / 795; binary with
// rock 80^3 240 / 235 / 234, 128^3 988 / 976 / 919; binary 72^3 76 / 77 / 78, 128^3
// 411 / 405 / 410, sheared 97x66x63 154 / 155 / 162, 128^3 607 / 598 / 616.
static int fp64_block(const DevParams &P) {
  if (P.nsites > 300000) return P.nc == 3 || P.any_rock ? 256 : 128;
  return P.nsites > 16384 ? 64 : 128;
}
// Up to here all components stream in one launch: its saved launch is worth more
// than the occupancy that red and blue lose to the surfactant's registers (a step
// with one and with two: ternary 16^3 15.1 and 16.3 us, 40^3 28.3 and 32.6, 44^3
// 39.1 and 41.9, 64^3 109.0 and 109.9, 96^3 347 and 349; 112^3 552 and 551, 128^3
// 798 and 794, 160x128x128 1010 and 1002).
static bool fp64_small(const DevParams &P) { return P.nsites <= 1000000; }

// The stream kernel over all components: red and blue in one launch and the
// surfactant, whose dipole flux takes more registers, in another (ternary 128^3:
// 58 + 58 + 107 us as three launches); small lattices all three in one.
template <bool STORE>
static cudaError_t launch_stream(const DevParams &P, const double *fin, double *fout, double *rho, double *psi,
                                 double *mom, double *da, const double *db, const uint8_t *rock, const double *hlo,
                                 const double *hhi, cudaStream_t st, bool pdl = false, bool chain = false) {
  const int bs = fp64_block(P);
  const unsigned gr = grid_for(P.nsites, bs);
  auto go = [&](auto rocky, auto plain, unsigned ny, int c0) {
    const cudaError_t e = launch(P.any_rock ? rocky : plain, dim3(gr, ny), bs, st, pdl, P, fin, fout, rho, psi, mom,
                                 da, db, rock, hlo, hhi, c0);
    pdl = chain;
    return e;
  };
  if (P.nc == 2)
    return P.le ? go(k_stream<2, true, false, true, STORE>, k_stream<2, true, false, false, STORE>, 2, 0)
                : go(k_stream<2, false, false, true, STORE>, k_stream<2, false, false, false, STORE>, 2, 0);
  if (fp64_small(P)) return go(k_stream<3, false, true, true, STORE>, k_stream<3, false, true, false, STORE>, 3, 0);
  const cudaError_t e = go(k_stream<3, false, false, true, STORE>, k_stream<3, false, false, false, STORE>, 2, 0);
  return e != cudaSuccess ? e
                          : go(k_stream<3, false, true, true, STORE>, k_stream<3, false, true, false, STORE>, 1, 2);
}

int fp64_stream_launches(const DevParams &P) { return P.nc == 2 || fp64_small(P) ? 1 : 2; }

cudaError_t fp64_zouhe_flux(const DevParams &P, double *g, double *da, const double *db,
                            const uint8_t *rock, cudaStream_t st) {
  const int n = 2 * P.nx * P.ny;
  if (P.nc == 2)
    k_zouhe_flux<2><<<grid_for(n, 128), 128, 0, st>>>(P, g, da, db, rock);
  else
    k_zouhe_flux<3><<<grid_for(n, 128), 128, 0, st>>>(P, g, da, db, rock);
  return cudaGetLastError();
}

cudaError_t fp64_zouhe_density(const DevParams &P, double *g, const uint8_t *rock, double fr,
                               double fb, double pr, double pb, cudaStream_t st) {
  const int n = 2 * P.nx * P.ny;
  k_zouhe_density<<<grid_for(n, 128), 128, 0, st>>>(P, g, rock, fr, fb, pr, pb);
  return cudaGetLastError();
}

cudaError_t fp64_recolour(const DevParams &P, double *g, const uint8_t *rock, double mr, double mb,
                          cudaStream_t st) {
  const int n = P.nx * P.ny;
  k_recolour<<<grid_for(n, 128), 128, 0, st>>>(P, g, rock, mr, mb);
  return cudaGetLastError();
}

cudaError_t fp64_stream(const DevParams &P, const double *fin, double *fout, double *rho,
                        double *psi, double *mom, double *da, const double *db,
                        const uint8_t *rock, const double *hlo, const double *hhi,
                        cudaStream_t st) {
  return launch_stream<true>(P, fin, fout, rho, psi, mom, da, db, rock, hlo, hhi, st);
}

cudaError_t fp64_step_pull(const DevParams &P, const double *fin, double *fout, double *rho,
                           double *psi, double *mom, double *da, double *db, const uint8_t *rock,
                           cudaStream_t st, const Fp64Le *le, bool chained) {
  if (P.zouhe || (P.le != 0) != (le != nullptr)) return cudaErrorInvalidValue;
  const int bs = fp64_block(P);
  const unsigned gr = grid_for(P.nsites, bs);
  const bool rk = P.any_rock != 0;
  // moments pass: densities, psi, momenta and (surfactant) the advected dipole flux
  cudaError_t e = launch_stream<false>(P, fin, le ? le->post : nullptr, rho, psi, mom, da, db, rock,
                                       le ? le->hlo : nullptr, le ? le->hhi : nullptr, st, chained, true);
  if (e == cudaSuccess && P.nc == 3) e = fp64_dipole(P, rho, da, db, st, true);
  if (e == cudaSuccess && le)
    e = fp64_le_halo(P, le->step, le->post, true, nullptr, nullptr, le->rlo, le->rhi, le->plo, le->phi, st, true);
  if (e != cudaSuccess) return e;
  const double *plo = le ? le->plo : nullptr, *phi = le ? le->phi : nullptr;
  const double *hlo = le ? le->hlo : nullptr, *hhi = le ? le->hhi : nullptr;
  auto go = [&](auto rocky, auto plain) {
    return launch(rk ? rocky : plain, dim3(gr), bs, st, true, P, fin, fout, rho, psi, mom, db, rock, plo, phi, hlo,
                  hhi);
  };
  if (P.nc == 3) return go(k_collide<3, false, true, true>, k_collide<3, false, true, false>);
  if (le) return go(k_collide<2, true, true, true>, k_collide<2, true, true, false>);
  return go(k_collide<2, false, true, true>, k_collide<2, false, true, false>);
}

cudaError_t fp64_dipole(const DevParams &P, const double *rho, const double *da, double *db,
                        cudaStream_t st, bool pdl) {
  const int bs = fp64_block(P);
  return launch(k_dipole, dim3(grid_for(P.nsites, bs)), bs, st, pdl, P, rho, da, db);
}

cudaError_t fp64_collide(const DevParams &P, const double *g, double *f, const double *rho,
                         const double *psi, const double *mom, const double *db,
                         const uint8_t *rock, const double *plo, const double *phi,
                         cudaStream_t st) {
  const int bs = fp64_block(P);
  const unsigned gr = grid_for(P.nsites, bs);
  if (P.nc == 2) {
    if (P.le)
      k_collide<2, true><<<gr, bs, 0, st>>>(P, g, f, rho, psi, mom, db, rock, plo, phi);
    else
      k_collide<2, false><<<gr, bs, 0, st>>>(P, g, f, rho, psi, mom, db, rock, plo, phi);
  } else {
    k_collide<3, false><<<gr, bs, 0, st>>>(P, g, f, rho, psi, mom, db, rock, plo, phi);
  }
  return cudaGetLastError();
}

cudaError_t fp64_dump(const DevParams &P, int field, const double *f, const double *rho,
                      const double *psi, const double *db, const uint8_t *rock, double *out,
                      cudaStream_t st) {
  unsigned gr = grid_for(P.nsites, 256);
  if (P.nc == 2)
    k_dump<2><<<gr, 256, 0, st>>>(P, field, f, rho, psi, db, rock, out);
  else
    k_dump<3><<<gr, 256, 0, st>>>(P, field, f, rho, psi, db, rock, out);
  return cudaGetLastError();
}

cudaError_t fp64_moments(const DevParams &P, const double *f, double *rho, double *psi,
                         double *mom, cudaStream_t st) {
  unsigned gr = grid_for(P.nsites, 256);
  if (P.nc == 2)
    k_moments<2><<<gr, 256, 0, st>>>(P, f, rho, psi, mom);
  else
    k_moments<3><<<gr, 256, 0, st>>>(P, f, rho, psi, mom);
  return cudaGetLastError();
}

cudaError_t fp64_detmath(int fn, const double *x, double *y, long long n, cudaStream_t st) {
  k_detmath<<<grid_for(n, 256), 256, 0, st>>>(fn, x, y, n);
  return cudaGetLastError();
}

}  // namespace lb3d
