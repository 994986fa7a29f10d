// fp32_path.cu -- FP32 deviation storage: the fused stream-collide pass, and the
// host side of every FP32 strategy (fp32_split.cuh: strategies 1 and 2,
// fp32_eqstate.cu: strategy 3).
//
// Populations are stored as FP32 deviations delta_{c,i} = n_{c,i} - w_i rho0
// from the rest state (w_i = 1/36 moving, 1/3 rest), so the stored values
// and the moment sums carry the small variations at full FP32 relative
// precision.  One kernel launch advances a step: each CTA owns a TX x TY
// column tile and a range of z planes and marches in z with three stages
// per plane, keeping every intermediate field on chip:
//
//   A(k)   post-stream moments on the tile plus a halo of H sites
//          (H = 2 ternary, 1 binary): pull 19*nc deviations, densities,
//          psi deviations dpsi = psi(rho) - psi(rho0) = -e^{-rho0}
//          expm1(-drho), and (ternary) the advected dipole flux da using the
//          previous dipoles staged in shared memory.
//   B(k-1) (ternary) dipole relaxation on the tile plus a one-site halo
//          from the A ring (code/lb3d_collision.F90:296-403).
//   C(k-H) Shan-Chen force from the on-chip psi/dipole rings, body force,
//          the pull of the own site's populations (an L2 hit: the same
//          values were pulled by stage A two planes earlier), the
//          equilibrium of code/lb3d_bdist.F90:301-370 in deviation form
//          and the BGK update, written to the other buffer.
//
// HBM traffic per site and step is therefore one read and one write of the
// 19*nc deviations (plus the dipoles and a rock byte), against ~800 B for a
// three-kernel split.  Nothing in the path is a dense contraction, so there
// are no tensor cores; the roofline is HBM bandwidth.
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <cmath>
#include <cstring>
#include <vector>

#include "fp32_device.cuh"
#include "fp32_eqstate.h"
#include "fp32_path.h"
#include "reduce.h"
#include "fp64_path.h"
#include "le_common.cuh"

namespace lb3d {
namespace f32 {

// ---------------------------------------------------------------------------
// The fused kernel.  Grid: persistent CTAs over a tile list.  Populations
// of lattice L live at f[(c*19+q)*S + L.base + site]; each component's
// base is a 64-bit pointer and the offsets within a component are unsigned
// 32-bit, which bounds the packed capacity at 19*S < 2^32 sites.
//
// On-chip rings (float4 entries, one per site):
//   A  ternary: {rho_b - rho_r, da_x, da_y, da_z}, {drho_s, dpsi_r, dpsi_b,
//      dpsi_s} on the tile + 2 halo, 4 planes;  binary: {dpsi_r, dpsi_b, -, -}
//      on the tile + 1 halo, 3 planes
//   B  ternary: new dipoles {d_x, d_y, d_z, -} on the tile + 1 halo, 3 planes
//   D  ternary: previous dipoles on the tile + 3 halo, 3 planes
// ---------------------------------------------------------------------------
#include "inflow.cuh"

// Stage-8 inflow boundaries of one site on the FP32 path
// (code/lb3d_bc.F90:125-133 runs them between advection and collision):
// applied to the site's post-stream deviations after its own moments were
// taken, as the reference's collision keeps the advection moments.  Each
// closure works on the populations n = d + w rho0 in FP32 and writes the
// deviations back.  Recolouring (code/lb3d_invasion.F90:1257-1358) visits
// z = 0, 1 and then z = nz - 2, nz - 1 in that order, so planes that are
// both are recoloured twice as the reference's two loops do; the Zou-He
// closures (inflow.cuh) act on z = 0 and z = nz - 1 per component,
// surfactant first.
template <int NC>
__device__ __forceinline__ void inflow_site(float2 d01[19], float ds[19], const LatDesc &Lg, int gz,
                                            int nz) {
  const float r0 = Lg.rho0;
  if (Lg.invk == 1) {
    const float mr = Lg.inv_fluid == 7 ? 1.0f : 0.0f, mb = 1.0f - mr;
    const int zs[4] = {0, 1, nz - 2, nz - 1};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (gz != zs[k]) continue;
      const float a = k < 2 ? mr : mb, b = k < 2 ? mb : mr;
#pragma unroll
      for (int q = 0; q < 19; ++q) {
        const float w = wq(q) * r0;
        const float pop = (d01[q].x + w) + (d01[q].y + w);
        d01[q].x = a * pop - w;
        d01[q].y = b * pop - w;
      }
    }
    return;
  }
  const bool bottom = gz == 0;
  if (!bottom && gz != nz - 1) return;
  float F[19];
  if (NC == 3 && Lg.invk == 3) {
#pragma unroll
    for (int q = 0; q < 19; ++q) F[q] = (ds[q] + wq(q) * r0) * (float)gw(q);
    zouhe_flux_site<float>(F, Lg.zh_uz[2], bottom, Lg.inv_type);
#pragma unroll
    for (int q = 0; q < 19; ++q) ds[q] = F[q] / (float)gw(q) - wq(q) * r0;
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
#pragma unroll
    for (int q = 0; q < 19; ++q) F[q] = ((c ? d01[q].y : d01[q].x) + wq(q) * r0) * (float)gw(q);
    if (Lg.invk == 3)
      zouhe_flux_site<float>(F, Lg.zh_uz[c], bottom, Lg.inv_type);
    else
      zouhe_density_site<float>(F, bottom ? Lg.zh_in[c] : Lg.zh_uz[c], Lg.amass[c],
                                bottom ? Lg.amass[0] : Lg.amass[c], Lg.tau[c], bottom);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
      const float d = F[q] / (float)gw(q) - wq(q) * r0;
      if (c) d01[q].y = d; else d01[q].x = d;
    }
  }
}

// Kernel modes.  FUSED: one pass per step (moments recomputed on the halo).
// MOMENTS + COLLIDE: the split strategy, two passes per step: MOMENTS
// writes each site's post-stream moment entry (the A-ring entry) to a
// global field M exactly once, COLLIDE loads M with its halo into the same
// rings and runs the dipole, force and BGK stages.
constexpr int MODE_FUSED = 0, MODE_MOMENTS = 1, MODE_COLLIDE = 2;

template <int NC, int TX, int TY, int MODE>
struct FusedGeom {
  static constexpr int NT = TX * TY;
  static constexpr int H = (MODE == MODE_MOMENTS) ? 0 : ((NC == 3) ? 2 : 1);
  static constexpr int AW = TX + 2 * H, AH = TY + 2 * H, AN = AW * AH;
  static constexpr int AV = (NC == 3) ? 2 : 1;  // float4 per A entry
  static constexpr int AR = (NC == 3) ? 4 : 3;  // A ring depth
  static constexpr int BW = TX + 2, BH = TY + 2, BN = BW * BH;
  static constexpr int DH_ = (MODE == MODE_MOMENTS) ? 1 : 3;  // D-ring halo
  static constexpr int DW = TX + 2 * DH_, DH = TY + 2 * DH_, DN = DW * DH;
  static constexpr int A_F4 = (MODE == MODE_MOMENTS) ? 0 : AR * AV * AN;
  static constexpr int B_F4 = (NC == 3 && MODE != MODE_MOMENTS) ? 3 * BN : 0;
  static constexpr int D_F4 = (NC == 3 && MODE != MODE_COLLIDE) ? 3 * DN : 0;
  static constexpr int SMEM = 16 * (A_F4 + B_F4 + D_F4);
};

template <int NC, int TX, int TY, bool ROCK, bool BODY, int MODE, bool LE = false,
          bool NARROW = false>
__global__ void __launch_bounds__(TX *TY, (MODE == MODE_MOMENTS ? 1024 / (TX * TY) : (TX * TY >= 512 ? 1 : (TX * TY >= 256 ? 2 : 3))))
    k_fused(const LatDesc *__restrict__ lats, const Tile *__restrict__ tiles, int ntiles,
            float *f0, float *f1, float *db0, float *db1, const uint8_t *__restrict__ rock, unsigned S,
            float4 *__restrict__ Mf, float4 *__restrict__ Jf) {
  using G = FusedGeom<NC, TX, TY, MODE>;
  constexpr int NT = G::NT, H = G::H, AW = G::AW, AN = G::AN, AV = G::AV, AR = G::AR;
  constexpr int BW = G::BW, BN = G::BN, DW = G::DW, DN = G::DN, DHH = G::DH_;
  extern __shared__ float4 smem4[];
  float4 *ringA = smem4;              // [AR][AV][AN]
  float4 *ringB = ringA + G::A_F4;    // [3][BN]
  float4 *ringD = ringB + G::B_F4;    // [3][DN]
  const int tid = threadIdx.x;
  const int tx = tid % TX, ty = tid / TX;

  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const Tile T = tiles[t];
    const LatDesc &Lg = lats[T.lat];
    const int nx = Lg.nx, ny = Lg.ny, nz = Lg.nz;
    const int base = (int)Lg.base;
    const int par = Lg.parity;
    const float *__restrict__ F = (par ? f1 : f0) + base;
    float *__restrict__ Fo = (par ? f0 : f1) + base;
    const float *__restrict__ DBi = (NC == 3) ? (par ? db1 : db0) + base : nullptr;
    float *__restrict__ DBo = (NC == 3) ? (par ? db0 : db1) + base : nullptr;
    const uint8_t *__restrict__ RK = rock + base;
    const float rho0 = Lg.rho0, em0 = Lg.em0, psi0 = Lg.psi0;
    const int x0 = T.x0, y0 = T.y0, z0 = T.z0, zc = T.zc;
    const int zfirst = z0 - H;
    const int niter = zc + 2 * H;
    float4 *__restrict__ Mb = Mf ? Mf + base : nullptr;  // moment field of this lattice
    float4 *__restrict__ Jb = Jf ? Jf + base : nullptr;  // own-site moments
    // halo coordinates wrap with wrapz (a division only when the lattice is
    // narrower than the halo)
    auto wx = [&](int v) { return wrapz(v, nx); };
    auto wy = [&](int v) { return wrapz(v, ny); };

    auto load_db_plane = [&](int j) {
      const int gz = wrapz(zfirst - 1 + j, nz);
      float4 *dst = ringD + (j % 3) * DN;
      for (int s = tid; s < DN; s += NT) {
        const int gx = wx(x0 - DHH + s % DW), gy = wy(y0 - DHH + s / DW);
        const int i = gx + nx * (gy + ny * gz);
        dst[s] = make_float4(__ldg(DBi + i), __ldg(DBi + S + i), __ldg(DBi + 2 * S + i), 0.0f);
      }
    };
    if (NC == 3 && MODE != MODE_COLLIDE) {
      load_db_plane(0);
      load_db_plane(1);
    }

    for (int it = 0; it < niter; ++it) {
      const int zA = zfirst + it;
      if (NC == 3 && MODE != MODE_COLLIDE) load_db_plane(it + 2);
      __syncthreads();
      // ---------------- stage A: post-stream moments on the haloed tile ----
      {
        float4 *slot = ringA + (it % AR) * AV * AN;
        const int gz = wrapz(zA, nz);
        // D ring: plane zfirst - 1 + j sits in slot j % 3
        const float4 *Dm = ringD + (it % 3) * DN;        // plane zA - 1
        const float4 *D0 = ringD + ((it + 1) % 3) * DN;  // plane zA
        const float4 *Dp = ringD + ((it + 2) % 3) * DN;  // plane zA + 1
        for (int s = tid; s < AN; s += NT) {
          const int ax = s % AW, ay = s / AW;
          const int gx = wx(x0 - H + ax), gy = wy(y0 - H + ay);
          Nbr nb;
          make_nbr(nb, gx, gy, gz, nx, ny, nz);
          const int self = noff<18, 1>(nb);
          LeYZ lw;
          if constexpr (LE) make_leyz(lw, gy, gz, ny, nz);
          float dr[NC], jm[NC][3];
          float a0 = 0.f, a1 = 0.f, a2 = 0.f;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            float d[19];
            if constexpr (LE) {
              if (ROCK && __ldg(RK + self) != 0) {
                // a rock site keeps its (zero) populations
                // (code/lb3d_advection.F90:109-151 pulls into fluid sites only)
                const float *fc = F + (size_t)(c * 19) * S + self;
#pragma unroll
                for (int q = 0; q < 19; ++q) d[q] = __ldg(fc + q * S);
              } else {
                pull_comp_le<NARROW, ROCK>(F, S, c, nb, self, gx, nx, lw, Lg, ny * nz, d, RK);
              }
              // the post-stream populations of the x boundary planes, for
              // the stage-8 halo kernel
              if (MODE == MODE_MOMENTS && x0 + ax < nx && y0 + ay < ny)
                le_store_boundary(Lg, 2, c, gx, gy, gz, d);
            } else {
              pull_comp<ROCK, false, NARROW>(F, S, c, nb, self, RK, d);
            }
            if (MODE == MODE_MOMENTS) {
              own_moments<1>(d, dr[c], jm[c][0], jm[c][1], jm[c][2]);
            } else {
              float acc = 0.0f;
#pragma unroll
              for (int q = 0; q < 19; ++q) acc = fmaf((float)gw(q), d[q], acc);
              dr[c] = acc;
            }
            if (NC == 3 && c == 2) {
              // Zou-He flux boundaries change the surfactant's populations on
              // the z planes before its advected dipole flux is summed
              // (code/lb3d_invasion.F90:2143-2457 recomputes it there)
              if (MODE == MODE_MOMENTS && Lg.invk == 3 && (gz == 0 || gz == nz - 1)) {
                float Fs[19];
#pragma unroll
                for (int q = 0; q < 19; ++q) Fs[q] = (d[q] + wq(q) * rho0) * (float)gw(q);
                zouhe_flux_site<float>(Fs, Lg.zh_uz[2], gz == 0, Lg.inv_type);
#pragma unroll
                for (int q = 0; q < 19; ++q) d[q] = Fs[q] / (float)gw(q) - wq(q) * rho0;
              }
              // da = sum_q (n_s(x - c_q, q) g_q) db(x - c_q) + n_s(x, rest) db(x)
              // (code/lb3d_advection.F90:137-148)
              const int ds0 = (ax + 1) + DW * (ay + 1);  // A-local -> D-local
#pragma unroll
              for (int q = 0; q < 19; ++q) {
                const float4 *Dq = cz(q) == 1 ? Dm : (cz(q) == -1 ? Dp : D0);
                const float4 b = Dq[ds0 - cx(q) - DW * cy(q)];
                const float ng = (float)gw(q) * fmaf(wq(q), rho0, d[q]);
                a0 = fmaf(ng, b.x, a0);
                a1 = fmaf(ng, b.y, a1);
                a2 = fmaf(ng, b.z, a2);
              }
            }
          }
          float4 e0, e1;
          if (NC == 3) {
            e0 = make_float4(dr[1] - dr[0], a0, a1, a2);
            e1 = make_float4(dr[NC - 1], -em0 * expm1f(-dr[0]), -em0 * expm1f(-dr[1]),
                             -em0 * expm1f(-dr[NC - 1]));
          } else {
            e0 = make_float4(-em0 * expm1f(-dr[0]), -em0 * expm1f(-dr[1]), 0.f, 0.f);
          }
          if (MODE == MODE_MOMENTS) {
            // one entry per site, the tile only (H = 0)
            if (x0 + ax < nx && y0 + ay < ny) {
              if (NC == 3) {
                Mb[self] = e0;
                Mb[S + self] = e1;
                if (Jb) {
                  Jb[self] = make_float4(dr[0], dr[1], dr[2], jm[0][0]);
                  Jb[S + self] = make_float4(jm[0][1], jm[0][2], jm[1][0], jm[1][1]);
                  Jb[2 * S + self] = make_float4(jm[1][2], jm[NC - 1][0], jm[NC - 1][1], jm[NC - 1][2]);
                }
              } else {
                reinterpret_cast<float2 *>(Mb)[self] = make_float2(e0.x, e0.y);
                if (Jb) {
                  Jb[self] = make_float4(dr[0], dr[1], jm[0][0], jm[0][1]);
                  Jb[S + self] = make_float4(jm[0][2], jm[1][0], jm[1][1], jm[1][2]);
                }
              }
            }
          } else {
            slot[s] = e0;
            if (NC == 3) slot[AN + s] = e1;
          }
        }
      }  // stage A
      __syncthreads();
      if (MODE == MODE_MOMENTS) continue;
      // ---------------- stage B (ternary): dipole relaxation ----------------
      if constexpr (NC == 3) if (it >= 2) {
        float4 *slotB = ringB + (it % 3) * BN;
        const int zB = zA - 1;
        const float4 *Am = ringA + ((it - 2) % AR) * AV * AN;  // plane zB - 1
        const float4 *A0 = ringA + ((it - 1) % AR) * AV * AN;  // plane zB
        const float4 *Ap = ringA + ((it) % AR) * AV * AN;      // plane zB + 1
        for (int s = tid; s < BN; s += NT) {
          const int bx = s % BW, by = s / BW;
          const int as = (bx + 1) + AW * (by + 1);
          const float3 nd = dipole_site<AW>(Am, A0, Ap, as, Lg, rho0, A0[AN + as].x);
          const float n0 = nd.x, n1 = nd.y, n2 = nd.z;
          slotB[s] = make_float4(n0, n1, n2, 0.0f);
          if (bx >= 1 && bx <= TX && by >= 1 && by <= TY && zB >= z0 && zB < z0 + zc) {
            const int gx = x0 + bx - 1, gy = y0 + by - 1;
            if (gx < nx && gy < ny) {
              const int i = gx + nx * (gy + ny * wrapz(zB, nz));
              __stcs(DBo + i, n0);
              __stcs(DBo + S + i, n1);
              __stcs(DBo + 2 * S + i, n2);
            }
          }
        }
        __syncthreads();
      }
      // ---------------- stage C: force + BGK on the tile ---------------------
      const int itC = it - H;  // A iteration of plane zC
      const int zC = zA - H;
      if (zC >= z0 && zC < z0 + zc) {
        const int gx = x0 + tx, gy = y0 + ty;
        if (gx < nx && gy < ny) {
          const int gz = wrapz(zC, nz);
          Nbr nb;
          make_nbr(nb, gx, gy, gz, nx, ny, nz);
          const int self = noff<18, 1>(nb);
          bool own_rock = false;
          if (ROCK) own_rock = __ldg(RK + self) != 0;
          if (!own_rock) {
            const int as = (tx + H) + AW * (ty + H);
            const float4 *Am = ringA + ((itC + AR - 1) % AR) * AV * AN;
            const float4 *A0 = ringA + (itC % AR) * AV * AN;
            const float4 *Ap = ringA + ((itC + 1) % AR) * AV * AN;
            float Fx[NC][3];
            if constexpr (NC == 3) {
              // ---- ternary Shan-Chen force, code/lb3d_force_shanchen.F90:215-330
              const int itB = itC + 1;  // B computed plane zC at iteration itC + 1
              const int bs = (tx + 1) + BW * (ty + 1);
              force_ternary<AW, BW>(Am + AN, A0 + AN, Ap + AN, DipF4{ringB + ((itB + 2) % 3) * BN},
                                    DipF4{ringB + (itB % 3) * BN}, DipF4{ringB + ((itB + 1) % 3) * BN},
                                    as, bs, Lg, psi0, reinterpret_cast<float(*)[3]>(Fx));
            } else {
              // ---- binary Shan-Chen force with walls, :127-210
              force_binary<AW, ROCK>(Am, A0, Ap, as, nb, RK, Lg, psi0,
                                     reinterpret_cast<float(*)[3]>(Fx));
            }
            // ---- pass 1: moments of the own post-stream populations (the
            // pulls hit L2: stage A fetched them H planes earlier)
            float dr[NC], j[NC][3];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              float d[19];
              pull_comp<ROCK>(F, S, c, nb, self, RK, d);
              own_moments<1>(d, dr[c], j[c][0], j[c][1], j[c][2]);
            }
            float rho[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) rho[c] = rho0 + dr[c];
            if (BODY) {
              const int x1 = gx + 1, y1 = gy + 1, z1 = gz + 1;
              bool on;
              if (Lg.inv_fluid == 9)
                on = (z1 == 1) || (z1 == nz);
              else if (Lg.inv_fluid == 20 || Lg.inv_fluid == 21)
                on = z1 == 1;
              else
                on = z1 >= Lg.amin_z && z1 <= Lg.amax_z && x1 >= Lg.amin_x && x1 <= Lg.amax_x &&
                     y1 >= Lg.amin_y && y1 <= Lg.amax_y;
              if (on) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                  const float m = Lg.amass[c] * rho[c];
                  Fx[c][0] = fmaf(m, Lg.g_accn_x, Fx[c][0]);
                  Fx[c][1] = fmaf(m, Lg.g_accn_y, Fx[c][1]);
                  Fx[c][2] = fmaf(m, Lg.g_accn, Fx[c][2]);
                }
              }
            }
            // common velocity u~ (code/lb3d_collision.F90:560-587)
            float p0 = 0.f, p1 = 0.f, p2 = 0.f, rt = 0.f;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              const float am = Lg.amass[c] * Lg.omega[c];
              p0 = fmaf(am, j[c][0], p0);
              p1 = fmaf(am, j[c][1], p1);
              p2 = fmaf(am, j[c][2], p2);
              rt = fmaf(am, rho[c], rt);
            }
            const float irt = 1.0f / fmaxf(rt, 1.0e-8f);
            const float u0 = p0 * irt, u1 = p1 * irt, u2 = p2 * irt;
            // ---- pass 2: reload, relax, store
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              // du = tau F / (amass max(rho, 1e-8))  (:523-556)
              const float k = Lg.tau[c] / (Lg.amass[c] * fmaxf(rho[c], 1.0e-8f));
              float d[19];
              pull_comp<ROCK, true>(F, S, c, nb, self, RK, d);
              bgk_update(d, rho[c], dr[c], fmaf(k, Fx[c][0], u0), fmaf(k, Fx[c][1], u1),
                         fmaf(k, Fx[c][2], u2), Lg.omega[c]);
              float *fo = Fo + (size_t)(c * 19) * S + self;
              // streaming stores: the new populations are not read again in
              // this launch, so they should not displace the inputs from L2
#pragma unroll
              for (int q = 0; q < 19; ++q) __stcs(fo + q * S, d[q]);
            }
          }
        }
      }
      __syncthreads();
    }
  }
}

#include "fp32_split.cuh"

__global__ void k_flip(LatDesc *lats, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && (lats[i].flags & LAT_ACTIVE)) lats[i].parity ^= 1;
}

// FP32 state -> FP64 populations n = delta + w rho0 (dumps, reductions).
// The products and sums are rounded separately (no contraction), as the
// host-side conversions of the ensemble do, so both routes agree bit for bit.
__global__ void k_to_fp64(const float *__restrict__ f, double *__restrict__ n, long long S,
                          long long base, long long N, int nc, double rho0) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  for (int c = 0; c < nc; ++c)
    for (int q = 0; q < 19; ++q)
      n[((long long)c * 19 + q) * N + i] =
          __dadd_rn((double)f[((long long)c * 19 + q) * S + base + i],
                    __dmul_rn(q == 18 ? 1.0 / 3.0 : 1.0 / 36.0, rho0));
}

// FP64 populations -> FP32 deviations (upload); rock sites (rock[i] != 0,
// when rock is given) hold n = 0.
__global__ void k_from_fp64(const double *__restrict__ n, float *__restrict__ f, long long S,
                            long long base, long long N, int nc, double rho0,
                            const uint8_t *__restrict__ rock = nullptr) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const bool solid = rock && rock[i] != 0;
  for (int c = 0; c < nc; ++c)
    for (int q = 0; q < 19; ++q) {
      const double w = __dmul_rn(q == 18 ? 1.0 / 3.0 : 1.0 / 36.0, rho0);
      const double v = solid ? 0.0 : n[((long long)c * 19 + q) * N + i];
      f[((long long)c * 19 + q) * S + base + i] = (float)__dsub_rn(v, w);
    }
}

// One population plane FP64 <-> FP32 deviations (w = w_q rho0), rounded as
// k_to_fp64 / k_from_fp64; the upload writes both buffers.
__global__ void k_plane_from_fp64(const double *__restrict__ src, float *__restrict__ d0,
                                  float *__restrict__ d1, long long N, double w,
                                  const uint8_t *__restrict__ rock) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double v = (rock && rock[i] != 0) ? 0.0 : src[i];
  const float x = (float)__dsub_rn(v, w);
  d0[i] = x;
  d1[i] = x;
}
// One plane of a download, FP64: a population plane (the deviations of one
// direction plus w; rock sites hold no populations), a density or momentum
// plane (summed in FP64 over the populations in direction order, the
// products and sums rounded separately), or a dipole plane.  A density plane
// reads 76 B a site, so even the four moment planes of a component take less
// than the link needs for one of them (128^3: 25 us against 365 us).
struct PlaneJob {
  int kind;  // 0: population (src one plane), 1: density, 2..4: momentum x, y, z (src 19 planes), 5: as it is
  const float *src;
  double rho0;
};
__global__ void k_plane_to_fp64(PlaneJob J, long long S, double *__restrict__ dst, long long N, double w,
                                const uint8_t *__restrict__ rock) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const bool solid = rock && rock[i] != 0;
  if (J.kind == 0) {
    dst[i] = solid ? 0.0 : __dadd_rn((double)J.src[i], w);
    return;
  }
  if (J.kind == 5) {
    dst[i] = (double)J.src[i];
    return;
  }
  double m = 0.0;
#pragma unroll
  for (int q = 0; q < 19; ++q) {
    const int c = J.kind == 1 ? 1 : J.kind == 2 ? cx(q) : J.kind == 3 ? cy(q) : cz(q);
    const double wr = __dmul_rn(q == 18 ? 1.0 / 3.0 : 1.0 / 36.0, J.rho0);
    const double n = solid ? 0.0 : __dadd_rn((double)J.src[(long long)q * S + i], wr);
    m = __dadd_rn(m, __dmul_rn(__dmul_rn(n, (double)gw(q)), (double)c));
  }
  dst[i] = m;
}

}  // namespace f32

using namespace f32;

cudaError_t fp32_to_fp64(const float *f, double *out, long long S, long long base, long long N,
                         int nc, double rho0, cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  k_to_fp64<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(f, out, S, base, N, nc, rho0);
  return cudaGetLastError();
}

__global__ void k_planes_f2d(const float *__restrict__ src, double *__restrict__ dst, long long S,
                             long long base, long long N, int planes) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  for (int k = 0; k < planes; ++k) dst[(long long)k * N + i] = (double)src[(long long)k * S + base + i];
}

cudaError_t fp32_planes_to_fp64(const float *src, double *dst, long long S, long long base,
                                long long N, int planes, cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  k_planes_f2d<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(src, dst, S, base, N, planes);
  return cudaGetLastError();
}

cudaError_t fp32_from_fp64(const double *n, float *f, long long S, long long base, long long N,
                           int nc, double rho0, const uint8_t *rock, cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  k_from_fp64<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(n, f, S, base, N, nc, rho0, rock);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// launch table
// ---------------------------------------------------------------------------
constexpr int MODE_DIPOLE = 3, MODE_COLLIDE2 = 4;
// the moments pass with 32-bit component offsets (k_fused<..., NARROW>)
constexpr int MODE_MOMENTS32 = 5;

size_t fp32_mode_smem(int nc, const FusedShape &sh, int mode) {
  if (mode == MODE_MOMENTS32) mode = MODE_MOMENTS;
  const size_t AN1 = (size_t)(sh.tx + 2) * (sh.ty + 2);
  if (mode == MODE_DIPOLE) return 16 * 5 * AN1 + (size_t)4 * 5 * sh.tx * sh.ty;
  if (mode == MODE_COLLIDE2)  // Collide2Geom: ring slots x entry bytes + population stage
    return 5 * AN1 * (nc == 3 ? 16 + 12 : 8) + (size_t)19 * nc * sh.tx * sh.ty * 4;
  if (mode == MODE_COLLIDE) return 16 * 3 * AN1 * (nc == 3 ? 2 : 1);
  const int H = mode == MODE_MOMENTS ? 0 : (nc == 3 ? 2 : 1);
  const int dh = mode == MODE_MOMENTS ? 1 : 3;
  const size_t AN = (size_t)(sh.tx + 2 * H) * (sh.ty + 2 * H);
  const size_t BN = (size_t)(sh.tx + 2) * (sh.ty + 2);
  const size_t DN = (size_t)(sh.tx + 2 * dh) * (sh.ty + 2 * dh);
  size_t f4 = 0;
  if (mode != MODE_MOMENTS) f4 += (nc == 3 ? 4 * 2 : 3) * AN;
  if (nc == 3 && mode != MODE_MOMENTS) f4 += 3 * BN;
  if (nc == 3) f4 += 3 * DN;
  return 16 * f4;
}
size_t fp32_fused_smem(int nc, const FusedShape &sh) { return fp32_mode_smem(nc, sh, MODE_FUSED); }

template <int NC, int TX, int TY, bool ROCK, bool BODY, int MODE, bool LE, bool INF = false>
static const void *fused_ptr() {
  if constexpr (MODE == MODE_COLLIDE)
    return (const void *)k_split_collide<NC, TX, TY, ROCK, BODY>;
  else if constexpr (MODE == MODE_COLLIDE2)
    return (const void *)k_split_collide2<NC, TX, TY, ROCK, BODY, LE, INF>;
  else if constexpr (MODE == MODE_DIPOLE)
    return (const void *)k_split_dipole<TX, TY>;
  else if constexpr (MODE == MODE_MOMENTS32)
    return (const void *)k_fused<NC, TX, TY, ROCK, BODY, MODE_MOMENTS, LE, true>;
  else
    return (const void *)k_fused<NC, TX, TY, ROCK, BODY, MODE, LE>;
}

// LE: the Lees-Edwards variants, built for binary lattices without rock and
// only for the moments and staged collide passes (strategy 2).
// INF: the staged collide variant with the stage-8 inflow boundaries.
template <int MODE, bool LE = false, bool INF = false>
static const void *mode_fn(int nc, bool rock, bool body, const FusedShape &sh) {
#define LB3D_SHAPES(NC, R, B)                                                            \
  if (sh.tx == 32 && sh.ty == 8) return fused_ptr<NC, 32, 8, R, B, MODE, LE, INF>();     \
  if (sh.tx == 32 && sh.ty == 4) return fused_ptr<NC, 32, 4, R, B, MODE, LE, INF>();     \
  if (sh.tx == 16 && sh.ty == 16) return fused_ptr<NC, 16, 16, R, B, MODE, LE, INF>();   \
  if (sh.tx == 16 && sh.ty == 8) return fused_ptr<NC, 16, 8, R, B, MODE, LE, INF>();     \
  if (sh.tx == 64 && sh.ty == 4) return fused_ptr<NC, 64, 4, R, B, MODE, LE, INF>();
  // the moments and dipole passes do not apply the body force
  if (MODE == MODE_MOMENTS || MODE == MODE_MOMENTS32 || MODE == MODE_DIPOLE) body = false;
  if constexpr (LE) {
    static_assert(MODE == MODE_MOMENTS || MODE == MODE_MOMENTS32 || MODE == MODE_COLLIDE2,
                  "no Lees-Edwards variant");
    if (nc != 2) return nullptr;
    if (rock) {
      if (body) { LB3D_SHAPES(2, true, true) } else { LB3D_SHAPES(2, true, false) }
    } else {
      if (body) { LB3D_SHAPES(2, false, true) } else { LB3D_SHAPES(2, false, false) }
    }
    return nullptr;
  }
  if (MODE == MODE_DIPOLE) rock = false;
  if (nc == 3) {
    if (body) { LB3D_SHAPES(3, false, true) } else { LB3D_SHAPES(3, false, false) }
  } else {
    if (MODE == MODE_DIPOLE) return nullptr;
    if (rock) {
      if (body) { LB3D_SHAPES(2, true, true) } else { LB3D_SHAPES(2, true, false) }
    } else {
      if (body) { LB3D_SHAPES(2, false, true) } else { LB3D_SHAPES(2, false, false) }
    }
  }
#undef LB3D_SHAPES
  return nullptr;
}

static const void *kernel_fn(int nc, bool rock, bool body, const FusedShape &sh, int mode,
                             bool le = false, bool inf = false) {
  if (inf && mode == MODE_COLLIDE2) return mode_fn<MODE_COLLIDE2, false, true>(nc, rock, body, sh);
  if (le) {
    if (mode == MODE_MOMENTS) return mode_fn<MODE_MOMENTS, true>(nc, rock, body, sh);
    if (mode == MODE_MOMENTS32) return mode_fn<MODE_MOMENTS32, true>(nc, rock, body, sh);
    if (mode == MODE_COLLIDE2) return mode_fn<MODE_COLLIDE2, true>(nc, rock, body, sh);
    return nullptr;
  }
  if (mode == MODE_MOMENTS) return mode_fn<MODE_MOMENTS>(nc, rock, body, sh);
  if (mode == MODE_MOMENTS32) return mode_fn<MODE_MOMENTS32>(nc, rock, body, sh);
  if (mode == MODE_COLLIDE) return mode_fn<MODE_COLLIDE>(nc, rock, body, sh);
  if (mode == MODE_DIPOLE) return mode_fn<MODE_DIPOLE>(nc, rock, body, sh);
  if (mode == MODE_COLLIDE2) return mode_fn<MODE_COLLIDE2>(nc, rock, body, sh);
  return mode_fn<MODE_FUSED>(nc, rock, body, sh);
}
static const void *fused_fn(int nc, bool rock, bool body, const FusedShape &sh) {
  return kernel_fn(nc, rock, body, sh, MODE_FUSED);
}

static int mode_ctas_per_sm(int nc, bool rock, bool body, const FusedShape &sh, int mode) {
  const void *fn = kernel_fn(nc, rock, body, sh, mode);
  if (!fn) return 0;
  size_t smem = fp32_mode_smem(nc, sh, mode);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return 0;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, sh.tx * sh.ty, smem) != cudaSuccess) return 0;
  return n;
}

int fp32_fused_ctas_per_sm(int nc, bool rock, bool body, const FusedShape &sh) {
  int a = mode_ctas_per_sm(nc, rock, body, sh,
                           sh.split == 2 ? MODE_COLLIDE2 : (sh.split ? MODE_COLLIDE : MODE_FUSED));
  if (!sh.split) return a;
  int b = mode_ctas_per_sm(nc, rock, body, sh, MODE_MOMENTS);
  int c = nc == 3 ? mode_ctas_per_sm(nc, rock, body, sh, MODE_DIPOLE) : b;
  return std::min(a, std::min(b, c));
}

// Grid of one pass: as many CTAs as are resident at once (up to the tile
// count), from the pass's own occupancy, so a pass with a large shared
// memory stage does not throttle the others.  The dynamic shared memory
// attribute and the occupancy are set up once per kernel and device.
cudaError_t fp32_prepare_kernel(const void *fn, int nthreads, size_t smem, int *ctas_total) {
  static std::mutex mu;
  static std::map<std::tuple<const void *, size_t, int, int>, int> cache;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const auto key = std::make_tuple(fn, smem, nthreads, dev);
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *ctas_total = it->second;
    return cudaSuccess;
  }
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per = 0, nsm = 148;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, nthreads, smem);
  if (e != cudaSuccess) return e;
  if (per < 1) return cudaErrorInvalidConfiguration;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cache[key] = *ctas_total = per * nsm;
  return cudaSuccess;
}

static cudaError_t launch_mode(int mode, int nc, bool rock, bool body, const FusedShape &sh,
                               const LatDesc *d_lat, const Tile *d_tiles, int ntiles, int max_grid,
                               float *f0, float *f1, float *db0, float *db1, const uint8_t *rockp,
                               unsigned S, float4 *M, float4 *J, cudaStream_t st, bool le = false,
                               bool inf = false) {
  if (mode == MODE_MOMENTS && 19ull * nc * S < (1ull << 32)) mode = MODE_MOMENTS32;
  const void *fn = kernel_fn(nc, rock, body, sh, mode, le, inf);
  if (!fn) return cudaErrorInvalidConfiguration;
  size_t smem = fp32_mode_smem(nc, sh, mode);
  int resident = 0;
  cudaError_t e = fp32_prepare_kernel(fn, sh.tx * sh.ty, smem, &resident);
  if (e != cudaSuccess) return e;
  int grid = std::max(1, std::min(ntiles, resident));
  if (max_grid > 0) grid = std::min(grid, max_grid);
  if (mode == MODE_DIPOLE) {
    const float4 *Mc = M;
    void *args[] = {(void *)&d_lat, (void *)&d_tiles, (void *)&ntiles, (void *)&db0, (void *)&db1,
                    (void *)&Mc, (void *)&S};
    return cudaLaunchKernel(fn, dim3(grid), dim3(sh.tx * sh.ty), args, smem, st);
  }
  if (mode == MODE_COLLIDE2) {
    const float4 *Mc = M;
    void *args[] = {(void *)&d_lat, (void *)&d_tiles, (void *)&ntiles, (void *)&f0, (void *)&f1,
                    (void *)&db0, (void *)&db1, (void *)&rockp, (void *)&S, (void *)&Mc};
    return cudaLaunchKernel(fn, dim3(grid), dim3(sh.tx * sh.ty), args, smem, st);
  }
  if (mode == MODE_COLLIDE) {
    const float4 *Mc = M, *Jc = J;
    void *args[] = {(void *)&d_lat, (void *)&d_tiles, (void *)&ntiles, (void *)&f0, (void *)&f1,
                    (void *)&db0, (void *)&db1, (void *)&rockp, (void *)&S, (void *)&Mc, (void *)&Jc};
    return cudaLaunchKernel(fn, dim3(grid), dim3(sh.tx * sh.ty), args, smem, st);
  }
  void *args[] = {(void *)&d_lat, (void *)&d_tiles, (void *)&ntiles, (void *)&f0, (void *)&f1,
                  (void *)&db0, (void *)&db1, (void *)&rockp, (void *)&S, (void *)&M, (void *)&J};
  return cudaLaunchKernel(fn, dim3(grid), dim3(sh.tx * sh.ty), args, smem, st);
}

cudaError_t fp32_launch_fused(int nc, bool rock, bool body, const FusedShape &sh,
                              const LatDesc *d_lat, const Tile *d_tiles, int ntiles, int max_grid,
                              float *f0, float *f1, float *db0, float *db1, const uint8_t *rockp,
                              long long S64, cudaStream_t st, float4 *M, float4 *J,
                              const LEStep *le, const DevParams *P) {
  if (S64 * 19 >= (1LL << 32)) return cudaErrorInvalidValue;
  const unsigned S = (unsigned)S64;
  if (le) {
    // stage 6 halo, moments pass, stage 8 halo, staged collide pass
    if (!P || nc != 2 || sh.split != 2 || !M) return cudaErrorInvalidValue;
    // two threads per (y, z) of the x-halo planes (one per side): 64-thread
    // blocks spread the few thousand threads over every SM
    const unsigned g = (unsigned)((2 * P->ny * P->nz + 63) / 64);
    k_le_pre32<2><<<g, 64, 0, st>>>(*P, *le, d_lat, f0, f1, S);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
      e = launch_mode(MODE_MOMENTS, nc, rock, body, sh, d_lat, d_tiles, ntiles, max_grid, f0, f1, db0,
                      db1, rockp, S, M, nullptr, st, true);
    if (e != cudaSuccess) return e;
    k_le_post32<2><<<g, 64, 0, st>>>(*P, *le, d_lat, f0, f1, S);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return launch_mode(MODE_COLLIDE2, nc, rock, body, sh, d_lat, d_tiles, ntiles, max_grid, f0, f1,
                       db0, db1, rockp, S, M, nullptr, st, true);
  }
  // lattices with inflow boundaries run the staged collide's inflow variant
  const bool inf = P && P->invk != 0;
  if (inf && sh.split != 2) return cudaErrorInvalidValue;
  if (!sh.split)
    return launch_mode(MODE_FUSED, nc, rock, body, sh, d_lat, d_tiles, ntiles, max_grid, f0, f1, db0,
                       db1, rockp, S, nullptr, nullptr, st);
  if (!M || (sh.split == 1 && !J)) return cudaErrorInvalidValue;
  // strategy 2 recomputes the own moments in the collide pass: no J field
  if (sh.split == 2) J = nullptr;
  cudaError_t e = launch_mode(MODE_MOMENTS, nc, rock, body, sh, d_lat, d_tiles, ntiles, max_grid, f0,
                              f1, db0, db1, rockp, S, M, J, st);
  if (e == cudaSuccess && nc == 3)
    e = launch_mode(MODE_DIPOLE, nc, rock, body, sh, d_lat, d_tiles, ntiles, max_grid, f0, f1, db0,
                    db1, rockp, S, M, J, st);
  if (e != cudaSuccess) return e;
  return launch_mode(sh.split == 2 ? MODE_COLLIDE2 : MODE_COLLIDE, nc, rock, body, sh, d_lat,
                     d_tiles, ntiles, max_grid, f0, f1, db0, db1, rockp, S, M, J, st, false, inf);
}

cudaError_t fp32_flip_parity(LatDesc *d_lat, int nlat, cudaStream_t st) {
  k_flip<<<(nlat + 127) / 128, 128, 0, st>>>(d_lat, nlat);
  return cudaGetLastError();
}

void fp32_tiles_for(const LatDesc &L, int lat_id, const FusedShape &sh, std::vector<Tile> &out) {
  const int zc = std::min(sh.zc, L.nz);
  for (int z0 = 0; z0 < L.nz; z0 += zc)
    for (int y0 = 0; y0 < L.ny; y0 += sh.ty)
      for (int x0 = 0; x0 < L.nx; x0 += sh.tx) {
        Tile t;
        t.lat = lat_id;
        t.x0 = x0;
        t.y0 = y0;
        t.z0 = z0;
        t.zc = std::min(zc, L.nz - z0);
        out.push_back(t);
      }
}

LatDesc fp32_make_desc(const DevParams &P, double rho0, long long base, bool rock) {
  LatDesc L{};
  L.nx = P.nx;
  L.ny = P.ny;
  L.nz = P.nz;
  L.nc = P.nc;
  L.base = base;
  L.parity = 0;
  for (int c = 0; c < 3; ++c) {
    L.omega[c] = (float)P.omega[c];
    L.tau[c] = (float)P.tau[c];
    L.amass[c] = (float)P.amass[c];
  }
  L.g_br = (float)P.g_br;
  L.g_bs = (float)P.g_bs;
  L.g_ss = (float)P.g_ss;
  L.wall_r = (float)(-P.g_wr * P.tau_wr / P.tau[0]);
  L.wall_b = (float)(-P.g_wb * P.tau_wb / P.tau[1]);
  L.psiw_r = (float)(1.0 - std::exp(-P.rc_r));
  L.psiw_b = (float)(1.0 - std::exp(-P.rc_b));
  L.beta = (float)P.beta;
  L.d0 = (float)P.d_0;
  L.omega_d = (float)P.omega_d;
  L.g_accn = (float)P.g_accn;
  L.g_accn_x = (float)P.g_accn_x;
  L.g_accn_y = (float)P.g_accn_y;
  L.amin_x = P.g_accn_min_x;
  L.amax_x = P.g_accn_max_x;
  L.amin_y = P.g_accn_min_y;
  L.amax_y = P.g_accn_max_y;
  L.amin_z = P.g_accn_min;
  L.amax_z = P.g_accn_max;
  L.inv_fluid = P.inv_fluid;
  L.invk = P.invk;
  L.inv_type = P.inv_type;
  L.zh_in[0] = (float)P.zh_in[0];
  L.zh_in[1] = (float)P.zh_in[1];
  for (int c = 0; c < 3; ++c) L.zh_uz[c] = (float)P.zh_uz[c];
  L.rho0 = (float)rho0;
  L.em0 = (float)std::exp(-rho0);
  L.psi0 = (float)(1.0 - std::exp(-rho0));
  bool body = (P.g_accn != 0.0 || P.g_accn_x != 0.0 || P.g_accn_y != 0.0);
  L.flags = LAT_ACTIVE | (rock ? LAT_ROCK : 0) | (body ? LAT_BODY : 0);
  return L;
}

// ---------------------------------------------------------------------------
// single-lattice handle
// ---------------------------------------------------------------------------
// Bytes of strategy 3's fields per site beside the neighbour mask.
static long long eq_bytes(int nc) { return nc == 3 ? 44 : 20; }

long long fp32_footprint(const lb3dc_params &p) {
  const long long N = (long long)p.nx * p.ny * p.nz;
  const bool le = p.boundary_cond != 0 && (p.inv_fluid == 5 || p.inv_fluid == 6);
  const long long np = (long long)p.ny * p.nz;
  // the fields of strategy 3 when every component relaxes fully (with the
  // neighbour mask of a binary lattice with rock)
  const bool full = p.tau_r == 1.0 && p.tau_b == 1.0 && (p.ncomp == 2 || p.tau_s == 1.0);
  const long long mf = full ? N * (eq_bytes(p.ncomp) + (p.ncomp == 2 ? 4 : 0)) : 0;
  return 2LL * p.ncomp * 19 * N * 4 + (p.ncomp == 3 ? 6LL * N * 4 : 0) +
         N * fp32_moment_bytes(p.ncomp) + mf +
         (le ? 2 * np * (p.ncomp * 19 * 4 + 8) + 4 * np * p.ncomp * 19 * 4 : 0) + N * 16 + 4096;
}

// ---------------------------------------------------------------------------
// strategy 3: eligibility, fields, tile lists, steps
// ---------------------------------------------------------------------------
bool fp32_eq_eligible(const DevParams &P) {
  if ((P.le && P.nc != 2) || P.invk) return false;
  for (int c = 0; c < P.nc; ++c)
    if (P.omega[c] != 1.0) return false;
  return P.nx >= 2 && P.ny >= 2;
}

static void free_eq(Fp32State &s) {
  if (s.o1) s.bytes -= s.S * eq_bytes(s.lat.nc);
  if (s.mask) s.bytes -= s.S * 4;
  void *bufs[] = {s.o1, s.mask, s.eq_tiles};
  for (void *b : bufs)
    if (b) cudaFree(b);
  s.o1 = s.o3 = nullptr;
  s.o2 = nullptr;
  s.psi = nullptr;
  s.mask = nullptr;
  s.eq_tiles = nullptr;
}

bool fp32_make_room(Fp32State &s, cudaStream_t st) {
  if (!s.o1) return false;
  cudaStreamSynchronize(st);
  free_eq(s);
  if (s.split == 3) s.split = 2;  // d_tiles serve it as they are
  return true;
}

// A device allocation of the handle; strategy 3's fields make way for it.
static int alloc_device(Fp32State &s, void **p, size_t bytes, cudaStream_t st) {
  for (int k = 0; k < 2; ++k) {
    if (cudaMalloc(p, bytes) == cudaSuccess) return LB3DC_OK;
    cudaGetLastError();
    *p = nullptr;
    if (k || !fp32_make_room(s, st)) break;
  }
  return LB3DC_ENOMEM;
}

// The fields of strategy 3, allocated the first time a lattice is switched to
// it, and (with rock) the neighbour mask and the rock sites' psi entries.
static int ensure_eq(const DevParams &P, Fp32State &s, cudaStream_t st) {
  const size_t N = (size_t)P.nsites;
  if (!s.o1) {
    // one block: o1, o3 (float4), psi (ternary), o2
    if (cudaMalloc(&s.o1, N * eq_bytes(P.nc)) != cudaSuccess) {
      cudaGetLastError();
      s.o1 = nullptr;
      return LB3DC_ENOMEM;
    }
    if (P.nc == 3) {
      s.o3 = s.o1 + N;
      s.psi = reinterpret_cast<float2 *>(s.o3 + N);
      s.o2 = reinterpret_cast<float *>(s.psi + N);
    } else {
      s.o2 = reinterpret_cast<float *>(s.o1 + N);
    }
    s.bytes += (long long)N * eq_bytes(P.nc);
  }
  if (s.lat.flags & LAT_ROCK) {
    if (!s.mask) {
      if (cudaMalloc(&s.mask, N * sizeof(uint32_t)) != cudaSuccess) {
        s.mask = nullptr;
        cudaGetLastError();
        return LB3DC_ENOMEM;
      }
      s.bytes += (long long)N * 4;
    }
    if (eq_build_mask(P.nx, P.ny, P.nz, P.le != 0, s.rock, s.mask, reinterpret_cast<float2 *>(s.M), s.lat.psi0,
                      st) != cudaSuccess)
      return LB3DC_ECUDA;
  }
  return LB3DC_OK;
}

static bool eq_kernel_of(const DevParams &P, const Fp32State &s, int pass, bool first, int tx, int ty, EqKernel *k) {
  const bool rock = (s.lat.flags & LAT_ROCK) != 0;
  int ax = tx, ay = ty;
  if (pass <= EQ_SURFACTANT) eq_moments_tile(P.nx, P.le != 0, &ax, &ay);
  return eq_kernel(pass, first, P.nc, rock, s.le_h[0] != nullptr, ax, ay, 19ull * P.nc * s.S < (1ull << 32), k);
}

// One step of strategy 3: the moments pass (ternary: two of them after the
// first step of a loop), the dipole pass (ternary) and the collide pass, each on
// its own tile list and resident grid; with le (a binary Lees-Edwards lattice)
// the stage-6 halo kernel runs before the moments pass and the stage-8 one
// before the collide pass.  The halo kernels, bound by FP64 latency at 12 % of
// the issue slots, concern only the tiles on the sheared boundary (eq_edge of
// the moments tiles, at the end of the list): a lattice whose moments tiles fill
// more than one round of the resident CTAs runs halo, boundary tiles and halo on
// the copy stream while the other tiles run on st.  Where they fill about two
// rounds or more, a step takes 128^3 162 -> 155 us, 144x112x112 131 -> 126,
// 160x100x100 128 -> 123, 256x128x128 221 -> 211, 200^3 431 -> 407 (96x512x16 74
// and 74, 200x96x48 79 -> 81); where all run in one round, the boundary tiles take
// as long as the others and start a halo kernel later: 112^3 107 us unforked and
// 118 forked, 192x128x128 188 and 201, 224x160x128 261 and 292, 512x64x64 145 and
// 157, 64x192x192 170 and 172.
// The first pass of a loop launches plainly: everything before it on the stream,
// the parity flip of the loop before included, is complete and visible when it
// starts, and so when any later pass does, which is what lets those read the
// descriptor before their own wait.  Lattices with rock launch every pass
// plainly: the overlap of programmatic dependent launch measured 0.8 % slower on
// the porous lattice, 0.9-1 % faster on the others.
static cudaError_t eq_step(const DevParams &P, Fp32State &s, const uint8_t *rockp, bool first, bool last,
                           const LEStep *le, cudaStream_t st) {
  if (le && !s.le_h[0]) return cudaErrorInvalidValue;
  const bool rock = (s.lat.flags & LAT_ROCK) != 0;
  const unsigned leg = (unsigned)((2 * P.ny * P.nz + 63) / 64);  // two threads per (y, z)
  EqArgs a{};
  a.lats = s.d_lat;
  a.f0 = s.f[0], a.f1 = s.f[1], a.db0 = s.db[0], a.db1 = s.db[1];
  a.rock = rockp;
  a.mask = s.mask;
  a.X = EqFields{s.M, P.nc == 3 ? s.psi : reinterpret_cast<float2 *>(s.M), s.o1, s.o3, s.o2,
                 {reinterpret_cast<float4 *>(s.f[0]), reinterpret_cast<float4 *>(s.f[1])}, (unsigned)s.S};
  const bool fork = le && s.eq_edge > 0;
  cudaError_t e = cudaSuccess;
  for (int pass = 0; pass < EQ_PASSES && e == cudaSuccess; ++pass) {
    EqKernel k;
    if (!eq_kernel_of(P, s, pass, first, s.tx, s.ty, &k)) continue;
    a.tiles = s.eq_tiles + s.eq_off[pass];
    a.ntiles = s.eq_ntiles[pass];
    if (fork && pass == EQ_MOMENTS) {
      // xev[0]: the previous step is done; xev[1]: the boundary's part is done
      if ((e = cudaEventRecord(s.xev[0], st)) != cudaSuccess) break;
      if ((e = cudaStreamWaitEvent(s.xs, s.xev[0], 0)) != cudaSuccess) break;
      k_le_pre32<2><<<leg, 64, 0, s.xs>>>(P, *le, s.d_lat, s.f[0], s.f[1], a.X.S);
      EqArgs edge = a;
      edge.tiles = a.tiles + (a.ntiles - s.eq_edge);
      edge.ntiles = s.eq_edge;
      a.ntiles -= s.eq_edge;
      if ((e = cudaGetLastError()) == cudaSuccess) e = eq_launch(k, pass, first, last, edge, false, s.xs);
      if (e != cudaSuccess) break;
      k_le_post32<2><<<leg, 64, 0, s.xs>>>(P, *le, s.d_lat, s.f[0], s.f[1], a.X.S);
      if ((e = cudaGetLastError()) != cudaSuccess) break;
      if ((e = cudaEventRecord(s.xev[1], s.xs)) != cudaSuccess) break;
      if (a.ntiles) e = eq_launch(k, pass, first, last, a, false, st);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(st, s.xev[1], 0);
      continue;
    }
    if (le && !fork && pass == EQ_MOMENTS)
      k_le_pre32<2><<<leg, 64, 0, st>>>(P, *le, s.d_lat, s.f[0], s.f[1], a.X.S);
    if (le && !fork && pass == EQ_COLLIDE)
      k_le_post32<2><<<leg, 64, 0, st>>>(P, *le, s.d_lat, s.f[0], s.f[1], a.X.S);
    if ((e = cudaGetLastError()) == cudaSuccess)
      e = eq_launch(k, pass, first, last, a,
                    !rock && !(first && pass == EQ_MOMENTS) && !(fork && pass == EQ_COLLIDE), st);
  }
  return e;
}

// The z chunking of one pass of strategy 3: nxy column tiles, `resident`
// CTAs at once, `halo` planes each chunk reads beyond its own.  Chooses the
// number of chunks per column so that the tiles fill whole rounds of the
// resident grid (1 to 8 rounds), weighed against the halo planes that
// shorter chunks reload; the chunks of a column differ in length by at most
// one plane.
int fp32_z_chunks(int nz, int nxy, int resident, int halo) {
  int best = 1;
  double best_score = -1.0;
  for (int rounds = 1; rounds <= 8; ++rounds) {
    int k = std::min(nz, std::max(1, (int)((long long)rounds * resident / nxy)));
    const long long nt = (long long)nxy * k;
    const long long used = (nt + resident - 1) / resident * resident;
    const double zc = (double)nz / k;
    const double score = (double)nt / used * zc / (zc + halo);
    if (score > best_score + 1e-9) best_score = score, best = k;
  }
  return best;
}

// A tile list on the device; null when there is no room for it.
static Tile *upload_tiles(const std::vector<Tile> &tiles, cudaStream_t st, int *rc) {
  Tile *d = nullptr;
  *rc = LB3DC_OK;
  if (cudaMalloc(&d, tiles.size() * sizeof(Tile)) != cudaSuccess) {
    cudaGetLastError();
    *rc = LB3DC_ENOMEM;
    return nullptr;
  }
  if (cudaMemcpyAsync(d, tiles.data(), tiles.size() * sizeof(Tile), cudaMemcpyHostToDevice, st) == cudaSuccess &&
      cudaStreamSynchronize(st) == cudaSuccess)
    return d;
  cudaFree(d);
  *rc = LB3DC_ECUDA;
  return nullptr;
}

// The tile lists of strategy 3's passes, one after the other.
struct EqTiles {
  std::vector<Tile> all;
  int off[EQ_PASSES], ntiles[EQ_PASSES], edge = 0;
};

static int eq_build_tiles(const DevParams &P, const Fp32State &s, const FusedShape &sh, EqTiles &out) {
  const LatDesc &L = s.lat;
  std::vector<Tile> &all = out.all;
  // a chunk of any pass works on one plane beyond each of its ends
  for (int pass = 0; pass < EQ_PASSES; ++pass) {
    out.off[pass] = (int)all.size();
    out.ntiles[pass] = 0;
    EqKernel kn;
    if (!eq_kernel_of(P, s, pass, false, sh.tx, sh.ty, &kn)) {
      if (pass == EQ_MOMENTS || pass == EQ_COLLIDE) return LB3DC_EINVAL;
      continue;
    }
    int tx = sh.tx, ty = sh.ty, res = 0;
    if (pass <= EQ_SURFACTANT) eq_moments_tile(P.nx, P.le != 0, &tx, &ty);
    if (fp32_prepare_kernel(kn.fn, kn.threads, kn.smem, &res) != cudaSuccess) return LB3DC_ECUDA;
    const int nxt = (L.nx + tx - 1) / tx, nxy = nxt * ((L.ny + ty - 1) / ty);
    const int k = fp32_z_chunks(L.nz, nxy, res, 2);
    for (int c = 0; c < k; ++c) {
      const int z0 = (int)((long long)L.nz * c / k), z1 = (int)((long long)L.nz * (c + 1) / k);
      for (int yt = 0; yt * ty < L.ny; ++yt)
        for (int xt = 0; xt < nxt; ++xt) {
          Tile t;
          t.lat = 0;
          // sheared lattices: the tiles on the x boundary take longer; rotated
          // by row and chunk they do not all fall to the same CTAs
          t.x0 = (P.le ? (xt + yt + c) % nxt : xt) * tx;
          t.y0 = yt * ty;
          t.z0 = z0;
          t.zc = z1 - z0;
          all.push_back(t);
        }
    }
    out.ntiles[pass] = (int)all.size() - out.off[pass];
    if (pass == EQ_MOMENTS && P.le && out.ntiles[pass] > res) {
      auto inner = [&](const Tile &t) { return t.x0 != 0 && t.x0 + tx < L.nx; };
      const auto end = std::stable_partition(all.begin() + out.off[pass], all.end(), inner);
      const auto start = all.begin() + out.off[pass];
      out.edge = end > start ? (int)(all.end() - end) : 0;  // all on the boundary: nothing to run beside
    }
  }
  return LB3DC_OK;
}

// Lees-Edwards lattices: the compact pre-stream boundary planes from the
// current state (after an upload or a restore; the collide passes keep them
// current from then on).
static cudaError_t le_gather(const DevParams &P, Fp32State &s, cudaStream_t st) {
  const long long n = (long long)P.nc * 19 * P.ny * P.nz;
  k_le_gather32<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s.d_lat, s.f[0], s.f[1], (unsigned)s.S);
  return cudaGetLastError();
}

// The Lees-Edwards halo planes of a single lattice, referenced by its descriptor.
static void attach_le(Fp32State &s) {
  for (int b = 0; b < 2; ++b) {
    s.lat.le_h[b] = s.le_h[b];
    s.lat.le_p[b] = s.le_p[b];
  }
  for (int b = 0; b < 4; ++b) s.lat.le_b[b] = s.le_b[b];
}

// Shape before any autotuning.  Fully relaxing lattices: strategy 3 with 16x8
// tiles, the fastest or within 3 % of it on every lattice measured (ternary
// 32^3, 64^3, 75x67x87, 128^3: 0.019, 0.040, 0.062, 0.202 ms a step against
// 0.058, 0.082, 0.126, 0.384 for strategy 2; binary 256x128x128 0.157 against
// 0.432, sheared 0.211 against 0.564, porous 192^3 0.273 against 0.924).
// Others: the split strategy with the staged collide pass, the fastest of 0 to
// 2.
static FusedShape default_shape(const DevParams &P) {
  if (fp32_eq_eligible(P)) return FusedShape{16, 8, 16, 3};
  FusedShape sh{32, 4, P.nc == 3 ? 8 : 16, 2};
  if (P.nx < 32) sh.tx = 16, sh.ty = 8;
  return sh;
}

// The own-moment field J is read only by the plain split strategy (split 1);
// it is allocated the first time a lattice is switched to that strategy, so
// the other strategies hold no memory for it.
static int ensure_own(const DevParams &P, Fp32State &s) {
  if (s.J) return LB3DC_OK;
  const size_t b = (size_t)P.nsites * fp32_own_bytes(P.nc);
  if (cudaMalloc(&s.J, b) != cudaSuccess) {
    s.J = nullptr;
    cudaGetLastError();
    return LB3DC_ENOMEM;
  }
  s.bytes += (long long)b;
  return LB3DC_OK;
}

// Switches to a launch shape; where that fails the present one stays whole.
static int rebuild_tiles(const DevParams &P, Fp32State &s, const FusedShape &sh, cudaStream_t st) {
  const bool rock = (s.lat.flags & LAT_ROCK) != 0, body = (s.lat.flags & LAT_BODY) != 0;
  int rc = LB3DC_OK, per = 0;
  if (sh.split != 3 && (per = fp32_fused_ctas_per_sm(P.nc, rock, body, sh)) < 1) return LB3DC_EINVAL;
  if (sh.split == 1 && (rc = ensure_own(P, s))) return rc;
  EqTiles eq;
  Tile *d_eq = nullptr;
  if (sh.split == 3) {
    if (!fp32_eq_eligible(P)) return LB3DC_ENOTSUP;
    if ((rc = ensure_eq(P, s, st)) || (rc = eq_build_tiles(P, s, sh, eq))) return rc;
    if (!(d_eq = upload_tiles(eq.all, st, &rc))) return rc;
  }
  std::vector<Tile> tiles;
  fp32_tiles_for(s.lat, 0, sh, tiles);
  Tile *d = upload_tiles(tiles, st, &rc);
  if (!d) {
    if (d_eq) cudaFree(d_eq);
    return rc;
  }
  if (d_eq) {
    if (s.eq_tiles) cudaFree(s.eq_tiles);
    s.eq_tiles = d_eq;
    std::copy(eq.off, eq.off + EQ_PASSES, s.eq_off);
    std::copy(eq.ntiles, eq.ntiles + EQ_PASSES, s.eq_ntiles);
    s.eq_edge = eq.edge;
  }
  if (s.d_tiles) cudaFree(s.d_tiles);
  s.d_tiles = d;
  s.ntiles = (int)tiles.size();
  s.tx = sh.tx;
  s.ty = sh.ty;
  s.zc = sh.zc;
  s.split = sh.split;
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  // strategy 3: each pass sizes its own grid at launch
  s.grid = sh.split == 3 ? s.ntiles : std::min(s.ntiles, per * nsm);
  return LB3DC_OK;
}

int fp32_set_shape(const DevParams &P, Fp32State &s, const FusedShape &sh, cudaStream_t st) {
  if (!fused_fn(P.nc, false, false, sh)) return LB3DC_EINVAL;
  // Lees-Edwards lattices and lattices with inflow boundaries run the
  // staged split strategy only
  if ((s.le_h[0] && sh.split < 2) || (s.lat.invk && sh.split != 2)) return LB3DC_ENOTSUP;
  if (sh.split == 3 && !fp32_eq_eligible(P)) return LB3DC_ENOTSUP;
  if (sh.split && !s.M) return LB3DC_EINVAL;
  if (sh.split < 0 || sh.split > 3) return LB3DC_EINVAL;
  if (sh.zc < 1) return LB3DC_EINVAL;
  const FusedShape entry{s.tx, s.ty, s.zc, s.split};
  int rc = rebuild_tiles(P, s, sh, st);
  if (rc == LB3DC_ENOMEM && sh.split != 3 && fp32_make_room(s, st)) {
    rc = rebuild_tiles(P, s, sh, st);
    if (rc) rebuild_tiles(P, s, entry, st);
  }
  return rc;
}

std::vector<FusedShape> fp32_candidate_shapes(const DevParams &P) {
  std::vector<FusedShape> out;
  const int xy[5][2] = {{32, 8}, {32, 4}, {16, 16}, {16, 8}, {64, 4}};
  const int zcs[3] = {8, 16, 32};
  for (auto &t : xy) {
    if (t[0] > 2 * P.nx && t[0] > 16) continue;
    for (int zc : zcs) {
      if (zc > P.nz && zc != 8) continue;
      for (int split = (P.le || P.invk) ? 2 : 0; split < 3; ++split)
        out.push_back(FusedShape{t[0], t[1], zc, split});
    }
  }
  // strategy 3 chunks z per pass from each pass's resident grid: one
  // candidate per tile shape (its zc is not used)
  if (fp32_eq_eligible(P)) {
    for (auto &t : xy) {
      if (t[0] > 2 * P.nx && t[0] > 16) continue;
      out.push_back(FusedShape{t[0], t[1], 16, 3});
    }
  }
  return out;
}

// The project's autotuner: time each candidate shape with CUDA events on a
// saved copy of the state, keep the fastest and restore the state.
int fp32_autotune(const DevParams &P, Fp32State &s, const uint8_t *rock, double *ms_out,
                  int *ntried, cudaStream_t st, const LEStep *le) {
  const size_t pop = (size_t)P.nc * 19 * s.S * sizeof(float);
  const size_t dbs = P.nc == 3 ? 3 * (size_t)s.S * sizeof(float) : 0;
  float *save = nullptr;
  const FusedShape entry{s.tx, s.ty, s.zc, s.split};
  if (alloc_device(s, (void **)&save, pop + dbs, st)) return LB3DC_ENOMEM;
  const bool made_way = s.split != entry.split;
  const int cur0 = s.lat.parity;
  cudaMemcpyAsync(save, s.f[cur0], pop, cudaMemcpyDeviceToDevice, st);
  if (dbs) cudaMemcpyAsync((char *)save + pop, s.db[cur0], dbs, cudaMemcpyDeviceToDevice, st);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  FusedShape best{s.tx, s.ty, s.zc, s.split};
  float best_ms = 1e30f;
  KernelTimer *saved_timer = s.timer;
  s.timer = nullptr;
  int n = 0;
  for (const FusedShape &sh : fp32_candidate_shapes(P)) {
    if (rebuild_tiles(P, s, sh, st) != LB3DC_OK) continue;
    if (fp32_run(P, s, rock, 2, st, le) != LB3DC_OK) continue;
    cudaEventRecord(e0, st);
    const int reps = 5;
    if (fp32_run(P, s, rock, reps, st, le) != LB3DC_OK) continue;
    cudaEventRecord(e1, st);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    ms /= reps;
    if (ms_out && n < 64) ms_out[n] = ms;
    ++n;
    if (ms < best_ms) {
      best_ms = ms;
      best = sh;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  // restore the state into the buffer the lattice now reads from
  const int cur = s.lat.parity;
  cudaMemcpyAsync(s.f[cur], save, pop, cudaMemcpyDeviceToDevice, st);
  if (dbs) cudaMemcpyAsync(s.db[cur], (char *)save + pop, dbs, cudaMemcpyDeviceToDevice, st);
  if (s.le_b[0]) le_gather(P, s, st);
  cudaStreamSynchronize(st);
  cudaFree(save);
  if (ntried) *ntried = n;
  s.timer = saved_timer;
  // strategy 3, where it made way for the copy, was not timed: back to it
  int rc = made_way ? rebuild_tiles(P, s, entry, st) : LB3DC_ENOMEM;
  if (rc == LB3DC_ENOMEM) rc = rebuild_tiles(P, s, best, st);
  if (rc) return rc;
  return cudaStreamSynchronize(st) == cudaSuccess ? LB3DC_OK : LB3DC_ECUDA;
}

int fp32_alloc(const DevParams &P, const lb3dc_params &p, Fp32State &s, cudaStream_t st) {
  const long long N = P.nsites;
  s.S = N;
  const size_t pop = (size_t)P.nc * 19 * N * sizeof(float);
  for (int b = 0; b < 2; ++b) {
    if (cudaMalloc(&s.f[b], pop) != cudaSuccess) return LB3DC_ENOMEM;
    s.bytes += pop;
    cudaMemsetAsync(s.f[b], 0, pop, st);
  }
  if (P.nc == 3) {
    if (cudaMalloc(&s.db[0], 6 * N * sizeof(float)) != cudaSuccess) return LB3DC_ENOMEM;
    s.db[1] = s.db[0] + 3 * N;
    s.bytes += 6 * N * sizeof(float);
    cudaMemsetAsync(s.db[0], 0, 6 * N * sizeof(float), st);
  }
  // one block: M and the staging planes
  const size_t mb = (size_t)N * fp32_moment_bytes(P.nc), sb = 2 * (size_t)N * sizeof(double);
  if (cudaMalloc(&s.M, mb + sb) != cudaSuccess) return LB3DC_ENOMEM;
  s.stage = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(s.M) + mb);
  s.bytes += (long long)(mb + sb);
  if (cudaMalloc(&s.d_lat, sizeof(LatDesc)) != cudaSuccess) return LB3DC_ENOMEM;
  if (cudaStreamCreateWithFlags(&s.xs, cudaStreamNonBlocking) != cudaSuccess) return LB3DC_ECUDA;
  for (int i = 0; i < 4; ++i)
    if (cudaEventCreateWithFlags(&s.xev[i], cudaEventDisableTiming) != cudaSuccess) return LB3DC_ECUDA;
  if (P.le) {
    // one block: the psi planes and the 2 + 4 population planes
    const size_t np = (size_t)P.ny * P.nz, plane = (size_t)P.nc * 19 * np;
    const size_t bytes = 2 * np * sizeof(float2) + 6 * plane * sizeof(float);
    if (cudaMalloc(&s.le_p[0], bytes) != cudaSuccess) return LB3DC_ENOMEM;
    s.le_p[1] = s.le_p[0] + np;
    float *f = reinterpret_cast<float *>(s.le_p[1] + np);
    for (int b = 0; b < 2; ++b) s.le_h[b] = f + b * plane;
    for (int b = 0; b < 4; ++b) s.le_b[b] = f + (2 + b) * plane;
    s.bytes += (long long)bytes;
  }
  s.lat = fp32_make_desc(P, p.rho0 > 0 ? p.rho0 : 0.7, 0, false);
  attach_le(s);
  FusedShape sh = default_shape(P);
  int rc = rebuild_tiles(P, s, sh, st);
  if (rc == LB3DC_ENOMEM && sh.split == 3) {
    // no room for strategy 3's fields
    sh = FusedShape{sh.tx, sh.ty, sh.zc, 2};
    rc = rebuild_tiles(P, s, sh, st);
  }
  return rc;
}

void fp32_free(Fp32State &s) {
  for (int b = 0; b < 2; ++b) {
    if (s.f[b]) cudaFree(s.f[b]);
    s.f[b] = nullptr;
  }
  if (s.db[0]) cudaFree(s.db[0]);
  s.db[0] = s.db[1] = nullptr;
  if (s.d_lat) cudaFree(s.d_lat);
  if (s.d_tiles) cudaFree(s.d_tiles);
  if (s.M) cudaFree(s.M);
  if (s.J) cudaFree(s.J);
  free_eq(s);
  s.stage = nullptr;
  for (int i = 0; i < 4; ++i) {
    if (s.xev[i]) cudaEventDestroy(s.xev[i]);
    s.xev[i] = nullptr;
  }
  if (s.xs) cudaStreamDestroy(s.xs);
  s.xs = nullptr;
  if (s.le_p[0]) cudaFree(s.le_p[0]);
  for (int b = 0; b < 2; ++b) s.le_h[b] = nullptr, s.le_p[b] = nullptr;
  for (int b = 0; b < 4; ++b) s.le_b[b] = nullptr;
  s.d_lat = nullptr;
  s.d_tiles = nullptr;
  s.M = nullptr;
  s.J = nullptr;
}

int fp32_upload(const DevParams &P, const lb3dc_params &p, Fp32State &s, const double *n,
                const double *db, const uint8_t *rockp, cudaStream_t st) {
  const long long N = P.nsites;
  const double rho0 = s.lat.rho0;
  // the caller has uploaded the rock flags (rockp, device) and set any_rock
  const bool any = P.any_rock != 0;
  if (any && P.nc == 3) return LB3DC_EINVAL;
  const int flags = s.lat.flags;
  s.lat = fp32_make_desc(P, rho0, 0, any);
  attach_le(s);
  s.lat.parity = 0;
  s.rock = rockp;
  // one FP64 plane at a time through two staging planes: the copy of plane
  // cq + 1 (copy stream) overlaps the conversion of plane cq (populations to
  // deviations, dipoles rounded to FP32, into both buffers); xev[b] marks
  // staging plane b filled, xev[2 + b] drained
  const int nplanes = P.nc * 19 + (P.nc == 3 ? 3 : 0);
  cudaError_t e = cudaEventRecord(s.xev[2], st);
  if (e == cudaSuccess) e = cudaEventRecord(s.xev[3], st);
  for (int cq = 0; cq < nplanes && e == cudaSuccess; ++cq) {
    const int b = cq & 1;
    double *stg = s.stage + (size_t)b * N;
    const bool pop = cq < P.nc * 19;
    const double *src = pop ? n + (size_t)cq * N : db + (size_t)(cq - P.nc * 19) * N;
    float *d0 = pop ? s.f[0] + (size_t)cq * s.S : s.db[0] + (size_t)(cq - P.nc * 19) * s.S;
    float *d1 = pop ? s.f[1] + (size_t)cq * s.S : s.db[1] + (size_t)(cq - P.nc * 19) * s.S;
    const double w = pop ? (cq % 19 == 18 ? 1.0 / 3.0 : 1.0 / 36.0) * rho0 : 0.0;
    e = cudaStreamWaitEvent(s.xs, s.xev[2 + b], 0);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(stg, src, (size_t)N * sizeof(double), cudaMemcpyHostToDevice, s.xs);
    if (e == cudaSuccess) e = cudaEventRecord(s.xev[b], s.xs);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st, s.xev[b], 0);
    if (e != cudaSuccess) break;
    k_plane_from_fp64<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(stg, d0, d1, N, w,
                                                                    any ? rockp : nullptr);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaEventRecord(s.xev[2 + b], st);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s.xs);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return LB3DC_ECUDA;
  if (cudaMemcpyAsync(s.d_lat, &s.lat, sizeof(LatDesc), cudaMemcpyHostToDevice, st) != cudaSuccess)
    return LB3DC_ECUDA;
  if (s.le_b[0] && le_gather(P, s, st) != cudaSuccess) return LB3DC_ECUDA;
  // keep the launch shape chosen so far (set or autotuned); the kernel variant,
  // and with it the tile lists, may change with the rock flag, the neighbour
  // mask with every upload
  int rc = s.lat.flags != flags ? rebuild_tiles(P, s, FusedShape{s.tx, s.ty, s.zc, s.split}, st)
           : s.split == 3       ? ensure_eq(P, s, st)
                                : LB3DC_OK;
  if (rc == LB3DC_ENOMEM && s.split == 3) {  // no room for the neighbour mask
    fp32_make_room(s, st);
    rc = rebuild_tiles(P, s, FusedShape{s.tx, s.ty, s.zc, 2}, st);
  }
  if (rc) return rc;
  (void)p;
  return cudaStreamSynchronize(st) == cudaSuccess ? LB3DC_OK : LB3DC_ECUDA;
}

int fp32_download(const DevParams &P, const lb3dc_params &p, Fp32State &s, double *n, double *db,
                  double *rho, double *mom, double *da, const uint8_t *rockp, cudaStream_t st) {
  const long long N = P.nsites;
  const int nc = P.nc;
  const int cur = s.lat.parity;
  const double rho0 = s.lat.rho0;
  // one FP64 plane at a time through two staging planes: the conversion of a
  // plane (and the sums of the density and momentum planes) overlaps the copy
  // of the one before (copy stream); xev[b] marks staging plane b filled,
  // xev[2 + b] drained
  const uint8_t *rk = rockp && (s.lat.flags & LAT_ROCK) ? rockp : nullptr;
  cudaError_t e = cudaEventRecord(s.xev[2], s.xs);
  if (e == cudaSuccess) e = cudaEventRecord(s.xev[3], s.xs);
  int planes = 0;
  auto plane = [&](int kind, const float *src, double w, double *dst) {
    if (e != cudaSuccess) return;
    const int b = planes++ & 1;
    double *stg = s.stage + (size_t)b * N;
    e = cudaStreamWaitEvent(st, s.xev[2 + b], 0);
    if (e != cudaSuccess) return;
    k_plane_to_fp64<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(PlaneJob{kind, src, rho0}, s.S, stg, N, w, rk);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaEventRecord(s.xev[b], st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s.xs, s.xev[b], 0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dst, stg, (size_t)N * sizeof(double), cudaMemcpyDeviceToHost, s.xs);
    if (e == cudaSuccess) e = cudaEventRecord(s.xev[2 + b], s.xs);
  };
  for (int c = 0; c < nc; ++c) {
    const float *f = s.f[cur] + (size_t)c * 19 * s.S;
    for (int q = 0; n && q < 19; ++q)
      plane(0, f + (size_t)q * s.S, (q == 18 ? 1.0 / 3.0 : 1.0 / 36.0) * rho0, n + ((size_t)c * 19 + q) * N);
    if (rho) plane(1, f, 0.0, rho + (size_t)c * N);
    for (int k = 0; mom && k < 3; ++k) plane(2 + k, f, 0.0, mom + ((size_t)c * 3 + k) * N);
  }
  for (int k = 0; db && nc == 3 && k < 3; ++k) plane(5, s.db[cur] + (size_t)k * s.S, 0.0, db + (size_t)k * N);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s.xs);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return LB3DC_ECUDA;
  if (db && nc != 3) std::memset(db, 0, 3 * N * sizeof(double));
  if (da) std::memset(da, 0, 3 * N * sizeof(double));
  (void)p;
  return LB3DC_OK;
}

int fp32_step(const DevParams &P, Fp32State &s, const uint8_t *rock, cudaStream_t st,
              const LEStep *le) {
  return fp32_run(P, s, rock, 1, st, le);
}

int fp32_run(const DevParams &P, Fp32State &s, const uint8_t *rock, int nsteps, cudaStream_t st,
             const LEStep *le, bool le_per_step) {
  FusedShape sh{s.tx, s.ty, s.zc, s.split};
  const bool rk = (s.lat.flags & LAT_ROCK) != 0, body = (s.lat.flags & LAT_BODY) != 0;
  if (le && !s.le_h[0]) return LB3DC_ESTATE;
  // kernels per step: the pass(es) (ternary strategy 3: one more after its
  // first step; forked sheared lattices: the moments pass in two parts), two
  // Lees-Edwards halo kernels, and the parity flip (strategy 3: one for the
  // whole loop)
  const int passes = sh.split ? (P.nc == 3 ? 3 : 2) : 1;
  for (int i = 0; i < nsteps; ++i) {
    const LEStep *l = le ? le + (le_per_step ? i : 0) : nullptr;
    const bool flip = sh.split != 3 || i == nsteps - 1;
    if (s.timer) s.timer->start(st);
    cudaError_t e = sh.split == 3
                        ? eq_step(P, s, rock, i == 0, i == nsteps - 1, l, st)
                        : fp32_launch_fused(P.nc, rk, body, sh, s.d_lat, s.d_tiles, s.ntiles, 0,
                                            s.f[0], s.f[1], s.db[0], s.db[1], rock, s.S, st, s.M,
                                            s.J, l, &P);
    if (s.timer) {
      s.timer->stop(st);
      s.timer->launches += passes + (sh.split == 3 && P.nc == 3 && i > 0 ? 1 : 0) + (le ? 2 : 0) + (flip ? 1 : 0) +
                           (sh.split == 3 && l && s.eq_edge > 0 && s.eq_edge < s.eq_ntiles[EQ_MOMENTS] ? 1 : 0);
    }
    if (e != cudaSuccess) return LB3DC_ECUDA;
    if (!flip) continue;
    e = fp32_flip_parity(s.d_lat, 1, st);
    if (e != cudaSuccess) return LB3DC_ECUDA;
    s.lat.parity ^= 1;
  }
  return LB3DC_OK;
}

// Dumps of the FP32 state: the deviations are converted to FP64
// populations on the device and the FP64 dump kernels are applied, with the
// densities recomputed from the current populations (the FP32 path does not
// keep the post-stream moments between steps).
int fp32_dump(const DevParams &P, Fp32State &s, int field, const uint8_t *rock, double *out,
              cudaStream_t st) {
  const long long N = P.nsites;
  const int nc = P.nc;
  double *n = nullptr, *rho = nullptr, *psi = nullptr, *mom = nullptr, *db = nullptr;
  size_t bytes = ((size_t)nc * 19 * N + 2 * (size_t)nc * N + 3 * (size_t)nc * N + 3 * (size_t)N) * 8;
  const FusedShape entry{s.tx, s.ty, s.zc, s.split};
  if (alloc_device(s, (void **)&n, bytes, st)) return LB3DC_ENOMEM;
  rho = n + (size_t)nc * 19 * N;
  psi = rho + (size_t)nc * N;
  mom = psi + (size_t)nc * N;
  db = mom + 3 * (size_t)nc * N;
  const int cur = s.lat.parity;
  k_to_fp64<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(s.f[cur], n, s.S, 0, N, nc, s.lat.rho0);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = fp64_moments(P, n, rho, psi, mom, st);
  if (e == cudaSuccess && nc == 3) e = fp32_planes_to_fp64(s.db[cur], db, s.S, 0, N, 3, st);
  if (e == cudaSuccess) e = fp64_dump(P, field, n, rho, psi, db, rock, out, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFree(n);
  if (s.split != entry.split) rebuild_tiles(P, s, entry, st);  // strategy 3 again, where it had made way
  return e == cudaSuccess ? LB3DC_OK : LB3DC_ECUDA;
}

cudaError_t fp32_reduce_conservation(const DevParams &P, Fp32State &s, const uint8_t *rock,
                                     double *scratch, double mass[3], double mom[3],
                                     cudaStream_t st) {
  return reduce_conservation_fp32(P, s.f[s.lat.parity], s.S, 0, (double)s.lat.rho0, rock, scratch,
                                  mass, mom, st);
}

cudaError_t fp32_sanity_counts(const DevParams &P, Fp32State &s, unsigned long long *scratch,
                               unsigned long long cnt[2], cudaStream_t st) {
  return sanity_counts_fp32(P, s.f[s.lat.parity], s.S, 0, (double)s.lat.rho0, scratch, cnt, st);
}

cudaError_t fp32_sanity_velocity(const DevParams &P, Fp32State &s, const uint8_t *rock,
                                 void *scratch, SanityVelocity &out, cudaStream_t st) {
  return sanity_velocity_fp32(P, s.f[s.lat.parity], s.S, 0, (double)s.lat.rho0, rock, scratch, out,
                              st);
}

}  // namespace lb3d
