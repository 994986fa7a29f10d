// fp32_eqstate.cu -- strategy 3 of the FP32 deviation path: fully relaxing
// lattices (tau = 1) carry the equilibrium's arguments from step to step.
//
// With omega_c = 1 the BGK update (code/lb3d_collision.F90:258-284) leaves
// every component in equilibrium, so between two steps a site's 19 nc
// populations are a function of 4 nc numbers: the density deviation drho_c
// and the velocity v_c the equilibrium was taken at.  Inside a time loop
// the collide pass stores those ({drho_c, v_c}: 48 B a ternary site, 32 B a
// binary one, instead of 228 B and 152 B of populations), and the next
// moments pass evaluates the populations again where they are pulled, with
// eq_store's expressions on the same arguments: the same bits as stored and
// reloaded populations.  The first moments pass of a loop reads populations,
// the last collide pass writes them, so the lattice's state outside a loop is
// the populations, as with every other strategy.
//
// Passes per step (binary lattices skip the second):
//   moments   k_eq_moments0 (from populations) or k_eq_moments (ternary: two
//             launches, red with blue and the surfactant): the pulled
//             post-stream deviations (code/lb3d_advection.F90:109-151,
//             bounce-back of code/lb3d_bc_bounce.F90:53-90) reduced to the
//             densities, the weighted momentum P = sum_c amass_c omega_c j_c
//             (code/lb3d_collision.F90:560-587), the red and blue psi
//             deviations and (ternary) phi = rho_b - rho_r with the advected
//             dipole flux da (code/lb3d_advection.F90:137-148);
//   dipole    k_eq_dipole: the dipole relaxation (code/lb3d_collision.F90:
//             296-403) and the force-stencil entry {a = d psi_s, dpsi_s};
//   collide   k_eq_collide: Shan-Chen force (code/lb3d_force_shanchen.F90:
//             127-330), body force, velocities, and the arguments (or, in the
//             last step of a loop, the populations) of the next state.
//
// The arguments and the dipoles of the steps between lie in X.Q, which a
// single lattice lays over the buffer the loop's first pass has read (dead
// from then on), so a loop needs no memory beyond the pass fields, and flips
// the lattice's parity once.  Lattices of an ensemble share the launches
// through their descriptors and tile lists, as in the other strategies.
#include <algorithm>
#include <type_traits>

#include "fp32_device.cuh"
#include "fp32_eqstate.h"

namespace lb3d {
namespace f32 {

// Plane class of a direction and its index within the class: D (c_z = -1),
// Z (c_z = 0), U (c_z = +1).  The two directions along z (4, 5) are pulled
// by the thread that evaluated them and never leave its registers.
LB3D_HDI constexpr int dir_slot(int q) {
  return q == 9 ? 0 : q == 13 ? 1 : q == 15 ? 2 : q == 17 ? 3                    // D
       : q == 8 ? 0 : q == 12 ? 1 : q == 14 ? 2 : q == 16 ? 3                    // U
       : q < 4 ? q : q == 6 ? 4 : q == 7 ? 5 : q == 10 ? 6 : 7;                  // Z
}

// The deviation of a rock site's (zero) population q: as an upload stores it.
__device__ __forceinline__ float rock_dev(int q, float rho0) {
  return -(float)__dmul_rn(q == 18 ? 1.0 / 3.0 : 1.0 / 36.0, (double)rho0);
}

// The red and blue entries of a site: psi deviations, density deviations and
// their part of the weighted momentum P, summed as the other strategies'
// collide passes sum it.
__device__ __forceinline__ void put_rb(const EqFields &X, size_t i, const LatDesc &Lg, float2 dr, float2 j0, float2 j1,
                                       float2 j2) {
  const float am0 = Lg.amass[0] * Lg.omega[0], am1 = Lg.amass[1] * Lg.omega[1], em0 = Lg.em0;
  X.psi[i] = make_float2(-em0 * expm1f(-dr.x), -em0 * expm1f(-dr.y));
  X.o1[i] = make_float4(dr.x, dr.y, fmaf(am1, j0.y, fmaf(am0, j0.x, 0.f)), fmaf(am1, j1.y, fmaf(am0, j1.x, 0.f)));
  X.o2[i] = fmaf(am1, j2.y, fmaf(am0, j2.x, 0.f));
}

// ---------------------------------------------------------------------------
// Moments pass from populations (the first step of a loop): one thread per
// tile site, marching the tile's z range; the previous dipoles (ternary)
// stream through a four-plane ring with a one-site halo, refilled with
// cp.async one plane ahead.  HBM-bound: 19 nc deviations read per site.
// ---------------------------------------------------------------------------
template <int NC, int TX, int TY, bool ROCK, bool NARROW, bool LE>
__global__ void __launch_bounds__(TX *TY, 1024 / (TX * TY))
    k_eq_moments0(const LatDesc *__restrict__ lats, const Tile *__restrict__ tiles, int ntiles, const float *f0,
                  const float *f1, const float *db0, const float *db1, const uint8_t *__restrict__ rock,
                  const __grid_constant__ EqFields X) {
  constexpr int NT = TX * TY, DW = TX + 2, DN = DW * (TY + 2), DR = 4;
  extern __shared__ float4 smd[];  // previous dipoles [DR][DN] (ternary)
  const unsigned S = X.S;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  pdl_launch_next();
  pdl_wait_previous();
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const Tile T = tiles[t];
    const LatDesc &Lg = lats[T.lat];
    const int nx = Lg.nx, ny = Lg.ny, nz = Lg.nz;
    const int par = Lg.parity;
    const float *__restrict__ F = (par ? f1 : f0) + Lg.base;
    const float *__restrict__ DBi = (NC == 3) ? (par ? db1 : db0) + Lg.base : nullptr;
    const uint8_t *__restrict__ RK = rock + Lg.base;
    const float rho0 = Lg.rho0;
    const int x0 = T.x0, y0 = T.y0, z0 = T.z0, zc = T.zc;
    const int gx = x0 + tx, gy = y0 + ty;
    const bool act = gx < nx && gy < ny;
    const bool le_edge = x0 == 0 || x0 + TX >= nx;  // the tile holds x = 0 or x = nx - 1
    auto load_db_plane = [&](int j) {  // plane z0 - 1 + j in slot j % DR
      const int gz = wrapz(z0 - 1 + j, nz);
      float *dst = reinterpret_cast<float *>(smd + (j % DR) * DN);
      for (int s = tid; s < DN; s += NT) {
        const int ix = wrapz(x0 - 1 + s % DW, nx), iy = wrapz(y0 - 1 + s / DW, ny);
        const int i = ix + nx * (iy + ny * gz);
        cp_async4(dst + 4 * s, DBi + i);
        cp_async4(dst + 4 * s + 1, DBi + S + i);
        cp_async4(dst + 4 * s + 2, DBi + 2 * (size_t)S + i);
      }
    };
    if (NC == 3) {
      load_db_plane(0);
      load_db_plane(1);
      load_db_plane(2);
      cp_async_commit();
    }
    for (int it = 0; it < zc; ++it) {
      if (NC == 3) {
        if (it + 3 <= zc + 1) load_db_plane(it + 3);
        cp_async_commit();
        cp_async_wait<1>();  // planes up to it + 2 landed (this thread's copies)
        __syncthreads();     // ... and everybody's
      }
      bool fluid = act;
      Nbr nb;
      int self = 0, gz = 0;
      if (act) {
        gz = wrapz(z0 + it, nz);
        make_nbr(nb, gx, gy, gz, nx, ny, nz);
        self = noff<18, 1>(nb);
        // rock sites are never collided and their entries are never written
        // (psi: set once to the deviation of psi = 0): no pulls
        if (ROCK) fluid = __ldg(RK + self) == 0;
      }
      if (LE && ROCK && act && !fluid && le_edge) {
        // a rock site on the sheared boundary keeps its (zero) populations:
        // they go to the post-stream boundary plane as they are
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          float d[19];
#pragma unroll
          for (int q = 0; q < 19; ++q) d[q] = rock_dev(q, rho0);
          le_store_boundary(Lg, 2, c, gx, gy, gz, d);
        }
      }
      if (fluid) {
        float dr[NC], jm[NC][3];
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        const float4 *Dm = smd + (it % DR) * DN, *D0 = smd + ((it + 1) % DR) * DN,
                     *Dp = smd + ((it + 2) % DR) * DN;
        LeYZ lw;
        if constexpr (LE) make_leyz(lw, gy, gz, ny, nz);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          float d[19];
          // Lees-Edwards lattices pull across x = 0 and x = nx - 1 from the
          // sheared halo planes of this step; tiles away from those planes
          // pull as periodic lattices do
          if (LE && le_edge) {
            pull_comp_le<NARROW, ROCK>(F, S, c, nb, self, gx, nx, lw, Lg, ny * nz, d, RK);
            le_store_boundary(Lg, 2, c, gx, gy, gz, d);  // for the stage-8 halo kernel
          } else {
            pull_comp<ROCK, false, NARROW>(F, S, c, nb, self, RK, d);
          }
          own_moments<1>(d, dr[c], jm[c][0], jm[c][1], jm[c][2]);
          if (NC == 3 && c == 2) {
            // da = sum_q (n_s(x - c_q, q) g_q) db(x - c_q) + n_s(x, rest) db(x)
            const int ds0 = (tx + 1) + DW * (ty + 1);
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
        const size_t i = (size_t)Lg.base + self;
        put_rb(X, i, Lg, make_float2(dr[0], dr[1]), make_float2(jm[0][0], jm[1][0]),
               make_float2(jm[0][1], jm[1][1]), make_float2(jm[0][2], jm[1][2]));
        if constexpr (NC == 3) {
          float p[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            p[k] = 0.f;
#pragma unroll
            for (int c = 0; c < NC; ++c) p[k] = fmaf(Lg.amass[c] * Lg.omega[c], jm[c][k], p[k]);
          }
          X.o3[i] = make_float4(dr[2], p[0], p[1], p[2]);
          X.M[i] = make_float4(dr[1] - dr[0], a0, a1, a2);
        }
      }
      if (NC == 3) __syncthreads();  // the next iteration refills a ring slot read here
    }
    if (NC == 3) cp_async_wait<0>();
  }
}

// ---------------------------------------------------------------------------
// Moments pass from the equilibrium's arguments, one launch for red and blue
// (paired lanes) and one for the surfactant with the dipole flux.  A thread
// per site of the tile plus its one-site halo, marching z: each iteration
// evaluates the 19 populations of the newest plane m once per component, and
// after a CTA barrier the tile's threads sum the pulled ones of plane m - 1.
// 16 of the 18 moving populations cross shared memory, in planes by direction:
// D (c_z = -1) is pulled in the iteration that evaluates it, Z in the next, U
// in the one after (one iteration in registers, then two slots); the two
// along z stay in registers.  A halo thread evaluates only the five that
// enter the tile.
// ---------------------------------------------------------------------------
// Arithmetic on one component (float) or two (float2), lane for lane the same
// roundings.
__device__ __forceinline__ float vset(float, float v) { return v; }
__device__ __forceinline__ float2 vset(float2, float v) { return f2(v); }
__device__ __forceinline__ float vadd(float a, float b) { return a + b; }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return add2(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return a * b; }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return mul2(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return fma2(a, b, c); }
__device__ __forceinline__ float vlane(float a, int) { return a; }
__device__ __forceinline__ float vlane(float2 a, int k) { return k ? a.y : a.x; }
__device__ __forceinline__ float vneg(float a) { return -a; }
__device__ __forceinline__ float vsub(float a, float b) { return a - b; }
// one instruction: b scaled by -1 is exact
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return fma2(f2(-1.0f), b, a); }
__device__ __forceinline__ float2 vneg(float2 a) { return neg2(a); }

// The equilibrium of a site from its arguments: eq_store's arithmetic with
// omega = 1.
template <typename V>
struct EqSite {
  V tx, ty, tz, a, b, orw, obase, rest;
  __device__ __forceinline__ EqSite(float rho0, V dr, V vx, V vy, V vz) {
    auto k = [&](float v) { return vset(V(), v); };
    const V rho = vadd(k(rho0), dr);
    tx = vmul(k(3.0f), vx), ty = vmul(k(3.0f), vy), tz = vmul(k(3.0f), vz);
    const V uke = vmul(k(0.5f), vfma(tz, vz, vfma(ty, vy, vmul(tx, vx))));
    a = vneg(uke);
    b = vadd(k(1.0f), a);
    orw = vmul(rho, k(W1)), obase = vmul(dr, k(W1));
    rest = vfma(vmul(rho, k(W0)), a, vmul(dr, k(W0)));
  }
  // even and odd parts of the pair of populations along e
  __device__ __forceinline__ void pair(V e, V &ev, V &od) const {
    const V e2 = vmul(e, e);
    ev = vfma(orw, vfma(vset(V(), 0.5f), e2, a), obase);
    od = vmul(vmul(orw, e), vfma(e2, vset(V(), 1.0f / 6.0f), b));
  }
};

template <typename V, int TX, int TY, bool ROCK>
struct EqGeom {
  static constexpr bool SURF = sizeof(V) == 4;
  static constexpr int NT = TX * TY, AW = TX + 2, AN = AW * (TY + 2);
  static constexpr int NTH = (AN + 31) / 32 * 32;
  static constexpr int DS = ROCK ? 2 : 1;  // a bounced pull returns the own site's D populations
  static constexpr int PLANES = 4 * DS + 2 * 8 + 2 * 4;
  static constexpr int DIP = SURF ? 4 * AN * 16 : 0;
  // staged own entries, two slots: the arguments (red and blue: two float4),
  // for the surfactant the other launch's o1 and o2
  static constexpr int STAGE = SURF ? 2 * (NTH * 16 + NT * 20) : 2 * NTH * 32;
  static constexpr int SMEM = DIP + STAGE + PLANES * AN * (int)sizeof(V);
  // 80 registers a thread: two CTAs of 32 x 8 tiles, four of 16 x 8
  static constexpr int MINB = NTH > 192 ? 2 : 4;
};

// All threads of the CTA, from the tile's and the halo's loop alike.
template <int N>
__device__ __forceinline__ void cta_barrier() {
  asm volatile("bar.sync 1, %0;\n" ::"n"(N) : "memory");
}

template <typename V, int TX, int TY, bool ROCK, bool LE>
__global__ void __launch_bounds__(EqGeom<V, TX, TY, ROCK>::NTH, EqGeom<V, TX, TY, ROCK>::MINB)
    k_eq_moments(const LatDesc *__restrict__ lats, const Tile *__restrict__ tiles, int ntiles,
                 const uint32_t *__restrict__ mask, const __grid_constant__ EqFields X) {
  using G = EqGeom<V, TX, TY, ROCK>;
  constexpr bool SURF = G::SURF;
  constexpr int NT = G::NT, AW = G::AW, AN = G::AN, DS = G::DS, NTH = G::NTH;
  static_assert(NT % 32 == 0, "a warp holds tile sites or halo sites");
  extern __shared__ float4 sme[];
  __shared__ LatDesc sLat;
  float4 *dip = sme;                       // [4][AN] dipoles
  float4 *stA = sme + G::DIP / 16;         // [2][NTH] arguments
  float4 *stB = stA + 2 * NTH;             // [2][NTH] arguments, or [2][NT] o1
  float *stC = reinterpret_cast<float *>(stB + 2 * NT);  // surfactant: [2][NT] o2
  V *pD = reinterpret_cast<V *>(reinterpret_cast<unsigned char *>(stA) + G::STAGE);  // [DS][4][AN]
  V *pZ = pD + 4 * DS * AN;                          // [2][8][AN]
  V *pU = pZ + 16 * AN;                              // [2][4][AN]
  const size_t S = X.S;
  const int tid = threadIdx.x;
  // threads 0 .. NT - 1 own the tile's sites, the others the halo ring: its
  // bottom and top rows with the corners, then its left and right columns
  int hx, hy;
  if (tid < NT) {
    hx = tid % TX + 1, hy = tid / TX + 1;
  } else {
    const int r = tid - NT;
    if (r < 2 * AW)
      hx = r < AW ? r : r - AW, hy = r < AW ? 0 : TY + 1;
    else
      hx = r - 2 * AW < TY ? 0 : TX + 1, hy = (r - 2 * AW) % TY + 1;
  }
  const bool part = tid < AN;
  const int s = hx + AW * hy;
  // The first tile, its descriptor and offsets are set up before the previous
  // pass has finished: no pass of a loop writes them, and what did (the flip of
  // the loop before, an upload) completed before the loop's first pass, which is
  // launched plainly, could start.  A step of ternary 16^3 24.6 -> 15.2 us, 32^3 29.3 -> 19.5, 64^3 48.9 -> 39.8, 128^3
  // 214 -> 202.
  const Tile T0 = tiles[blockIdx.x];
  if (tid == 0) sLat = lats[T0.lat];
  pdl_launch_next();
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const Tile T = t == blockIdx.x ? T0 : tiles[t];
    if (tid == 0 && t != blockIdx.x) sLat = lats[T.lat];
    cta_barrier<NTH>();
    const LatDesc &Lg = sLat;
    const int nx = Lg.nx, ny = Lg.ny, nz = Lg.nz, pl = nx * ny;
    const float rho0 = Lg.rho0;
    const int x0 = T.x0, y0 = T.y0, z0 = T.z0, zc = T.zc;
    const int vx = x0 - 1 + hx, vy = y0 - 1 + hy;
    const int wy = wrapz(vy, ny), xy = wrapz(vx, nx) + nx * wy;
    const int side = !LE || !part ? -1 : vx == -1 ? 0 : vx == nx ? 1 : -1;  // a sheared halo site
    // the arguments of the plane evaluated next, copied one iteration ahead
    // (asynchronously into shared memory: held in registers, the 16-byte loads
    // were moved out of their register quads at once and their latency with
    // them); the dipoles go straight into their ring
    const float4 *qa = X.Q[Lg.parity] + (SURF ? 2 * S : 0) + Lg.base + xy, *qb = qa + S;
    int zl = wrapz(z0 - 1, nz);  // z of the plane copied next
    auto load = [&](int m) {
      const int i = pl * zl;
      cp_async16(stA + (m & 1) * NTH + tid, qa + i);
      cp_async16(SURF ? dip + (m & 3) * AN + s : stB + (m & 1) * NTH + tid, qb + i);
      zl = zl + 1 == nz ? 0 : zl + 1;
    };
    auto site = [&](int m) {
      const float4 la = stA[(m & 1) * NTH + tid];
      if constexpr (SURF) {
        return EqSite<V>(rho0, la.x, la.y, la.z, la.w);
      } else {
        const float4 lb = stB[(m & 1) * NTH + tid];
        return EqSite<V>(rho0, make_float2(la.x, la.y), make_float2(la.z, la.w), make_float2(lb.x, lb.y),
                         make_float2(lb.z, lb.w));
      }
    };
    // the populations of the stage-6 halo plane at a sheared halo site
    const unsigned NP = ny * nz;
    auto sheared = [&](int d, int z) {
      const float *h = Lg.le_h[side] + wy + ny * z;
      return make_float2(h[d * NP], h[(19 + d) * NP]);
    };
    pdl_wait_previous();  // from here on, data of earlier passes
    if (part) load(0);
    cp_async_commit();
    if (tid >= NT) {
      // ---- halo: lo, the site's side (left, bottom); its directions into the
      // tile: three in the plane, one up, one down
      const bool row = hy == 0 || hy == TY + 1, lo = row ? hy == 0 : hx == 0;
      const int hq[5] = {row ? (lo ? 2 : 3) : (lo ? 0 : 1), lo ? 6 : 11, row ? (lo ? 10 : 7) : (lo ? 7 : 10),
                         row ? (lo ? 14 : 16) : (lo ? 8 : 12), row ? (lo ? 15 : 17) : (lo ? 9 : 13)};
      int off[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        off[k] = s;
#pragma unroll
        for (int q = 0; q < 18; ++q)
          if (q != 4 && q != 5 && hq[k] == q) off[k] = dir_slot(q) * AN + s;
      }
      const V sg = vset(V(), lo ? 1.0f : -1.0f), sd = vset(V(), lo != row ? 1.0f : -1.0f);
      V up = vset(V(), 0.f);
      // a sheared halo site's populations, read one plane ahead (their latency
      // would hold up the whole CTA at the barrier)
      float2 ahead[5];
      auto read_sheared = [&](int z) {
#pragma unroll
        for (int k = 0; k < 5; ++k) ahead[k] = sheared(hq[k], z);
      };
      if constexpr (LE && !SURF)
        if (side >= 0) read_sheared(zl == 0 ? nz - 1 : zl - 1);
#pragma unroll 1
      for (int m = 0; m <= zc + 1; ++m) {
        if (part) {
          const int z = zl;  // of plane m + 1
          V *mD = pD + (m % DS) * 4 * AN, *mZ = pZ + (m & 1) * 8 * AN, *mU = pU + ((m - 1) & 1) * 4 * AN;
          if (m > 0) mU[off[3]] = up;
          cp_async_wait<0>();
          const EqSite<V> E = site(m);
          if (m <= zc) load(m + 1);
          cp_async_commit();
          const V t1 = row ? E.ty : E.tx;
          V ev, od, z0v, z1v, z2v;
          E.pair(t1, ev, od);
          z0v = vfma(sg, od, ev);
          E.pair(vadd(E.tx, E.ty), ev, od);
          z1v = vfma(sg, od, ev);
          E.pair(vsub(E.tx, E.ty), ev, od);
          z2v = vfma(sd, od, ev);
          E.pair(vadd(t1, E.tz), ev, od);
          const V A = vfma(sg, od, ev);
          E.pair(vsub(t1, E.tz), ev, od);
          const V B = vfma(sg, od, ev);
          up = lo ? A : B;
          V down = lo ? B : A;
          if constexpr (LE && !SURF)
            if (side >= 0) {
              z0v = ahead[0], z1v = ahead[1], z2v = ahead[2], up = ahead[3], down = ahead[4];
              if (m <= zc) read_sheared(z);
            }
          mZ[off[0]] = z0v;
          mZ[off[1]] = z1v;
          mZ[off[2]] = z2v;
          mD[off[4]] = down;
        }
        if (m < 2) continue;
        cta_barrier<NTH>();
        cta_barrier<NTH>();
      }
      continue;
    }
    // ---- tile.  Waiting: U of the last plane; those along z (4: last two
    // planes, 5: last plane and, for a bounce, the one before); at rest
    const bool act = vx < nx && vy < ny;
    V ur[4], u4 = vset(V(), 0.f), u4p = u4, d5 = u4, d5p = u4, rest = u4;
    ur[0] = ur[1] = ur[2] = ur[3] = u4;
    int zo = z0 == 0 ? nz - 1 : z0 - 1;  // z of the plane before the one summed next
    const size_t own = (size_t)Lg.base + xy;
    uint32_t mk = 0, mkn = 0;  // rock mask of the plane summed, summed next
    auto iterate = [&](auto parity, int m) {
      constexpr int P = decltype(parity)::value;  // m & 1
      const V rest1 = rest, u4q = u4p;            // plane m - 1, plane m - 2
      V *mD = pD + (DS == 2 ? P * 4 * AN : 0) + s, *mZ = pZ + P * 8 * AN + s, *mU = pU + (1 - P) * 4 * AN + s;
      const float4 *dm = dip + (m & 2) * AN + s, *dx = dip + (2 - (m & 2)) * AN + s;  // dipole slots of this pair, the last
      if (m > 0)
#pragma unroll
        for (int k = 0; k < 4; ++k) mU[k * AN] = ur[k];
      u4p = u4, d5p = d5;
      {
        cp_async_wait<0>();
        const EqSite<V> E = site(m);
        rest = E.rest;
        const int z = zl == 0 ? nz - 1 : zl - 1;  // of plane m
        if (m <= zc) load(m + 1);
        mk = mkn;
        if ((ROCK || SURF) && m >= 1 && m <= zc) {
          // of plane m, summed in the next iteration
          const int i = pl * z;
          if (ROCK) mkn = __ldg(mask + own + i);
          if (SURF && act) {
            cp_async16(stB + P * NT + tid, X.o1 + own + i);
            cp_async4(stC + P * NT + tid, X.o2 + own + i);
          }
        }
        cp_async_commit();
        V ev, od;
        auto put = [&](int d, V v) {
          if (d == 4) u4 = v;
          else if (d == 5) d5 = v;
          else if (cz(d) == 1) ur[dir_slot(d) % 4] = v;
          else (cz(d) ? mD : mZ)[dir_slot(d) * AN] = v;
        };
#define LB3D_EQP(E_, I, J)  \
  E.pair(E_, ev, od);       \
  put(I, vadd(ev, od));     \
  put(J, vsub(ev, od));
        LB3D_EQP(E.tx, 0, 1)
        LB3D_EQP(E.ty, 2, 3)
        LB3D_EQP(E.tz, 4, 5)
        LB3D_EQP(vadd(E.tx, E.ty), 6, 11)
        LB3D_EQP(vsub(E.tx, E.ty), 7, 10)
        LB3D_EQP(vadd(E.tx, E.tz), 8, 13)
        LB3D_EQP(vsub(E.tx, E.tz), 9, 12)
        LB3D_EQP(vadd(E.ty, E.tz), 14, 17)
        LB3D_EQP(vsub(E.ty, E.tz), 15, 16)
#undef LB3D_EQP
        if constexpr (LE && !SURF) {
          if (side >= 0) {  // x = nx lies inside the tile's span
            put(1, sheared(1, z)), put(10, sheared(10, z)), put(11, sheared(11, z));
            put(12, sheared(12, z)), put(13, sheared(13, z));
          }
        }
      }
      if (m < 2) return;
      zo = zo + 1 == nz ? 0 : zo + 1;  // z of plane m - 1
      cta_barrier<NTH>();
      if (act) {
        // the pulled populations of plane m - 1: U of plane m - 2, Z of plane
        // m - 1, D of plane m; the own site's (plane m - 1) for a bounce
        const size_t self = own + pl * zo;
        const bool fluid = !ROCK || !(mk >> 18 & 1u);
        auto plane = [&](int d, bool own_site) {
          if (cz(d) == 0) return pZ + ((1 - P) * 8 + dir_slot(d)) * AN + s;
          if (cz(d) == 1) return pU + ((own_site ? 1 - P : P) * 4 + dir_slot(d)) * AN + s;
          return pD + ((DS == 1 ? 0 : own_site ? 1 - P : P) * 4 + dir_slot(d)) * AN + s;
        };
        V r = vset(V(), 0.f), j0 = r, j1 = r, j2 = r;
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        // edge: the tile holds sites on the sheared boundary, which also leave
        // their populations for the stage-8 halo kernel (a rock site those it
        // keeps)
        auto sum = [&](auto edge) {
          float *lbp = nullptr;
          if (decltype(edge)::value && (vx == 0 || vx == nx - 1)) lbp = Lg.le_b[vx == 0 ? 3 : 2] + vy + ny * zo;
#pragma unroll
          for (int d = 0; d < 19; ++d) {
            V v;
            const bool hit = ROCK && d < 18 && (mk >> d & 1u);
            if (d == 18) {
              v = rest1;
            } else if (d == 4) {
              v = hit ? d5p : u4q;
            } else if (d == 5) {
              v = hit ? u4p : d5;
            } else {
              const V *p = plane(d, false) - cx(d) - AW * cy(d);
              if (hit) p = plane(bounce(d), true);
              v = *p;
            }
            if constexpr (decltype(edge)::value) {
              if (lbp) {
                lbp[d * NP] = fluid ? vlane(v, 0) : rock_dev(d, rho0);
                lbp[(19 + d) * NP] = fluid ? vlane(v, 1) : rock_dev(d, rho0);
              }
            }
            const float g = (float)gw(d);
            r = vfma(vset(V(), g), v, r);
            if (cx(d)) j0 = vfma(vset(V(), g * (float)cx(d)), v, j0);
            if (cy(d)) j1 = vfma(vset(V(), g * (float)cy(d)), v, j1);
            if (cz(d)) j2 = vfma(vset(V(), g * (float)cz(d)), v, j2);
            if constexpr (SURF) {
              // da = sum_q (n_s(x - c_q, q) g_q) db(x - c_q) + n_s(x, rest) db(x)
              // planes m - 2, m - 1, m
              const float4 *p = cz(d) == 1 ? dx + P * AN : cz(d) == 0 ? (P ? dm : dx + AN) : dm + P * AN;
              const float4 bb = p[-cx(d) - AW * cy(d)];
              const float ng = g * fmaf(wq(d), rho0, v);
              a0 = fmaf(ng, bb.x, a0);
              a1 = fmaf(ng, bb.y, a1);
              a2 = fmaf(ng, bb.z, a2);
            }
          }
        };
        if constexpr (LE && !SURF) {
          if (x0 == 0 || x0 + TX >= nx)
            sum(std::true_type());
          else
            sum(std::false_type());
        } else {
          sum(std::false_type());
        }
        if constexpr (SURF) {
          const float am = Lg.amass[2] * Lg.omega[2];
          const float4 o1 = stB[(1 - P) * NT + tid];
          const float o2 = stC[(1 - P) * NT + tid];
          X.o3[self] = make_float4(r, fmaf(am, j0, o1.z), fmaf(am, j1, o1.w), fmaf(am, j2, o2));
          X.M[self] = make_float4(o1.y - o1.x, a0, a1, a2);
        } else if (fluid) {
          put_rb(X, self, Lg, r, j0, j1, j2);
        }
      }
      cta_barrier<NTH>();  // the next iteration overwrites the planes read here
    };
#pragma unroll 1
    for (int m = 0; m <= zc + 1; m += 2) {
      iterate(std::integral_constant<int, 0>(), m);
      if (m + 1 <= zc + 1) iterate(std::integral_constant<int, 1>(), m + 1);
    }
  }
}

// ---------------------------------------------------------------------------
// Dipole pass (ternary): the {rho_b - rho_r, da} entries stream through a
// five-slot ring, refilled with cp.async three planes ahead of the plane
// being relaxed (one barrier per plane); dipole_site's arithmetic.
// ---------------------------------------------------------------------------
template <int TX, int TY>
__global__ void __launch_bounds__(TX *TY, 1024 / (TX * TY))
    k_eq_dipole(const LatDesc *__restrict__ lats, const Tile *__restrict__ tiles, int ntiles, float *db0,
                float *db1, const __grid_constant__ EqFields X, int last) {
  constexpr int NT = TX * TY, AW = TX + 2, AN = AW * (TY + 2), RS = 5, RE = (AN + NT - 1) / NT;
  extern __shared__ float4 sme[];  // [RS][AN]
  __shared__ LatDesc sLat;
  const unsigned S = X.S;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  // the first tile early, as in the moments pass
  const Tile T0 = tiles[blockIdx.x];
  if (tid == 0) sLat = lats[T0.lat];
  pdl_launch_next();
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const Tile T = t == blockIdx.x ? T0 : tiles[t];
    if (tid == 0 && t != blockIdx.x) sLat = lats[T.lat];
    __syncthreads();
    const LatDesc &Lg = sLat;
    const int nx = Lg.nx, ny = Lg.ny, nz = Lg.nz, pl = nx * ny;
    float *DBo = (Lg.parity ? db0 : db1) + Lg.base;
    float4 *Qd = X.Q[Lg.parity] + 3 * (size_t)S + Lg.base;
    const float4 *Mb = X.M + Lg.base;
    float4 *DD = X.M + (size_t)S + Lg.base;
    const float4 *O3 = X.o3 + Lg.base;
    const int x0 = T.x0, y0 = T.y0, z0 = T.z0, zc = T.zc;
    const int gx = x0 + tx, gy = y0 + ty;
    const bool act = gx < nx && gy < ny;
    int rxy[RE];  // the in-plane offsets of this thread's ring entries
#pragma unroll
    for (int e = 0; e < RE; ++e) {
      const int s = tid + e * NT;
      rxy[e] = s < AN ? wrapz(x0 - 1 + s % AW, nx) + nx * wrapz(y0 - 1 + s / AW, ny) : 0;
    }
    const int own_xy = gx + nx * gy;
    auto load_ring = [&](int r) {  // plane z0 - 1 + r in slot r % RS
      const float4 *plane = Mb + pl * wrapz(z0 - 1 + r, nz);
      float4 *slot = sme + (r % RS) * AN;
#pragma unroll
      for (int e = 0; e < RE; ++e)
        if (tid + e * NT < AN) cp_async16(slot + tid + e * NT, plane + rxy[e]);
    };
    pdl_wait_previous();  // from here on, data of earlier passes
    load_ring(0);
    load_ring(1);
    load_ring(2);
    cp_async_commit();
    float drs = act ? O3[own_xy + pl * z0].x : 0.f;
    for (int k = 0; k < zc; ++k) {
      if (k + 3 <= zc + 1) load_ring(k + 3);
      cp_async_commit();
      const float own = drs;
      if (act && k + 1 < zc) drs = O3[own_xy + pl * wrapz(z0 + k + 1, nz)].x;
      cp_async_wait<1>();  // ring planes up to k + 2 landed (this thread's copies)
      __syncthreads();     // ... and everybody's
      if (act) {
        const int as = (tx + 1) + AW * (ty + 1);
        const float3 d = dipole_site<AW>((const float4 *)sme + (k % RS) * AN, (const float4 *)sme + ((k + 1) % RS) * AN,
                                         (const float4 *)sme + ((k + 2) % RS) * AN, as, Lg, Lg.rho0, own);
        const int i = own_xy + pl * wrapz(z0 + k, nz);
        Qd[i] = make_float4(d.x, d.y, d.z, 0.f);
        if (last) {
          DBo[i] = d.x;
          DBo[(size_t)S + i] = d.y;
          DBo[2 * (size_t)S + i] = d.z;
        }
        const float pse = -Lg.em0 * expm1f(-own);
        const float ps = Lg.psi0 + pse;
        const float2 a01 = mul2(make_float2(d.x, d.y), f2(ps));
        DD[i] = make_float4(a01.x, a01.y, d.z * ps, pse);
      }
    }
    cp_async_wait<0>();
    __syncthreads();  // the next tile refills ring slots 0..2
  }
}

// ---------------------------------------------------------------------------
// Collide pass: psi deviations and (ternary) {a, dpsi_s} entries stream
// through five-slot rings as in the dipole pass, and the own entries with
// them (prefetched in registers the 16-byte ones exposed their latency: 78
// against 70 us at ternary 128^3).  to_pops: write the populations (the last
// step of a loop) instead of the equilibrium's arguments, EQ_POPS_AFTER_ARGS
// where earlier steps of the loop wrote those.  Ternary 128^3: 70
// us at 16 warps per SM and 62 % issue (the pass that wrote populations every
// step: 154 us); binary 256x128x128: 66 us (172 us).
// ---------------------------------------------------------------------------
// force_ternary with the neighbours' a = d (psi0 + dpsi_s) from the dipole
// pass: the same operations in the same order.
template <int W>
__device__ __forceinline__ void force_ternary_pre(const float2 *Pm, const float2 *P0, const float2 *Pp,
                                                  const float4 *Am, const float4 *A0, const float4 *Ap,
                                                  int ap, float3 dd, const LatDesc &Lg, float psi0,
                                                  float Fx[3][3]) {
  // FB[k] = (f_br, f_rb)_k, SA01 = (SA_x, SA_y), M01[k] = (M_xk, M_yk),
  // TQ[K] = (T_K, Q_K)
  float2 FB[3] = {f2(0.f), f2(0.f), f2(0.f)}, M01[3] = {f2(0.f), f2(0.f), f2(0.f)};
  float2 TQ[6] = {f2(0.f), f2(0.f), f2(0.f), f2(0.f), f2(0.f), f2(0.f)};
  float2 SA01 = f2(0.f);
  float SA2 = 0.f, V[3] = {0, 0, 0}, M2[3] = {0, 0, 0}, SG = 0.f;
#pragma unroll
  for (int q = 0; q < 18; ++q) {
    const float2 *Pq = cz(q) == 1 ? Pp : (cz(q) == -1 ? Pm : P0);
    const float4 *Aq = cz(q) == 1 ? Ap : (cz(q) == -1 ? Am : A0);
    const float g = (float)gw(q);
    const int c[3] = {cx(q), cy(q), cz(q)};
    const float2 e = Pq[ap + cx(q) + W * cy(q)];
    const float4 av = Aq[ap + cx(q) + W * cy(q)];
    const float2 a01 = make_float2(av.x, av.y);
    const float a2 = av.z;
    const float a[3] = {a01.x, a01.y, a2};
    float ac = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (c[k]) ac = fmaf((float)c[k], a[k], ac);
    const float Gq = g * (e.y - e.x);
    const float g8 = 8.0f * g;
    SG += Gq;
    SA01 = fma2(f2(g), a01, SA01);
    SA2 = fmaf(g, a2, SA2);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (c[k]) {
        FB[k] = fma2(f2(g * (float)c[k]), e, FB[k]);
        V[k] = fmaf(g * (float)c[k], ac, V[k]);
        M01[k] = fma2(f2(g8 * (float)c[k]), a01, M01[k]);
        M2[k] = fmaf(g8 * (float)c[k], a2, M2[k]);
      }
    }
    const float2 gq = make_float2(Gq, g8 * ac);
#define LB3D_SYM(I, J, K)                                  \
  if (c[I] && c[J]) TQ[K] = fma2(gq, f2((float)(c[I] * c[J])), TQ[K]);
    LB3D_SYM(0, 0, 0) LB3D_SYM(1, 1, 1) LB3D_SYM(2, 2, 2)
    LB3D_SYM(0, 1, 3) LB3D_SYM(0, 2, 4) LB3D_SYM(1, 2, 5)
#undef LB3D_SYM
  }
  const float frb[3] = {FB[0].y, FB[1].y, FB[2].y}, fbr[3] = {FB[0].x, FB[1].x, FB[2].x};
  const float SA[3] = {SA01.x, SA01.y, SA2};
  const float T[6] = {TQ[0].x, TQ[1].x, TQ[2].x, TQ[3].x, TQ[4].x, TQ[5].x};
  const float Q[6] = {TQ[0].y, TQ[1].y, TQ[2].y, TQ[3].y, TQ[4].y, TQ[5].y};
  const float M[3][3] = {{M01[0].x, M01[1].x, M01[2].x}, {M01[0].y, M01[1].y, M01[2].y},
                         {M2[0], M2[1], M2[2]}};
  const float d[3] = {dd.x, dd.y, dd.z};
  const float2 own = P0[ap];
  const float psr = psi0 + own.x, psb = psi0 + own.y, pss = psi0 + A0[ap].w;
  auto dot3 = [&](float a0, float a1, float a2) { return fmaf(a2, d[2], fmaf(a1, d[1], a0 * d[0])); };
  const float Td[3] = {dot3(T[0], T[3], T[4]), dot3(T[3], T[1], T[5]), dot3(T[4], T[5], T[2])};
  const float Qd[3] = {dot3(Q[0], Q[3], Q[4]), dot3(Q[3], Q[1], Q[5]), dot3(Q[4], Q[5], Q[2])};
  const float trM = M[0][0] + M[1][1] + M[2][2];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float MTd = dot3(M[0][k], M[1][k], M[2][k]);
    const float Md = dot3(M[k][0], M[k][1], M[k][2]);
    const float fcs = fmaf(-2.0f, V[k], SA[k]);
    const float fsc = fmaf(SG, d[k], -2.0f * Td[k]);
    const float fss = fmaf(-2.0f, Qd[k], fmaf(trM, d[k], MTd + Md));
    const float cs = (-2.0f * Lg.g_bs) * fcs;
    Fx[1][k] = fmaf(-Lg.g_br, fbr[k], cs) * psb;
    Fx[0][k] = fmaf(-Lg.g_br, frb[k], -cs) * psr;
    Fx[2][k] = fmaf(2.0f * Lg.g_bs, fsc, -Lg.g_ss * fss) * pss;
  }
}

// force_binary (fp32_stencil.cuh) with the neighbours' rock flags as a mask
// (bit q: the upstream site x - c_q is rock, so the neighbour x + c_q is bit
// bounce(q)) and psi = 0 already in the rock sites' entries; red and blue on
// paired lanes, the same roundings (the weights are powers of two).
template <int W, bool ROCK, bool LE>
__device__ __forceinline__ void force_binary_masked(const float2 *Pm, const float2 *P0, const float2 *Pp, int as,
                                                    uint32_t mk, const LatDesc &Lg, float psi0, float Fx[2][3],
                                                    int gy, int gz) {
  float2 FB[3] = {f2(0.f), f2(0.f), f2(0.f)};  // (f_br, f_rb)_k
#pragma unroll
  for (int q = 0; q < 18; ++q) {
    const float2 *Pq = cz(q) == 1 ? Pp : (cz(q) == -1 ? Pm : P0);
    const float2 e = Pq[as + cx(q) + W * cy(q)];
    const int c[3] = {cx(q), cy(q), cz(q)};
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (c[k]) FB[k] = fma2(f2((float)(gw(q) * c[k])), e, FB[k]);
  }
  float fwr[3] = {0, 0, 0}, fwb[3] = {0, 0, 0};
  if (ROCK && (mk & 0x3ffffu)) {
#pragma unroll
    for (int q = 0; q < 18; ++q) {
      bool wall = mk >> bounce(q) & 1u;
      if (LE && wall)
        wall = !(gy + cy(q) < 0 || gy + cy(q) >= Lg.ny || gz + cz(q) < 0 || gz + cz(q) >= Lg.nz);
      const int c[3] = {cx(q), cy(q), cz(q)};
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (c[k] && wall) {
          fwb[k] = fmaf(Lg.psiw_b * (float)gw(q), (float)c[k], fwb[k]);
          fwr[k] = fmaf(Lg.psiw_r * (float)gw(q), (float)c[k], fwr[k]);
        }
    }
  }
  const float2 own = P0[as];
  const float psr = psi0 + own.x, psb = psi0 + own.y;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    Fx[1][k] = fmaf(-Lg.g_br, FB[k].x, Lg.wall_b * fwb[k]) * psb;
    Fx[0][k] = fmaf(-Lg.g_br, FB[k].y, Lg.wall_r * fwr[k]) * psr;
  }
}

constexpr int EQ_POPS = 1, EQ_POPS_AFTER_ARGS = 2;

template <int NC, int TX, int TY>
struct EqCollideGeom {
  static constexpr int NT = TX * TY, AW = TX + 2, AN = AW * (TY + 2), RS = 5;
  // rings of {a, dpsi_s} (ternary) and psi; the own entries: ternary
  // {drho_s, P}, the dipole and {drho_r, drho_b}, binary o1 and o2
  static constexpr int SMEM = RS * (AN * (NC == 3 ? 24 : 8) + NT * (NC == 3 ? 40 : 20));
  static constexpr int MINB = NC == 3 ? 512 / NT : 768 / NT;
};

template <int NC, int TX, int TY, bool ROCK, bool LE>
__global__ void __launch_bounds__(TX *TY, EqCollideGeom<NC, TX, TY>::MINB)
    k_eq_collide(const LatDesc *__restrict__ lats, const Tile *__restrict__ tiles, int ntiles, float *f0, float *f1,
                 const uint32_t *__restrict__ mask, const __grid_constant__ EqFields X, int to_pops) {
  using G = EqCollideGeom<NC, TX, TY>;
  constexpr int NT = G::NT, AW = G::AW, AN = G::AN, RS = G::RS, RE = (AN + NT - 1) / NT;
  extern __shared__ float4 sme[];
  float4 *ringA = sme;                                                  // [RS][AN] (ternary)
  float4 *own1 = sme + (NC == 3 ? RS * AN : 0), *own2 = own1 + (NC == 3 ? RS * NT : 0);  // [RS][NT] each
  float2 *ringP = reinterpret_cast<float2 *>(own2 + RS * NT);                           // [RS][AN]
  float2 *own3 = ringP + RS * AN;                                                       // [RS][NT]
  __shared__ LatDesc sLat;
  const unsigned S = X.S;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  // the first tile early, as in the moments pass
  const Tile T0 = tiles[blockIdx.x];
  if (tid == 0) sLat = lats[T0.lat];
  pdl_launch_next();
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const Tile T = t == blockIdx.x ? T0 : tiles[t];
    if (tid == 0 && t != blockIdx.x) sLat = lats[T.lat];
    __syncthreads();
    const LatDesc &Lg = sLat;
    const int nx = Lg.nx, ny = Lg.ny, nz = Lg.nz, pl = nx * ny;
    const int par = Lg.parity;
    const size_t base = (size_t)Lg.base;
    const float psi0 = Lg.psi0;
    const float2 *PS = X.psi + base;
    const float4 *DD = NC == 3 ? X.M + (size_t)S + base : nullptr;
    const float4 *O1 = X.o1 + base, *O3 = X.o3 + base;
    const float *O2 = X.o2 + base;
    float4 *Q = X.Q[par] + base;
    const int x0 = T.x0, y0 = T.y0, z0 = T.z0, zc = T.zc;
    const int gx = x0 + tx, gy = y0 + ty;
    const bool act = gx < nx && gy < ny;
    // the in-plane offsets of this thread's ring entries; the psi entries of
    // sheared halo columns come from the stage-8 halo planes
    int rxy[RE];
    const float2 *rps[RE];
    int rpl[RE];
#pragma unroll
    for (int e = 0; e < RE; ++e) {
      const int s = tid + e * NT;
      const int ry = wrapz(y0 - 1 + s / AW, ny);
      rxy[e] = s < AN ? wrapz(x0 - 1 + s % AW, nx) + nx * ry : 0;
      rps[e] = PS + rxy[e];
      rpl[e] = pl;
      const int vx = x0 - 1 + s % AW;
      if (LE && s < AN && (vx == -1 || vx == nx)) rps[e] = Lg.le_p[vx < 0 ? 0 : 1] + ry, rpl[e] = ny;
    }
    const int own_xy = gx + nx * gy;
    auto load_ring = [&](int r) {  // plane z0 - 1 + r in slot r % RS
      const int gz = wrapz(z0 - 1 + r, nz), sl = (r % RS) * AN;
#pragma unroll
      for (int e = 0; e < RE; ++e) {
        const int s = tid + e * NT;
        if (s >= AN) break;
        if (NC == 3) cp_async16(ringA + sl + s, DD + rxy[e] + pl * gz);
        cp_async8(ringP + sl + s, rps[e] + (LE ? rpl[e] : pl) * gz);
      }
      if (act) {
        const int i = own_xy + pl * gz, o = (r % RS) * NT + tid;
        if (NC == 3) {
          cp_async16(own1 + o, O3 + i);
          cp_async16(own2 + o, Q + 3 * (size_t)S + i);
          cp_async8(own3 + o, O1 + i);
        } else {
          cp_async16(own1 + o, O1 + i);
          cp_async4(reinterpret_cast<float *>(own3) + o, O2 + i);
        }
      }
    };
    pdl_wait_previous();  // from here on, data of earlier passes
    load_ring(0);
    load_ring(1);
    load_ring(2);
    cp_async_commit();
    uint32_t mkn = 0;  // rock mask of the plane collided next
    if (ROCK && act) mkn = __ldg(mask + base + own_xy + pl * z0);
    for (int k = 0; k < zc; ++k) {
      if (k + 3 <= zc + 1) load_ring(k + 3);
      cp_async_commit();
      const uint32_t mk = mkn;
      if (ROCK && act && k + 1 < zc) mkn = __ldg(mask + base + own_xy + pl * wrapz(z0 + k + 1, nz));
      cp_async_wait<1>();  // ring planes up to k + 2 landed (this thread's copies)
      __syncthreads();     // ... and everybody's
      if (!act) continue;
      const int gz = wrapz(z0 + k, nz);
      const int self = own_xy + pl * gz;
      if (ROCK && (mk >> 18 & 1u)) {
        // a rock site's populations stay zero; the arguments between a loop's
        // steps were laid over the first 8 planes of the buffer it read (all 38
        // planes of both buffers rewritten in every loop: a one-step loop of the
        // porous 128^3 lattice 430 us, this way 208)
        if (to_pops == EQ_POPS_AFTER_ARGS) {
          float *fi = (par ? f1 : f0) + base + self;
#pragma unroll
          for (int q = 0; q < 8; ++q) fi[(size_t)q * S] = rock_dev(q, Lg.rho0);
        }
        continue;
      }
      const int as = (tx + 1) + AW * (ty + 1), o = ((k + 1) % RS) * NT + tid;
      float Fx[NC][3];
      const float2 *Pm = ringP + (k % RS) * AN, *P0 = ringP + ((k + 1) % RS) * AN, *Pp = ringP + ((k + 2) % RS) * AN;
      float4 pp = own1[o];  // drho_s (ternary), P
      float2 drb;
      float3 dd = make_float3(0.f, 0.f, 0.f);
      if (NC == 3) {
        const float4 d = own2[o];
        dd = make_float3(d.x, d.y, d.z);
        drb = own3[o];
      } else {
        drb = make_float2(pp.x, pp.y);
        pp = make_float4(0.f, pp.z, pp.w, reinterpret_cast<const float *>(own3)[o]);
      }
      if constexpr (NC == 3)
        force_ternary_pre<AW>(Pm, P0, Pp, ringA + (k % RS) * AN, ringA + ((k + 1) % RS) * AN,
                              ringA + ((k + 2) % RS) * AN, as, dd, Lg, psi0, reinterpret_cast<float(*)[3]>(Fx));
      else
        force_binary_masked<AW, ROCK, LE>(Pm, P0, Pp, as, mk, Lg, psi0, reinterpret_cast<float(*)[3]>(Fx), gy, gz);
      float dr[NC], rho[NC];
      dr[0] = drb.x, dr[1] = drb.y;
      if (NC == 3) dr[NC - 1] = pp.x;
#pragma unroll
      for (int c = 0; c < NC; ++c) rho[c] = Lg.rho0 + dr[c];
      if (Lg.flags & LAT_BODY) {
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
      float rt = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) rt = fmaf(Lg.amass[c] * Lg.omega[c], rho[c], rt);
      const float irt = 1.0f / fmaxf(rt, 1.0e-8f);
      const float u0 = pp.y * irt, u1 = pp.z * irt, u2 = pp.w * irt;
      float vx[NC], vy[NC], vz[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const float kf = Lg.tau[c] / (Lg.amass[c] * fmaxf(rho[c], 1.0e-8f));
        vx[c] = fmaf(kf, Fx[c][0], u0);
        vy[c] = fmaf(kf, Fx[c][1], u1);
        vz[c] = fmaf(kf, Fx[c][2], u2);
      }
      const float2 rho2 = make_float2(rho[0], rho[1]), dr2 = make_float2(dr[0], dr[1]), one = f2(1.0f);
      const float2 vx2 = make_float2(vx[0], vx[1]), vy2 = make_float2(vy[0], vy[1]), vz2 = make_float2(vz[0], vz[1]);
      if (LE && (gx == 0 || gx == nx - 1)) {
        // the next step's pre-stream boundary plane of its stage-6 halo kernel
        const unsigned NP = ny * nz;
        float *b = Lg.le_b[gx == nx - 1 ? 0 : 1] + gy + ny * gz;
        eq_store2(b, b + 19 * NP, NP, rho2, dr2, vx2, vy2, vz2, one);
      }
      if (to_pops) {
        float *fo = (par ? f0 : f1) + base + self;
        eq_store2(fo, fo + (size_t)19 * S, S, rho2, dr2, vx2, vy2, vz2, one);
        if (NC == 3)
          eq_store(fo + (size_t)38 * S, S, rho[NC - 1], dr[NC - 1], vx[NC - 1], vy[NC - 1], vz[NC - 1], 1.0f);
      } else {
        Q[self] = make_float4(dr2.x, dr2.y, vx2.x, vx2.y);
        Q[S + self] = make_float4(vy2.x, vy2.y, vz2.x, vz2.y);
        if (NC == 3) Q[2 * (size_t)S + self] = make_float4(dr[NC - 1], vx[NC - 1], vy[NC - 1], vz[NC - 1]);
      }
    }
    cp_async_wait<0>();
    __syncthreads();  // sLat and ring slots 0..2 are reused by the next tile
  }
}

// Bit q (q < 18) of a site's mask: its upstream site x - c_q is rock; bit 18:
// the site itself is.  Under Lees-Edwards a site across the sheared boundary
// is never rock (code/lb3d_bc_leesedwards.F90:678,866).  Rock sites also get
// their psi entry, the deviation of psi = 0.
__global__ void k_eq_mask(int nx, int ny, int nz, int le, const uint8_t *__restrict__ rock, uint32_t *mask,
                          float2 *psi, float psi0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nx * ny * nz) return;
  const int x = i % nx, y = i / nx % ny, z = i / (nx * ny);
  uint32_t m = 0;
  for (int q = 0; q < 18; ++q) {
    const int ux = x - cx(q);
    if (le && (ux < 0 || ux >= nx)) continue;
    if (rock[wrap(ux, nx) + nx * (wrap(y - cy(q), ny) + ny * wrap(z - cz(q), nz))]) m |= 1u << q;
  }
  if (rock[i]) {
    m |= 1u << 18;
    psi[i] = make_float2(-psi0, -psi0);
  }
  mask[i] = m;
}

}  // namespace f32

using namespace f32;

// ---------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------
// Tile of the moments passes: 32 x 8, or 16 x 8 where that pads the lattice's
// x side less.  At equal padding the wider tile is 3 % faster (ternary 128^3,
// a step: 0.213 against 0.220 ms; binary 256x128x128: 0.162 against 0.164):
// its halo is 0.33 of the tile's sites, the narrower one's 0.41.  Sheared
// lattices: 16 x 8, whose variant does not spill.
void eq_moments_tile(int nx, bool le, int *tx, int *ty) {
  *tx = le || 1.03 * ((nx + 15) / 16 * 16) < (double)((nx + 31) / 32 * 32) ? 16 : 32;
  *ty = 8;
}

template <int NC, bool ROCK, bool LE, int TX, int TY>
static bool eq_moments_fn(int pass, bool first, bool narrow, EqKernel *k) {
  if (first) {
    if (pass == EQ_SURFACTANT) return false;
    k->fn = narrow ? (const void *)k_eq_moments0<NC, TX, TY, ROCK, true, LE>
                   : (const void *)k_eq_moments0<NC, TX, TY, ROCK, false, LE>;
    k->threads = TX * TY;
    k->smem = NC == 3 ? 4 * (TX + 2) * (TY + 2) * 16 : 0;
  } else if (pass == EQ_MOMENTS) {
    k->fn = (const void *)k_eq_moments<float2, TX, TY, ROCK, LE>;
    k->threads = EqGeom<float2, TX, TY, ROCK>::NTH;
    k->smem = EqGeom<float2, TX, TY, ROCK>::SMEM;
  } else {
    k->fn = (const void *)k_eq_moments<float, TX, TY, false, false>;
    k->threads = EqGeom<float, TX, TY, false>::NTH;
    k->smem = EqGeom<float, TX, TY, false>::SMEM;
  }
  return true;
}

template <int NC, bool ROCK, bool LE>
static bool eq_fn(int pass, bool first, int tx, int ty, bool narrow, EqKernel *k) {
  if (pass == EQ_MOMENTS || pass == EQ_SURFACTANT) {
    if (ty != 8 || (tx != 16 && (LE || tx != 32)) || (pass == EQ_SURFACTANT && NC != 3)) return false;
    if constexpr (!LE)
      if (tx == 32) return eq_moments_fn<NC, ROCK, LE, 32, 8>(pass, first, narrow, k);
    return eq_moments_fn<NC, ROCK, LE, 16, 8>(pass, first, narrow, k);
  }
#define LB3D_EQ_SHAPE(TX, TY)                                            \
  if (tx == TX && ty == TY) {                                            \
    k->threads = TX * TY;                                                \
    if (pass == EQ_DIPOLE) {                                             \
      if (NC != 3) return false;                                         \
      k->fn = (const void *)k_eq_dipole<TX, TY>;                         \
      k->smem = (size_t)5 * (TX + 2) * (TY + 2) * 16;                    \
    } else {                                                             \
      k->fn = (const void *)k_eq_collide<NC, TX, TY, ROCK, LE>;          \
      k->smem = EqCollideGeom<NC, TX, TY>::SMEM;                         \
    }                                                                    \
    return true;                                                         \
  }
  LB3D_EQ_SHAPE(32, 8) LB3D_EQ_SHAPE(32, 4) LB3D_EQ_SHAPE(16, 16) LB3D_EQ_SHAPE(16, 8) LB3D_EQ_SHAPE(64, 4)
#undef LB3D_EQ_SHAPE
  return false;
}

bool eq_kernel(int pass, bool first, int nc, bool rock, bool le, int tx, int ty, bool narrow, EqKernel *k) {
  k->fn = nullptr;
  if (nc == 3) return !rock && !le && eq_fn<3, false, false>(pass, first, tx, ty, narrow, k);
  if (rock) return le ? eq_fn<2, true, true>(pass, first, tx, ty, narrow, k)
                      : eq_fn<2, true, false>(pass, first, tx, ty, narrow, k);
  return le ? eq_fn<2, false, true>(pass, first, tx, ty, narrow, k)
            : eq_fn<2, false, false>(pass, first, tx, ty, narrow, k);
}

cudaError_t eq_launch(const EqKernel &k, int pass, bool first, bool last, const EqArgs &a, bool pdl, cudaStream_t st) {
  if (a.ntiles <= 0) return cudaSuccess;  // every CTA reads a tile
  int resident = 0;
  cudaError_t e = fp32_prepare_kernel(k.fn, k.threads, k.smem, &resident);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min(a.ntiles, resident));
  cfg.blockDim = dim3((unsigned)k.threads);
  cfg.dynamicSmemBytes = k.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  int l = last ? (first ? EQ_POPS : EQ_POPS_AFTER_ARGS) : 0;
  void *p00[] = {(void *)&a.lats, (void *)&a.tiles, (void *)&a.ntiles, (void *)&a.f0, (void *)&a.f1,
                 (void *)&a.db0, (void *)&a.db1, (void *)&a.rock, (void *)&a.X};
  void *p0[] = {(void *)&a.lats, (void *)&a.tiles, (void *)&a.ntiles, (void *)&a.mask, (void *)&a.X};
  void *p1[] = {(void *)&a.lats, (void *)&a.tiles, (void *)&a.ntiles, (void *)&a.db0, (void *)&a.db1, (void *)&a.X,
                (void *)&l};
  void *p2[] = {(void *)&a.lats, (void *)&a.tiles, (void *)&a.ntiles, (void *)&a.f0, (void *)&a.f1,
                (void *)&a.mask, (void *)&a.X, (void *)&l};
  return cudaLaunchKernelExC(&cfg, k.fn,
                             pass == EQ_DIPOLE ? p1 : pass == EQ_COLLIDE ? p2 : first ? p00 : p0);
}

cudaError_t eq_build_mask(int nx, int ny, int nz, bool le, const uint8_t *rock, uint32_t *mask, float2 *psi,
                          float psi0, cudaStream_t st) {
  const long long n = (long long)nx * ny * nz;
  k_eq_mask<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(nx, ny, nz, le ? 1 : 0, rock, mask, psi, psi0);
  return cudaGetLastError();
}

}  // namespace lb3d
