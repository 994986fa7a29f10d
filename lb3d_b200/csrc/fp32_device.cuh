// fp32_device.cuh -- per-site device code shared by the FP32 kernels of
// fp32_path.cu (the strategies that carry populations from step to step) and
// fp32_eqstate.cu (the strategy that carries the equilibrium's arguments):
// weights, the BGK update, own moments, pulls, the Lees-Edwards pulls and
// asynchronous copies, and the stencils of fp32_stencil.cuh.
#ifndef LB3D_FP32_DEVICE_CUH
#define LB3D_FP32_DEVICE_CUH

#include "fp32_path.h"

namespace lb3d {
namespace f32 {

constexpr float W1 = 1.0f / 36.0f;
constexpr float W0 = 1.0f / 3.0f;
LB3D_HDI constexpr float wq(int q) { return q == 18 ? W0 : W1; }

__device__ __forceinline__ int pmod(int v, int n) {
  int r = v % n;
  return r < 0 ? r + n : r;
}
// Periodic wrap without a division when v lies within one period of the
// lattice (-n <= v < 2n), the case of every tile and halo coordinate of a
// lattice at least as large as the halo; pmod otherwise.
__device__ __forceinline__ int wrapz(int v, int n) {
  if (v >= -n && v < 2 * n) return v < 0 ? v + n : (v >= n ? v - n : v);
  return pmod(v, n);
}

// Langevin function L(x) = coth x - 1/x, accurate in FP32 for small x.
__device__ __forceinline__ float langevin(float x) {
  if (x < 0.3f) {
    float x2 = x * x;
    return x * fmaf(x2, fmaf(x2, fmaf(x2, -1.0f / 4725.0f, 2.0f / 945.0f), -1.0f / 45.0f), 1.0f / 3.0f);
  }
  float t = tanhf(x);
  return 1.0f / t - 1.0f / x;
}

// Equilibrium deviation for one component: deq_i = rho*(E_i(v) - w_i) + drho*w_i
// with E of bdist = 2 (code/lb3d_bdist.F90:301-370), then the BGK update
// d_i <- d_i + omega (deq_i - d_i), evaluated as (1 - omega) d_i + omega deq_i
// with omega folded into the equilibrium's coefficients.  Every multiply-add
// is written out (fmaf), so bgk_update2 below can repeat the same roundings
// lane by lane.
__device__ __forceinline__ void bgk_update(float d[19], float rho, float drho, float vx, float vy,
                                           float vz, float omega) {
  const float tx = 3.0f * vx, ty = 3.0f * vy, tz = 3.0f * vz;
  const float uke = 0.5f * fmaf(tz, vz, fmaf(ty, vy, tx * vx));
  const float a = -uke;          // even part minus w
  const float b = 1.0f + a;      // odd linear coefficient
  const float orw = (omega * rho) * W1;
  const float obase = (omega * drho) * W1;
  const float om1 = 1.0f - omega;
#define LB3D_PAIR32(CD, I, J)                                             \
  {                                                                       \
    const float e = (CD);                                                 \
    const float e2 = e * e;                                               \
    const float ev = fmaf(orw, fmaf(0.5f, e2, a), obase);                 \
    const float od = (orw * e) * fmaf(e2, 1.0f / 6.0f, b);                \
    d[I] = fmaf(om1, d[I], ev + od);                                      \
    d[J] = fmaf(om1, d[J], ev - od);                                      \
  }
  LB3D_PAIR32(tx, 0, 1)
  LB3D_PAIR32(ty, 2, 3)
  LB3D_PAIR32(tz, 4, 5)
  LB3D_PAIR32(tx + ty, 6, 11)
  LB3D_PAIR32(tx - ty, 7, 10)
  LB3D_PAIR32(tx + tz, 8, 13)
  LB3D_PAIR32(tx - tz, 9, 12)
  LB3D_PAIR32(ty + tz, 14, 17)
  LB3D_PAIR32(ty - tz, 15, 16)
#undef LB3D_PAIR32
  const float oeq0 = fmaf((omega * rho) * W0, a, (omega * drho) * W0);
  d[18] = fmaf(om1, d[18], oeq0);
}

// Paired FP32 arithmetic (sm_100 FADD2/FMUL2/FFMA2: two lanes per
// instruction, each rounded as its scalar counterpart).
__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 neg2(float2 v) { return make_float2(-v.x, -v.y); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// bgk_update for two components at once (lane x, lane y), bit for bit the
// scalar routine on each lane.
__device__ __forceinline__ void bgk_update2(float2 d[19], float2 rho, float2 drho, float2 vx,
                                            float2 vy, float2 vz, float2 omega) {
  const float2 tx = mul2(f2(3.0f), vx), ty = mul2(f2(3.0f), vy), tz = mul2(f2(3.0f), vz);
  const float2 uke = mul2(f2(0.5f), fma2(tz, vz, fma2(ty, vy, mul2(tx, vx))));
  const float2 a = neg2(uke);
  const float2 b = add2(f2(1.0f), a);
  const float2 orw = mul2(mul2(omega, rho), f2(W1));
  const float2 obase = mul2(mul2(omega, drho), f2(W1));
  const float2 om1 = add2(f2(1.0f), neg2(omega));
#define LB3D_PAIR2(CD, I, J)                                                  \
  {                                                                           \
    const float2 e = (CD);                                                    \
    const float2 e2 = mul2(e, e);                                             \
    const float2 ev = fma2(orw, fma2(f2(0.5f), e2, a), obase);                \
    const float2 od = mul2(mul2(orw, e), fma2(e2, f2(1.0f / 6.0f), b));       \
    d[I] = fma2(om1, d[I], add2(ev, od));                                     \
    d[J] = fma2(om1, d[J], add2(ev, neg2(od)));                               \
  }
  LB3D_PAIR2(tx, 0, 1)
  LB3D_PAIR2(ty, 2, 3)
  LB3D_PAIR2(tz, 4, 5)
  LB3D_PAIR2(add2(tx, ty), 6, 11)
  LB3D_PAIR2(add2(tx, neg2(ty)), 7, 10)
  LB3D_PAIR2(add2(tx, tz), 8, 13)
  LB3D_PAIR2(add2(tx, neg2(tz)), 9, 12)
  LB3D_PAIR2(add2(ty, tz), 14, 17)
  LB3D_PAIR2(add2(ty, neg2(tz)), 15, 16)
#undef LB3D_PAIR2
  const float2 oeq0 = fma2(mul2(mul2(omega, rho), f2(W0)), a, mul2(mul2(omega, drho), f2(W0)));
  d[18] = fma2(om1, d[18], oeq0);
}

// Equilibrium deviations of one component written straight to the output
// (full relaxation: the BGK update with omega = 1), with bgk_update's
// arithmetic; out[q * S] receives population q.
__device__ __forceinline__ void eq_store(float *out, unsigned S, float rho, float drho, float vx, float vy,
                                         float vz, float omega) {
  const float tx = 3.0f * vx, ty = 3.0f * vy, tz = 3.0f * vz;
  const float uke = 0.5f * fmaf(tz, vz, fmaf(ty, vy, tx * vx));
  const float a = -uke;
  const float b = 1.0f + a;
  const float orw = (omega * rho) * W1;
  const float obase = (omega * drho) * W1;
#define LB3D_EQ32(CD, I, J)                                               \
  {                                                                       \
    const float e = (CD);                                                 \
    const float e2 = e * e;                                               \
    const float ev = fmaf(orw, fmaf(0.5f, e2, a), obase);                 \
    const float od = (orw * e) * fmaf(e2, 1.0f / 6.0f, b);                \
    __stcs(out + (I) * S, ev + od);                                       \
    __stcs(out + (J) * S, ev - od);                                       \
  }
  LB3D_EQ32(tx, 0, 1)
  LB3D_EQ32(ty, 2, 3)
  LB3D_EQ32(tz, 4, 5)
  LB3D_EQ32(tx + ty, 6, 11)
  LB3D_EQ32(tx - ty, 7, 10)
  LB3D_EQ32(tx + tz, 8, 13)
  LB3D_EQ32(tx - tz, 9, 12)
  LB3D_EQ32(ty + tz, 14, 17)
  LB3D_EQ32(ty - tz, 15, 16)
#undef LB3D_EQ32
  __stcs(out + 18 * S, fmaf((omega * rho) * W0, a, (omega * drho) * W0));
}
// eq_store for two components (lanes x, y) with bgk_update2's paired
// arithmetic; lane x goes to outA, lane y to outB.
__device__ __forceinline__ void eq_store2(float *outA, float *outB, unsigned S, float2 rho, float2 drho,
                                          float2 vx, float2 vy, float2 vz, float2 omega) {
  const float2 tx = mul2(f2(3.0f), vx), ty = mul2(f2(3.0f), vy), tz = mul2(f2(3.0f), vz);
  const float2 uke = mul2(f2(0.5f), fma2(tz, vz, fma2(ty, vy, mul2(tx, vx))));
  const float2 a = neg2(uke);
  const float2 b = add2(f2(1.0f), a);
  const float2 orw = mul2(mul2(omega, rho), f2(W1));
  const float2 obase = mul2(mul2(omega, drho), f2(W1));
#define LB3D_EQ2(CD, I, J)                                                    \
  {                                                                           \
    const float2 e = (CD);                                                    \
    const float2 e2 = mul2(e, e);                                             \
    const float2 ev = fma2(orw, fma2(f2(0.5f), e2, a), obase);                \
    const float2 od = mul2(mul2(orw, e), fma2(e2, f2(1.0f / 6.0f), b));       \
    const float2 p = add2(ev, od), m = add2(ev, neg2(od));                    \
    __stcs(outA + (I) * S, p.x);                                              \
    __stcs(outB + (I) * S, p.y);                                              \
    __stcs(outA + (J) * S, m.x);                                              \
    __stcs(outB + (J) * S, m.y);                                              \
  }
  LB3D_EQ2(tx, 0, 1)
  LB3D_EQ2(ty, 2, 3)
  LB3D_EQ2(tz, 4, 5)
  LB3D_EQ2(add2(tx, ty), 6, 11)
  LB3D_EQ2(add2(tx, neg2(ty)), 7, 10)
  LB3D_EQ2(add2(tx, tz), 8, 13)
  LB3D_EQ2(add2(tx, neg2(tz)), 9, 12)
  LB3D_EQ2(add2(ty, tz), 14, 17)
  LB3D_EQ2(add2(ty, neg2(tz)), 15, 16)
#undef LB3D_EQ2
  const float2 oeq0 = fma2(mul2(mul2(omega, rho), f2(W0)), a, mul2(mul2(omega, drho), f2(W0)));
  __stcs(outA + 18 * S, oeq0.x);
  __stcs(outB + 18 * S, oeq0.y);
}

// Own-site moments of one component's post-stream deviations d[q * ST]:
// drho = sum_q g_q d_q and j = sum_q g_q c_q d_q, in q order, one fused
// multiply-add per term.
template <int ST>
__device__ __forceinline__ void own_moments(const float *d, float &dr, float &j0, float &j1,
                                            float &j2) {
  float r = 0.f, a0 = 0.f, a1 = 0.f, a2 = 0.f;
#pragma unroll
  for (int q = 0; q < 19; ++q) {
    const float v = d[q * ST], g = (float)gw(q);
    r = fmaf(g, v, r);
    if (cx(q)) a0 = fmaf(g * (float)cx(q), v, a0);
    if (cy(q)) a1 = fmaf(g * (float)cy(q), v, a1);
    if (cz(q)) a2 = fmaf(g * (float)cz(q), v, a2);
  }
  dr = r;
  j0 = a0;
  j1 = a1;
  j2 = a2;
}
// own_moments of two components (lanes x, y) with paired instructions.
__device__ __forceinline__ void own_moments2(const float2 v[19], float2 &dr, float2 &j0,
                                                 float2 &j1, float2 &j2) {
  float2 r = f2(0.f), a0 = f2(0.f), a1 = f2(0.f), a2 = f2(0.f);
#pragma unroll
  for (int q = 0; q < 19; ++q) {
    const float g = (float)gw(q);
    r = fma2(f2(g), v[q], r);
    if (cx(q)) a0 = fma2(f2(g * (float)cx(q)), v[q], a0);
    if (cy(q)) a1 = fma2(f2(g * (float)cy(q)), v[q], a1);
    if (cz(q)) a2 = fma2(f2(g * (float)cz(q)), v[q], a2);
  }
  dr = r;
  j0 = a0;
  j1 = a1;
  j2 = a2;
}
// Site offsets (32-bit, relative to the lattice base) of the -1, 0, +1
// neighbours along each axis, with the periodic wrap applied once.
struct Nbr {
  int cx[3], ry[3], rz[3];
};

__device__ __forceinline__ void make_nbr(Nbr &n, int gx, int gy, int gz, int nx, int ny, int nz) {
  const int pl = nx * ny;
  n.cx[0] = gx == 0 ? nx - 1 : gx - 1;
  n.cx[1] = gx;
  n.cx[2] = gx == nx - 1 ? 0 : gx + 1;
  n.ry[0] = (gy == 0 ? ny - 1 : gy - 1) * nx;
  n.ry[1] = gy * nx;
  n.ry[2] = (gy == ny - 1 ? 0 : gy + 1) * nx;
  n.rz[0] = (gz == 0 ? nz - 1 : gz - 1) * pl;
  n.rz[1] = gz * pl;
  n.rz[2] = (gz == nz - 1 ? 0 : gz + 1) * pl;
}
// site offset of x + s*c_q (s = +1 neighbour, s = -1 upstream)
template <int Q, int SGN>
__device__ __forceinline__ int noff(const Nbr &n) {
  return n.cx[1 + SGN * cx(Q)] + n.ry[1 + SGN * cy(Q)] + n.rz[1 + SGN * cz(Q)];
}

// Pulls the post-stream deviations of component C of one site (with
// half-way bounce-back when ROCK): d[q] = delta*(x - c_q, q), or
// delta*(x, bounce(q)) when x - c_q is rock (code/lb3d_bc_bounce.F90:53-90
// with code/lb3d_advection.F90:109-151).  F points at component 0 of the
// lattice; the component stride is 19*S.
// LAST selects the last-use load hint (the final read of these values by
// this CTA), which lets L2 drop the lines early.  NARROW forms the component
// offset c*19*S in 32 bits (lattices with 19*nc*S < 2^32), which keeps the
// register-capped moments pass free of 64-bit products.
template <bool ROCK, bool LAST = false, bool NARROW = false>
__device__ __forceinline__ void pull_comp(const float *__restrict__ F, unsigned S, int c, const Nbr &n,
                                          int self, const uint8_t *__restrict__ rk, float d[19]) {
  const float *fc = NARROW ? F + (unsigned)(c * 19) * S : F + (size_t)(c * 19) * S;
  d[18] = LAST ? __ldlu(fc + 18 * S + self) : __ldg(fc + 18 * S + self);
#define LB3D_PULL(Q)                                                     \
  {                                                                      \
    const int up = noff<Q, -1>(n);                                       \
    bool uf = true;                                                      \
    if (ROCK) uf = __ldg(rk + up) == 0;                                  \
    const float *a_ = fc + (uf ? Q * S + up : bounce(Q) * S + self);     \
    d[Q] = LAST ? __ldlu(a_) : __ldg(a_);                                \
  }
  LB3D_PULL(0) LB3D_PULL(1) LB3D_PULL(2) LB3D_PULL(3) LB3D_PULL(4) LB3D_PULL(5)
  LB3D_PULL(6) LB3D_PULL(7) LB3D_PULL(8) LB3D_PULL(9) LB3D_PULL(10) LB3D_PULL(11)
  LB3D_PULL(12) LB3D_PULL(13) LB3D_PULL(14) LB3D_PULL(15) LB3D_PULL(16) LB3D_PULL(17)
#undef LB3D_PULL
}

// Lees-Edwards pulls (binary, no rock; code/lb3d_bc_leesedwards.F90:147-1315
// feeding code/lb3d_advection.F90:109-151): across x = 0 (c_x = +1) and
// x = nx - 1 (c_x = -1) the upstream site lies in the sheared halo planes
// Lg.le_h[0] / Lg.le_h[1], [nc][19][nz][ny], at the wrapped (y - c_y, z - c_z).
// Offsets within a set of planes, [nc][19][nz][ny], are unsigned 32-bit: at most
// 38 ny nz, and a lattice of at least two sites across stays below.
static_assert(38ull * (((1ull << 32) - 1) / 19 / 2) < (1ull << 32), "19 sites < 2^32, two sites across");
struct LeYZ {
  int y[3], z[3];  // wrap(gy + k - 1) and ny * wrap(gz + k - 1)
};
__device__ __forceinline__ void make_leyz(LeYZ &w, int gy, int gz, int ny, int nz) {
  w.y[0] = gy == 0 ? ny - 1 : gy - 1;
  w.y[1] = gy;
  w.y[2] = gy == ny - 1 ? 0 : gy + 1;
  w.z[0] = ny * (gz == 0 ? nz - 1 : gz - 1);
  w.z[1] = ny * gz;
  w.z[2] = ny * (gz == nz - 1 ? 0 : gz + 1);
}
// With ROCK (walls) the sheared halo sites are never rock, as the
// reference's exchange leaves them (code/lb3d_bc_leesedwards.F90:678,866),
// and a pull from a rock site inside the lattice bounces back.
template <int Q, bool ROCK = false>
__device__ __forceinline__ const float *le_src(const float *fc, unsigned S, int c, const Nbr &n, int gx,
                                               int nx, const LeYZ &w, const LatDesc &Lg, unsigned NP,
                                               int self = 0, const uint8_t *__restrict__ rk = nullptr) {
  if (cx(Q) == 1 && gx == 0) return Lg.le_h[0] + (c * 19 + Q) * NP + w.y[1 - cy(Q)] + w.z[1 - cz(Q)];
  if (cx(Q) == -1 && gx == nx - 1)
    return Lg.le_h[1] + (c * 19 + Q) * NP + w.y[1 - cy(Q)] + w.z[1 - cz(Q)];
  const int up = noff<Q, -1>(n);
  if (ROCK && __ldg(rk + up) != 0) return fc + bounce(Q) * S + self;
  return fc + Q * S + up;
}
template <bool NARROW = false, bool ROCK = false>
__device__ __forceinline__ void pull_comp_le(const float *__restrict__ F, unsigned S, int c, const Nbr &n,
                                             int self, int gx, int nx, const LeYZ &w,
                                             const LatDesc &Lg, unsigned NP, float d[19],
                                             const uint8_t *__restrict__ rk = nullptr) {
  const float *fc = NARROW ? F + (unsigned)(c * 19) * S : F + (size_t)(c * 19) * S;
  d[18] = __ldg(fc + 18 * S + self);
#define LB3D_PULL_LE(Q) d[Q] = __ldg(le_src<Q, ROCK>(fc, S, c, n, gx, nx, w, Lg, NP, self, rk));
  LB3D_PULL_LE(0) LB3D_PULL_LE(1) LB3D_PULL_LE(2) LB3D_PULL_LE(3) LB3D_PULL_LE(4) LB3D_PULL_LE(5)
  LB3D_PULL_LE(6) LB3D_PULL_LE(7) LB3D_PULL_LE(8) LB3D_PULL_LE(9) LB3D_PULL_LE(10) LB3D_PULL_LE(11)
  LB3D_PULL_LE(12) LB3D_PULL_LE(13) LB3D_PULL_LE(14) LB3D_PULL_LE(15) LB3D_PULL_LE(16) LB3D_PULL_LE(17)
#undef LB3D_PULL_LE
}

// Writes one component's 19 deviations of a site on the x boundary of a
// Lees-Edwards lattice to the compact boundary planes: set 0 (pre-stream,
// le_b[0] at x = nx - 1, le_b[1] at x = 0) or set 2 (post-stream, le_b[2],
// le_b[3]); sites elsewhere write nothing.
__device__ __forceinline__ void le_store_boundary(const LatDesc &Lg, int set, int c, int gx, int gy,
                                                  int gz, const float d[19]) {
  const int nx = Lg.nx;
  const unsigned NP = Lg.ny * Lg.nz, o = (c * 19) * NP + gy + Lg.ny * gz;
  if (gx == nx - 1) {
    float *b = Lg.le_b[set] + o;
#pragma unroll
    for (int q = 0; q < 19; ++q) b[q * NP] = d[q];
  }
  if (gx == 0) {
    float *b = Lg.le_b[set + 1] + o;
#pragma unroll
    for (int q = 0; q < 19; ++q) b[q * NP] = d[q];
  }
}

// Asynchronous copies global -> shared (cp.async, 4/8/16 bytes) in commit
// groups; a thread waits for its own groups, a barrier then publishes them.
__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

#include "fp32_stencil.cuh"

}  // namespace f32
}  // namespace lb3d
#endif
