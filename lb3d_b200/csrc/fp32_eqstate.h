// fp32_eqstate.h -- launches of the FP32 strategy that carries the
// equilibrium's arguments (fp32_eqstate.cu).
#ifndef LB3D_FP32_EQSTATE_H
#define LB3D_FP32_EQSTATE_H

#include "fp32_path.h"

namespace lb3d {

// Fields between the passes of a step, indexed by base + site of the packed
// site space (stride S):
//   M    ternary: float4 [S] {rho_b - rho_r, da}, then float4 [S] {a, dpsi_s}
//   psi  {dpsi_r, dpsi_b}
//   o1   {drho_r, drho_b, P_x, P_y}, o2: P_z, P of red and blue
//   o3   ternary: {drho_s, P}, P of all components
// and between the steps of a loop, for lattices of parity 0 and 1,
//   Q    float4 [4][S]: {drho_r, drho_b, vx_r, vx_b}, {vy_r, vy_b, vz_r, vz_b},
//        ternary: {drho_s, v_s}, {d}
struct EqFields {
  float4 *M;
  float2 *psi;
  float4 *o1, *o3;
  float *o2;
  float4 *Q[2];
  unsigned S;
};

struct EqKernel {
  const void *fn;
  int threads;
  size_t smem;
};

struct EqArgs {
  const LatDesc *lats;
  const Tile *tiles;
  int ntiles;
  float *f0, *f1, *db0, *db1;
  const uint8_t *rock;
  const uint32_t *mask;
  EqFields X;
};

// The passes of a step, in order; the surfactant's moments pass and the dipole
// pass exist for ternary lattices, and a first step (from populations) takes
// all moments in EQ_MOMENTS.
enum { EQ_MOMENTS, EQ_SURFACTANT, EQ_DIPOLE, EQ_COLLIDE, EQ_PASSES };
// Tile of the moments passes for a lattice nx sites wide (le: Lees-Edwards).
void eq_moments_tile(int nx, bool le, int *tx, int *ty);
// The kernel of a pass for a lattice kind and tile; false if there is none.
// narrow: 19 nc S < 2^32.
bool eq_kernel(int pass, bool first, int nc, bool rock, bool le, int tx, int ty, bool narrow, EqKernel *k);
cudaError_t eq_launch(const EqKernel &k, int pass, bool first, bool last, const EqArgs &a, bool pdl,
                      cudaStream_t st);
// Neighbour masks of a lattice with rock (base 0), and its rock sites' psi entries.
cudaError_t eq_build_mask(int nx, int ny, int nz, bool le, const uint8_t *rock, uint32_t *mask, float2 *psi,
                          float psi0, cudaStream_t st);

}  // namespace lb3d
#endif
