// fp64_path.h -- host launchers of the FP64 drop-in kernels (fp64_path.cu).
#ifndef LB3D_FP64_PATH_H
#define LB3D_FP64_PATH_H

#include "common.cuh"

namespace lb3d {

// Lees-Edwards x-halo planes from the populations src (compact: from the
// boundary planes [2][nc][19][nz][ny] of x = nx - 1 and x = 0), their
// densities and psi when rlo is given; binary lattices.
cudaError_t fp64_le_halo(const DevParams &P, const LEStep &S, const double *src, bool compact, double *hlo,
                         double *hhi, double *rlo, double *rhi, double *plo, double *phi,
                         cudaStream_t st, bool pdl = false);
// Zou-He flux boundaries on the z = 1 and z = nz planes (inv_fluid 12),
// applied to the post-stream populations g and the advected dipole flux da.
cudaError_t fp64_zouhe_density(const DevParams &P, double *g, const uint8_t *rock, double fr,
                               double fb, double pr, double pb, cudaStream_t st);
cudaError_t fp64_recolour(const DevParams &P, double *g, const uint8_t *rock, double mr, double mb,
                          cudaStream_t st);
cudaError_t fp64_zouhe_flux(const DevParams &P, double *g, double *da, const double *db,
                            const uint8_t *rock, cudaStream_t st);
cudaError_t fp64_stream(const DevParams &P, const double *fin, double *fout, double *rho,
                        double *psi, double *mom, double *da, const double *db,
                        const uint8_t *rock, const double *hlo, const double *hhi,
                        cudaStream_t st);
// Kernels of fp64_stream, and of fp64_step_pull's moments pass.
int fp64_stream_launches(const DevParams &P);
// Lees-Edwards planes of a pulling step: the stage-6 halo (filled), the
// step's offset, the post-stream boundary planes [2][nc][19][nz][ny] and the
// stage-8 halo densities and psi (filled by the step).
struct Fp64Le {
  LEStep step;
  const double *hlo, *hhi;
  double *post, *rlo, *rhi, *plo, *phi;
};
// One time step with streaming fused into the collision (lattices without
// inflow boundaries; le under Lees-Edwards): moments pass (rho, psi, momenta,
// dipole flux), dipole relaxation (ternary), stage-8 halo (Lees-Edwards), pull
// + forces + BGK from fin into fout.  Every buffer ends up as after fp64_stream
// + fp64_dipole + fp64_collide, bit for bit, except that the post-stream
// populations are never stored.  The kernels of a step follow each other with
// programmatic dependent launch; chained: the kernel launched before on the
// stream is one of this step's kind, and the first one follows it so, too.
cudaError_t fp64_step_pull(const DevParams &P, const double *fin, double *fout, double *rho,
                           double *psi, double *mom, double *da, double *db, const uint8_t *rock,
                           cudaStream_t st, const Fp64Le *le = nullptr, bool chained = false);
cudaError_t fp64_dipole(const DevParams &P, const double *rho, const double *da, double *db,
                        cudaStream_t st, bool pdl = false);
cudaError_t fp64_collide(const DevParams &P, const double *g, double *f, const double *rho,
                         const double *psi, const double *mom, const double *db,
                         const uint8_t *rock, const double *plo, const double *phi,
                         cudaStream_t st);
// field: 0 od, 1 wd, 2 sur, 3 dir, 4 vel, 5 arr, 6 rock
cudaError_t fp64_dump(const DevParams &P, int field, const double *f, const double *rho,
                      const double *psi, const double *db, const uint8_t *rock, double *out,
                      cudaStream_t st);
cudaError_t fp64_moments(const DevParams &P, const double *f, double *rho, double *psi,
                         double *mom, cudaStream_t st);
cudaError_t fp64_detmath(int fn, const double *x, double *y, long long n, cudaStream_t st);

}  // namespace lb3d

#endif
