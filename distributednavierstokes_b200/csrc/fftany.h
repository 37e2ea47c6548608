// fftany.h -- launches of the run-time-split transform kernels (fftany.cuh).
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace dnsb {

// A line length as N1 x N2 register transforms and the kernel tier it needs;
// tier 0: no split (the Stockham kernels run).
struct AnySplit {
  int n1 = 0, n2 = 0, tier = 0;
};
AnySplit any_split(int n);

// opt in to the shared memory of the kernels of one split
cudaError_t any_allow(int device, const AnySplit &x, const AnySplit &y, const AnySplit &z);

// lines per block of the transforms along x, y and z (over nkx kx planes): `asked`
// within what fits, or with 0 the launch's own rule.  What they return gives
// itself when asked for.
int any_lines_x(const Geo &g, const AnySplit &sp, int asked);
int any_lines_y(const Geo &g, const AnySplit &sp, int nkx, int asked);
int any_lines_z(const Geo &g, const AnySplit &sp, int nkx, int asked);

// Each returns the launch's status; the launches are launch_pdl's.  nkx: kx planes transformed; lines: lines per
// block (0: the launch's own rule).
cudaError_t any_fftz(const Geo &g, const AnySplit &sp, int nkx, int lines, bool inv, double2 *S,
                     const double2 *twz, cudaStream_t stream);
// mode: YFourierMode
cudaError_t any_y(const Geo &g, const AnySplit &sp, int nkx, int lines, int mode, double2 *S,
                  const double2 *twy, const double *lam1, const double *lam2, const double *lam3,
                  cudaStream_t stream);
// mode: RInMode
cudaError_t any_rfftx(const Geo &g, const AnySplit &sp, int lines, int mode, double2 *S,
                      const double *a,
                      const double *b, const double *c, const double2 *twM, const double2 *twN,
                      cudaStream_t stream);
// mode: ROutMode
cudaError_t any_irfftx(const Geo &g, const AnySplit &sp, int lines, int mode, const double2 *S, double *out,
                       const double2 *twM, const double2 *twN, cudaStream_t stream);

}  // namespace dnsb
