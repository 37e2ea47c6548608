// spany.h -- the pseudo-spectral solver's right-hand side on the run-time
// split transforms, truncated to the retained modes (spany.cuh).
#pragma once
#include <cuda_runtime.h>

#include "fftany.h"

namespace dnsb {

// cube side, retained wavenumbers, compact sizes, 2 pi / l
struct SpCube {
  int n, kcut, m;  // m = 2 kcut + 1
  long long nc;    // (kcut + 1) m m
  double kfac;
};

struct SpPlan {
  SpCube s{};
  AnySplit x, yz;  // n/2 and n
  const double2 *twM = nullptr, *twN = nullptr, *twn = nullptr;
  double2 *buf[6] = {};  // (kcut + 1) n n values each
  bool ok() const { return x.tier && yz.tier; }
};

cudaError_t sp_any_allow(int device, const SpPlan &p);

// v[c] <- the physical velocity of the compact state uh (three components)
cudaError_t sp_any_phys(const SpPlan &p, const double2 *uh, double *const v[3], cudaStream_t st);

// buf[f] <- the retained modes of the six products v_a v_b (xx yy zz xy yz
// zx), unnormalised, at [kx][ky][kz] with pitches n; with vmax the maximum of
// |v_1| + |v_2| + |v_3| is folded into it (ordered bits)
cudaError_t sp_any_products(const SpPlan &p, double *const v[3], unsigned long long *vmax,
                            cudaStream_t st);

// du <- the right-hand side from buf
cudaError_t sp_any_rhs(const SpPlan &p, double2 *du, cudaStream_t st);

// One Wray stage from buf: uh <- project(phi (start + a dt du)), and with
// next != nullptr next <- phi (start + b dt du).  start may be uh or next.
cudaError_t sp_any_stage(const SpPlan &p, double2 *uh, const double2 *start, double2 *next, double a,
                         double b, double nudcdt, double dt, cudaStream_t st);

}  // namespace dnsb
