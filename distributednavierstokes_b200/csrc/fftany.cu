// fftany.cu -- splits, launch shapes and launches of fftany.cuh.
#include "fftany.h"

#include <algorithm>

#include "fftany.cuh"
#include "launch.h"
#include "tiers.h"

namespace dnsb {
namespace {

// Lines per block: enough for FA_THREADS register transforms, fewer where
// the grid would leave SMs without a block (small boxes: latency, not
// throughput, is what their transforms cost), and within shared memory.
int lines_for(const AnySplit &sp, int asked, long long lines, int least, size_t bytes_per_line, size_t fixed) {
  int L = asked > 0 ? asked : std::max(least, FA_THREADS / std::max(sp.n1, sp.n2));
  const long long few = 2LL * sm_count();
  while (asked <= 0 && L > least && (lines + L - 1) / L < few && L / 2 * std::max(sp.n1, sp.n2) >= 64)
    L = std::max(least, L / 2);
  while (L > 1 && fixed + L * bytes_per_line > kSmemPerBlock) L--;
  return L;
}

// the same number of blocks per row of nz lines with the lines spread evenly
int even(int nz, int L) {
  const int groups = (nz + L - 1) / L;
  return (nz + groups - 1) / groups;
}

size_t smem_z(const AnySplit &sp, int L) {
  return sizeof(double2) * ((size_t)L * sp.n1 * fa_pitch(sp.n2) + sp.n1 * sp.n2);
}

size_t smem_y(const AnySplit &sp, int L) {
  return sizeof(double2) * (size_t)(L + 1) * sp.n1 * sp.n2;
}

size_t line_x(const AnySplit &sp) {
  return sizeof(double2) * ((size_t)sp.n1 * fa_pitch(sp.n2) + sp.n1 * sp.n2 + 1);
}
size_t fixed_x(const AnySplit &sp) { return sizeof(double2) * (2 * (size_t)sp.n1 * sp.n2 + 1); }
size_t smem_x(const AnySplit &sp, int L) { return fixed_x(sp) + L * line_x(sp); }

}  // namespace

int any_lines_x(const Geo &g, const AnySplit &sp, int asked) {
  return even(g.nz, std::min(16, lines_for(sp, asked, (long long)g.ny * g.nz, 4, line_x(sp), fixed_x(sp))));
}

int any_lines_y(const Geo &g, const AnySplit &sp, int nkx, int asked) {
  const int n = sp.n1 * sp.n2;
  const int L = lines_for(sp, asked, (long long)nkx * g.nz, 4, sizeof(double2) * n, sizeof(double2) * n);
  return even(g.nz, std::min(L, 16));
}

int any_lines_z(const Geo &g, const AnySplit &sp, int nkx, int asked) {
  const int n = sp.n1 * sp.n2;
  return lines_for(sp, asked, (long long)g.ny * nkx, 2, sizeof(double2) * sp.n1 * fa_pitch(sp.n2),
                   sizeof(double2) * n);
}

AnySplit any_split(int n) {
#define FA_LIST(R) R,
  static const int sizes[] = {FA_RADICES(FA_LIST)};
#undef FA_LIST
  AnySplit best;
  for (int a : sizes) {
    if (n % a) continue;
    const int b = n / a;
    if (std::find(std::begin(sizes), std::end(sizes), b) == std::end(sizes)) continue;
    if (best.n1 == 0 || std::max(a, b) < std::max(best.n1, best.n2)) {
      best.n1 = a;
      best.n2 = b;
    }
  }
  if (best.n1) {
    const int m = std::max(best.n1, best.n2);
    best.tier = m <= 10 ? 10 : m <= 16 ? 16 : 25;
  }
  return best;
}

cudaError_t any_allow(int device, const AnySplit &x, const AnySplit &y, const AnySplit &z) {
  cudaError_t e = cudaSuccess;
  auto allow = [&](auto kernel) {
    if (e == cudaSuccess) e = raise_smem(device, kernel, kSmemPerBlock);
    return e;
  };
  if (z.tier) by_tier(z.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    allow(k_fftz_any<T, false>);
    return allow(k_fftz_any<T, true>);
  });
  if (y.tier) by_tier(y.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    allow(k_y_any<T, YF_SOLVE>);
    allow(k_y_any<T, YF_FORWARD>);
    return allow(k_y_any<T, YF_INVERSE>);
  });
  if (x.tier) by_tier(x.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    allow(k_rfftx_any<T, RIN_DIVERGENCE>);
    allow(k_rfftx_any<T, RIN_REAL>);
    allow(k_rfftx_any<T, RIN_FIELD>);
    allow(k_rfftx_any<T, RIN_PRODUCT>);
    allow(k_irfftx_any<T, ROUT_INTERIOR>);
    allow(k_irfftx_any<T, ROUT_IMAGES>);
    return allow(k_irfftx_any<T, ROUT_REAL>);
  });
  return e;
}

cudaError_t any_fftz(const Geo &g, const AnySplit &sp, int nkx, int lines, bool inv, double2 *S,
                     const double2 *twz, cudaStream_t stream) {
  const long long nlines = (long long)g.ny * nkx;
  const int L = any_lines_z(g, sp, nkx, lines);
  const dim3 grid((unsigned)((nlines + L - 1) / L)), block(threads_for(L * std::max(sp.n1, sp.n2)));
  return by_tier(sp.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    return launch_pdl(inv ? k_fftz_any<T, true> : k_fftz_any<T, false>, grid, block,
                            smem_z(sp, L), stream, g.nz, sp.n1, sp.n2, L, nlines, S, twz);
  });
}

cudaError_t any_y(const Geo &g, const AnySplit &sp, int nkx, int lines, int mode, double2 *S, const double2 *twy,
                  const double *lam1, const double *lam2, const double *lam3, cudaStream_t stream) {
  const int L = any_lines_y(g, sp, nkx, lines);
  const dim3 grid((unsigned)(nkx * ((g.nz + L - 1) / L))), block(threads_for(L * std::max(sp.n1, sp.n2)));
  return by_tier(sp.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    auto k = mode == YF_SOLVE ? k_y_any<T, YF_SOLVE>
             : mode == YF_FORWARD ? k_y_any<T, YF_FORWARD> : k_y_any<T, YF_INVERSE>;
    return launch_pdl(k, grid, block, smem_y(sp, L), stream, g, sp.n1, sp.n2, L, S, twy, lam1,
                            lam2, lam3);
  });
}

cudaError_t any_rfftx(const Geo &g, const AnySplit &sp, int lines, int mode, double2 *S,
                      const double *a,
                      const double *b, const double *c, const double2 *twM, const double2 *twN,
                      cudaStream_t stream) {
  const int L = any_lines_x(g, sp, lines);
  const dim3 grid((unsigned)(g.ny * ((g.nz + L - 1) / L)));
  return by_tier(sp.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    auto k = mode == RIN_DIVERGENCE ? k_rfftx_any<T, RIN_DIVERGENCE>
             : mode == RIN_REAL     ? k_rfftx_any<T, RIN_REAL>
             : mode == RIN_FIELD    ? k_rfftx_any<T, RIN_FIELD>
                                    : k_rfftx_any<T, RIN_PRODUCT>;
    return launch_pdl(k, grid, dim3(FA_THREADS), smem_x(sp, L), stream, g, sp.n1, sp.n2, L, S, a,
                            b, c, twM, twN);
  });
}

cudaError_t any_irfftx(const Geo &g, const AnySplit &sp, int lines, int mode, const double2 *S, double *out,
                       const double2 *twM, const double2 *twN, cudaStream_t stream) {
  const int L = any_lines_x(g, sp, lines);
  const dim3 grid((unsigned)(g.ny * ((g.nz + L - 1) / L)));
  return by_tier(sp.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    auto k = mode == ROUT_INTERIOR ? k_irfftx_any<T, ROUT_INTERIOR>
             : mode == ROUT_IMAGES ? k_irfftx_any<T, ROUT_IMAGES>
                                   : k_irfftx_any<T, ROUT_REAL>;
    return launch_pdl(k, grid, dim3(FA_THREADS), smem_x(sp, L), stream, g, sp.n1, sp.n2, L, S,
                            out, twM, twN);
  });
}

}  // namespace dnsb
