// spany.cu -- launches of spany.cuh.
#include "spany.h"

#include <algorithm>

#include "launch.h"
#include "spany.cuh"
#include "tiers.h"

namespace dnsb {
namespace {

// lines per block: FA_THREADS register transforms, within shared memory, at
// most `most`
int lines_for(const AnySplit &sp, int most, size_t per_line, size_t fixed) {
  int L = std::min(most, std::max(2, FA_THREADS / std::max(sp.n1, sp.n2)));
  while (L > 1 && fixed + L * per_line > kSmemPerBlock) L--;
  return L;
}

constexpr size_t C = sizeof(double2);
size_t buf_line(const AnySplit &sp) { return C * sp.n1 * fa_pitch(sp.n2); }

}  // namespace

cudaError_t sp_any_allow(int device, const SpPlan &p) {
  cudaError_t e = cudaSuccess;
  auto allow = [&](auto kernel) {
    if (e == cudaSuccess) e = raise_smem(device, kernel, kSmemPerBlock);
    return e;
  };
  by_tier(p.yz.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    allow(k_sp_yinv<T>);
    allow(k_sp_z<T, true>);
    allow(k_sp_z<T, false>);
    return allow(k_sp_yfwd<T>);
  });
#define ALLOW4(A, B_)                       \
  if (p.s.n == 2 * A * B_) {                \
    if (e == cudaSuccess) e = raise_smem(device, k_sp_xinv4<A, B_>, XWarp<A, B_>::smem);           \
    if (e == cudaSuccess) e = raise_smem(device, k_sp_xprod4<A, B_>, sp_xprod4_smem<A, B_>());     \
  }
  SP4_SPLITS(ALLOW4)
#undef ALLOW4
  by_tier(p.x.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    allow(k_sp_xinv<T>);
    return allow(k_sp_xprod<T>);
  });
  return e;
}

cudaError_t sp_any_phys(const SpPlan &p, const double2 *uh, double *const v[3], cudaStream_t st) {
  const SpCube &s = p.s;
  const int n = s.n, h = s.kcut + 1;
  const SpBufs A{{p.buf[0], p.buf[1], p.buf[2]}}, B{{p.buf[3], p.buf[4], p.buf[5]}};
  cudaError_t e = by_tier(p.yz.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    const dim3 grid((unsigned)((h + 1) / 2 * ((s.m + 3) / 4)), 1, 3);
    return launch_pdl(k_sp_yinv<T>, grid, dim3(threads_for(8 * std::max(p.yz.n1, p.yz.n2))),
                            C * 9 * n, st, s, p.yz.n1, p.yz.n2, uh, A, p.twn);
  });
  if (e != cudaSuccess) return e;
  e = by_tier(p.yz.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    const int L = lines_for(p.yz, 64, buf_line(p.yz), C * n);
    const long long nlines = (long long)n * h;
    const dim3 grid((unsigned)((nlines + L - 1) / L), 1, 3);
    return launch_pdl(k_sp_z<T, true>, grid, dim3(threads_for(L * std::max(p.yz.n1, p.yz.n2))),
                            L * buf_line(p.yz) + C * n, st, s, p.yz.n1, p.yz.n2, L, A, B, p.twn);
  });
  if (e != cudaSuccess) return e;
#define XINV4(A, B_)                                                                             \
  if (n == 2 * A * B_) {                                                                           \
    const dim3 grid(n * ((n + XWarp<A, B_>::LINES - 1) / XWarp<A, B_>::LINES), 1, 3);              \
    return launch_pdl(k_sp_xinv4<A, B_>, grid, dim3(128), XWarp<A, B_>::smem, st, s, B,            \
                      SpFields{{v[0], v[1], v[2]}}, p.twM, p.twN);                                 \
  }
  SP4_SPLITS(XINV4)
#undef XINV4
  return by_tier(p.x.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    const int M = n / 2;
    const size_t line = buf_line(p.x) + C * (M + 1), fixed = C * (2 * M + 1);
    const int L = lines_for(p.x, 16, line, fixed);
    const dim3 grid((unsigned)(n * ((n + L - 1) / L)), 1, 3);
    return launch_pdl(k_sp_xinv<T>, grid, dim3(FA_THREADS), fixed + L * line, st, s, p.x.n1, p.x.n2,
                            L, B, SpFields{{v[0], v[1], v[2]}}, p.twM, p.twN);
  });
}

cudaError_t sp_any_products(const SpPlan &p, double *const v[3], unsigned long long *vmax,
                            cudaStream_t st) {
  const SpCube &s = p.s;
  const int n = s.n, h = s.kcut + 1;
  SpBufs F;
  std::copy(p.buf, p.buf + 6, F.b);
  bool by_warps = false;
  cudaError_t e = cudaSuccess;
#define XPROD4(A, B_)                                                                              \
  if (n == 2 * A * B_) {                                                                           \
    const dim3 grid(n * ((n + XWarp<A, B_>::LINES - 1) / XWarp<A, B_>::LINES));                    \
    by_warps = true;                                                                               \
    e = launch_pdl(k_sp_xprod4<A, B_>, grid, dim3(128), sp_xprod4_smem<A, B_>(), st, s,            \
                   SpFields{{v[0], v[1], v[2]}}, F, vmax, p.twM, p.twN);                           \
  }
  SP4_SPLITS(XPROD4)
#undef XPROD4
  if (!by_warps) e = by_tier(p.x.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    const int M = n / 2;
    const size_t line = buf_line(p.x) + C * (4 * M + 1), fixed = C * (2 * M + 1);
    const int L = lines_for(p.x, 16, line, fixed);
    const dim3 grid((unsigned)(n * ((n + L - 1) / L)));
    return launch_pdl(k_sp_xprod<T>, grid, dim3(FA_THREADS), fixed + L * line, st, s, p.x.n1, p.x.n2,
                            L, SpFields{{v[0], v[1], v[2]}}, F, vmax, p.twM, p.twN);
  });
  if (e != cudaSuccess) return e;
  e = by_tier(p.yz.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    const int L = lines_for(p.yz, 64, buf_line(p.yz), C * n);
    const long long nlines = (long long)n * h;
    const dim3 grid((unsigned)((nlines + L - 1) / L), 1, 6);
    return launch_pdl(k_sp_z<T, false>, grid, dim3(threads_for(L * std::max(p.yz.n1, p.yz.n2))),
                            L * buf_line(p.yz) + C * n, st, s, p.yz.n1, p.yz.n2, L, F, F, p.twn);
  });
  if (e != cudaSuccess) return e;
  return by_tier(p.yz.tier, [&](auto t) {
    constexpr int T = decltype(t)::value;
    const int L = std::max(4, lines_for(p.yz, 16, C * n, C * n));
    const dim3 grid((unsigned)(h * ((s.m + L - 1) / L)), 1, 6);
    return launch_pdl(k_sp_yfwd<T>, grid, dim3(threads_for(L * std::max(p.yz.n1, p.yz.n2))),
                            C * (L + 1) * n, st, s, p.yz.n1, p.yz.n2, L, F, p.twn);
  });
}

namespace {
dim3 stage_grid(const SpCube &s) {
  return dim3((unsigned)((s.kcut + SPS_T) / SPS_T), (unsigned)((s.m + SPS_T - 1) / SPS_T), (unsigned)s.m);
}
}  // namespace

cudaError_t sp_any_rhs(const SpPlan &p, double2 *du, cudaStream_t st) {
  SpBufs F;
  std::copy(p.buf, p.buf + 6, F.b);
  return launch_pdl(k_sp_stage<true>, stage_grid(p.s), dim3(SPS_T * SPS_T), 0, st, p.s, F, du,
                          (const double2 *)nullptr, (double2 *)nullptr, 0.0, 0.0, 0.0, 0.0);
}

cudaError_t sp_any_stage(const SpPlan &p, double2 *uh, const double2 *start, double2 *next, double a,
                         double b, double nudcdt, double dt, cudaStream_t st) {
  SpBufs F;
  std::copy(p.buf, p.buf + 6, F.b);
  return launch_pdl(k_sp_stage<false>, stage_grid(p.s), dim3(SPS_T * SPS_T), 0, st, p.s, F, uh, start,
                          next, a, b, nudcdt, dt);
}

}  // namespace dnsb
