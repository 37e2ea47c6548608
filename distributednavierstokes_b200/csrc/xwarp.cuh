// xwarp.cuh -- real FFTs along x by warps (the kernels are in spectral4.cuh
// and spany.cuh).
//
// A warp owns LW lines (row j, kz = k0 + LW w ..)
// from load to store: its lanes stage the lines, run both register steps of
// the half-length transform (M = N1 N2 = nx/2) and the real transform's pass,
// ordered by __syncwarp alone.
//
// Why by warps: with a CTA of 256 threads per tile the two steps kept 96 and
// 128 of them busy (M = 192, 8 lines) between CTA barriers, and the kernel
// was bound by those phases' latency at 2-3 CTAs per SM, not by HBM (52 % of
// its rate forward, 40 % inverse).  Here LW = 32 / max(N1, N2) lines fill the
// lanes of both steps, warps drift apart so that one's loads run under
// another's arithmetic, and the buffer of a step is reused by the next (every
// lane reads its inputs before any writes).  At 256^3 the divergence and forward
// transform then take 129 us (4.0 TB/s of DRAM, 0.61 of the copy rate), the inverse
// 97 (its spectrum partly in L2); the shared-memory pipe is 66 % busy in both (74 %
// at M = 192), with 16 warps per SM held by the registers.  The spectrum is touched LW lines
// of 16 bytes at a time (32 or 64 bytes: whole sectors); the CTA's four warps
// take adjacent lines.
#pragma once
#include "fft4.cuh"

namespace dnsb {

template <int N1, int N2>
struct XWarp {
  static constexpr int M = N1 * N2, P = fft4_pitch<N2>();
  static constexpr int LW = 32 / (N1 > N2 ? N1 : N2);  // lines per warp
  static constexpr int WARPS = 4;
  static constexpr int LINES = WARPS * LW;  // per CTA
  // complex values per line: the larger of the ordered line and the transpose
  // buffer, with the residue mod 8 that gives the step-2 reads (8 lanes = LW
  // lines x 8/LW rows of pitch P) distinct banks
  static constexpr int need = N1 * P > M + 1 ? N1 * P : M + 1;
  static constexpr int res = LW == 1 ? 0 : 8 / LW;
  static constexpr int LS = need + ((res - need) % 8 + 8) % 8;
  static constexpr size_t smem = sizeof(double2) * (2 * M + 1 + (size_t)LINES * LS);
  static constexpr int BLOCKS = (N1 > 16 || N2 > 16) ? 3 : 4;  // per SM: registers
};

// Step 1 of the warp's lines: ld(l, e) is element e of line l; the result is
// the transpose buffer [l][k1][j2] in buf (which ld may read: all lanes load
// before any stores).
template <int N1, int N2, bool INV, class Ld>
__device__ __forceinline__ void xw_step1(double2 *buf, const double2 *tw, int lane, Ld ld) {
  using W = XWarp<N1, N2>;
  const bool act = lane < W::LW * N2;
  const int l = act ? lane / N2 : 0, j2 = act ? lane - l * N2 : 0;
  double2 v[N1];
#pragma unroll
  for (int j1 = 0; j1 < N1; j1++) v[j1] = ld(l, j1 * N2 + j2);
  reg_fft<N1, INV>(v, tw, N2);
  __syncwarp();
  if (act) {
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) {
      double2 w = tw[j2 * k1];
      if (INV) w = cconj(w);
      buf[l * W::LS + k1 * W::P + j2] = k1 == 0 ? v[0] : cmul(v[k1], w);
    }
  }
  __syncwarp();
}

// Step 2 of a forward transform with the real output X[kx] = E + w^kx O formed
// in registers: lane (column k1, line l, l fastest) holds Z[k1 + N1 k2];
// Z[M - k1 - N1 k2] is element N2-1-k2 of column N1-k1, one shuffle away;
// columns 0 and N1/2 are their own partners.  st(kx, X) per retained lane of
// line lane % LW, kx = M from column 0.
template <int N1, int N2, class St>
__device__ __forceinline__ void xw_real_out(const double2 *buf, const double2 *tw, const double2 *tn,
                                            int lane, St st) {
  using W = XWarp<N1, N2>;
  constexpr int M = W::M, LW = W::LW;
  const int l = lane % LW, k1 = (lane / LW) % N1;
  double2 v[N2];
#pragma unroll
  for (int j2 = 0; j2 < N2; j2++) v[j2] = buf[l * W::LS + k1 * W::P + j2];
  reg_fft<N2, false>(v, tw, N1);
  const int partner = l + LW * ((N1 - k1) % N1);
  const bool self0 = k1 == 0, selfh = 2 * k1 == N1;
  const bool mine_out = lane < LW * N1;
#pragma unroll
  for (int k2 = 0; k2 < N2; k2++) {
    const double2 mine = v[N2 - 1 - k2];
    double2 other;
    other.x = __shfl_sync(0xffffffffu, mine.x, partner);
    other.y = __shfl_sync(0xffffffffu, mine.y, partner);
    const double2 zm = self0 ? v[(N2 - k2) % N2] : (selfh ? mine : other);
    const int kx = k1 + N1 * k2;
    const double2 zk = v[k2], zc = cconj(zm);
    const double2 e = make_double2(0.5 * (zk.x + zc.x), 0.5 * (zk.y + zc.y));
    const double2 d = csub(zk, zc);
    const double2 o = make_double2(0.5 * d.y, -0.5 * d.x);
    if (mine_out) st(kx, cadd(e, cmul(tn[kx], o)));
    if (self0 && k2 == 0 && mine_out) {  // kx = M from Z[0]
      const double2 z0c = cconj(zk);
      const double2 e0 = make_double2(0.5 * (zk.x + z0c.x), 0.5 * (zk.y + z0c.y));
      const double2 d0 = csub(zk, z0c);
      st(M, cadd(e0, cmul(tn[M], make_double2(0.5 * d0.y, -0.5 * d0.x))));
    }
  }
}

// The twiddle tables tw (M) and tn (M + 1) of a block of 128 threads, in two
// parts: the loads, and behind the loads of the lines the stores (the caller
// then synchronises the block).  In one part ahead of the lines they cost a
// memory latency of their own per block.
template <int N1, int N2>
struct XTables {
  static constexpr int M = N1 * N2, N = (2 * M + 1 + 127) / 128;
  double2 v[N];
  __device__ __forceinline__ void load(const double2 *__restrict__ twM, const double2 *__restrict__ twN) {
#pragma unroll
    for (int i = 0; i < N; i++) {
      const int t = threadIdx.x + 128 * i;
      if (t < 2 * M + 1) v[i] = t < M ? __ldg(twM + t) : __ldg(twN + t - M);
    }
  }
  __device__ __forceinline__ void store(double2 *tw) {
#pragma unroll
    for (int i = 0; i < N; i++) {
      const int t = threadIdx.x + 128 * i;
      if (t < 2 * M + 1) tw[t] = v[i];
    }
  }
};

// Spectrum of line lane % LW -> packed input of the inverse transform, in
// order in buf: Z[k] = E[k] + i O[k], E = h (X[k] + conj X[M-k]),
// O = h (X[k] - conj X[M-k]) conj(w^k), from ld(k) = X[k]; h = 1/2 for the
// normalised transform, 1 for the sum over the full spectrum.  All of a lane's
// pairs (up to 9) are loaded before `ready` (the tables' store and the block's
// barrier) is called.
template <int N1, int N2, class Ld, class Ready>
__device__ __forceinline__ void xw_pairs(double2 *buf, const double2 *tn, int lane, double h, Ld ld,
                                         Ready ready) {
  using W = XWarp<N1, N2>;
  constexpr int M = W::M;
  double2 *Z = buf + (lane % W::LW) * W::LS;
  constexpr int half = M / 2 + 1, STEP = 32 / W::LW, IT = (half + STEP - 1) / STEP;
  static_assert(IT <= 9, "one batch of pairs per lane");
  double2 a[IT], b[IT];
#pragma unroll
  for (int u = 0; u < IT; u++) {
    const int k = lane / W::LW + STEP * u;
    a[u] = b[u] = make_double2(0.0, 0.0);
    if (k < half) {
      a[u] = ld(k);
      b[u] = ld(M - k);
    }
  }
  ready();
#pragma unroll
  for (int u = 0; u < IT; u++) {
    const int k = lane / W::LW + STEP * u, k2 = M - k;
    if (k >= half) continue;
    const double2 bc = cconj(b[u]);
    const double2 e = cscale(cadd(a[u], bc), h);
    const double2 o = cmul(cscale(csub(a[u], bc), h), cconj(tn[k]));
    // k = 0 takes the real parts of X[0] and X[M] only
    Z[k] = k == 0 ? make_double2(h * (a[u].x + b[u].x), h * (a[u].x - b[u].x))
                  : make_double2(e.x - o.y, e.y + o.x);
    if (k != 0 && k2 != k) {
      const double2 ac = cconj(a[u]);
      const double2 e2 = cscale(cadd(b[u], ac), h);
      const double2 o2 = cmul(cscale(csub(b[u], ac), h), cconj(tn[k2]));
      Z[k2] = make_double2(e2.x - o2.y, e2.y + o2.x);
    }
  }
  __syncwarp();
}

// Step 2 of an inverse transform, scaled, back into buf in order.
template <int N1, int N2>
__device__ __forceinline__ void xw_ordered(double2 *buf, const double2 *tw, int lane, double sc) {
  using W = XWarp<N1, N2>;
  const int l = lane % W::LW, k1 = (lane / W::LW) % N1;
  double2 v[N2];
#pragma unroll
  for (int j2 = 0; j2 < N2; j2++) v[j2] = buf[l * W::LS + k1 * W::P + j2];
  reg_fft<N2, true>(v, tw, N1);
  __syncwarp();
  if (lane < W::LW * N1) {
#pragma unroll
    for (int k2 = 0; k2 < N2; k2++) buf[l * W::LS + k1 + N1 * k2] = cscale(v[k2], sc);
  }
  __syncwarp();
}

// the splits of nx/2 = N1 N2 with a compile-time x-kernel
#define FFT4_SPLITS(X) X(16, 24) X(16, 16) X(16, 12) X(16, 8) X(8, 12) X(8, 8) X(8, 6) X(8, 4)

}  // namespace dnsb
