// spectral4.cuh -- the Poisson transform kernels on the four-step engine.
//
// Same contracts as k_fftz / k_rfftx / k_irfftx in spectral.cuh (which
// remain the path for lengths without a specialised split), with the
// transforms of fft4.cuh: every element crosses shared memory once per
// transform, so these kernels stay bound by HBM traffic.
#pragma once
#include "fft4.cuh"
#include "pdl.cuh"
#include "spectral.cuh"
#include "xwarp.cuh"

namespace dnsb {

constexpr int F4_THREADS = 256;

// the splits of nz that k_fftz4 is compiled for: those below 128 (from there on the
// run-time split is the faster, launch_fftz)
#define FFTZ4_SPLITS(X) X(8, 12) X(8, 8) X(8, 6) X(8, 4)

// Complex FFT along z of L contiguous lines of S (n = N1*N2 = nz); INV
// scales by 1/nz.  Shared memory: transpose buffer + n twiddles.
template <int N1, int N2, bool INV>
__global__ void __launch_bounds__(F4_THREADS, 2) k_fftz4(Geo g, double2 *S, int L,
                                                         const double2 *__restrict__ twz, int dep) {
  constexpr int n = N1 * N2;
  extern __shared__ double2 smem[];
  double2 *buf = smem;
  double2 *tw = smem + fft4_buf<N1, N2>(L);
  const long long nlines = (long long)g.ny * g.nkx;
  const long long l0 = (long long)blockIdx.x * L;
  const int Lv = (int)min((long long)L, nlines - l0);
  pdl_trigger(dep);
  for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = twz[t];
  __syncthreads();
  pdl_wait(dep);
  double2 *src = S + l0 * n;
  const double sc = 1.0 / n;
  fft4_lines<N1, N2, INV>(
      [&](int l, int e) { return l < Lv ? src[l * n + e] : make_double2(0.0, 0.0); },
      [&](int l, int e, double2 v) {
        if (l < Lv) src[l * n + e] = INV ? cscale(v, sc) : v;
      },
      buf, L, tw);
}

// Forward: r = divergence of in0..in2, a ghost-free real array, the product
// of two, or a field's interior (INMODE, see k_rfftx), packed z[m] = r[2m] +
// i r[2m+1].  Step 2 forms the output X[k] in registers: its lane (line,
// column k1) holds Z[k1 + N1 k2]; Z[M - k1 - N1 k2] is element N2-1-k2 of
// column N1-k1, one shuffle away; columns 0 and N1/2 are their own partners.
template <int N1, int N2, int INMODE>
__global__ void __launch_bounds__(128, (XWarp<N1, N2>::BLOCKS))
    k_rfftx4(Geo g, double2 *__restrict__ S, const double *in0, const double *in1, const double *in2,
             const double2 *__restrict__ twM, const double2 *__restrict__ twN, int dep) {
  using W = XWarp<N1, N2>;
  constexpr int M = W::M, LW = W::LW, LS = W::LS;
  extern __shared__ double2 smem[];
  double2 *tw = smem, *tn = smem + M;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2 *buf = smem + 2 * M + 1 + warp * (LW * LS);
  const int ngrp = (g.nz + W::LINES - 1) / W::LINES;
  const int j = blockIdx.x / ngrp;
  const int k0 = (blockIdx.x - j * ngrp) * W::LINES + warp * LW;
  pdl_trigger(dep);
  XTables<N1, N2> tables;
  tables.load(twM, twN);
  const double rdyJ = __ldg(g.rdy + j + 1);
  pdl_wait(dep);
  const int sy = g.NX, sz = g.NX * g.NY;
  constexpr int IT = M / 16;  // values of a line per lane
  constexpr int B = IT % 6 == 0 ? 6 : IT % 4 == 0 ? 4 : IT % 3 == 0 ? 3 : 2;
#pragma unroll 1
  for (int l = 0; l < LW; l++) {
    if (k0 + l >= g.nz) break;
    double *z = reinterpret_cast<double *>(buf + l * LS);
    const long long ro = (long long)g.nx * (j + (long long)g.ny * (k0 + l));
    const int c0 = gidx(g, 1, j + 1, k0 + l + 1);
#pragma unroll 1
    for (int t = 0; t < IT; t += B) {
      double v[B];
#pragma unroll
      for (int u = 0; u < B; u++) {
        const int i = lane + 32 * (t + u);
        if constexpr (INMODE == RIN_REAL) {
          v[u] = in0[ro + i];
        } else if constexpr (INMODE == RIN_PRODUCT) {
          v[u] = in0[ro + i] * in1[ro + i];
        } else if constexpr (INMODE == RIN_FIELD) {
          v[u] = in0[c0 + i];
        } else {
          const int c = c0 + i;
          v[u] = (in0[c] - in0[c - 1]) * g.rdx + (in1[c] - in1[c - sy]) * rdyJ + (in2[c] - in2[c - sz]) * g.rdz;
        }
      }
#pragma unroll
      for (int u = 0; u < B; u++) z[lane + 32 * (t + u)] = v[u];
    }
  }
  tables.store(tw);
  __syncthreads();
  if (k0 >= g.nz) return;
  xw_step1<N1, N2, false>(buf, tw, lane, [&](int l, int e) { return buf[l * LS + e]; });
  const bool in = k0 + lane % LW < g.nz;
  double2 *dst = S + sidx(g, 0, j, k0 + lane % LW);
  const long long skx = (long long)g.nz * g.ny;
  xw_real_out<N1, N2>(buf, tw, tn, lane, [&](int kx, double2 v) {
    if (in) dst[kx * skx] = v;
  });
}

// Inverse (OUTMODE, see k_irfftx): each pair X[k], X[M-k] becomes Z[k],
// Z[M-k] on its way to shared memory, the two steps transform, and the
// ordered line leaves by whole 256-byte segments with its ghost images.
template <int N1, int N2, int OUTMODE>
__global__ void __launch_bounds__(128, (XWarp<N1, N2>::BLOCKS))
    k_irfftx4(Geo g, const double2 *S, double *__restrict__ out, const double2 *__restrict__ twM,
              const double2 *__restrict__ twN, int dep) {
  using W = XWarp<N1, N2>;
  constexpr int M = W::M, LW = W::LW, LS = W::LS;
  extern __shared__ double2 smem[];
  double2 *tw = smem, *tn = smem + M;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2 *buf = smem + 2 * M + 1 + warp * (LW * LS);
  const int ngrp = (g.nz + W::LINES - 1) / W::LINES;
  const int j = blockIdx.x / ngrp;
  const int k0 = (blockIdx.x - j * ngrp) * W::LINES + warp * LW;
  pdl_trigger(dep);
  XTables<N1, N2> tables;
  tables.load(twM, twN);
  pdl_wait(dep);
  const long long skx = (long long)g.nz * g.ny;
  const bool in = k0 + lane % LW < g.nz;
  const double2 *src = S + sidx(g, 0, j, k0 + lane % LW);
  xw_pairs<N1, N2>(buf, tn, lane, 0.5, [&](int k) { return in ? src[k * skx] : make_double2(0.0, 0.0); },
                   [&] {
                     tables.store(tw);
                     __syncthreads();
                   });
  if (k0 >= g.nz) return;
  xw_step1<N1, N2, true>(buf, tw, lane, [&](int l, int e) { return buf[l * LS + e]; });
  xw_ordered<N1, N2>(buf, tw, lane, 1.0 / M);
#pragma unroll 1
  for (int l = 0; l < LW; l++) {
    const int K = k0 + l + 1, J = j + 1;
    if (K > g.nz) break;
    const double *x = reinterpret_cast<const double *>(buf + l * LS);
    if constexpr (OUTMODE == ROUT_REAL) {
      double *row = out + (long long)g.nx * (j + (long long)g.ny * (K - 1));
#pragma unroll 4
      for (int i = lane; i < 2 * M; i += 32) row[i] = x[i];
    } else {
      double *row = out + gidx(g, 1, J, K);
#pragma unroll 4
      for (int i = lane; i < 2 * M; i += 32) row[i] = x[i];
      if (OUTMODE == ROUT_IMAGES) {
        // ghost images: whole lines on the box's edges, else the line's ends
        const bool edge = (J == 1) | (J >= g.ny - 1) | (K == 1) | (K == g.nz);
        for (int i = lane; i < 2 * M; i += 32)
          if (edge || i == 0 || i == 2 * M - 1)
            store_images_core(out, g.nx, g.ny, g.nz, g.NX, g.NY, g.wall, i + 1, J, K, x[i], STAG_P);
      }
    }
  }
}

}  // namespace dnsb
