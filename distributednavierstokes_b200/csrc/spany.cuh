// spany.cuh -- right-hand side and stage of the pseudo-spectral solver
// (spectral_rhs!, src/spectral/operators.jl:66-96; ifstage_kernel! and
// project_kernel!, src/spectral/step.jl:22-43, operators.jl:10-23) on
// transforms that carry the retained modes only.
//
// What bounds it is memory: n^3 fields and their half spectra.  Transforming
// the six velocity products one at a time over the full half spectrum reads
// every velocity four times, writes planes kx > kcut that are dropped, clears
// and scatters a full spectrum per component and passes over the state seven
// times per stage.  Here
//   inverse: y (from the compact state) -> z -> x, three components per
//     launch; a line's absent modes are zeros in registers, never memory;
//   forward: one x-kernel reads the three velocities once and writes the six
//     products' kx <= kcut; z and y (six spectra per launch, in place) keep
//     m of n lines;
//   stage: one kernel reads the six spectra and the state and writes the
//     projected state and the next start.
// 4 + 3 launches per stage instead of 42; passes (n^3 values of 8 bytes, kcut
// = n/3) 15 + 17 + 6 instead of about 90.  256^3 step 6.84 -> 4.03 ms, 128^3 1.49
// -> 0.57 ms, 32^3 0.71 -> 0.12 ms.
// Per launch at 256^3 (counters: DRAM bytes over time, share of the shared-memory
// and L1 pipe, of the FP64 pipe):
//   six products 417 us, 2.2 TB/s, 83 %, 35 %: the shared-memory pipe (each product
//     reads two velocities and crosses the buffer twice; 3 blocks of 72 KB, 12
//     warps per SM)
//   inverse x 219 us, 2.8 TB/s, 83 %, 30 %: the same pipe
//   inverse z 188 us, 2.1 TB/s, 32 %, 12 %: latency of the loads from the compact
//     lines (m values of 16 bytes, every other one off its 32-byte sector)
//   forward z 178 us, 4.8 TB/s; forward y 151, 3.8; inverse y 93, 2.8; stage 107, 5.3
// The kernels are those of fftany.cuh with other load and store maps.
#pragma once
#include "fftany.cuh"
#include "spany.h"
#include "xwarp.cuh"

namespace dnsb {

struct SpBufs {
  double2 *b[6];
};
struct SpFields {
  double *v[3];
};

// compact index of full index e, or -1 where the mode is not retained
__device__ __forceinline__ int sp_kept(int e, int n, int kcut, int m) {
  return e <= kcut ? e : e >= n - kcut ? e - n + m : -1;
}

// Inverse along y: the compact state (kx fastest) -> A[kzc + m (y + n kx)].
// A block takes 2 kx x 4 kz lines: 32-byte reads of the state, 64-byte
// writes of A.  grid (groups, 1, component)
template <int TIER>
__global__ void __launch_bounds__(FA_THREADS, fa_blocks(TIER))
    k_sp_yinv(SpCube s, int N1, int N2, const double2 *uh, SpBufs A, const double2 *__restrict__ twn, int dep) {
  constexpr int L = 8;
  extern __shared__ double2 smem[];
  const int n = s.n, h = s.kcut + 1, m = s.m;
  double2 *buf = smem, *tw = smem + L * n;
  pdl_trigger(dep);
  for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = twn[t];
  __syncthreads();
  pdl_wait(dep);
  const int gx = (h + 1) / 2;
  const int kx0 = (blockIdx.x % gx) * 2, kz0 = (blockIdx.x / gx) * 4;
  const double2 *src = uh + blockIdx.z * s.nc;
  double2 *dst = A.b[blockIdx.z];
  fa_dispatch<TIER>(N1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < L * N2; it += blockDim.x) {
      const int j2 = it / L, l = it - j2 * L;
      const int kx = kx0 + (l & 1), kz = kz0 + (l >> 1);
      const bool in = kx < h && kz < m;
      double2 v[R];
#pragma unroll
      for (int j1 = 0; j1 < R; j1++) {
        const int j = sp_kept(j1 * N2 + j2, n, s.kcut, m);
        v[j1] = in && j >= 0 ? src[kx + h * (j + (long long)m * kz)] : make_double2(0.0, 0.0);
      }
      reg_fft<R, true>(v, tw, N2);
#pragma unroll
      for (int k1 = 0; k1 < R; k1++)
        buf[(k1 * N2 + j2) * L + l] = k1 == 0 ? v[0] : cmul(v[k1], cconj(tw[j2 * k1]));
    }
  });
  __syncthreads();
  fa_dispatch<TIER>(N2, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < L * N1; it += blockDim.x) {
      const int k1 = it / L, q = it - k1 * L;
      const int l = (q >> 2) + 2 * (q & 3);  // four kz of one kx in a row
      const int kx = kx0 + (l & 1), kz = kz0 + (l >> 1);
      double2 v[R];
#pragma unroll
      for (int j2 = 0; j2 < R; j2++) v[j2] = buf[(k1 * N2 + j2) * L + l];
      reg_fft<R, true>(v, tw, N1);
      if (kx < h && kz < m) {
#pragma unroll
        for (int k2 = 0; k2 < R; k2++)
          dst[kz + (long long)m * ((k1 + N1 * k2) + (long long)n * kx)] = v[k2];
      }
    }
  });
}

// Along z, L lines per block; grid (groups, 1, field).
// Inverse: line A[.. m values] -> B[.. n values].  Forward, in place: a line
// of n values keeps its m retained modes at its front.
template <int TIER, bool INV>
__global__ void __launch_bounds__(FA_THREADS, fa_blocks(TIER))
    k_sp_z(SpCube s, int N1, int N2, int L, SpBufs in, SpBufs out, const double2 *__restrict__ twn, int dep) {
  extern __shared__ double2 smem[];
  const int n = s.n, m = s.m, P = fa_pitch(N2), LS = N1 * P;
  double2 *buf = smem, *tw = smem + L * LS;
  pdl_trigger(dep);
  for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = twn[t];
  __syncthreads();
  pdl_wait(dep);
  const long long nlines = (long long)n * (s.kcut + 1), l0 = (long long)blockIdx.x * L;
  const int Lv = (int)min((long long)L, nlines - l0);
  const double2 *src = in.b[blockIdx.z] + l0 * (INV ? m : n);
  double2 *dst = out.b[blockIdx.z] + l0 * n;
  fa_step1<TIER, INV>(N1, N2, P, LS, Lv, tw, buf, [&](int l, int e) {
    if constexpr (!INV) return src[(long long)l * n + e];
    const int q = sp_kept(e, n, s.kcut, m);
    return q >= 0 ? src[l * m + q] : make_double2(0.0, 0.0);
  });
  __syncthreads();
  fa_step2<TIER, INV>(N1, N2, P, LS, Lv, tw, buf, [&](int l, int e, double2 v) {
    if constexpr (INV) {
      dst[l * n + e] = v;
    } else {
      const int q = sp_kept(e, n, s.kcut, m);
      if (q >= 0) dst[l * n + q] = v;
    }
  });
}

// Inverse real FFT along x: kx <= kcut of B -> v, unnormalised (Z = (X[k] +
// conj X[M-k]) + i (X[k] - conj X[M-k]) conj(w^k): twice E + i O, which with
// the half-length transform is the sum over the full spectrum).
template <int TIER>
__global__ void __launch_bounds__(FA_THREADS, fa_blocks(TIER))
    k_sp_xinv(SpCube s, int N1, int N2, int L, SpBufs B, SpFields out, const double2 *__restrict__ twM,
              const double2 *__restrict__ twN, int dep) {
  extern __shared__ double2 smem[];
  const int n = s.n, M = N1 * N2, ls = M + 1, P = fa_pitch(N2), LS = N1 * P;
  double2 *buf = smem, *zb = buf + L * LS, *tw = zb + L * ls, *tn = tw + M;
  const int ngrp = (n + L - 1) / L;
  const int j = blockIdx.x / ngrp, k0 = (blockIdx.x - j * ngrp) * L;
  const int Lv = min(L, n - k0);
  pdl_trigger(dep);
  for (int t = threadIdx.x; t < M; t += blockDim.x) tw[t] = twM[t];
  for (int t = threadIdx.x; t <= M; t += blockDim.x) tn[t] = twN[t];
  __syncthreads();
  pdl_wait(dep);
  const double2 *src = B.b[blockIdx.z] + k0 + (long long)n * j;
  const long long skx = (long long)n * n;
  const int half = M / 2 + 1;
  constexpr int U = 4;  // pairs in flight per thread
  for (FaWalk w(L); w.q < half;) {
    double2 a[U], b[U];
    FaWalk v = w;
#pragma unroll
    for (int u = 0; u < U; u++) {
      a[u] = b[u] = make_double2(0.0, 0.0);
      if (w.q < half && w.r < Lv) {
        if (w.q <= s.kcut) a[u] = src[w.q * skx + w.r];
        if (M - w.q <= s.kcut) b[u] = src[(M - w.q) * skx + w.r];
      }
      w.next();
    }
#pragma unroll
    for (int u = 0; u < U; u++, v.next()) {
      const int k = v.q, l = v.r;
      if (k >= half || l >= Lv) continue;
      double2 *Z = zb + l * ls;
      if (k == 0) {  // the imaginary parts of kx = 0 and n/2 do not enter
        Z[0] = make_double2(a[u].x + b[u].x, a[u].x - b[u].x);
        continue;
      }
      const int k2 = M - k;
      const double2 bc = cconj(b[u]), e = cadd(a[u], bc), o = cmul(csub(a[u], bc), cconj(tn[k]));
      Z[k] = make_double2(e.x - o.y, e.y + o.x);
      if (k2 != k) {
        const double2 ac = cconj(a[u]), e2 = cadd(b[u], ac), o2 = cmul(csub(b[u], ac), cconj(tn[k2]));
        Z[k2] = make_double2(e2.x - o2.y, e2.y + o2.x);
      }
    }
  }
  __syncthreads();
  fa_step1<TIER, true>(N1, N2, P, LS, Lv, tw, buf, [&](int l, int e) { return zb[l * ls + e]; });
  __syncthreads();
  fa_step2<TIER, true>(N1, N2, P, LS, Lv, tw, buf,
                       [&](int l, int e, double2 v) { zb[l * ls + e] = v; });
  __syncthreads();
  double *dst = out.v[blockIdx.z];
  for (FaWalk w(M); w.q < Lv; w.next()) {
    const int l = w.q, e = w.r;
    *reinterpret_cast<double2 *>(dst + (long long)n * (j + (long long)n * (k0 + l)) + 2 * e) = zb[l * ls + e];
  }
}

// The same by warps, for the sides with a compile-time split of n/2 (xwarp.cuh);
// n = 512 and 768 have no run-time split along y and z, so that neither takes these
// transforms.
#define SP4_SPLITS(X) X(16, 12) X(16, 8) X(8, 12) X(8, 8) X(8, 6) X(8, 4)
template <int N1, int N2>
__global__ void __launch_bounds__(128, (XWarp<N1, N2>::BLOCKS))
    k_sp_xinv4(SpCube s, SpBufs B, SpFields out, const double2 *__restrict__ twM,
               const double2 *__restrict__ twN, int dep) {
  using W = XWarp<N1, N2>;
  constexpr int M = W::M, LW = W::LW, LS = W::LS;
  extern __shared__ double2 smem[];
  double2 *tw = smem, *tn = smem + M;
  const int n = s.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2 *buf = smem + 2 * M + 1 + warp * (LW * LS);
  const int ngrp = (n + W::LINES - 1) / W::LINES;
  const int j = blockIdx.x / ngrp;
  const int k0 = (blockIdx.x - j * ngrp) * W::LINES + warp * LW;
  pdl_trigger(dep);
  XTables<N1, N2> tables;
  tables.load(twM, twN);
  pdl_wait(dep);
  const bool in = k0 + lane % LW < n;
  const double2 *src = B.b[blockIdx.z] + (k0 + lane % LW) + (long long)n * j;
  const long long skx = (long long)n * n;
  xw_pairs<N1, N2>(buf, tn, lane, 1.0, [&](int k) {
    return in && k <= s.kcut ? src[k * skx] : make_double2(0.0, 0.0);
  }, [&] {
    tables.store(tw);
    __syncthreads();
  });
  if (k0 >= n) return;
  xw_step1<N1, N2, true>(buf, tw, lane, [&](int l, int e) { return buf[l * LS + e]; });
  xw_ordered<N1, N2>(buf, tw, lane, 1.0);
#pragma unroll 1
  for (int l = 0; l < LW && k0 + l < n; l++) {
    const double *x = reinterpret_cast<const double *>(buf + l * LS);
    double *row = out.v[blockIdx.z] + (long long)n * (j + (long long)n * (k0 + l));
#pragma unroll 4
    for (int i = lane; i < 2 * M; i += 32) row[i] = x[i];
  }
}

// The six products of L lines (row j, z = k0..): velocities read once into
// shared memory, then per product the half-length transform of its pairs and
// kx <= kcut of the real transform's output.
template <int TIER>
__global__ void __launch_bounds__(FA_THREADS, fa_blocks(TIER))
    k_sp_xprod(SpCube s, int N1, int N2, int L, SpFields v, SpBufs F, unsigned long long *vmax,
               const double2 *__restrict__ twM, const double2 *__restrict__ twN, int dep) {
  extern __shared__ double2 smem[];
  const int n = s.n, M = N1 * N2, ls = M + 1, P = fa_pitch(N2), LS = N1 * P;
  double2 *buf = smem, *res = buf + L * LS, *vel = res + L * ls, *tw = vel + 3 * L * M, *tn = tw + M;
  const int ngrp = (n + L - 1) / L;
  const int j = blockIdx.x / ngrp, k0 = (blockIdx.x - j * ngrp) * L;
  const int Lv = min(L, n - k0);
  pdl_trigger(dep);
  for (int t = threadIdx.x; t < M; t += blockDim.x) tw[t] = twM[t];
  for (int t = threadIdx.x; t <= M; t += blockDim.x) tn[t] = twN[t];
  pdl_wait(dep);
  double big = 0.0;
  for (FaWalk w(M); w.q < Lv; w.next()) {
    const int l = w.q, e = w.r;
    const long long o = (long long)n * (j + (long long)n * (k0 + l)) + 2 * e;
    double2 x[3];
#pragma unroll
    for (int c = 0; c < 3; c++) x[c] = *reinterpret_cast<const double2 *>(v.v[c] + o);
#pragma unroll
    for (int c = 0; c < 3; c++) vel[(c * L + l) * M + e] = x[c];
    big = fmax(big, fmax((fabs(x[0].x) + fabs(x[1].x)) + fabs(x[2].x),
                         (fabs(x[0].y) + fabs(x[1].y)) + fabs(x[2].y)));
  }
  if (vmax) {
    for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
    if ((threadIdx.x & 31) == 0) atomicMax(vmax, (unsigned long long)__double_as_longlong(big));
  }
  __syncthreads();
#pragma unroll 1
  for (int f = 0; f < 6; f++) {
    const int a = f < 3 ? f : f - 3, b = f < 3 ? f : (f == 5 ? 0 : f - 2);
    const double2 *va = vel + a * L * M, *vb = vel + b * L * M;
    fa_step1<TIER, false>(N1, N2, P, LS, Lv, tw, buf, [&](int l, int e) {
      const double2 x = va[l * M + e], y = vb[l * M + e];
      return make_double2(x.x * y.x, x.y * y.y);
    });
    __syncthreads();  // (also: everyone is past the previous product's reads of res)
    fa_step2<TIER, false>(N1, N2, P, LS, Lv, tw, buf,
                          [&](int l, int e, double2 z) { res[l * ls + e] = z; });
    __syncthreads();
    double2 *dst = F.b[f] + k0 + (long long)n * j;
    for (FaWalk w(L); w.q <= s.kcut; w.next()) {
      const int kx = w.q, l = w.r;
      if (l >= Lv) continue;
      const double2 zk = res[l * ls + kx], zc = cconj(res[l * ls + (kx == 0 ? 0 : M - kx)]);
      const double2 e = make_double2(0.5 * (zk.x + zc.x), 0.5 * (zk.y + zc.y));
      const double2 d = csub(zk, zc);
      const double2 o = make_double2(0.5 * d.y, -0.5 * d.x);
      dst[(long long)n * n * kx + l] = cadd(e, cmul(tn[kx], o));
    }
  }
}

// The same by warps: a warp holds its LW lines of the three velocities and one
// product's buffer; six products without a block barrier.
template <int N1, int N2>
constexpr size_t sp_xprod4_smem() {
  using W = XWarp<N1, N2>;
  return sizeof(double2) * (2 * W::M + 1 + (size_t)W::LINES * (W::LS + 3 * W::M));
}
template <int N1, int N2>
__global__ void __launch_bounds__(128, (XWarp<N1, N2>::BLOCKS))
    k_sp_xprod4(SpCube s, SpFields v, SpBufs F, unsigned long long *vmax, const double2 *__restrict__ twM,
                const double2 *__restrict__ twN, int dep) {
  using W = XWarp<N1, N2>;
  constexpr int M = W::M, LW = W::LW, LS = W::LS;
  extern __shared__ double2 smem[];
  double2 *tw = smem, *tn = smem + M;
  const int n = s.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2 *buf = smem + 2 * M + 1 + warp * (LW * (LS + 3 * M)), *vel = buf + LW * LS;
  const int ngrp = (n + W::LINES - 1) / W::LINES;
  const int j = blockIdx.x / ngrp;
  const int k0 = (blockIdx.x - j * ngrp) * W::LINES + warp * LW;
  pdl_trigger(dep);
  XTables<N1, N2> tables;
  tables.load(twM, twN);
  pdl_wait(dep);
  double big = 0.0;
#pragma unroll 1
  for (int l = 0; l < LW && k0 + l < n; l++) {
    const long long o = (long long)n * (j + (long long)n * (k0 + l));
#pragma unroll 2
    for (int e = lane; e < M; e += 32) {
      double2 x[3];
#pragma unroll
      for (int c = 0; c < 3; c++) x[c] = *reinterpret_cast<const double2 *>(v.v[c] + o + 2 * e);
#pragma unroll
      for (int c = 0; c < 3; c++) vel[(c * LW + l) * M + e] = x[c];
      big = fmax(big, fmax((fabs(x[0].x) + fabs(x[1].x)) + fabs(x[2].x),
                           (fabs(x[0].y) + fabs(x[1].y)) + fabs(x[2].y)));
    }
  }
  if (vmax) {
    for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
    if (lane == 0) atomicMax(vmax, (unsigned long long)__double_as_longlong(big));
  }
  tables.store(tw);
  __syncthreads();
  if (k0 >= n) return;
  const bool in = k0 + lane % LW < n;
  const long long at = (k0 + lane % LW) + (long long)n * j, skx = (long long)n * n;
#pragma unroll 1
  for (int f = 0; f < 6; f++) {
    const int a = f < 3 ? f : f - 3, b = f < 3 ? f : (f == 5 ? 0 : f - 2);
    const double2 *va = vel + a * LW * M, *vb = vel + b * LW * M;
    xw_step1<N1, N2, false>(buf, tw, lane, [&](int l, int e) {
      const double2 x = va[l * M + e], y = vb[l * M + e];
      return make_double2(x.x * y.x, x.y * y.y);
    });
    double2 *dst = F.b[f] + at;
    xw_real_out<N1, N2>(buf, tw, tn, lane, [&](int kx, double2 x) {
      if (in && kx <= s.kcut) dst[kx * skx] = x;
    });
    __syncwarp();  // the columns are read before the next product overwrites them
  }
}

// Forward along y of the retained kz, in place: column (kx, kzc) of n values
// (stride n) keeps its m retained modes at its front.  grid (groups, 1, field)
template <int TIER>
__global__ void __launch_bounds__(FA_THREADS, fa_blocks(TIER))
    k_sp_yfwd(SpCube s, int N1, int N2, int L, SpBufs F, const double2 *__restrict__ twn, int dep) {
  extern __shared__ double2 smem[];
  const int n = s.n, m = s.m;
  double2 *buf = smem, *tw = smem + L * n;
  const int ngrp = (m + L - 1) / L;
  const int kx = blockIdx.x / ngrp, k0 = (blockIdx.x - kx * ngrp) * L;
  pdl_trigger(dep);
  for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = twn[t];
  __syncthreads();
  pdl_wait(dep);
  double2 *line0 = F.b[blockIdx.z] + (long long)n * n * kx + k0;
  fa_dispatch<TIER>(N1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < L * N2; it += blockDim.x) {
      const int j2 = it / L, l = it - j2 * L;
      const bool in = k0 + l < m;
      double2 v[R];
#pragma unroll
      for (int j1 = 0; j1 < R; j1++)
        v[j1] = in ? line0[(long long)(j1 * N2 + j2) * n + l] : make_double2(0.0, 0.0);
      reg_fft<R, false>(v, tw, N2);
#pragma unroll
      for (int k1 = 0; k1 < R; k1++)
        buf[(k1 * N2 + j2) * L + l] = k1 == 0 ? v[0] : cmul(v[k1], tw[j2 * k1]);
    }
  });
  __syncthreads();
  fa_dispatch<TIER>(N2, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < L * N1; it += blockDim.x) {
      const int k1 = it / L, l = it - k1 * L;
      double2 v[R];
#pragma unroll
      for (int j2 = 0; j2 < R; j2++) v[j2] = buf[(k1 * N2 + j2) * L + l];
      reg_fft<R, false>(v, tw, N1);
      if (k0 + l < m) {
#pragma unroll
        for (int k2 = 0; k2 < R; k2++) {
          const int q = sp_kept(k1 + N1 * k2, n, s.kcut, m);
          if (q >= 0) line0[(long long)q * n + l] = v[k2];
        }
      }
    }
  });
}

// Stage (or right-hand side) from the six spectra.  A block takes 16 kx x 16
// kz at one ky: the spectra (kz fastest) cross shared memory into the state's
// order (kx fastest), 256-byte segments on both sides.
constexpr int SPS_T = 16;
template <bool RHS>
__global__ void __launch_bounds__(SPS_T *SPS_T)
    k_sp_stage(SpCube s, SpBufs F, double2 *uh, const double2 *start, double2 *next, double a, double b,
               double nudcdt, double dt, int dep) {
  __shared__ double2 tile[6][SPS_T][SPS_T + 1];
  pdl_trigger(dep);
  pdl_wait(dep);
  const int h = s.kcut + 1, m = s.m, n = s.n;
  const int jy = blockIdx.z, kx0 = blockIdx.x * SPS_T, kz0 = blockIdx.y * SPS_T;
  const int tx = threadIdx.x % SPS_T, ty = threadIdx.x / SPS_T;
  if (kx0 + ty < h && kz0 + tx < m) {
    const long long o = kz0 + tx + (long long)n * (jy + (long long)n * (kx0 + ty));
#pragma unroll
    for (int f = 0; f < 6; f++) tile[f][ty][tx] = F.b[f][o];
  }
  __syncthreads();
  const int kx = kx0 + tx, kzc = kz0 + ty;
  if (kx >= h || kzc >= m) return;
  const int ky = jy <= s.kcut ? jy : jy - m, kz = kzc <= s.kcut ? kzc : kzc - m;
  const double k1 = s.kfac * kx, k2 = s.kfac * ky, k3 = s.kfac * kz;
  const double n1 = (double)n, sc = 1.0 / (n1 * n1 * n1);
  double2 sg[6];
#pragma unroll
  for (int f = 0; f < 6; f++) sg[f] = cscale(tile[f][tx][ty], sc);
  // du_i = -i k_j sigma_ij with sigma = xx yy zz xy yz zx
  auto force = [](double ka, double2 x, double kb, double2 y, double kc, double2 z) {
    return make_double2((ka * x.y + kb * y.y) + kc * z.y, -((ka * x.x + kb * y.x) + kc * z.x));
  };
  const double2 d[3] = {force(k1, sg[0], k2, sg[3], k3, sg[5]), force(k2, sg[1], k1, sg[3], k3, sg[4]),
                        force(k3, sg[2], k1, sg[5], k2, sg[4])};
  const long long q = kx + h * (jy + (long long)m * kzc);
  if constexpr (RHS) {
#pragma unroll
    for (int c = 0; c < 3; c++) uh[c * s.nc + q] = d[c];
    return;
  }
  const double kk = k1 * k1 + k2 * k2 + k3 * k3;
  const double phi = exp(-nudcdt * kk);
  double2 w[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const double2 st = start[c * s.nc + q];
    w[c] = make_double2(phi * (st.x + a * dt * d[c].x), phi * (st.y + a * dt * d[c].y));
    if (next) next[c * s.nc + q] = make_double2(phi * (st.x + b * dt * d[c].x), phi * (st.y + b * dt * d[c].y));
  }
  double2 p = make_double2(0.0, 0.0);
  if (kk != 0)
    p = make_double2((k1 * w[0].x + k2 * w[1].x + k3 * w[2].x) / kk,
                     (k1 * w[0].y + k2 * w[1].y + k3 * w[2].y) / kk);
  uh[q] = make_double2(w[0].x - k1 * p.x, w[0].y - k1 * p.y);
  uh[s.nc + q] = make_double2(w[1].x - k2 * p.x, w[1].y - k2 * p.y);
  uh[2 * s.nc + q] = make_double2(w[2].x - k3 * p.x, w[2].y - k3 * p.y);
}

}  // namespace dnsb
