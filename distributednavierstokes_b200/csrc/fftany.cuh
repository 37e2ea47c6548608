// fftany.cuh -- the Poisson transform kernels for every line length
// N = N1 * N2 whose factors are register-resident transform sizes
// (FA_RADICES), with the split chosen at run time.
//
// The four-step transform of fft4.cuh is specialised per length at compile
// time, which covers eight lengths; every other one took the Stockham
// kernels (spectral.cuh), where a line crosses shared memory once per radix
// stage behind a barrier each.  Here each of the two register steps switches
// on its size once per block, so one kernel serves all lengths and a line
// still crosses shared memory once per transform.
//
// Index maps (n = j1 N2 + j2 input, k = k1 + N1 k2 output):
//   forward: thread (line, j2) transforms x[j1 N2 + j2] over j1, multiplies
//     by W_N^(j2 k1), writes [k1][j2]; thread (line, k1) transforms over j2
//     and holds X[k1 + N1 k2].
//   inverse of a spectrum held that way (y-solve): thread (line, k1) inverse
//     transforms over k2 in place, multiplies by W_N^(-j2 k1), writes back
//     [k1][j2]; thread (line, j2) inverse transforms over k1 and holds
//     x[j1 N2 + j2].  Forward, division and inverse cross shared memory
//     twice, where the Stockham form took 2 (stages) + 1 crossings.
//
// Measured on B200 against the Stockham kernels: a 100 x 75 x 90 implicit step
// 543 -> 386 us, 32^3 periodic 137 -> 98 us, an 8-step 96 x 72 x 80 solve 2569 ->
// 2149 us; lengths with a compile-time split keep it (spectral4.cuh), where
// index arithmetic on constants is cheaper.
//
// TIER bounds the register sizes a kernel can switch to (10, 16 or 25) so
// that short lines do not pay the register count of the long ones: blocks of
// at most 128 threads at 6, 4 and 3 per SM.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "fft4.cuh"
#include "pdl.cuh"

namespace dnsb {

#define FA_RADICES(X) \
  X(2) X(3) X(4) X(5) X(6) X(8) X(9) X(10) X(12) X(15) X(16) X(18) X(20) X(24) X(25)

constexpr int FA_THREADS = 128;
__host__ __device__ constexpr int fa_blocks(int tier) { return tier <= 10 ? 6 : tier <= 16 ? 4 : 3; }
__host__ __device__ constexpr int fa_pitch(int n2) { return n2 | 1; }

// t = tid, tid + nth, ... as (t / n, t % n) with one division for the loop
// (n is a run-time value: a division per element cost as much as its loads)
struct FaWalk {
  int q, r, n, dq, dr;
  __device__ __forceinline__ FaWalk(int n_) : n(n_) {
    q = threadIdx.x / n;
    r = threadIdx.x - q * n;
    dq = blockDim.x / n;
    dr = blockDim.x - dq * n;
  }
  __device__ __forceinline__ void next() {
    q += dq;
    r += dr;
    if (r >= n) {
      r -= n;
      q++;
    }
  }
};

// f(integral_constant<r>) for the register size r
template <int TIER, class F>
__device__ __forceinline__ void fa_dispatch(int r, F f) {
#define FA_CASE(R)                                                   \
  case R:                                                            \
    if constexpr (R <= TIER) f(std::integral_constant<int, R>());    \
    break;
  switch (r) {
    FA_RADICES(FA_CASE)
    default: break;  // not chosen by the host
  }
#undef FA_CASE
}

// x[j1 N2 + j2] over j1 -> buf(l, k1, j2): line-major layout, rows padded to
// an odd pitch (P), LS values per line
template <int TIER, bool INV, class Ld>
__device__ __forceinline__ void fa_step1(int N1, int N2, int P, int LS, int L, const double2 *tw,
                                         double2 *buf, Ld ld) {
  fa_dispatch<TIER>(N1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < L * N2; it += blockDim.x) {
      const int l = it / N2, j2 = it - l * N2;
      double2 v[R];
#pragma unroll
      for (int j1 = 0; j1 < R; j1++) v[j1] = ld(l, j1 * N2 + j2);
      reg_fft<R, INV>(v, tw, N2);
      double2 *row = buf + l * LS + j2;
#pragma unroll
      for (int k1 = 0; k1 < R; k1++) {
        double2 w = tw[j2 * k1];
        if (INV) w = cconj(w);
        row[k1 * P] = k1 == 0 ? v[0] : cmul(v[k1], w);
      }
    }
  });
}

// buf(l, k1, j2) over j2 -> st(l, k1 + N1 k2, value)
template <int TIER, bool INV, class St>
__device__ __forceinline__ void fa_step2(int N1, int N2, int P, int LS, int L, const double2 *tw,
                                         const double2 *buf, St st) {
  fa_dispatch<TIER>(N2, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < L * N1; it += blockDim.x) {
      const int l = it / N1, k1 = it - l * N1;
      const double2 *col = buf + l * LS + k1 * P;
      double2 v[R];
#pragma unroll
      for (int j2 = 0; j2 < R; j2++) v[j2] = col[j2];
      reg_fft<R, INV>(v, tw, N1);
#pragma unroll
      for (int k2 = 0; k2 < R; k2++) st(l, k1 + N1 * k2, v[k2]);
    }
  });
}

// Complex FFT along z of L contiguous lines of S, in place (k_fftz).  256^3: 46 us,
// DRAM at 0.69 of the copy rate, the shared-memory pipe 70 % busy.
template <int TIER, bool INV>
__global__ void __launch_bounds__(FA_THREADS, fa_blocks(TIER))
    k_fftz_any(int n, int N1, int N2, int L, long long nlines, double2 *S,
               const double2 *__restrict__ twz, int dep) {
  extern __shared__ double2 smem[];
  const int P = fa_pitch(N2), LS = N1 * P;
  double2 *buf = smem, *tw = smem + L * LS;
  pdl_trigger(dep);
  for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = twz[t];
  __syncthreads();
  pdl_wait(dep);
  const long long l0 = (long long)blockIdx.x * L;
  const int Lv = (int)min((long long)L, nlines - l0);
  double2 *src = S + l0 * n;
  const double sc = 1.0 / n;
  fa_step1<TIER, INV>(N1, N2, P, LS, Lv, tw, buf, [&](int l, int e) { return src[l * n + e]; });
  __syncthreads();
  fa_step2<TIER, INV>(N1, N2, P, LS, Lv, tw, buf, [&](int l, int e, double2 v) {
    src[l * n + e] = INV ? cscale(v, sc) : v;
  });
}

// Periodic y (k_yfourier): per block L consecutive kz of one kx with all ny
// rows.  Lines lie across threads (l fastest): L = 8 values of 16 bytes are
// one 128-byte segment, in memory and as one conflict-free shared-memory
// wavefront, so the buffer needs no padding.
// Bound by the latency of its loads at 16 warps per SM (128 registers): DRAM at 0.33
// of the copy rate, the FP64 pipe 31 % busy.  256^3 (16 x 16, L = 8): 170.6 us with
// the Stockham k_yfourier, 98 here (two passes at the copy rate: 41 us); 32^3: 6.8
// -> 5.8 us.
template <int TIER, int YMODE>
__global__ void __launch_bounds__(FA_THREADS, fa_blocks(TIER))
    k_y_any(Geo g, int N1, int N2, int L, double2 *S, const double2 *__restrict__ twy,
            const double *__restrict__ lam1, const double *__restrict__ lam2,
            const double *__restrict__ lam3, int dep) {
  extern __shared__ double2 smem[];
  const int n = g.ny;
  double2 *buf = smem, *tw = smem + L * n;  // buf[(k1 N2 + j2) L + l]
  const int ngrp = (g.nz + L - 1) / L;
  const int bid = gridDim.x - 1 - blockIdx.x;  // last kx plane first: still in L2 from the z-transform
  const int kx = bid / ngrp, k0 = (bid - kx * ngrp) * L;
  pdl_trigger(dep);
  for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = twy[t];
  __syncthreads();
  pdl_wait(dep);
  constexpr bool INV = YMODE == YF_INVERSE;
  const double sc = YMODE == YF_FORWARD ? 1.0 : 1.0 / n;
  double2 *line0 = S + sidx(g, kx, 0, k0);
  fa_dispatch<TIER>(N1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < L * N2; it += blockDim.x) {
      const int j2 = it / L, l = it - j2 * L;
      const bool in = k0 + l < g.nz;
      double2 v[R];
#pragma unroll
      for (int j1 = 0; j1 < R; j1++)
        v[j1] = in ? line0[(long long)(j1 * N2 + j2) * g.nz + l] : make_double2(0.0, 0.0);
      reg_fft<R, INV>(v, tw, N2);
#pragma unroll
      for (int k1 = 0; k1 < R; k1++) {
        double2 w = tw[j2 * k1];
        if (INV) w = cconj(w);
        buf[(k1 * N2 + j2) * L + l] = k1 == 0 ? v[0] : cmul(v[k1], w);
      }
    }
  });
  __syncthreads();
  const double l1 = YMODE == YF_SOLVE ? lam1[kx] : 0.0;
  fa_dispatch<TIER>(N2, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int it = threadIdx.x; it < L * N1; it += blockDim.x) {
      const int k1 = it / L, l = it - k1 * L;
      double2 *col = buf + (k1 * N2) * L + l;
      double2 v[R];
#pragma unroll
      for (int j2 = 0; j2 < R; j2++) v[j2] = col[j2 * L];
      reg_fft<R, INV>(v, tw, N1);
      if constexpr (YMODE == YF_SOLVE) {
        // divide by lambda (0 for the mean mode) and go back
        const double l3 = lam3[min(k0 + l, g.nz - 1)];
#pragma unroll
        for (int k2 = 0; k2 < R; k2++) {
          const double lam = (l1 + lam2[k1 + N1 * k2]) + l3;
          v[k2] = cscale(v[k2], lam == 0.0 ? 0.0 : sc / lam);
        }
        reg_fft<R, true>(v, tw, N1);
#pragma unroll
        for (int j2 = 0; j2 < R; j2++)
          col[j2 * L] = cmul(v[j2], cconj(tw[j2 * k1]));
      } else {
        if (k0 + l < g.nz) {
#pragma unroll
          for (int k2 = 0; k2 < R; k2++)
            line0[(long long)(k1 + N1 * k2) * g.nz + l] = INV ? cscale(v[k2], sc) : v[k2];
        }
      }
    }
  });
  if constexpr (YMODE == YF_SOLVE) {
    __syncthreads();
    fa_dispatch<TIER>(N1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
      for (int it = threadIdx.x; it < L * N2; it += blockDim.x) {
        const int j2 = it / L, l = it - j2 * L;
        double2 v[R];
#pragma unroll
        for (int k1 = 0; k1 < R; k1++) v[k1] = buf[(k1 * N2 + j2) * L + l];
        reg_fft<R, true>(v, tw, N2);
        if (k0 + l < g.nz) {
#pragma unroll
          for (int j1 = 0; j1 < R; j1++) line0[(long long)(j1 * N2 + j2) * g.nz + l] = v[j1];
        }
      }
    });
  }
}

// Real forward FFT along x (k_rfftx) of L lines (row j, kz = k0..): the
// input is staged by all threads, transformed at half length, and the real
// transform's output pass stores S(kx, j, k0 + l), l fastest.
template <int TIER, int INMODE>
__global__ void __launch_bounds__(FA_THREADS, fa_blocks(TIER))
    k_rfftx_any(Geo g, int N1, int N2, int L, double2 *__restrict__ S, const double *in0,
                const double *in1, const double *in2,
                const double2 *__restrict__ twM, const double2 *__restrict__ twN, int dep) {
  extern __shared__ double2 smem[];
  const int M = N1 * N2, ls = M + 1, P = fa_pitch(N2), LS = N1 * P;
  double2 *buf = smem, *res = buf + L * LS, *tw = res + L * ls, *tn = tw + M;
  const int ngrp = (g.nz + L - 1) / L;
  const int j = blockIdx.x / ngrp, k0 = (blockIdx.x - j * ngrp) * L;
  const int Lv = min(L, g.nz - k0);
  pdl_trigger(dep);
  for (int t = threadIdx.x; t < M; t += blockDim.x) tw[t] = twM[t];
  for (int t = threadIdx.x; t <= M; t += blockDim.x) tn[t] = twN[t];
  const long long sy = g.NX, sz = (long long)g.NX * g.NY;
  const int J = j + 1;
  const double rdyJ = __ldg(g.rdy + J);
  pdl_wait(dep);
  auto load = [&](int l, int m) {
    const int k = k0 + l;
    if constexpr (INMODE == RIN_REAL || INMODE == RIN_PRODUCT) {
      const long long ro = (long long)g.nx * (j + (long long)g.ny * k);
      double2 z = *reinterpret_cast<const double2 *>(in0 + ro + 2 * m);
      if constexpr (INMODE == RIN_PRODUCT) {
        const double2 w = *reinterpret_cast<const double2 *>(in1 + ro + 2 * m);
        z = make_double2(z.x * w.x, z.y * w.y);
      }
      return z;
    } else {
      const int c0 = gidx(g, 2 * m + 1, J, k + 1);
      if constexpr (INMODE == RIN_FIELD) return make_double2(in0[c0], in0[c0 + 1]);
      const double a0 = in0[c0 - 1], a1 = in0[c0], a2 = in0[c0 + 1];
      const double b0 = in1[c0], b1 = in1[c0 - sy];
      const double b2 = in1[c0 + 1], b3 = in1[c0 + 1 - sy];
      const double d0 = in2[c0], d1 = in2[c0 - sz];
      const double d2 = in2[c0 + 1], d3 = in2[c0 + 1 - sz];
      return make_double2((a1 - a0) * g.rdx + (b0 - b1) * rdyJ + (d0 - d1) * g.rdz,
                          (a2 - a1) * g.rdx + (b2 - b3) * rdyJ + (d2 - d3) * g.rdz);
    }
  };
  constexpr int B = 4;  // values in flight per thread
  for (FaWalk w(M); w.q < Lv;) {
    double2 z[B];
    int o[B];
#pragma unroll
    for (int u = 0; u < B; u++) {
      o[u] = w.q < Lv ? w.q * ls + w.r : -1;
      if (o[u] >= 0) z[u] = load(w.q, w.r);
      w.next();
    }
#pragma unroll
    for (int u = 0; u < B; u++)
      if (o[u] >= 0) res[o[u]] = z[u];
  }
  __syncthreads();
  fa_step1<TIER, false>(N1, N2, P, LS, Lv, tw, buf, [&](int l, int m) { return res[l * ls + m]; });
  __syncthreads();
  fa_step2<TIER, false>(N1, N2, P, LS, Lv, tw, buf,
                        [&](int l, int e, double2 v) { res[l * ls + e] = v; });
  __syncthreads();
  for (FaWalk w(L); w.q <= M; w.next()) {
    const int kx = w.q, l = w.r;
    if (l >= Lv) continue;
    const double2 zk = res[l * ls + (kx == M ? 0 : kx)];
    const double2 zc = cconj(res[l * ls + (kx == 0 ? 0 : M - kx)]);
    const double2 e = make_double2(0.5 * (zk.x + zc.x), 0.5 * (zk.y + zc.y));
    const double2 d = csub(zk, zc);
    const double2 o = make_double2(0.5 * d.y, -0.5 * d.x);
    S[sidx(g, kx, j, k0 + l)] = cadd(e, cmul(tn[kx], o));
  }
}

// Inverse real FFT along x (k_irfftx) of L lines: each pair X[k], X[M-k] is
// loaded together and turned into Z[k], Z[M-k] on its way to shared memory.
template <int TIER, int OUTMODE>
__global__ void __launch_bounds__(FA_THREADS, fa_blocks(TIER))
    k_irfftx_any(Geo g, int N1, int N2, int L, const double2 *S, double *__restrict__ out,
                 const double2 *__restrict__ twM, const double2 *__restrict__ twN, int dep) {
  extern __shared__ double2 smem[];
  const int M = N1 * N2, ls = M + 1, P = fa_pitch(N2), LS = N1 * P;
  double2 *buf = smem, *zb = buf + L * LS, *tw = zb + L * ls, *tn = tw + M;
  const int ngrp = (g.nz + L - 1) / L;
  const int j = blockIdx.x / ngrp, k0 = (blockIdx.x - j * ngrp) * L;
  const int Lv = min(L, g.nz - k0);
  pdl_trigger(dep);
  for (int t = threadIdx.x; t < M; t += blockDim.x) tw[t] = twM[t];
  for (int t = threadIdx.x; t <= M; t += blockDim.x) tn[t] = twN[t];
  __syncthreads();
  pdl_wait(dep);
  // Z[k] = E + i O, E = (X[k] + conj X[M-k])/2, O = (X[k] - conj X[M-k]) conj(w^k)/2
  const int half = M / 2 + 1;
  const double2 *src = S + sidx(g, 0, j, k0);
  const long long skx = (long long)g.nz * g.ny;
  constexpr int B = 4;  // pairs in flight per thread
  for (FaWalk w(L); w.q < half;) {
    double2 a[B], b[B];
    FaWalk v = w;
#pragma unroll
    for (int u = 0; u < B; u++) {
      a[u] = b[u] = make_double2(0.0, 0.0);
      if (w.q < half && w.r < Lv) {
        a[u] = src[w.q * skx + w.r];
        b[u] = src[(M - w.q) * skx + w.r];
      }
      w.next();
    }
#pragma unroll
    for (int u = 0; u < B; u++, v.next()) {
      const int k = v.q, l = v.r;
      if (k >= half || l >= Lv) continue;
      double2 *Z = zb + l * ls;
      if (k == 0) {
        Z[0] = make_double2(0.5 * (a[u].x + b[u].x), 0.5 * (a[u].x - b[u].x));
        continue;
      }
      const int k2 = M - k;
      const double2 bc = cconj(b[u]), e = cscale(cadd(a[u], bc), 0.5);
      const double2 o = cmul(cscale(csub(a[u], bc), 0.5), cconj(tn[k]));
      Z[k] = make_double2(e.x - o.y, e.y + o.x);
      if (k2 != k) {
        const double2 ac = cconj(a[u]), e2 = cscale(cadd(b[u], ac), 0.5);
        const double2 o2 = cmul(cscale(csub(b[u], ac), 0.5), cconj(tn[k2]));
        Z[k2] = make_double2(e2.x - o2.y, e2.y + o2.x);
      }
    }
  }
  __syncthreads();
  fa_step1<TIER, true>(N1, N2, P, LS, Lv, tw, buf, [&](int l, int m) { return zb[l * ls + m]; });
  __syncthreads();
  const double sc = 1.0 / M;
  const int J = j + 1;
  const bool row_edge = (J == 1) | (J >= g.ny - 1);
  // The output is put in order in shared memory and stored by whole rows.
  fa_step2<TIER, true>(N1, N2, P, LS, Lv, tw, buf,
                       [&](int l, int m, double2 z) { zb[l * ls + m] = cscale(z, sc); });
  __syncthreads();
  for (FaWalk w(M); w.q < Lv; w.next()) {
    const int l = w.q, m = w.r;
    const double2 z = zb[l * ls + m];
    const int K = k0 + l + 1;
    if constexpr (OUTMODE == ROUT_REAL) {
      double *row = out + (long long)g.nx * (j + (long long)g.ny * (K - 1));
      *reinterpret_cast<double2 *>(row + 2 * m) = z;
    } else {
      const int c0 = gidx(g, 2 * m + 1, J, K);
      out[c0] = z.x;
      out[c0 + 1] = z.y;
      if (OUTMODE == ROUT_IMAGES && (row_edge | (K == 1) | (K == g.nz) | (m == 0) | (m == M - 1))) {
        store_images_core(out, g.nx, g.ny, g.nz, g.NX, g.NY, g.wall, 2 * m + 1, J, K, z.x, STAG_P);
        store_images_core(out, g.nx, g.ny, g.nz, g.NX, g.NY, g.wall, 2 * m + 2, J, K, z.y, STAG_P);
      }
    }
  }
}

}  // namespace dnsb
