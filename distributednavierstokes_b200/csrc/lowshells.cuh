// lowshells.cuh -- the shell-clamp forcing of a periodic FV box for the
// lowest shells by direct partial Fourier sums instead of 3-D FFTs.
//
// shellforcing (src/spectral/forcing.jl:37-56) only touches the modes with
// floor(|k|) < nb, nb <= 4: at most 4 x 7 x 7 of the half spectrum.  Their
// coefficients u_hat(k) = sum_x u(x) e^{-i k.x} (the unnormalised FFT of the
// interior, as the transform path computes them) are formed separably:
//   1. per (y, z) line, the x-sums for kx = 0..KM (one read of the field; a
//      thread per line and component, the tile staged in shared memory);
//   2. the y-sums (ky = -KM..KM), then the z-sums (kz = -KM..KM), a thread per
//      row, output and part of the row (PARTS), the parts added in order;
//   3. one block: the shell energies (1/2 w |u_hat|^2 / N^2, w the rfft
//      double count; a warp per shell), the clamp factors f = sqrt(eref / E),
//      the corrections G(k) = (f(shell) - 1) u_hat(k) / N;
//   4. per block of 16 lines of one plane, the z- and y-sums of G back to
//      physical space (cooperatively, in shared memory), then
//      u += Re sum_kx w P(kx) e^{i kx x} per point with the periodic ghost
//      images.
// Two passes over each component instead of three forward and three
// inverse 3-D transforms.  KM = nb - 1 <= 3 and 2 KM < n in every direction.
// Every sum has a fixed order.  What bounded the first form was not memory:
// the x-sums spent 240 shuffles per line on reducing 12 complex partial sums,
// the correction formed each line's 12 plane sums on 12 lanes of its warp
// from 7 global loads and 14 integer remainders, the shell sums ran on one
// thread.  128^3, shells 1-2, before -> now: x-sums 32.0 -> 20.4, y 9.1 -> 8.4,
// z 4.3 -> 3.2, modes 16.1 -> 3.3, correction 56.5 -> 29.6 us.
#pragma once
#include "common.cuh"
#include "fft.cuh"
#include "pdl.cuh"

namespace dnsb {

constexpr int LS_KX = 4;             // kx = 0..3
constexpr int LS_KY = 7;             // ky, kz = -3..3
constexpr int LS_TILE = 1024;        // points per component of a block's tile of the x-sums
constexpr int LS_CLINES = 16;        // lines (one plane) per block of the correction

// the phases e^{+2 pi i r / n} = (cos, sin) for r = 0..n-1 of one direction,
// formed once per context (the expression the partial sums evaluated per
// point before)
__global__ void k_ls_phases(int n, double2 *__restrict__ ph) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    double sn, cs;
    sincospi(2.0 * (double)i / (double)n, &sn, &cs);
    ph[i] = make_double2(cs, sn);
  }
}

// e^{-2 pi i m / n} (sign -1) or e^{+2 pi i m / n} (sign +1) for integer m
// (|m| < 2^31, 32-bit reduction) from the direction's table
__device__ __forceinline__ double2 ls_phase_tab(int m, int n, double sign, const double2 *__restrict__ ph) {
  int r = m % n;
  if (r < 0) r += n;
  const double2 e = ph[r];
  return make_double2(e.x, sign * e.y);
}

// A[((c * (KM+1) + kx) * nz + (K-1)) * ny + (J-1)] = sum_i u_c(i, J, K) e^{-2 pi i kx i / nx}
// LINES lines per block, staged LS_TILE / LINES points at a time; a thread sums 32
// points of a line's tile, the 32 / LINES threads of a line are added at the end.
// A tile costs about 2 us at few blocks per SM, so few long lines want few tiles
// each: 32 lines a block, and 8 where those are less than two blocks per SM and a
// line fills the longer tile (512 x 16 x 16 34.0 -> 9.9 us, 512 x 64 x 64 35.4 ->
// 18.3, 256 x 32 x 32 18.2 -> 6.1).
template <int LINES>
__global__ void __launch_bounds__(128) k_ls_xsums(Geo g, CFields3 u, int KM, const double2 *__restrict__ xph,
                                                  double2 *__restrict__ A, int dep) {
  constexpr int ROWS = 3 * LINES, XT = LS_TILE / LINES, SEG = XT / 32;  // SEG warps side by side on a line
  static_assert(4 % SEG == 0 && ROWS * SEG == 96, "four warps load, 96 threads sum");
  __shared__ double tile[ROWS][XT + 1];
  __shared__ double2 ph[LS_KX][XT];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int line0 = blockIdx.x * LINES, nlines = g.ny * g.nz;
  const int l0 = warp / SEG, xs = 32 * (warp % SEG) + lane;    // loads: line l0, l0 + 4 / SEG, .., point xs
  const int row = tid % ROWS, part = tid / ROWS;               // sums: points 32 part ..
  // the first cell of each staged line
  __shared__ int first[LINES];
  if (tid < LINES) {
    const int line = min(line0 + tid, nlines - 1);
    first[tid] = gidx(g, 1, line % g.ny + 1, line / g.ny + 1);
  }
  pdl_trigger(dep);
  pdl_wait(dep);
  __syncthreads();
  double a0 = 0.0;
  double2 acc[LS_KX] = {};
  for (int x0 = 0; x0 < g.nx; x0 += XT) {
    const int x = x0 + xs;
    const bool in = x < g.nx;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double *f = c == 0 ? u.x : c == 1 ? u.y : u.z;
      double v[8];
#pragma unroll
      for (int r = 0; r < 8; r++) v[r] = in ? f[first[l0 + 4 / SEG * r] + x] : 0.0;
#pragma unroll
      for (int r = 0; r < 8; r++) tile[c * LINES + l0 + 4 / SEG * r][xs] = v[r];
    }
    if (warp < SEG) {
      const double2 e = in ? xph[x] : make_double2(1.0, 0.0);
      const double2 z1 = make_double2(e.x, -e.y), z2 = cmul(z1, z1);
      ph[1][xs] = z1;
      ph[2][xs] = z2;
      ph[3][xs] = cmul(z2, z1);
    }
    __syncthreads();
    if (tid < ROWS * SEG) {
      const double *t = &tile[row][32 * part];
      const double2(*e)[XT] = reinterpret_cast<const double2(*)[XT]>(&ph[0][32 * part]);
#pragma unroll 8
      for (int i = 0; i < 32; i++) {
        const double v = t[i];
        a0 += v;
#pragma unroll
        for (int kx = 1; kx < LS_KX; kx++) {
          acc[kx].x = fma(v, e[kx][i].x, acc[kx].x);
          acc[kx].y = fma(v, e[kx][i].y, acc[kx].y);
        }
      }
    }
    __syncthreads();
  }
  acc[0] = make_double2(a0, 0.0);
  if constexpr (SEG > 1) {  // the parts of a line, in order (the tile is free)
    double2(*sums)[LS_KX][ROWS] = reinterpret_cast<double2(*)[LS_KX][ROWS]>(&ph[0][0]);
    static_assert(sizeof(double2) * SEG * LS_KX * ROWS <= sizeof ph, "the parts' sums fit the phases");
    if (part > 0 && part < SEG) {
#pragma unroll
      for (int kx = 0; kx < LS_KX; kx++) sums[part][kx][row] = acc[kx];
    }
    __syncthreads();
#pragma unroll
    for (int q = 1; q < SEG; q++)
#pragma unroll
      for (int kx = 0; kx < LS_KX; kx++)
        if (part == 0) acc[kx] = cadd(acc[kx], sums[q][kx][row]);
  }
  if (part == 0 && line0 + row % LINES < nlines) {
    const int c = row / LINES, line = line0 + row % LINES;
#pragma unroll
    for (int kx = 0; kx < LS_KX; kx++)
      if (kx <= KM) A[(long long)(c * (KM + 1) + kx) * nlines + line] = acc[kx];
  }
}

// out[r W + q] = sum_i in[base(r) + i stride] e^{-2 pi i (q - KM) i / n}, with
// base(r) = (r / inner) outer + r % inner: the y-sums (rows of A: inner 1)
// and the z-sums (rows of B, k strided by W: inner W).  Thread (row, output
// q < W, part of the row): 8 rows in quarters for the many y-rows, one row in
// 32 parts for the at most 84 z-rows and for y-rows of 128 or more points too few
// to fill half the GPU (clamp of 40 x 250 x 16 46.5 -> 28-34 us, 16 x 512 x 16
// 44.5 -> 25.4, 64 x 256 x 64 64.8 -> 46.2).
constexpr int LS_STHREADS = 8 * LS_KY * 4;
template <int ROWS, int PARTS>
__global__ void __launch_bounds__(LS_STHREADS)
    k_ls_sums(int rows, int n, int inner, long long outer, int stride, const double2 *in, int KM,
              const double2 *__restrict__ ph, double2 *__restrict__ out, int dep) {
  const int W = 2 * KM + 1;
  static_assert(ROWS * PARTS * LS_KY == LS_STHREADS, "one thread per row, part and output");
  __shared__ double2 part[PARTS][ROWS][LS_KY];
  const int tid = threadIdx.x;
  const int q = tid % LS_KY, p = (tid / LS_KY) % PARTS, rl = tid / (LS_KY * PARTS);
  const int r = blockIdx.x * ROWS + rl;
  pdl_trigger(dep);
  pdl_wait(dep);
  if (r < rows && q < W) {
    const double2 *a = in + (r / inner) * outer + r % inner;
    const int per = (n + PARTS - 1) / PARTS, i0 = p * per, i1 = min(n, i0 + per);
    // phase index ky i mod n, advanced by ky mod n per term
    const int ky = q - KM, step = ky < 0 ? ky + n : ky;
    int m = (int)((long long)step * i0 % n);
    double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int i = i0; i < i1; i++) {
      acc = cadd(acc, cmul(a[(long long)i * stride], cconj(ph[m])));
      m += step;
      if (m >= n) m -= n;
    }
    part[p][rl][q] = acc;
  }
  __syncthreads();
  if (r < rows && q < W && p == 0) {
    double2 sum = part[0][rl][q];
    for (int i = 1; i < PARTS; i++) sum = cadd(sum, part[i][rl][q]);
    out[(long long)r * W + q] = sum;
  }
}

// floor(sqrt(k2)) for the small integers here
__device__ __forceinline__ int ls_shell(int k2) {
  int sh = (int)sqrtf((float)k2);
  while (sh * sh > k2) sh--;
  while ((sh + 1) * (sh + 1) <= k2) sh++;
  return sh;
}

// One block: the shell energies of the modes u_hat in Gm into E[0..nb), clamp
// factors into f, the corrections G = (f(shell) - 1) u_hat / N in place;
// eref[s] < 0 leaves shell s unforced.
__global__ void __launch_bounds__(256) k_ls_modes(Geo g, int KM, double2 *Gm, double *E,
                                                  const double *eref, double *f, int nb, int dep) {
  const int W = 2 * KM + 1, H = KM + 1;
  const double N = (double)g.nx * g.ny * g.nz;
  const int nM = 3 * H * W * W;
  __shared__ double em[3 * LS_KX * LS_KY * LS_KY];
  __shared__ signed char sm[3 * LS_KX * LS_KY * LS_KY];
  __shared__ double fs[LS_KX];
  pdl_trigger(dep);
  pdl_wait(dep);
  for (int t = threadIdx.x; t < nM; t += blockDim.x) {
    const int kzi = t % W, r = t / W;
    const int kx = (r / W) % H, ky = r % W - KM, kz = kzi - KM;
    const double2 a = Gm[t];
    em[t] = (kx > 0 ? 2.0 : 1.0) * (a.x * a.x + a.y * a.y) / 2 / (N * N);
    sm[t] = (signed char)ls_shell(kx * kx + ky * ky + kz * kz);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < nb) {
    double acc = 0.0;
    for (int t = lane; t < nM; t += 32) acc += sm[t] == warp ? em[t] : 0.0;
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      const double fac = (eref[warp] >= 0 && acc > 0) ? sqrt(eref[warp] / acc) : 1.0;
      E[warp] = acc;
      f[warp] = fac;
      fs[warp] = fac;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nM; t += blockDim.x)
    Gm[t] = cscale(Gm[t], sm[t] < nb ? (fs[sm[t]] - 1.0) / N : 0.0);
}

// u_c(i, J, K) += Re sum_{kx, ky, kz} w(kx) G e^{+2 pi i (kx i/nx + ky j/ny + kz k/nz)},
// then the periodic ghost images of the updated cells.  grid (groups of
// LS_CLINES rows, nz, parts of x): few long lines are split along x, 64 points a
// part at the least, into two blocks per SM (512 x 16 x 16 48.3 -> 9.4 us, 1024 x
// 16 x 16 94.1 -> 9.9; at 48^3 parts of 24 points were no faster)
__global__ void __launch_bounds__(256, 4) k_ls_correct(Geo g, Fields3 u, int KM, const double2 *Gm,
                                                    const double2 *__restrict__ xph,
                                                    const double2 *__restrict__ yph,
                                                    const double2 *__restrict__ zph, int dep) {
  const int W = 2 * KM + 1, H = KM + 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int k = blockIdx.y, j0 = blockIdx.x * LS_CLINES;
  __shared__ double2 Hz[3 * LS_KX * LS_KY];          // [c H + kx][ky]: sum over kz at this k
  __shared__ double2 P[LS_CLINES][3][LS_KX];         // sum over ky at each line, w(kx) applied
  pdl_trigger(dep);
  pdl_wait(dep);
  if (tid < 3 * H * W) {
    double2 a = make_double2(0.0, 0.0);
    for (int kzi = 0; kzi < W; kzi++)
      a = cadd(a, cmul(Gm[tid * W + kzi], ls_phase_tab((kzi - KM) * k, g.nz, 1.0, zph)));
    Hz[tid] = a;
  }
  __syncthreads();
  if (tid < LS_CLINES * 3 * LS_KX) {
    const int kx = tid % LS_KX, c = (tid / LS_KX) % 3, l = tid / (3 * LS_KX), j = j0 + l;
    double2 a = make_double2(0.0, 0.0);
    if (kx <= KM && j < g.ny) {
      for (int kyi = 0; kyi < W; kyi++)
        a = cadd(a, cmul(Hz[(c * H + kx) * W + kyi], ls_phase_tab((kyi - KM) * j, g.ny, 1.0, yph)));
      if (kx > 0) a = cscale(a, 2.0);
    }
    P[l][c][kx] = a;
  }
  __syncthreads();
  double *fc[3] = {u.x, u.y, u.z};
  for (int i = lane + 32 * blockIdx.z; i < g.nx; i += 32 * gridDim.z) {
    const double2 z1 = xph[i], z2 = cmul(z1, z1), z3 = cmul(z2, z1);
#pragma unroll
    for (int q = 0; q < LS_CLINES / 8; q++) {
      const int l = warp + 8 * q, J = j0 + l + 1;
      if (J > g.ny) continue;
      const int c0 = gidx(g, i + 1, J, k + 1);
      double v[3];
#pragma unroll
      for (int c = 0; c < 3; c++) v[c] = fc[c][c0];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double2 *p = P[l][c];
        const double d = p[0].x + ((p[1].x * z1.x - p[1].y * z1.y) +
                                   ((p[2].x * z2.x - p[2].y * z2.y) + (p[3].x * z3.x - p[3].y * z3.y)));
        fc[c][c0] = v[c] + d;
        if (img_edge(g, i + 1, J, k + 1))
          store_images_of(fc[c], g.nx, g.ny, g.nz, g.NX, g.NY, g.wall, i + 1, J, k + 1, v[c] + d, STAG_P);
      }
    }
  }
}

}  // namespace dnsb
