// cnn.cu -- the sub-filter-stress CNN closure: context, TMA tensor maps,
// the small kernels around the tensor-core convolutions (crops, packing,
// Adam, split-K reduction, loss) and the C ABI of include/dnsb_cnn.h.
//
// No counterpart in the reference (DistributedNavierStokes has no learned
// closure); its training pairs follow the reference's SFS sampler
// (src/spectral/les.jl:302-370).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/dnsb.h"
#include "../../include/dnsb_cnn.h"
#include "cnn.cuh"
#include "cnn_host.h"
#include "launch.h"
#include "pdl.cuh"

using namespace dnsb::cnn;

namespace {

constexpr int NL = 4;
constexpr int CIN[NL] = {3, 32, 32, 32};
constexpr int COUT[NL] = {32, 32, 32, 6};
constexpr int CICH[NL] = {2, 4, 4, 4};  // input chunks of 8 channels (3 -> 16 padded)
constexpr int COCH[NL] = {4, 4, 4, 2};  // output chunks (6 -> 16 padded)
constexpr int HALO = 4;
constexpr long LOSS_CAP = 1L << 18;     // loss history ring
constexpr unsigned WAIT_LIMIT = 1u << 21;   // polls of up to 1 us each
constexpr int MAX_SMEM = 227 * 1024;

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  });
  return fn;
}

// parameter offsets: per layer W[27][cout][cin] then b[cout]
struct Layout {
  long w[NL], b[NL], total;
  Layout() {
    long o = 0;
    for (int L = 0; L < NL; L++) {
      w[L] = o;
      o += 27L * COUT[L] * CIN[L];
      b[L] = o;
      o += COUT[L];
    }
    total = o;
  }
};
const Layout LAYOUT;

// element offsets (BF16) of the packed B operands of layer L: per (dz, dy)
// pair g and K chunk, the N = 3 x 8 NCH rows (dx, output channel) of 8 K
// values each, in the K-major core-matrix order of the convolution kernel
// (tap t = 3 g + dx; the transposed convolution reads tap 26 - t).
__host__ __device__ inline long pack_fwd(int L, int t, int co, int ci) {
  const int cich = L == 0 ? 2 : 4, coch = L == 3 ? 2 : 4;
  const int g = t / 3, dx = t % 3;
  return (((long)g * cich + ci / 8) * (3 * coch) + dx * coch + co / 8) * 64 + (co % 8) * 8 + ci % 8;
}
__host__ __device__ inline long pack_bwd(int L, int t, int co, int ci) {
  const int cich = L == 0 ? 2 : 4, coch = L == 3 ? 2 : 4;
  const int g = (26 - t) / 3, dx = (26 - t) % 3;
  return (((long)g * coch + co / 8) * (3 * cich) + dx * cich + ci / 8) * 64 + (ci % 8) * 8 + co % 8;
}

struct KernelLayout {  // passed by value to the element-wise kernels
  long w[NL], b[NL], total;
  int cin[NL], cout[NL];
};

KernelLayout kernel_layout() {
  KernelLayout k;
  for (int L = 0; L < NL; L++) {
    k.w[L] = LAYOUT.w[L];
    k.b[L] = LAYOUT.b[L];
    k.cin[L] = CIN[L];
    k.cout[L] = COUT[L];
  }
  k.total = LAYOUT.total;
  return k;
}

struct Packs {
  __nv_bfloat16 *f[NL];  // forward B operands
  __nv_bfloat16 *d[NL];  // transposed (backward-data) B operands, L >= 1
};

// the split-K partials of the four weight gradients (k_wgrad's layout)
struct Partials {
  const float *part[NL];
  int nsplit[NL];
};

// With `reduce` every parameter's gradient from the split-K partials of its
// layer, with `adam` the Adam update, and the BF16 packing of every weight.
// Work is numbered over quads of the partials' columns (dy, co), rows (dx, ci)
// fastest, so that a thread reads 16 bytes of each split and a warp 512; 8 threads share a quad's splits (each
// adds every 8th, the sums are added in order), seven loads in flight at once.
// An ordinary launch, as k_tail, k_crops and k_batch_in behind it are, and without a
// trigger: k_conv loads the weights ahead of its wait (test_dependent_launches.py).
// One launch at the step's end: as four reductions between the backward kernels
// (5.2 us each, ordinary launches that kept the next convolution from starting
// early) and an Adam launch (5.9 us, two double pow per thread) they were 27 us
// of a 545 us training step.  15 us for the 49 MB of the splits' sums, in one
// wave of blocks (26 us with 16 threads a quad and twice the blocks, 23 us with columns
// fastest in the partials).
constexpr int UP_PARTS = 8, UP_QUADS = 32;
__host__ __device__ inline int up_quads(int L, int cin) {  // of layer L: weights, then biases
  const int coch = L == 3 ? 2 : 4;
  return 3 * 3 * cin * (3 * 2 * coch) + 2 * coch;
}
__global__ void __launch_bounds__(UP_PARTS *UP_QUADS)
    k_update(const __grid_constant__ KernelLayout k, const __grid_constant__ Partials pt, int reduce, float *params,
             float *grads, float *m, float *v, int adam, float lr, const long long *step,
             const __grid_constant__ Packs packs) {
  __shared__ float corr[2];
  __shared__ float4 sums[UP_PARTS][UP_QUADS];
  const int tid = threadIdx.x;
  if (adam && tid < 2) {  // 1 - beta^(step + 1), by squaring
    double b = tid ? (double)0.999f : (double)0.9f, q = 1.0;
    for (unsigned long long n = (unsigned long long)*step + 1; n; n >>= 1, b *= b)
      if (n & 1) q *= b;
    corr[tid] = (float)(1.0 - q);
  }
  // quad -> layer, tap, ci, first co and its place in a split's partials
  struct Quad {
    int L, t, ci, co;  // t < 0: bias; L = NL: none
    long at;
  };
  auto locate = [&](int lq) {
    Quad q{NL, -1, 0, 0, 0};
    int r = blockIdx.x * UP_QUADS + lq;
    for (int L = 0; L < NL; L++) {
      const int n = up_quads(L, k.cin[L]);
      if (r >= n) {
        r -= n;
        continue;
      }
      const int cich = L == 0 ? 2 : 4, coch = L == 3 ? 2 : 4, cin = k.cin[L], N = 24 * coch, N4 = N / 4;
      q.L = L;
      if (r >= 9 * cin * N4) {
        q.co = 4 * (r - 9 * cin * N4);
        q.at = 128L * q.co + 4 * 24 * cich;
      } else {
        // rows fastest, as in the partials
        const int row = r % (3 * cin), n4 = r / (3 * cin) % N4, dz = r / (3 * cin * N4), dx = row / cin;
        q.ci = row - dx * cin;
        q.co = 4 * n4 % (8 * coch);
        q.t = (dz * 3 + 4 * n4 / (8 * coch)) * 3 + dx;
        q.at = ((long)(dz * N4 + n4) * 128 + 8 * cich * dx + q.ci) * 4;
      }
      break;
    }
    return q;
  };
  if (reduce) {
    const int lq = tid % UP_QUADS, part = tid / UP_QUADS;
    const Quad q = locate(lq);
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    if (q.L < NL) {
      const long stride = 3L * 128 * (24 * (q.L == 3 ? 2 : 4));
      const int ns = pt.nsplit[q.L];
      const float *src = pt.part[q.L] + q.at;
#pragma unroll 7
      for (int sp = part; sp < ns; sp += UP_PARTS) {
        const float4 x = *reinterpret_cast<const float4 *>(src + sp * stride);
        g.x += x.x;
        g.y += x.y;
        g.z += x.z;
        g.w += x.w;
      }
    }
    sums[part][lq] = g;
  }
  __syncthreads();
  // one thread per parameter
  if (tid >= 4 * UP_QUADS) return;
  const Quad q = locate(tid / 4);
  if (q.L == NL) return;
  const int L = q.L, co = q.co + tid % 4;
  if (co >= k.cout[L]) return;
  const bool bias = q.t < 0;
  const long p = bias ? k.b[L] + co : k.w[L] + ((long)q.t * k.cout[L] + co) * k.cin[L] + q.ci;
  float w = params[p], g;
  if (reduce) {
    g = 0.f;
#pragma unroll
    for (int i = 0; i < UP_PARTS; i++) g += reinterpret_cast<const float *>(&sums[i][tid / 4])[tid % 4];
    grads[p] = g;
  } else {
    g = grads[p];
  }
  if (adam) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mm = b1 * m[p] + (1.f - b1) * g;
    const float vv = b2 * v[p] + (1.f - b2) * g * g;
    m[p] = mm;
    v[p] = vv;
    w = w - lr * ((mm / corr[0]) / (sqrtf(vv / corr[1]) + eps));
    params[p] = w;
  }
  if (bias) return;
  const __nv_bfloat16 wb = __float2bfloat16_rn(w);
  packs.f[L][pack_fwd(L, q.t, co, q.ci)] = wb;
  if (L > 0) packs.d[L][pack_bwd(L, q.t, co, q.ci)] = wb;
}

__device__ inline unsigned long long splitmix(unsigned long long x) {
  unsigned long long z = x + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ inline uint4 chunk3(float a, float b, float c) {
  return make_uint4(pack2(make_float2(a, b)), pack2(make_float2(c, 0.f)), 0u, 0u);
}

// random crops of the dataset: input with its halo (chunk 0 of x0) and the
// normalised targets of the crop.  A block takes one z plane of one sample
// (grid z: 0 input, 1 targets), draws the crop once and walks its rows; one
// thread per voxel with the draw's four 64-bit remainders and the index
// divisions of its own took 22.2 us per batch of 8 crops of 32^3.
__global__ void __launch_bounds__(256) k_crops(const float *data, int nsnap, int n, int crop, int P,
                                               unsigned long long seed, const long long *step, uint4 *x0,
                                               float4 *tgt) {
  const int b = blockIdx.y, z = blockIdx.x;
  const bool tpart = blockIdx.z;
  const int side = tpart ? crop : P, h = tpart ? 0 : HALO;
  if (z >= side) return;
  __shared__ int draw[4];  // snapshot, origin x, y, z
  if (threadIdx.x < 4) {
    const unsigned long long key = (unsigned long long)(*step) * 64ull + (unsigned long long)b;
    const unsigned long long h0 = splitmix(seed ^ splitmix(4 * key));
    const int i = threadIdx.x;
    draw[i] = i == 0 ? (int)(h0 % (unsigned long long)nsnap)
                     : (int)(splitmix(h0 + i) % (unsigned long long)n);
  }
  __syncthreads();
  const long n3 = (long)n * n * n, P3 = (long)P * P * P;
  const float *s = data + (long)draw[0] * 9 * n3;
  // (crop + 2 HALO may exceed n: the box wraps as often as it takes)
  auto wrap = [n](int a) { return a >= 0 && a < n ? a : ((a % n) + n) % n; };
  const float *plane = s + (long)wrap(draw[3] + z - h) * n * n;
  for (int i = threadIdx.x; i < side * side; i += blockDim.x) {
    const int y = i / side, x = i - y * side;
    const int gi = wrap(draw[2] + y - h) * n + wrap(draw[1] + x - h);
    if (!tpart) {
      x0[(long)b * 2 * P3 + ((long)z * P + y) * P + x] = chunk3(plane[gi], plane[n3 + gi], plane[2 * n3 + gi]);
    } else {
      const long o = (((long)b * P + z) * P + y) * P + x;
      tgt[2 * o] = make_float4(plane[3 * n3 + gi], plane[4 * n3 + gi], plane[5 * n3 + gi], plane[6 * n3 + gi]);
      tgt[2 * o + 1] = make_float4(plane[7 * n3 + gi], plane[8 * n3 + gi], 0.f, 0.f);
    }
  }
}

// a caller batch: x [B][3][P^3], t [B][6][crop^3]
__global__ void k_batch_in(const float *x, const float *t, int B, int crop, int P, uint4 *x0,
                           float4 *tgt) {
  const long P3 = (long)P * P * P, c3 = (long)crop * crop * crop;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)B * (P3 + c3)) return;
  if (i < (long)B * P3) {
    const int b = (int)(i / P3);
    const long v = i % P3;
    const float *xb = x + (long)b * 3 * P3;
    x0[(long)b * 2 * P3 + v] = chunk3(xb[v], xb[P3 + v], xb[2 * P3 + v]);
  } else {
    const long r = i - (long)B * P3;
    const int b = (int)(r / c3);
    const long v = r % c3;
    const int x = (int)(v % crop), y = (int)((v / crop) % crop), z = (int)(v / ((long)crop * crop));
    const float *tb = t + (long)b * 6 * c3;
    const long o = (((long)b * P + z) * P + y) * P + x;
    tgt[2 * o] = make_float4(tb[v], tb[c3 + v], tb[2 * c3 + v], tb[3 * c3 + v]);
    tgt[2 * o + 1] = make_float4(tb[4 * c3 + v], tb[5 * c3 + v], 0.f, 0.f);
  }
}

// the periodic field with a halo of 4: from cell-centred values v[3][n^3]
// or from the staggered ghosted FV fields (the cell average of the two
// faces, operators.jl:71-72); scaled by in_scale
// grid (ceil(P / blockDim.x), P, P): x along the threads, y and z from the
// block (no division per voxel); the halo (HALO < n) wraps by one correction
__global__ void k_infer_in(const double *v, const double *ux, const double *uy, const double *uz,
                           int n, int P, const float *in_scale, uint4 *x0, int dep) {
  dnsb::pdl_wait(dep);
  dnsb::pdl_trigger(dep);  // past the wait, as the convolution reads the weights ahead of its own
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, z = blockIdx.z;
  if (x >= P) return;
  const long i = ((long)z * P + y) * P + x;
  auto wrap = [n](int a) { return a < 0 ? a + n : (a >= n ? a - n : a); };
  const int cx = wrap(x - HALO), cy = wrap(y - HALO), cz = wrap(z - HALO);
  double a, b, c;
  if (v) {
    const long n3 = (long)n * n * n, gi = ((long)cz * n + cy) * n + cx;
    a = v[gi];
    b = v[n3 + gi];
    c = v[2 * n3 + gi];
  } else {
    const long NX = n + 2, NY = n + 2;
    auto G = [&](int I, int J, int K) { return ((long)K * NY + J) * NX + I; };
    const int I = cx + 1, J = cy + 1, K = cz + 1;
    a = 0.5 * (ux[G(I - 1, J, K)] + ux[G(I, J, K)]);
    b = 0.5 * (uy[G(I, J - 1, K)] + uy[G(I, J, K)]);
    c = 0.5 * (uz[G(I, J, K - 1)] + uz[G(I, J, K)]);
  }
  x0[i] = chunk3((float)a * in_scale[0], (float)b * in_scale[1], (float)c * in_scale[2]);
}

// loss of the step (partials in a fixed order) into the history ring; the
// step counter advances when `advance`
__global__ void k_tail(const float *part, int nparts, float inv_count, float *hist, long long *step,
                       int advance) {
  __shared__ float sh[256];
  float s = 0.f;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) s += part[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    hist[*step % LOSS_CAP] = sh[0] * inv_count;
    if (advance) *step += 1;
  }
}

// ---------------------------------------------------------------- host --

struct Volume {
  int P = 0, B = 0, side = 0;  // side: crop (training) or field (inference)
  uint4 *in[NL] = {};          // input of layer L: x0 (2 chunks), h1..h3 (4)
  uint4 *z[3] = {};            // pre-activations of layers 1..3
  uint4 *gz[NL] = {};          // gradients of the layer outputs (training)
  float4 *tgt = nullptr;       // targets (training)
  CUtensorMap fwd[NL], bwd[NL], flatA[NL], flatB[NL];
  int Rf = 0, Rb = 0;          // patch rows of forward / transposed reads
  int subf = 1, subb = 1;      // 126-output sub-tiles per plane load (1-4), forward / transposed
  int Rw[NL] = {};             // weight gradient: rows per K-block
};

struct Prof {
  cudaEvent_t a, b;
  int kind;
  double flops;
};

}  // namespace

struct dnsb_cnn {
  int device = 0;
  cudaStream_t stream = nullptr;
  int nsm = 148;
  std::string err;
  std::vector<void *> allocs;
  long launches = 0;
  Volume tr, inf;
  bool have_tr = false, have_inf = false;
  float *params = nullptr, *grads = nullptr, *m = nullptr, *v = nullptr;
  Packs packs{};
  Partials parts{};            // of the last backward pass
  float *scales = nullptr;     // in[3] (pad 4), out[6]
  float *partial[NL] = {};
  long partial_n[NL] = {};
  float *loss_part = nullptr;
  int loss_nparts = 0, loss_nparts_used = 0;
  float *hist = nullptr;
  long long *step = nullptr;
  long h_steps = 0;
  int *deverr = nullptr;
  const float *data = nullptr;
  int nsnap = 0, ndata = 0;
  bool prof_on = false;
  std::vector<Prof> prof_pending;
  std::vector<cudaEvent_t> evpool;
  double prof_ms[4] = {}, prof_flops[4] = {};
  long prof_n[4] = {};
  unsigned long long serial = 0;  // creation number, unique in the process
  bool pdl = true;  // convolutions launched as programmatic dependents (DNSB_CNN_PDL=0: ordinary)
};

namespace dnsb_internal {

unsigned long long cnn_serial(const dnsb_cnn *c) { return c->serial; }
bool cnn_profiling(const dnsb_cnn *c) { return c->prof_on; }

}  // namespace dnsb_internal

namespace {

std::mutex g_err_mu;
std::string g_create_err;

int cfail(dnsb_cnn *c, int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (c) c->err = buf;
  else {
    std::lock_guard<std::mutex> l(g_err_mu);
    g_create_err = buf;
  }
  return code;
}

#define CC(c, call)                                                                             \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess)                                                                      \
      return cfail(c, DNSB_ECUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__,   \
                   __LINE__);                                                                   \
  } while (0)

template <typename T>
int dal(dnsb_cnn *c, T **p, size_t count) {
  void *q = nullptr;
  const size_t bytes = std::max<size_t>(count * sizeof(T), 16);
  if (cudaMalloc(&q, bytes) != cudaSuccess) {
    cudaGetLastError();
    return cfail(c, DNSB_ENOMEM, "cudaMalloc of %zu bytes failed", bytes);
  }
  c->allocs.push_back(q);
  CC(c, cudaMemset(q, 0, bytes));
  *p = (T *)q;
  return 0;
}

int ensure_dev(dnsb_cnn *c) {
  int d = -1;
  if (cudaGetDevice(&d) != cudaSuccess) return cfail(c, DNSB_ECUDA, "cudaGetDevice failed");
  if (d != c->device) CC(c, cudaSetDevice(c->device));
  return 0;
}

int deverr_check(dnsb_cnn *c) {
  int e = 0;
  CC(c, cudaMemcpy(&e, c->deverr, sizeof(int), cudaMemcpyDeviceToHost));
  if (e) {
    cudaMemset(c->deverr, 0, sizeof(int));
    return cfail(c, DNSB_ECUDA, "a tensor-core kernel's device-side wait ran out of its limit (code %d)", e);
  }
  return 0;
}

// patch rows of a tile of `sub` sub-tiles: offsets x0 + s + (dy + e) P + 126 sb
// + m, x0 < P, sb < sub, m < 128
int patch_rows(int P, int s, int e, int sub) {
  const long M = (long)(P - 1) + (long)(sub - 1) * TILE_OUT + (TILE_M - 1) + s + (long)(2 + e) * P;
  return (int)(M / P) + 1;
}

// The chunked-voxel tensors are described with 8-byte elements so that the
// innermost box dimension is a whole x-row (16 P bytes) or a whole run of
// positions (1 KB): TMA moves long rows instead of 16-byte pieces.  The
// copy is byte-exact (no conversion; out-of-bounds elements read as zero).
// Conv plane: dims {2P (x and 8 channels), P (y), P (z), chunks * B}, box
// {2P, R, 1, chunks} -> shared memory [chunk][row][x][16 B] (one ring slot).
// The weight gradient takes R rows of one box of all chunks, or of one.
int make_map_patch(dnsb_cnn *c, CUtensorMap *m, void *base, int P, int chunks, int B, int R, int boxch) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return cfail(c, DNSB_ECUDA, "cuTensorMapEncodeTiled is not available");
  if (2 * P > 256 || R > 256 || chunks > 256) return cfail(c, DNSB_EUNSUP, "TMA box beyond 256 (P %d, R %d)", P, R);
  const cuuint64_t dims[4] = {2ull * P, (cuuint64_t)P, (cuuint64_t)P, (cuuint64_t)chunks * B};
  const cuuint64_t strides[3] = {16ull * P, 16ull * P * P, 16ull * P * P * P};
  const cuuint32_t box[4] = {(cuuint32_t)(2 * P), (cuuint32_t)R, 1, (cuuint32_t)boxch};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT64, 4, base, dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cfail(c, DNSB_ECUDA, "cuTensorMapEncodeTiled (patch) failed: %d", (int)r);
  return 0;
}

constexpr int RING_MAX = 12, RING_GOOD = 6, RING_MIN = 4;
constexpr size_t CONV_EXTRA = CONV_BARS + CONV_XBUF + 1024;  // barriers, exchange, alignment slack

// shared memory of a convolution with the largest plane ring that fits
// (at most RING_MAX slots); 0 when not even RING_MIN slots fit
size_t conv_smem(int ci, int co, int P, int R, int *nslot, uint32_t *slot, uint32_t *stride,
                 uint32_t *wbytes) {
  *slot = (uint32_t)ci * R * P * 16;
  *stride = (*slot + 1023) & ~1023u;
  *wbytes = 27u * ci * co * 128;
  const long room = (long)MAX_SMEM - (long)*wbytes - (long)CONV_EXTRA;
  const int n = (int)std::min<long>(RING_MAX, room / (long)*stride);
  *nslot = n;
  if (n < RING_MIN) return 0;
  return (size_t)*wbytes + (size_t)n * *stride + CONV_EXTRA;
}

template <int CI, int CO, int MODE>
int setup_conv_attr(dnsb_cnn *c, size_t smem) {
  if (smem > (size_t)MAX_SMEM) return cfail(c, DNSB_EUNSUP, "convolution needs %zu bytes of shared memory", smem);
  // the limit is the kernel's, not this closure's: only ever raised, so that a
  // closure of another side in another thread cannot lower it before the launch
  CC(c, dnsb::raise_smem(c->device, k_conv<CI, CO, MODE>, smem));
  return 0;
}

// Weight gradient: shared memory of K-blocks of R rows, and the rows with the
// least estimated time: a plane's Do + 2 rows in ceil((Do + 2) / R) blocks of
// R P positions padded to 16, about 48 positions' worth of waits per block, and
// 15 % where the padding needs a copy per chunk.  Against every number of rows that
// fits (1 to 16; crops of 12 to 80, odd ones among them, 1 to 8 of them) the choice
// is within 0.5 % of the best step, 2.4 % at crop 12; with one row a step takes 1.4
// to 3.5 times as long.
size_t wgrad_smem(int P, int R, int ci, int co) {
  const size_t chunk = (size_t)((R * P + 15) / 16 * 16) * 16;
  return WG_PLANES * 3 * ci * chunk + WG_GRADS * 3 * co * chunk + 256 + 1024;
}
int wgrad_rows(int P, int Do, int ci, int co) {
  int best = 0;
  double least = 0;
  for (int r = 1; r <= std::min(16, P); r++) {
    if (wgrad_smem(P, r, ci, co) > (size_t)MAX_SMEM) break;
    const int kb = r * P, kbp = (kb + 15) / 16 * 16;
    const double t = (Do + 2 + r - 1) / r * (kbp + 48) * (kb == kbp ? 1.0 : 1.15);
    if (!best || t <= least) {
      best = r;
      least = t;
    }
  }
  return best;
}

int alloc_volume(dnsb_cnn *c, Volume &V, int side, int B, bool training) {
  V.side = side;
  V.B = B;
  V.P = side + 2 * HALO;
  const int P = V.P;
  const size_t P3 = (size_t)P * P * P;
  int rc;
  if ((rc = dal(c, &V.in[0], (size_t)B * 2 * P3))) return rc;
  for (int L = 1; L < NL; L++)
    if ((rc = dal(c, &V.in[L], (size_t)B * 4 * P3))) return rc;
  if (training) {
    for (int L = 0; L < 3; L++)
      if ((rc = dal(c, &V.z[L], (size_t)B * 4 * P3))) return rc;
    for (int L = 0; L < NL; L++)
      if ((rc = dal(c, &V.gz[L], (size_t)B * COCH[L] * P3))) return rc;
    if ((rc = dal(c, &V.tgt, (size_t)B * P3 * 2))) return rc;
  }
  // up to four 126-output sub-tiles per plane load (fewer copies per
  // output): the most whose wider patch fits the plane and a ring of
  // RING_GOOD planes, else of at least RING_MIN.  Three planes are in use; with
  // one or two ahead the next plane's copy is not done in time: an inference of
  // 64^3 takes 85.6 us with 3 sub-tiles and 4 slots, 84.8 with 2 and 5, 81.7 with 1
  // and 7 (training on 8 crops of 32^3 about the same, 358 and 360 us).  Where no
  // choice reaches RING_GOOD, one sub-tile has 5 slots and is no faster than two
  // with 4 (side 80 144.2 against 138.5 us, 84 162.6 and 159.2, 88 178.3 and 177.3).
  {
    auto most = [&](int s, int e) {
      for (int want : {RING_GOOD, RING_MIN})
        for (int sub = 4; sub > (want == RING_GOOD ? 0 : 1); sub--) {
          int ns;
          uint32_t sl, st, wb;
          const int r = patch_rows(P, s, e, sub);
          if (r <= P && conv_smem(4, 4, P, r, &ns, &sl, &st, &wb) && ns >= want) return sub;
        }
      return 1;
    };
    V.subf = most(0, 0);
    V.subb = most(-2, 1);
  }
  V.Rf = patch_rows(P, 0, 0, V.subf);
  V.Rb = patch_rows(P, -2, 1, V.subb);
  if (V.Rf > P || V.Rb > P)
    return cfail(c, DNSB_EUNSUP, "side %d too small: the 128-position tiles need %d patch rows", side,
                 std::max(V.Rf, V.Rb));
  {
    int ns;
    uint32_t sl, st, wb;
    if (!conv_smem(4, 4, P, V.Rf, &ns, &sl, &st, &wb) ||
        (training && !conv_smem(4, 4, P, V.Rb, &ns, &sl, &st, &wb)))
      return cfail(c, DNSB_EUNSUP, "side %d too large: a convolution's plane ring (%d slots of %u bytes) "
                   "does not fit in shared memory", side, RING_MIN, sl);
  }
  if (training)
    for (int L = 0; L < NL; L++)
      if (!(V.Rw[L] = wgrad_rows(P, P - 2 * (L + 1), CICH[L], COCH[L])))
        return cfail(c, DNSB_EUNSUP, "crop side %d: no weight-gradient block of whole rows fits", side);
  for (int L = 0; L < NL; L++) {
    if ((rc = make_map_patch(c, &V.fwd[L], V.in[L], P, CICH[L], B, V.Rf, CICH[L]))) return rc;
    if (training) {
      const bool whole = V.Rw[L] * P % 16 == 0;
      if ((rc = make_map_patch(c, &V.flatA[L], V.in[L], P, CICH[L], B, V.Rw[L], whole ? CICH[L] : 1))) return rc;
      if ((rc = make_map_patch(c, &V.flatB[L], V.gz[L], P, COCH[L], B, V.Rw[L], whole ? COCH[L] : 1))) return rc;
      if (L > 0 && (rc = make_map_patch(c, &V.bwd[L], V.gz[L], P, COCH[L], B, V.Rb, COCH[L]))) return rc;
    }
  }
  return 0;
}

cudaEvent_t ev_get(dnsb_cnn *c) {
  if (!c->evpool.empty()) {
    cudaEvent_t e = c->evpool.back();
    c->evpool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}

void prof_begin(dnsb_cnn *c, Prof &p, int kind, double flops) {
  p.kind = kind;
  p.flops = flops;
  if (!c->prof_on) return;
  p.a = ev_get(c);
  p.b = ev_get(c);
  cudaEventRecord(p.a, c->stream);
}
void prof_end(dnsb_cnn *c, Prof &p) {
  c->launches++;
  if (!c->prof_on) return;
  cudaEventRecord(p.b, c->stream);
  c->prof_pending.push_back(p);
}

int grid_for(dnsb_cnn *c, const void *kernel, size_t smem, long work, int threads) {
  int per = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess || per < 1) {
    cudaGetLastError();
    per = 1;
  }
  return (int)std::max<long>(1, std::min<long>(work, (long)c->nsm * per));
}

// one forward / transposed convolution of layer L on volume V
template <int CI, int CO, int MODE>
int run_conv(dnsb_cnn *c, Volume &V, int L, const CUtensorMap &map, bool transposed, uint4 *out,
             uint4 *zout, const uint4 *zin, double *infer_out, int kind) {
  ConvArgs a{};
  a.P = V.P;
  a.Pz = V.P;
  a.B = V.B;
  a.s = transposed ? -2 : 0;
  a.e = transposed ? 1 : 0;
  a.R = transposed ? V.Rb : V.Rf;
  a.sub = transposed ? V.subb : V.subf;
  // output box of a forward layer L: P - 2 (L+1); of the transposed one: the
  // box of layer L's input (layer L-1's output)
  a.Do = transposed ? V.P - 2 * L : V.P - 2 * (L + 1);
  a.spp = (a.Do * a.P + TILE_OUT - 1) / TILE_OUT;
  a.tpp = (a.spp + a.sub - 1) / a.sub;
  a.nsub = V.B * a.Do * a.spp;
  const size_t smem = conv_smem(CI, CO, a.P, a.R, &a.nslot, &a.slot_bytes, &a.slot_stride, &a.w_bytes);
  if (!smem) return cfail(c, DNSB_EUNSUP, "convolution plane ring does not fit in shared memory");
  a.wait_limit = WAIT_LIMIT;
  a.wpack = reinterpret_cast<const uint4 *>(transposed ? c->packs.d[L] : c->packs.f[L]);
  a.bias = c->params + LAYOUT.b[L];
  a.out = out;
  a.zout = zout;
  a.zin = zin;
  a.target = V.tgt;
  a.loss_scale = 2.0f / (float)((double)V.B * V.side * V.side * V.side * 6);
  a.loss_part = c->loss_part;
  a.infer_out = infer_out;
  a.oscale = c->scales + 4;
  a.err = c->deverr;
  int rc = setup_conv_attr<CI, CO, MODE>(c, smem);
  if (rc) return rc;
  const int grid = grid_for(c, (const void *)k_conv<CI, CO, MODE>, smem, a.nsub, CONV_THREADS);
  if (MODE == FWD_LOSS) {
    if (grid > c->loss_nparts) return cfail(c, DNSB_EUNSUP, "loss partials: grid %d > %d", grid, c->loss_nparts);
    c->loss_nparts_used = grid;
  }
  const double flops = 2.0 * 27 * CIN[L] * COUT[L] * V.B * pow((double)(V.P - 2 * (L + 1)), 3);
  Prof p;
  prof_begin(c, p, kind, flops);
  {
    // programmatic dependent launch (the kernel waits before any memory access)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(CONV_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = c->pdl ? 1 : 0;
    CC(c, cudaLaunchKernelEx(&cfg, k_conv<CI, CO, MODE>, map, a));
  }
  prof_end(c, p);
  CC(c, cudaGetLastError());
  return 0;
}

template <int CI, int CO>
int run_wgrad(dnsb_cnn *c, Volume &V, int L) {
  WgradArgs a{};
  a.P = V.P;
  a.B = V.B;
  a.Do = V.P - 2 * (L + 1);
  a.R = V.Rw[L];
  a.KB = a.R * V.P;
  a.KBp = (a.KB + 15) / 16 * 16;
  a.whole = a.KB == a.KBp;
  a.kpp = (a.Do + 2 + a.R - 1) / a.R;
  a.h_bytes = 3u * CI * a.KBp * 16;
  a.g_bytes = 3u * CO * a.KBp * 16;
  a.wait_limit = WAIT_LIMIT;
  a.err = c->deverr;
  const size_t smem = wgrad_smem(V.P, a.R, CI, CO);
  CC(c, dnsb::raise_smem(c->device, k_wgrad<CI, CO>, smem));
  a.nsplit = (int)std::max(1LL, std::min<long long>(c->nsm, (long long)a.B * a.kpp * a.Do));
  const long need = (long)a.nsplit * 3 * 128 * (3 * 8 * CO);
  if (need > c->partial_n[L]) return cfail(c, DNSB_EUNSUP, "weight-gradient partials: %ld > %ld", need, c->partial_n[L]);
  a.partial = c->partial[L];
  const double flops = 2.0 * 27 * CIN[L] * COUT[L] * V.B * pow((double)a.Do, 3);
  Prof p;
  prof_begin(c, p, 2, flops);
  {
    // programmatic dependent launch (the kernel waits before any memory access)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)a.nsplit);
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = c->pdl ? 1 : 0;
    CC(c, cudaLaunchKernelEx(&cfg, k_wgrad<CI, CO>, V.flatA[L], V.flatB[L], a));
  }
  prof_end(c, p);
  CC(c, cudaGetLastError());
  c->parts.part[L] = c->partial[L];
  c->parts.nsplit[L] = a.nsplit;
  return 0;
}

// forward with the loss, backward, weight gradients as split-K partials
// (training volume)
int fwd_bwd(dnsb_cnn *c) {
  Volume &V = c->tr;
  int rc;
  if ((rc = run_conv<2, 4, FWD_GELU>(c, V, 0, V.fwd[0], false, V.in[1], V.z[0], nullptr, nullptr, 0)) ||
      (rc = run_conv<4, 4, FWD_GELU>(c, V, 1, V.fwd[1], false, V.in[2], V.z[1], nullptr, nullptr, 0)) ||
      (rc = run_conv<4, 4, FWD_GELU>(c, V, 2, V.fwd[2], false, V.in[3], V.z[2], nullptr, nullptr, 0)) ||
      (rc = run_conv<4, 2, FWD_LOSS>(c, V, 3, V.fwd[3], false, V.gz[3], nullptr, nullptr, nullptr, 0)))
    return rc;
  if ((rc = run_wgrad<4, 2>(c, V, 3)) ||
      (rc = run_conv<2, 4, DGRAD>(c, V, 3, V.bwd[3], true, V.gz[2], nullptr, V.z[2], nullptr, 1)) ||
      (rc = run_wgrad<4, 4>(c, V, 2)) ||
      (rc = run_conv<4, 4, DGRAD>(c, V, 2, V.bwd[2], true, V.gz[1], nullptr, V.z[1], nullptr, 1)) ||
      (rc = run_wgrad<4, 4>(c, V, 1)) ||
      (rc = run_conv<4, 4, DGRAD>(c, V, 1, V.bwd[1], true, V.gz[0], nullptr, V.z[0], nullptr, 1)) ||
      (rc = run_wgrad<2, 4>(c, V, 0)))
    return rc;
  return 0;
}

// gradients from the partials (reduce), Adam (adam), BF16 weights
int update(dnsb_cnn *c, bool reduce, bool adam, float lr) {
  const KernelLayout kl = kernel_layout();
  Prof p;
  prof_begin(c, p, 3, 0);
  int quads = 0;
  for (int L = 0; L < NL; L++) quads += up_quads(L, CIN[L]);
  k_update<<<(quads + UP_QUADS - 1) / UP_QUADS, UP_PARTS * UP_QUADS, 0, c->stream>>>(
      kl, c->parts, reduce ? 1 : 0, c->params, c->grads, c->m, c->v, adam ? 1 : 0, lr, c->step, c->packs);
  prof_end(c, p);
  CC(c, cudaGetLastError());
  return 0;
}

int tail(dnsb_cnn *c, bool advance) {
  Volume &V = c->tr;
  const double count = (double)V.B * V.side * V.side * V.side * 6;
  Prof p;
  prof_begin(c, p, 3, 0);
  k_tail<<<1, 256, 0, c->stream>>>(c->loss_part, c->loss_nparts_used, (float)(1.0 / count), c->hist,
                                   c->step, advance ? 1 : 0);
  prof_end(c, p);
  CC(c, cudaGetLastError());
  return 0;
}

int prof_harvest(dnsb_cnn *c) {
  if (c->prof_pending.empty()) return 0;
  CC(c, cudaStreamSynchronize(c->stream));
  for (auto &p : c->prof_pending) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, p.a, p.b);
    c->prof_ms[p.kind] += ms;
    c->prof_n[p.kind] += 1;
    c->prof_flops[p.kind] += p.flops;
    c->evpool.push_back(p.a);
    c->evpool.push_back(p.b);
  }
  c->prof_pending.clear();
  return 0;
}

}  // namespace

extern "C" {

int dnsb_cnn_create(int device, void *stream, int batch, int crop, int nfield, dnsb_cnn **out) {
  if (!out) return cfail(nullptr, DNSB_EINVAL, "null output");
  *out = nullptr;
  if (batch < 0 || crop < 0 || nfield < 0 || (batch > 0) != (crop > 0) || (batch == 0 && nfield == 0))
    return cfail(nullptr, DNSB_EINVAL, "need batch > 0 with crop > 0, or nfield > 0");
  if (crop + 2 * HALO > 256 || nfield + 2 * HALO > 256 || batch > 64)
    return cfail(nullptr, DNSB_EUNSUP, "crop + 8 and nfield + 8 must be <= 256, batch <= 64");
  if (!encode_fn()) return cfail(nullptr, DNSB_ECUDA, "cuTensorMapEncodeTiled is not available");
  dnsb_cnn *c = new dnsb_cnn();
  static std::atomic<unsigned long long> created{0};
  c->serial = ++created;
  c->device = device;
  c->stream = (cudaStream_t)stream;
  {
    const char *e = getenv("DNSB_CNN_PDL");
    if (e && atoi(e) == 0) c->pdl = false;
  }
  auto bail = [&](int rc) {
    if (!c->err.empty()) cfail(nullptr, rc, "%s", c->err.c_str());
    dnsb_cnn_destroy(c);
    return rc;
  };
  if (cudaSetDevice(device) != cudaSuccess) return bail(cfail(c, DNSB_ECUDA, "cudaSetDevice(%d) failed", device));
  int major = 0;
  cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device);
  if (major < 10) return bail(cfail(c, DNSB_EUNSUP, "the tensor-core kernels need sm_100 (compute capability %d)", major));
  cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, device);
  int rc;
  if ((rc = dal(c, &c->params, LAYOUT.total)) || (rc = dal(c, &c->grads, LAYOUT.total)) ||
      (rc = dal(c, &c->m, LAYOUT.total)) || (rc = dal(c, &c->v, LAYOUT.total)) ||
      (rc = dal(c, &c->scales, 16)) || (rc = dal(c, &c->hist, LOSS_CAP)) ||
      (rc = dal(c, &c->step, 1)) || (rc = dal(c, &c->deverr, 4)))
    return bail(rc);
  for (int L = 0; L < NL; L++) {
    if ((rc = dal(c, &c->packs.f[L], 27L * CICH[L] * COCH[L] * 64))) return bail(rc);
    if (L > 0 && (rc = dal(c, &c->packs.d[L], 27L * CICH[L] * COCH[L] * 64))) return bail(rc);
  }
  const float ones[16] = {1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1};
  if (cudaMemcpy(c->scales, ones, sizeof ones, cudaMemcpyHostToDevice) != cudaSuccess)
    return bail(cfail(c, DNSB_ECUDA, "scale upload failed"));
  if (batch > 0) {
    if ((rc = alloc_volume(c, c->tr, crop, batch, true))) return bail(rc);
    c->have_tr = true;
    for (int L = 0; L < NL; L++) {
      c->partial_n[L] = (long)c->nsm * 3 * 128 * 3 * 8 * COCH[L];
      if ((rc = dal(c, &c->partial[L], c->partial_n[L]))) return bail(rc);
    }
  }
  c->loss_nparts = 2 * c->nsm + 8;
  if ((rc = dal(c, &c->loss_part, c->loss_nparts))) return bail(rc);
  if (nfield > 0) {
    if ((rc = alloc_volume(c, c->inf, nfield, 1, false))) return bail(rc);
    c->have_inf = true;
  }
  *out = c;
  return 0;
}

void dnsb_cnn_destroy(dnsb_cnn *c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  else cudaDeviceSynchronize();
  for (auto &p : c->prof_pending) {
    cudaEventDestroy(p.a);
    cudaEventDestroy(p.b);
  }
  for (auto e : c->evpool) cudaEventDestroy(e);
  for (void *p : c->allocs) cudaFree(p);
  delete c;
}

const char *dnsb_cnn_last_error(const dnsb_cnn *c) {
  if (c) return c->err.c_str();
  std::lock_guard<std::mutex> l(g_err_mu);
  return g_create_err.c_str();
}

int dnsb_cnn_set_stream(dnsb_cnn *c, void *stream) {
  if (!c) return DNSB_EINVAL;
  c->stream = (cudaStream_t)stream;
  return 0;
}

int dnsb_cnn_sync(dnsb_cnn *c) {
  if (!c) return DNSB_EINVAL;
  int rc;
  if ((rc = ensure_dev(c))) return rc;
  CC(c, cudaStreamSynchronize(c->stream));
  return deverr_check(c);
}

long dnsb_cnn_launch_count(const dnsb_cnn *c) { return c ? c->launches : 0; }

int dnsb_cnn_param_count(const dnsb_cnn *) { return (int)LAYOUT.total; }

int dnsb_cnn_set_params(dnsb_cnn *c, const float *params) {
  if (!c || !params) return c ? cfail(c, DNSB_EINVAL, "null params") : DNSB_EINVAL;
  int rc;
  if ((rc = ensure_dev(c))) return rc;
  CC(c, cudaMemcpyAsync(c->params, params, LAYOUT.total * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  CC(c, cudaMemsetAsync(c->m, 0, LAYOUT.total * sizeof(float), c->stream));
  CC(c, cudaMemsetAsync(c->v, 0, LAYOUT.total * sizeof(float), c->stream));
  CC(c, cudaMemsetAsync(c->step, 0, sizeof(long long), c->stream));
  c->h_steps = 0;
  if ((rc = update(c, false, false, 0.f))) return rc;
  CC(c, cudaStreamSynchronize(c->stream));
  return 0;
}

int dnsb_cnn_init(dnsb_cnn *c, unsigned long long seed) {
  if (!c) return DNSB_EINVAL;
  std::vector<float> h(LAYOUT.total);
  for (int L = 0; L < NL; L++) {
    const double bound = 1.0 / std::sqrt(27.0 * CIN[L]);
    for (long i = LAYOUT.w[L]; i < LAYOUT.w[L] + 27L * COUT[L] * CIN[L] + COUT[L]; i++) {
      unsigned long long z = seed + (unsigned long long)i + 0x9E3779B97F4A7C15ull;
      z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
      z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
      z ^= z >> 31;
      const double u = ((double)(z >> 11) + 0.5) * 0x1.0p-53;
      h[i] = (float)((2 * u - 1) * bound);
    }
  }
  return dnsb_cnn_set_params(c, h.data());
}

int dnsb_cnn_get_params(dnsb_cnn *c, float *params) {
  if (!c || !params) return c ? cfail(c, DNSB_EINVAL, "null params") : DNSB_EINVAL;
  int rc;
  if ((rc = ensure_dev(c))) return rc;
  CC(c, cudaMemcpyAsync(params, c->params, LAYOUT.total * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
  CC(c, cudaStreamSynchronize(c->stream));
  return deverr_check(c);
}

int dnsb_cnn_set_scales(dnsb_cnn *c, const float *in3, const float *out6) {
  if (!c || !in3 || !out6) return c ? cfail(c, DNSB_EINVAL, "null scales") : DNSB_EINVAL;
  int rc;
  if ((rc = ensure_dev(c))) return rc;
  float h[16] = {in3[0], in3[1], in3[2], 1.f, out6[0], out6[1], out6[2], out6[3], out6[4], out6[5]};
  CC(c, cudaMemcpyAsync(c->scales, h, sizeof h, cudaMemcpyHostToDevice, c->stream));
  CC(c, cudaStreamSynchronize(c->stream));
  return 0;
}

int dnsb_cnn_set_dataset(dnsb_cnn *c, const float *data, int nsnap, int n) {
  if (!c || !data || nsnap < 1 || n < 1) return c ? cfail(c, DNSB_EINVAL, "bad dataset") : DNSB_EINVAL;
  c->data = data;
  c->nsnap = nsnap;
  c->ndata = n;
  return 0;
}

int dnsb_cnn_train(dnsb_cnn *c, int nsteps, float lr, unsigned long long seed) {
  if (!c) return DNSB_EINVAL;
  if (!c->have_tr) return cfail(c, DNSB_EINVAL, "no training geometry (batch = 0)");
  if (!c->data) return cfail(c, DNSB_EINVAL, "no dataset");
  if (nsteps < 0 || !(lr > 0)) return cfail(c, DNSB_EINVAL, "need nsteps >= 0, lr > 0");
  int rc;
  if ((rc = ensure_dev(c))) return rc;
  Volume &V = c->tr;
  for (int s = 0; s < nsteps; s++) {
    Prof p;
    prof_begin(c, p, 3, 0);
    k_crops<<<dim3(V.P, V.B, 2), 256, 0, c->stream>>>(c->data, c->nsnap, c->ndata, V.side, V.P, seed,
                                                      c->step, V.in[0], V.tgt);
    prof_end(c, p);
    CC(c, cudaGetLastError());
    if ((rc = fwd_bwd(c)) || (rc = update(c, true, true, lr)) || (rc = tail(c, true))) return rc;
    c->h_steps++;
  }
  return 0;
}

int dnsb_cnn_steps(dnsb_cnn *c, long *steps) {
  if (!c || !steps) return DNSB_EINVAL;
  int rc;
  if ((rc = ensure_dev(c))) return rc;
  long long s = 0;
  CC(c, cudaMemcpyAsync(&s, c->step, sizeof s, cudaMemcpyDeviceToHost, c->stream));
  CC(c, cudaStreamSynchronize(c->stream));
  *steps = (long)s;
  return deverr_check(c);
}

int dnsb_cnn_losses(dnsb_cnn *c, float *out, long first, long count) {
  if (!c || !out || first < 0 || count < 0) return c ? cfail(c, DNSB_EINVAL, "bad range") : DNSB_EINVAL;
  long steps = 0;
  int rc;
  if ((rc = dnsb_cnn_steps(c, &steps))) return rc;
  if (first + count > steps || first < steps - LOSS_CAP)
    return cfail(c, DNSB_EINVAL, "losses %ld..%ld not held (steps %ld, history %ld)", first,
                 first + count, steps, LOSS_CAP);
  for (long i = 0; i < count;) {
    const long s = (first + i) % LOSS_CAP;
    const long n = std::min(count - i, LOSS_CAP - s);
    CC(c, cudaMemcpy(out + i, c->hist + s, n * sizeof(float), cudaMemcpyDeviceToHost));
    i += n;
  }
  return 0;
}

int dnsb_cnn_batch(dnsb_cnn *c, const float *x, const float *t, int nadam, float lr, float *loss_out,
                   float *grads_out) {
  if (!c || !x || !t || nadam < 0) return c ? cfail(c, DNSB_EINVAL, "bad argument") : DNSB_EINVAL;
  if (!c->have_tr) return cfail(c, DNSB_EINVAL, "no training geometry (batch = 0)");
  if (nadam > 0 && !(lr > 0)) return cfail(c, DNSB_EINVAL, "need lr > 0");
  int rc;
  if ((rc = ensure_dev(c))) return rc;
  Volume &V = c->tr;
  const long P3 = (long)V.P * V.P * V.P, c3 = (long)V.side * V.side * V.side;
  const long work = (long)V.B * (P3 + c3);
  Prof p;
  prof_begin(c, p, 3, 0);
  k_batch_in<<<(unsigned)((work + 255) / 256), 256, 0, c->stream>>>(x, t, V.B, V.side, V.P, V.in[0], V.tgt);
  prof_end(c, p);
  CC(c, cudaGetLastError());
  for (int i = 0; i < std::max(1, nadam); i++) {
    if ((rc = fwd_bwd(c)) || (rc = update(c, true, false, 0.f))) return rc;
    if (i == 0) {
      if ((rc = tail(c, false))) return rc;
      if (grads_out)
        CC(c, cudaMemcpyAsync(grads_out, c->grads, LAYOUT.total * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
      if (loss_out) {
        CC(c, cudaStreamSynchronize(c->stream));
        long long s = 0;
        CC(c, cudaMemcpy(&s, c->step, sizeof s, cudaMemcpyDeviceToHost));
        CC(c, cudaMemcpy(loss_out, c->hist + s % LOSS_CAP, sizeof(float), cudaMemcpyDeviceToHost));
      }
    }
    if (nadam > 0) {
      if ((rc = update(c, false, true, lr)) || (rc = tail(c, true))) return rc;
      c->h_steps++;
    }
  }
  CC(c, cudaStreamSynchronize(c->stream));
  return deverr_check(c);
}

static int infer_common(dnsb_cnn *c, const double *v, const double *ux, const double *uy,
                        const double *uz, double *tau) {
  if (!c || !tau) return c ? cfail(c, DNSB_EINVAL, "null argument") : DNSB_EINVAL;
  if (!c->have_inf) return cfail(c, DNSB_EINVAL, "no inference geometry (nfield = 0)");
  int rc;
  if ((rc = ensure_dev(c))) return rc;
  Volume &V = c->inf;
  if (V.side <= HALO) return cfail(c, DNSB_EUNSUP, "inference side %d <= halo %d", V.side, HALO);
  Prof p;
  prof_begin(c, p, 3, 0);
  {
    const unsigned bx = std::min(256u, (unsigned)(V.P + 31) / 32 * 32);
    CC(c, dnsb::launch_as(c->pdl, k_infer_in, dim3((V.P + bx - 1) / bx, V.P, V.P), dim3(bx), 0, c->stream, v, ux,
                          uy, uz, V.side, V.P, c->scales, V.in[0], c->pdl ? 1 : 0));
  }
  prof_end(c, p);
  CC(c, cudaGetLastError());
  // inference keeps no pre-activations (zout = nullptr)
  if ((rc = run_conv<2, 4, FWD_GELU>(c, V, 0, V.fwd[0], false, V.in[1], nullptr, nullptr, nullptr, 0)) ||
      (rc = run_conv<4, 4, FWD_GELU>(c, V, 1, V.fwd[1], false, V.in[2], nullptr, nullptr, nullptr, 0)) ||
      (rc = run_conv<4, 4, FWD_GELU>(c, V, 2, V.fwd[2], false, V.in[3], nullptr, nullptr, nullptr, 0)) ||
      (rc = run_conv<4, 2, FWD_INFER>(c, V, 3, V.fwd[3], false, nullptr, nullptr, nullptr, tau, 0)))
    return rc;
  return 0;
}

int dnsb_cnn_infer_cells(dnsb_cnn *c, const double *v, double *tau) {
  if (!v) return c ? cfail(c, DNSB_EINVAL, "null v") : DNSB_EINVAL;
  return infer_common(c, v, nullptr, nullptr, nullptr, tau);
}

int dnsb_cnn_infer(dnsb_cnn *c, const double *ux, const double *uy, const double *uz, double *tau) {
  if (!ux || !uy || !uz) return c ? cfail(c, DNSB_EINVAL, "null field") : DNSB_EINVAL;
  return infer_common(c, nullptr, ux, uy, uz, tau);
}

int dnsb_cnn_profile(dnsb_cnn *c, int enable) {
  if (!c) return DNSB_EINVAL;
  int rc;
  if ((rc = prof_harvest(c))) return rc;
  c->prof_on = enable != 0;
  for (int k = 0; k < 4; k++) c->prof_ms[k] = c->prof_flops[k] = 0, c->prof_n[k] = 0;
  return 0;
}

int dnsb_cnn_profile_read(dnsb_cnn *c, int kind, double *ms, long *launches, double *flops) {
  if (!c || kind < 0 || kind > 3) return DNSB_EINVAL;
  int rc;
  if ((rc = prof_harvest(c))) return rc;
  if (ms) *ms = c->prof_ms[kind];
  if (launches) *launches = c->prof_n[kind];
  if (flops) *flops = c->prof_flops[kind];
  return 0;
}

}  // extern "C"
