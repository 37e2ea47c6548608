// cnn.cuh -- tensor-core kernels of the sub-filter-stress CNN closure.
//
// The network (no counterpart in the reference, which has no learned
// closure): 4 layers of 3x3x3 convolutions, channels 3 -> 32 -> 32 -> 32 ->
// 6, bias, GELU (tanh form) after the first three, periodic padding on the full
// field.  Every convolution is an implicit GEMM on the 5th-generation tensor
// cores: BF16 operands staged in shared memory by TMA, FP32 accumulators in
// tensor memory (tcgen05.mma, cta_group::1, M = 128), read back with
// tcgen05.ld for a fused epilogue.
//
// Activation layout ("chunked voxels"): a volume of P x P x Pz voxels per
// sample; channels in chunks of 8 BF16 values (16 bytes); element
// [b][chunk][z][y][x][8].  Every layer of a network lives in the same
// geometry (same P, Pz): layer L's output occupies the box [0, Do)^3, Do =
// P - 2L, and the input voxel of output (x, y, z) for tap (dx, dy, dz) is
// (x + s + dx, y + s + dy, z + s + dz) with s = 0 (forward, "valid"
// convolution) or s = -2 (the transposed convolution of the backward pass;
// the box of the input is surrounded by zeros).  Voxels outside an output's
// box hold zeros: the buffers are cleared once and every kernel writes zeros
// at the positions of its tiles that are outside the box.
//
// Forward / transposed convolution (k_conv): one tile = 128 consecutive
// positions f = y*P + x of one plane of one sample (rows of the GEMM).  With
// the input patch of that tile staged as whole rows [chunk][dz][row][x][16 B]
// (one 4-D TMA box: x-rows of 16 P bytes x R rows x 3 planes x CI chunks), the 128
// GEMM rows of every (dy, dz) tap pair are 128 consecutive 16-byte rows of
// the patch starting at offset x0 + s + (dy + e) P, e = 1 for s < 0 (one
// extra row below the tile so that offsets stay >= 0).  So the A operand is a
// K-major canonical layout without swizzle (8-row core matrices of 128
// contiguous bytes, SBO = 128 B, LBO = the chunk stride), addressed by its
// start alone: no im2col copy.  The three x-taps are columns of the GEMM
// (N = 3 x output channels), and the epilogue adds row m + dx of column
// block dx into output m, so a tile yields 126 outputs.  Positions with
// x >= Do inside a row compute garbage that the epilogue replaces by zeros.
// B (the weights) is resident in shared memory for the whole persistent
// CTA, packed in the K-major core-matrix order.
//
// Weight gradient (k_wgrad): dW[dz, dy, dx][ci][co] = sum_o h[o + (dz, dy,
// dx)][ci] g[o][co] over the output positions o (the GEMM's K).  With o' = o
// + (0, dy, 0) the taps split over both operands: the GEMM's rows are (dx,
// ci) of h shifted by dx, its columns (dy, co) of g shifted by -dy, and one
// accumulator per dz takes h's plane z + dz against g's plane z.  Both are
// MN-major canonical layouts without swizzle, straight from the chunked
// activations: a K-block of R whole rows of one plane (R P positions, padded
// to a multiple of 16) is one TMA box [chunk][R rows][x] per shift; an x
// shift runs past the row end into zeros where g is zero anyway, a y shift
// starts above or below the volume in zeros.  A CTA marches up z, so that
// each plane of h is copied once for its three dz.  The bias gradient is the
// sum of g, formed by the epilogue warps while the MMAs run.  Split-K partials are reduced in a fixed order.
//
// Warp roles: warp 0 issues the TMA copies; warps 1 and 2 of the convolution,
// 1 to 3 of the weight gradient issue the MMAs (the whole warp runs the loop,
// one elected lane issues) and warp 1 owns the tensor memory; the other warps
// run the epilogue (a warp reads TMEM lanes 32 (w % 4) .. + 31): four groups of
// four taking the convolution's sub-tiles in turn (608 threads), warps 4-7 of
// the weight gradient (256 threads).  Every
// mbarrier wait is bounded; a wait that runs out raises the CTA's abort flag
// and the global error word, every role leaves its loop, the copies and MMAs
// in flight are waited for (bounded), the tensor memory is freed and the CTA
// returns.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace dnsb {
namespace cnn {

constexpr int NTHREADS = 256;       // weight gradient: TMA, three MMA, four epilogue warps
constexpr int CONV_GROUPS = 4;      // convolution epilogue: groups of 4 warps taking tiles in turn
constexpr int CONV_THREADS = 96 + 128 * CONV_GROUPS;  // TMA, two MMA, epilogue warps
constexpr int NTAPS = 27;
constexpr int TILE_M = 128;      // GEMM rows (positions) of a convolution tile
constexpr int TILE_OUT = 126;    // outputs of a convolution tile (rows m, m + 1, m + 2 feed output m)
constexpr int CONV_BARS = 512;   // bytes of barriers and flags after the plane ring
constexpr int CONV_XBUF = CONV_GROUPS * 2 * 3 * 2 * 32 * 4;  // lane-quarter boundary exchange, bytes
enum { DEVERR_CNN_TIMEOUT = 2 };

enum Mode { FWD_GELU = 0, FWD_LOSS = 1, FWD_INFER = 2, DGRAD = 3 };

// ----------------------------------------------------------- PTX helpers --

__device__ __forceinline__ uint32_t saddr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mb_init(uint64_t *b, uint32_t n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void mb_expect(uint64_t *b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(b)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mb_arrive(uint64_t *b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(b)) : "memory");
}
// try_wait that may suspend the thread for up to `ns` nanoseconds while the
// phase is incomplete (returns as soon as it completes)
__device__ __forceinline__ bool mb_try_sleep(uint64_t *b, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity), "r"(ns)
      : "memory");
  return ok != 0;
}
// non-blocking test of the phase (no suspension)
__device__ __forceinline__ bool mb_test(uint64_t *b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: a test first (a phase already complete costs no
// suspending try, measured at ~300 cycles on a completed phase), then at
// most `limit` polls, each suspending up to 1 us (so a waiting role takes
// no issue slots from the working warps); gives up early once the CTA's
// abort flag is raised.
__device__ __forceinline__ bool mb_wait(uint64_t *b, uint32_t parity, unsigned limit,
                                        volatile int *abort_flag) {
  if (mb_test(b, parity)) return true;
  for (unsigned it = 0; it < limit; it++) {
    if (mb_try_sleep(b, parity, 1000)) return true;
    if ((it & 15) == 15 && *abort_flag) return false;
  }
  return false;
}
// The same by a whole warp, with one answer for all its lanes (so that the
// loops around it stay uniform)
__device__ __forceinline__ bool warp_wait(uint64_t *b, uint32_t parity, unsigned limit,
                                          volatile int *abort_flag) {
  if (__all_sync(0xffffffffu, mb_test(b, parity))) return true;
  for (unsigned it = 0; it < limit; it++) {
    if (__all_sync(0xffffffffu, mb_try_sleep(b, parity, 1000))) return true;
    if ((it & 15) == 15 && __any_sync(0xffffffffu, *abort_flag != 0)) return false;
  }
  return false;
}
// one lane of a converged warp, the same every time
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
  return r != 0;
}
// named barrier over `n` threads that also ORs a predicate across them
__device__ __forceinline__ bool bar_or(int id, int n, bool pred) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.red.or.pred q, %2, %3, p;\n selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)pred), "r"(id), "r"(n)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void tma4(void *dst, const CUtensorMap *m, int c0, int c1, int c2, int c3,
                                     uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
          saddr(dst)),
      "l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(saddr(bar))
      : "memory");
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          saddr(dst)),
      "l"(src), "r"(bytes), "r"(saddr(bar))
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// shared-memory matrix descriptor, no swizzle (layout type 0), version 1
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
// instruction descriptor of kind::f16: BF16 x BF16 -> FP32, M = 128
__host__ __device__ constexpr uint32_t idesc_bf16(int n, bool a_mn, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   saddr(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(slot)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
// The tensor memory of a block, then the programmatic dependents' launch: they
// may start once every block of this grid (one wave: grid_for) has its columns,
// and wait for its completion before touching memory.  In the other order a
// dependent block on the same SM could take the columns first (a kernel takes 256
// or 512 of the 512) and wait for this grid, one of whose blocks then waits for
// the columns: no end.  With it a grid that holds tensor memory and waits for
// another waits for one that holds all of its own, also beside other streams'.
__device__ __forceinline__ void tmem_alloc_then_trigger(uint32_t *slot, uint32_t ncols) {
  tmem_alloc(slot, ncols);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
// 32 lanes x N columns of FP32 (this warp's lane quarter), into v[0..N)
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float *v);
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, float *v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}
template <>
__device__ __forceinline__ void tmem_ld<32>(uint32_t taddr, float *v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// three 32-lane x 8-column loads (columns c0, c1, c2) and one wait, into v[0..24)
__device__ __forceinline__ void tmem_ld3x8(uint32_t c0, uint32_t c1, uint32_t c2, float *v) {
  uint32_t r[24];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%24];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%25];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%26];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23])
      : "r"(c0), "r"(c1), "r"(c2)
      : "memory");
#pragma unroll
  for (int i = 0; i < 24; i++) v[i] = __uint_as_float(r[i]);
}

// GELU in its tanh form, 0.5 z (1 + tanh(u)) with u = sqrt(2/pi) (z +
// 0.044715 z^3), on the hardware tanh (tanh.approx.f32: about 2^-11
// relative, below the BF16 rounding that follows): six instructions, one
// of them on the special-function unit.
constexpr float GELU_C = 0.7978845608028654f;  // sqrt(2 / pi)
constexpr float GELU_A = 0.044715f;
__device__ __forceinline__ float tanh_hw(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Two FP32 values per instruction (fma / mul / add .rn.f32x2, each rounded as
// the scalar operation): the convolutions' epilogue is bound by its
// instructions.
__device__ __forceinline__ unsigned long long bits2(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 float2_of(unsigned long long r) {
  float2 a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
  return a;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)), "l"(bits2(c)));
  return float2_of(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)));
  return float2_of(d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)));
  return float2_of(d);
}
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 tanh2(float2 u) { return make_float2(tanh_hw(u.x), tanh_hw(u.y)); }
__device__ __forceinline__ float2 gelu2(float2 z) {
  const float2 u = mul2(z, fma2(both(GELU_C * GELU_A), mul2(z, z), both(GELU_C)));
  const float2 h = mul2(both(0.5f), z);
  return fma2(h, tanh2(u), h);
}
// d/dz [0.5 z (1 + t)] = s + s (1 - t) z u'(z) with s = 0.5 (1 + t); s (1 - t) z
// first: it is 0 where t is 1 or -1, and z u' alone passes the largest FP32 value
// from |z| = 1.5e13 on (0 x infinity)
__device__ __forceinline__ float2 gelu_grad2(float2 z) {
  const float2 z2 = mul2(z, z);
  const float2 t = tanh2(mul2(z, fma2(both(GELU_C * GELU_A), z2, both(GELU_C))));
  const float2 du = fma2(both(3.f * GELU_C * GELU_A), z2, both(GELU_C));
  const float2 s = fma2(both(0.5f), t, both(0.5f));
  return fma2(mul2(mul2(s, fma2(both(-1.f), t, both(1.f))), z), du, s);
}

__device__ __forceinline__ uint32_t pack2(float2 v) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(v.x, v.y);
  return *reinterpret_cast<const uint32_t *>(&t);
}
__device__ __forceinline__ uint4 pack8(const float2 *v) {
  return make_uint4(pack2(v[0]), pack2(v[1]), pack2(v[2]), pack2(v[3]));
}
__device__ __forceinline__ float2 unpack2(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}

// ------------------------------------------------------------ geometry --

struct ConvArgs {
  int P, Pz, B;        // volume pitch (x, y), planes, samples
  int Do;              // output box side
  int s, e, R;         // input offset (0 / -2), extra patch row, patch rows
  int sub;             // 126-output sub-tiles per tile (1 to 4), one plane load each tile
  int spp;             // sub-tiles per plane: ceil(Do * P / 126)
  int tpp;             // tiles per plane: ceil(spp / sub), the last with the sub-tiles left over
  int nsub;            // B * Do * spp sub-tiles, z fastest (see SubWalk)
  int nslot;           // input planes held in the shared-memory ring
  uint32_t slot_bytes;   // one input plane: CI * R * P * 16 (one TMA box)
  uint32_t slot_stride;  // slot_bytes rounded up to 1 KB
  uint32_t w_bytes;      // 27 * CI * CO * 128
  unsigned wait_limit;
  const uint4 *wpack;    // packed weights (B operand), w_bytes
  const float *bias;     // Cout values (forward modes)
  uint4 *out;            // [b][CO][Pz][P^2] x 16 B (FWD_GELU, FWD_LOSS, DGRAD)
  uint4 *zout;           // FWD_GELU: the pre-activation, same layout
  const uint4 *zin;      // DGRAD: the pre-activation of the output's layer
  const float4 *target;  // FWD_LOSS: [b][Pz][P^2][8] floats
  float loss_scale;      // FWD_LOSS: 2 / count
  float *loss_part;      // FWD_LOSS: one partial sum per CTA
  double *infer_out;     // FWD_INFER: 6 arrays of Do^3 values ([z][y][x])
  const float *oscale;   // FWD_INFER: per-component output scale
  int *err;
};

// A CTA's sub-tiles, in order: tile (b, j) of a plane marches up z, and a
// tile is up to `sub` sub-tiles of one plane.  The CTAs' ranges are cut at
// sub-tiles: cut at whole tiles, the busiest CTA had 21 sub-tiles of an average
// 18.9 (side 64, three a tile).  tile() gives the sub-tiles [lo, hi) of the
// next tile, `fresh` where its first two planes are not in the ring yet, `last`
// where all three are used for the last time.
struct SubWalk {
  int b, j, z;       // the tile given last
  int lo, hi;        // its sub-tiles
  bool fresh, last;
  int left, n;       // sub-tiles to come; sub-tiles of a whole tile of column j
  bool first;
  __device__ __forceinline__ void start(const ConvArgs &a, int s0, int s1) {
    b = s0 / (a.spp * a.Do);
    int r = s0 - b * a.spp * a.Do;
    j = r / (a.sub * a.Do);
    r -= j * a.sub * a.Do;
    n = min(a.sub, a.spp - j * a.sub);
    z = r / n - 1;
    lo = r - (z + 1) * n;
    left = s1 - s0;
    first = true;
  }
  __device__ __forceinline__ bool tile(const ConvArgs &a) {
    if (left <= 0) return false;
    if (++z == a.Do) {
      z = 0;
      if (++j == a.tpp) j = 0, b++;
      n = min(a.sub, a.spp - j * a.sub);
    }
    if (!first) lo = 0;
    hi = min(n, lo + left);
    left -= hi - lo;
    fresh = first || z == 0;
    last = left == 0 || z == a.Do - 1;
    first = false;
    return true;
  }
};

// Forward / transposed convolution, CI input chunks (the GEMM's K, 16
// channels per MMA), CO output chunks.  One MMA covers the three x-taps of
// a (dz, dy) pair: its N = 3 * 8 CO columns are (dx, output channel), so
// D[m][(dx, c)] = sum over (dz, dy, ci) of in[m + x0 + s + (dy + e) P, plane
// z + s + dz][ci] W[dz, dy, dx][c][ci], and the convolution at position m
// is D[m][(0, c)] + D[m + 1][(1, c)] + D[m + 2][(2, c)].  The epilogue forms
// that sum with warp shuffles (rows of a TMEM lane quarter are the lanes
// of one warp) and, for the two rows that cross into the next quarter,
// through shared memory; a tile of 128 rows thus yields TILE_OUT = 126
// outputs and costs 9 CI / 2 MMAs of N = 24 CO instead of 27 CI / 2 of N =
// 8 CO (the tensor core takes about as long for N = 96 as for N = 32).
// Tiles are numbered z fastest and every CTA takes one contiguous range of
// their sub-tiles (SubWalk), marching up z: the input planes
// z+s .. z+s+2 of a tile sit in a ring of nslot shared-memory slots, so a
// tile loads one new plane (three at the start of a column) and the planes
// are released to the producer after their last use.
// Bound by the issue of the MMAs and the epilogue's instructions about alike
// (32 -> 32 channels, per sub-tile: 18 MMAs of about 50 cycles; 16 epilogue warps,
// 2.3k cycles of arithmetic and stores and 1.1k of tensor-memory reads and
// shuffles each, every fourth sub-tile).  64^3 inference, four layers, before ->
// now 90.3 -> 81.6 us: ranges cut at sub-tiles and a ring of seven slots (86.2 -> 81.6),
// MMAs issued by a whole warp's uniform loop (88.5 -> 86.2), packed FP32 pairs, two
// shuffles per output instead of three and the weights ahead of the wait
// (90.2 -> 88.5).  Training on 8 crops of 32^3: with these 428 -> 360 us a step.
// The tensor pipe is active 31 % of a 32 -> 32 layer at 64^3 (29 us on its own).
template <int CI, int CO, int MODE>
__global__ void __launch_bounds__(CONV_THREADS, 1)
    k_conv(const __grid_constant__ CUtensorMap tin, const ConvArgs a) {
  constexpr int NW = 8 * CO;                            // outputs per position
  constexpr int N = 3 * NW;                             // MMA columns: 96 or 48
  constexpr int NACC = 4;                               // accumulators in flight
  // one epilogue group per accumulator: a group then waits for its
  // accumulator's phases in order, so a parity wait never meets a barrier
  // two phases behind (with fewer groups than accumulators it can)
  static_assert(CONV_GROUPS == NACC, "one epilogue group per accumulator");
  constexpr uint32_t ACC_STRIDE = N <= 64 ? 64 : 128;   // TMEM columns per accumulator
  constexpr uint32_t NCOLS = NACC * ACC_STRIDE;         // 256 or 512 columns
  constexpr int MAXSLOT = 12;
  constexpr int CU = MODE == FWD_LOSS || MODE == FWD_INFER ? 1 : CO;  // chunks used: 6 components there
  constexpr int NU = 8 * CU;
  constexpr int XB = 3 * 2 * NW;                        // exchange floats per group and buffer
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // 1 KB-aligned base (TMA destinations; the host adds 1 KB of slack)
  unsigned char *smem = smem_raw + ((1024u - (saddr(smem_raw) & 1023u)) & 1023u);
  unsigned char *wsm = smem;
  unsigned char *ring = smem + a.w_bytes;
  uint64_t *bars = reinterpret_cast<uint64_t *>(ring + a.nslot * a.slot_stride);
  uint64_t *full = bars, *empty = bars + MAXSLOT, *tfull = bars + 2 * MAXSLOT,
           *tempty = bars + 2 * MAXSLOT + NACC, *wbar = bars + 2 * MAXSLOT + 2 * NACC;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bars + 2 * MAXSLOT + 2 * NACC + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 2 * MAXSLOT + 2 * NACC + 2);
  float *lsum = reinterpret_cast<float *>(bars + 2 * MAXSLOT + 2 * NACC + 3);  // 16 floats
  float *bsm = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(bars) + 352);  // 32 biases
  // boundary rows handed between TMEM lane quarters: [group][buffer][quarter
  // 1..3][2][NW] (for lanes 30 and 31 of the quarter below: row 32q's x-shift
  // 2; row 32q's x-shift 1 + row 32q + 1's x-shift 2)
  float *xbuf = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(bars) + CONV_BARS);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp-uniform
  // this CTA's sub-tiles
  SubWalk w;
  w.start(a, (int)((long long)a.nsub * blockIdx.x / gridDim.x),
          (int)((long long)a.nsub * (blockIdx.x + 1) / gridDim.x));

  if (threadIdx.x == 0) {
    for (int i = 0; i < a.nslot; i++) {
      mb_init(&full[i], 1);
      mb_init(&empty[i], 2);  // released by both issuing lanes
    }
    for (int i = 0; i < NACC; i++) {
      mb_init(&tfull[i], 1);
      mb_init(&tempty[i], 4);
    }
    mb_init(wbar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc_then_trigger(tslot, NCOLS);
  // The weights, by the lane that set the barriers.  They are written by an
  // ordinary launch (k_update), and the kernel that follows it in the chain is
  // an ordinary launch too or lets its dependents start only past its own wait
  // (k_infer_in), so this kernel starts with them complete and visible.  Every
  // kernel between them is held to that by tests/test_dependent_launches.py
  if (threadIdx.x == 0) {
    mb_expect(wbar, a.w_bytes);
    bulk_load(wsm, a.wpack, a.w_bytes, wbar);
  }
  // programmatic dependent launch: the barrier set-up, the tensor-memory
  // allocation and the weights above overlap the tail of the previous
  // convolution; every other read of global memory (biases, input planes,
  // zin, targets) and every write follows the wait (a no-op for an ordinary
  // launch)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (warp == 2) bsm[lane] = MODE != DGRAD && lane < (CO == 4 ? 32 : 6) ? __ldg(a.bias + lane) : 0.f;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = __shfl_sync(0xffffffffu, *tslot, 0);
  const int P2 = a.P * a.P;

  if (warp == 0) {
    if (lane == 0) {
      // the input planes of the tiles in order; one lane runs this loop
      // serially: the ring slot advances by increments (no division per plane)
      int g = 0, sl = 0, ph = 0;  // planes issued; slot and phase of the next
      int y0 = 0;
      bool ok = true;
      while (ok && w.tile(a)) {
        if (w.fresh) y0 = (w.j * a.sub * TILE_OUT) / a.P;
        for (int zp = w.fresh ? 0 : 2; zp < 3; zp++, g++) {
          if (*abort_flag || !mb_wait(&empty[sl], ph ^ 1, a.wait_limit, abort_flag)) {
            ok = false;
            break;
          }
          mb_expect(&full[sl], a.slot_bytes);
          tma4(ring + sl * a.slot_stride, &tin, 0, y0 + a.s - a.e, w.z + a.s + zp, w.b * CI, &full[sl]);
          if (++sl == a.nslot) sl = 0, ph ^= 1;
        }
      }
      if (!ok) {
        *abort_flag = 1;
        atomicExch(a.err, DEVERR_CNN_TIMEOUT);
      }
      // the copies issued last land before the CTA may leave
      for (int g2 = g - a.nslot < 0 ? 0 : g - a.nslot; g2 < g; g2++)
        mb_wait(&full[g2 % a.nslot], (g2 / a.nslot) & 1, a.wait_limit, abort_flag);
      mb_wait(wbar, 0, a.wait_limit, abort_flag);
    }
  } else if (warp == 1 || warp == 2) {
    // Two issuing warps (1 and 2) take the sub-tiles in turn (sub-tile
    // i on warp i % 2): while one does its waits and bookkeeping, the
    // other's MMAs keep the tensor pipe fed.  Both wait for every plane and
    // both release it (the empty barriers count two arrivals: a commit
    // arrives once that warp's earlier MMAs are done).  The whole warp runs
    // the loop with warp-uniform values and one elected lane issues: the
    // descriptors then stay in uniform registers.  Run by a single lane, an
    // MMA took 71-130 cycles to issue for 18-36 of the tensor pipe.
    const int r = warp - 1;
    constexpr uint32_t idesc = idesc_bf16(N, false, false);
    // Descriptors are built once; per MMA only the start-address field
    // (bits 0-13, 16-byte units) moves, by an offset added to the whole
    // 64-bit word (starts stay below 256 KB, so the field never carries).
    const uint32_t cstride_u = (uint32_t)a.R * a.P;  // chunk stride in a slot, 16-byte units
    const uint64_t bdesc0 = sdesc(saddr(wsm), 3 * CO * 128u, 128);
    const uint64_t adesc_st = sdesc(0, cstride_u * 16u, 128);  // start 0
    const uint32_t ring_u = saddr(ring) >> 4, stride_u = a.slot_stride >> 4;
    uint32_t yrow[3];  // (dy + e) P, 16-byte units
#pragma unroll
    for (int q = 0; q < 3; q++) yrow[q] = (uint32_t)((q + a.e) * a.P);
    // plane slots, tile coordinates and accumulators advance by increments
    // (no division per tile)
    int i = 0, last_a = -1, last_aph = 0;
    int gs = 0, gph = 0;  // slot and phase of the next plane to arrive
    int ac = r, aph = 0;  // accumulator (i % NACC) of this warp's next sub-tile and its phase
    // phases seen complete ahead of their wait, by tests placed among the
    // MMAs: the next accumulator's release, the next plane
    bool acc_ready = false, plane_ready = false;
    int x0 = 0;  // the tile's first position in patch row y0
    bool ok = warp_wait(wbar, 0, a.wait_limit, abort_flag);
    while (ok && w.tile(a)) {
      if (w.fresh) x0 = (w.j * a.sub * TILE_OUT) % a.P;
      for (int q = w.fresh ? 0 : 2; q < 3 && ok; q++) {
        if (!plane_ready) ok = warp_wait(&full[gs], gph, a.wait_limit, abort_flag);
        plane_ready = false;
        if (++gs == a.nslot) gs = 0, gph ^= 1;
      }
      if (!ok) break;
      // slots of the last three planes loaded: planes z+s, z+s+1, z+s+2
      int sz[3];
      sz[2] = gs == 0 ? a.nslot - 1 : gs - 1;
      sz[1] = sz[2] == 0 ? a.nslot - 1 : sz[2] - 1;
      sz[0] = sz[1] == 0 ? a.nslot - 1 : sz[1] - 1;
      uint64_t ab[3];
#pragma unroll
      for (int dz = 0; dz < 3; dz++)
        ab[dz] = adesc_st + (uint64_t)(ring_u + (uint32_t)sz[dz] * stride_u + (uint32_t)(x0 + a.s));
      for (int sb = w.lo; sb < w.hi; sb++, i++) {
        if ((i & 1) != r) continue;
        if (!acc_ready && !warp_wait(&tempty[ac], aph ^ 1, a.wait_limit, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t dacc = tbase + (uint32_t)ac * ACC_STRIDE;
        const uint64_t so = (uint64_t)(sb * TILE_OUT);  // the sub-tile's rows, 16-byte units
        const int nac = ac + 2 >= NACC ? ac + 2 - NACC : ac + 2, naph = ac + 2 >= NACC ? aph ^ 1 : aph;
        auto taps = [&](int zy) {
          const uint64_t at = ab[zy / 3] + so + (uint64_t)yrow[zy % 3];
#pragma unroll
          for (int k = 0; k < CI / 2; k++)
            mma_bf16(dacc, at + (uint64_t)(2 * k) * cstride_u,
                     bdesc0 + (uint64_t)((zy * CI + 2 * k) * 3 * CO * 8), idesc, (zy | k) != 0 ? 1u : 0u);
        };
        if (elect_one()) {
#pragma unroll
          for (int zy = 0; zy < 6; zy++) taps(zy);
        }
        __syncwarp();
        acc_ready = __all_sync(0xffffffffu, mb_test(&tempty[nac], naph ^ 1));
        if (sb + 2 >= w.hi && w.left > 0) plane_ready = __all_sync(0xffffffffu, mb_test(&full[gs], gph));
        if (elect_one()) {
#pragma unroll
          for (int zy = 6; zy < 9; zy++) taps(zy);
          mma_commit(&tfull[ac]);
        }
        __syncwarp();
        last_a = ac;
        last_aph = aph;
        ac = nac;
        aph = naph;
      }
      if (!ok) break;
      // release the planes this tile used for the last time
      if (elect_one()) {
        mma_commit(&empty[sz[0]]);
        if (w.last) {
          mma_commit(&empty[sz[1]]);
          mma_commit(&empty[sz[2]]);
        }
      }
      __syncwarp();
    }
    if (!ok && lane == 0) {
      *abort_flag = 1;
      atomicExch(a.err, DEVERR_CNN_TIMEOUT);
    }
    // the MMAs issued last complete before the tensor memory is freed
    if (last_a >= 0) warp_wait(&tfull[last_a], last_aph, a.wait_limit, abort_flag);
  } else {
    // epilogue: CONV_GROUPS groups of 4 warps take the tiles in turn (group
    // e / 4 the tiles with local index i % CONV_GROUPS == e / 4); warp w
    // reads TMEM lanes 32 (w % 4) .. + 31 (rows m = 32 (w % 4) + lane of its
    // tile), 8 columns of each x-shift at a time
    const int e = warp - 3, q = warp & 3, grp = e >> 2;
    const int m = q * 32 + lane;
    const float2 keep = both(lane < 31 ? 1.f : 0.f);
    float osc[6];
#pragma unroll
    for (int k = 0; k < 6; k++) osc[k] = MODE == FWD_INFER ? __ldg(a.oscale + k) : 0.f;
    const bool store_z = a.zout != nullptr;
    float *xg = xbuf + grp * 2 * XB;
    float lacc = 0.f;
    // this thread's positions in the tile's sub-tiles, updated as z marches
    int fA = 0, xA = 0, yA = 0;  // this thread's row in sub-tile 0: offset, x, y
    // a sub-tile further: TILE_OUT = q126 rows of P + r126
    const int q126 = TILE_OUT / a.P, r126 = TILE_OUT - q126 * a.P;
    const long long cstr = (long long)a.Pz * P2;  // one chunk of 8 channels further
    const float2 *bias2 = reinterpret_cast<const float2 *>(bsm);
    bool stop = false;
    int i = 0, own = 0;
    while (!stop && w.tile(a)) {
      if (w.fresh) {
        fA = w.j * a.sub * TILE_OUT + m;
        yA = fA / a.P;
        xA = fA - yA * a.P;
      }
      int x = xA, y = yA;
      for (int sb = 0; sb < w.lo; sb++) {  // a range that starts inside a tile
        x += r126;
        y += q126;
        if (x >= a.P) x -= a.P, y++;
      }
      for (int sb = w.lo; sb < w.hi; sb++, i++, x += r126, y += q126) {
        if (x >= a.P) x -= a.P, y++;
        const bool mine = (i % CONV_GROUPS) == grp;
        const int ac = i % NACC, aph = (i / NACC) & 1;
        if (!mine) continue;
        const int f = fA + sb * TILE_OUT;
        const bool inside = m < TILE_OUT && f < P2;
        const bool valid = inside && x < a.Do && y < a.Do;
        const long long vox = (long long)w.z * P2 + f;
        const long long o0 = (long long)w.b * CO * cstr + vox;
        // what the tile's outputs need from memory is on its way while the MMAs run
        uint4 zq[CO];
        float4 tq[2];
        if (MODE == DGRAD) {
#pragma unroll
          for (int c = 0; c < CO; c++) zq[c] = valid ? a.zin[o0 + c * cstr] : make_uint4(0, 0, 0, 0);
        }
        if (MODE == FWD_LOSS) {
          const float4 *tp = a.target + ((long long)w.b * a.Pz * P2 + vox) * 2;
#pragma unroll
          for (int k = 0; k < 2; k++) tq[k] = valid ? tp[k] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float2 v[NU / 2];
        {
          float *xw = xg + (own & 1) * XB;
          bool ok = !*abort_flag && mb_wait(&tfull[ac], aph, a.wait_limit, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (ok) {
            tc_fence_after();
            const uint32_t ta = tbase + ((uint32_t)(q * 32) << 16) + (uint32_t)ac * ACC_STRIDE;
#pragma unroll
            for (int c = 0; c < CU; c++) {
              float d[24];  // columns 8c.. of x-shift 0, 1, 2
              tmem_ld3x8(ta + 8 * c, ta + NW + 8 * c, ta + 2 * NW + 8 * c, d);
              // out[m] = d0[m] + (d1 + d2[. + 1])[m + 1]
              float2 w[4];
#pragma unroll
              for (int k = 0; k < 4; k++) {
                const float2 s2 = make_float2(__shfl_down_sync(0xffffffffu, d[16 + 2 * k], 1),
                                              __shfl_down_sync(0xffffffffu, d[17 + 2 * k], 1));
                w[k] = fma2(s2, keep, make_float2(d[8 + 2 * k], d[9 + 2 * k]));
              }
              if (q > 0 && lane == 0) {
                float4 *xs = reinterpret_cast<float4 *>(xw + 2 * (q - 1) * NW + 8 * c);
                xs[0] = make_float4(d[16], d[17], d[18], d[19]);
                xs[1] = make_float4(d[20], d[21], d[22], d[23]);
                xs[NW / 4] = make_float4(w[0].x, w[0].y, w[1].x, w[1].y);
                xs[NW / 4 + 1] = make_float4(w[2].x, w[2].y, w[3].x, w[3].y);
              }
#pragma unroll
              for (int k = 0; k < 4; k++) {
                const float2 s1 = make_float2(__shfl_down_sync(0xffffffffu, w[k].x, 1),
                                              __shfl_down_sync(0xffffffffu, w[k].y, 1));
                v[4 * c + k] = fma2(s1, keep, make_float2(d[2 * k], d[2 * k + 1]));
              }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mb_arrive(&tempty[ac]);
          }
          // the group's four warps agree on going on, and the boundary rows
          // written above are visible after this barrier
          if (bar_or(1 + grp, 128, !ok)) {
            *abort_flag = 1;
            atomicExch(a.err, DEVERR_CNN_TIMEOUT);
            stop = true;
            break;
          }
          if (q < 3 && lane >= 30) {
            const float4 *xr = reinterpret_cast<const float4 *>(xw + 2 * q * NW + (lane - 30) * NW);
#pragma unroll
            for (int c = 0; c < NU / 4; c++) {  // quarter q + 1's rows
              const float4 h = xr[c];
              v[2 * c] = add2(v[2 * c], make_float2(h.x, h.y));
              v[2 * c + 1] = add2(v[2 * c + 1], make_float2(h.z, h.w));
            }
          }
          own++;
        }
        if (!inside) continue;
        if (MODE == FWD_GELU) {
#pragma unroll
          for (int c = 0; c < CO; c++) {
            float2 zv[4], hv[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
              zv[k] = add2(v[4 * c + k], bias2[4 * c + k]);
              hv[k] = gelu2(zv[k]);
            }
            const uint4 none = make_uint4(0, 0, 0, 0);
            const long long o = o0 + c * cstr;
            if (store_z) a.zout[o] = valid ? pack8(zv) : none;
            a.out[o] = valid ? pack8(hv) : none;
          }
        } else if (MODE == FWD_LOSS) {
          // 6 output components in chunk 0 (N = 16: chunk 1 stays zero)
          const float tv[6] = {tq[0].x, tq[0].y, tq[0].z, tq[0].w, tq[1].x, tq[1].y};
          float2 gv[4] = {both(0.f), both(0.f), both(0.f), both(0.f)};
          if (valid) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
              const float2 d = make_float2(v[k].x + bsm[2 * k] - tv[2 * k], v[k].y + bsm[2 * k + 1] - tv[2 * k + 1]);
              lacc += d.x * d.x;
              lacc += d.y * d.y;
              gv[k] = make_float2(a.loss_scale * d.x, a.loss_scale * d.y);
            }
          }
          a.out[o0] = pack8(gv);
        } else if (MODE == FWD_INFER) {
          if (valid) {
            const long long n3 = (long long)a.Do * a.Do * a.Do;
            const long long o = ((long long)w.z * a.Do + y) * a.Do + x;
#pragma unroll
            for (int k = 0; k < 3; k++) {
              a.infer_out[2 * k * n3 + o] = (double)((v[k].x + bsm[2 * k]) * osc[2 * k]);
              a.infer_out[(2 * k + 1) * n3 + o] = (double)((v[k].y + bsm[2 * k + 1]) * osc[2 * k + 1]);
            }
          }
        } else {  // DGRAD: g = dL/dh * gelu'(z) of the output's layer
#pragma unroll
          for (int c = 0; c < CO; c++) {
            const uint32_t zw[4] = {zq[c].x, zq[c].y, zq[c].z, zq[c].w};
            float2 gv[4];
#pragma unroll
            for (int k = 0; k < 4; k++) gv[k] = mul2(v[4 * c + k], gelu_grad2(unpack2(zw[k])));
            a.out[o0 + c * cstr] = valid ? pack8(gv) : make_uint4(0, 0, 0, 0);
          }
        }
      }
    }
    if (MODE == FWD_LOSS) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) lacc += __shfl_xor_sync(0xffffffffu, lacc, o);
      if (lane == 0) lsum[e] = lacc;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (MODE == FWD_LOSS && threadIdx.x == 0) {
    float l = 0.f;
    for (int k = 0; k < 4 * CONV_GROUPS; k++) l += lsum[k];
    a.loss_part[blockIdx.x] = l;
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_free(tbase, NCOLS);
  }
}

// ------------------------------------------------------ weight gradient --

constexpr int WG_PLANES = 4;  // planes of h in shared memory: three in use, one ahead
constexpr int WG_GRADS = 3;   // planes of g

struct WgradArgs {
  int P, B;         // volume geometry
  int Do;           // output box side (of g)
  int R, KB, KBp;   // rows per K-block, its positions R P, padded to a multiple of 16
  int whole;        // one TMA box per shift holds all chunks (KB == KBp), else one per chunk
  int kpp;          // K-blocks per plane: ceil((Do + 2) / R)
  int nsplit;       // K splits = CTAs
  uint32_t h_bytes, g_bytes;  // one plane of h and of g (three shifts each)
  unsigned wait_limit;
  float *partial;   // [split][dz][N / 4][128][4]: a warp stores 512 contiguous bytes
  int *err;
};

// h: CI chunks (A operand, shifted in x), g: CO chunks (B operand, shifted in
// y): per step (one plane of one row block) six boxes of 64-byte positions and
// 3 KBp / 16 MMAs of N = 96 (48 cycles each) for 27 taps.
// Of a 32 x 32-channel layer of 8 crops of 32^3 (56k cycles, 29-32 us) the tensor
// pipe takes 24k (43 %; 51 % of the first layer), set-up and the partial sums' stores
// about 5k each; the rest is spent waiting for planes.  With the taps stacked four
// at a time on the rows (N = 32) every position was copied 34 times and took 7 MMAs
// of 52 cycles per 16 positions: 85.6 us (959 MB of copies, 11.7 TB/s); 53.4 us
// with one issuing lane for the three dz, 34.1 with an issuing warp each, 33.1 with
// a third plane of g in flight and 29.3 with the partial sums stored 512 contiguous
// bytes a warp instead of 16 a lane at a stride of 384.
template <int CI, int CO>
__global__ void __launch_bounds__(NTHREADS, 1)
    k_wgrad(const __grid_constant__ CUtensorMap th, const __grid_constant__ CUtensorMap tg,
            const WgradArgs a) {
  constexpr int N = 3 * 8 * CO;
  constexpr uint32_t ACC = 128, NCOLS = 512;  // columns between the dz accumulators, allocated
  const uint32_t chunk = (uint32_t)a.KBp * 16;  // bytes of one chunk of a K-block
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((1024u - (saddr(smem_raw) & 1023u)) & 1023u);
  unsigned char *gs = smem + WG_PLANES * a.h_bytes;
  uint64_t *bars = reinterpret_cast<uint64_t *>(gs + WG_GRADS * a.g_bytes);
  uint64_t *hfull = bars, *hempty = hfull + WG_PLANES, *gfull = hempty + WG_PLANES,
           *gempty = gfull + WG_GRADS, *done = gempty + WG_GRADS;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(done + 2);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp-uniform
  const int split = blockIdx.x;
  // steps (sample, row block, z), z fastest
  const long long nsteps = (long long)a.B * a.kpp * a.Do;
  const int s0 = (int)(nsteps * split / a.nsplit), s1 = (int)(nsteps * (split + 1) / a.nsplit);

  if (threadIdx.x == 0) {
    for (int i = 0; i < WG_PLANES; i++) {
      mb_init(&hfull[i], 1);
      mb_init(&hempty[i], 3);  // one arrival per issuing lane
    }
    for (int i = 0; i < WG_GRADS; i++) {
      mb_init(&gfull[i], 1);
      mb_init(&gempty[i], 3 + 4);  // and one per summing warp
    }
    mb_init(done, 3);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (!a.whole) {
    // the padding positions of every chunk stay zero
    uint4 *z = reinterpret_cast<uint4 *>(smem);
    const int n = (int)((WG_PLANES * a.h_bytes + WG_GRADS * a.g_bytes) / 16);
    for (int i = threadIdx.x; i < n; i += NTHREADS) z[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 1) tmem_alloc_then_trigger(tslot, NCOLS);
  // the previous kernel's outputs (activations, gradients) complete and
  // visible past this (a no-op for an ordinary launch)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = __shfl_sync(0xffffffffu, *tslot, 0);

  if (warp == 0) {
    if (lane == 0) {
      const uint32_t hb = 3u * CI * a.KB * 16, gb = 3u * CO * a.KB * 16;
      int pl = 0, gi = 0;  // planes of h and of g issued
      bool ok = true;
      for (int s = s0; ok && s < s1; s++) {
        const int col = s / a.Do, z = s - col * a.Do;
        const int b = col / a.kpp, y0 = (col - b * a.kpp) * a.R;
        // the first step of a column loads three planes, the others one
        for (int pz = s == s0 || z == 0 ? z : z + 2; ok && pz <= z + 2; pz++) {
          const int sl = pl % WG_PLANES;
          ok = !*abort_flag && mb_wait(&hempty[sl], ((pl / WG_PLANES) & 1) ^ 1, a.wait_limit, abort_flag);
          if (!ok) break;
          mb_expect(&hfull[sl], hb);
          unsigned char *d = smem + sl * a.h_bytes;
          for (int dx = 0; dx < 3; dx++)
            for (int c = 0; c < (a.whole ? 1 : CI); c++)
              tma4(d + (dx * CI + c) * chunk, &th, 2 * dx, y0, pz, b * CI + c, &hfull[sl]);
          pl++;
        }
        if (ok) {
          const int st = gi % WG_GRADS;
          ok = !*abort_flag && mb_wait(&gempty[st], ((gi / WG_GRADS) & 1) ^ 1, a.wait_limit, abort_flag);
          if (!ok) break;
          mb_expect(&gfull[st], gb);
          unsigned char *d = gs + st * a.g_bytes;
          for (int dy = 0; dy < 3; dy++)
            for (int c = 0; c < (a.whole ? 1 : CO); c++)
              tma4(d + (dy * CO + c) * chunk, &tg, 0, y0 - dy, z, b * CO + c, &gfull[st]);
          gi++;
        }
      }
      if (!ok) {
        *abort_flag = 1;
        atomicExch(a.err, DEVERR_CNN_TIMEOUT);
      }
      // let the last copies of every slot land before leaving
      for (int i = pl < WG_PLANES ? 0 : pl - WG_PLANES; i < pl; i++)
        mb_wait(&hfull[i % WG_PLANES], (i / WG_PLANES) & 1, a.wait_limit, abort_flag);
      for (int i = gi < WG_GRADS ? 0 : gi - WG_GRADS; i < gi; i++)
        mb_wait(&gfull[i % WG_GRADS], (i / WG_GRADS) & 1, a.wait_limit, abort_flag);
    }
  } else if (warp <= 3) {
    // One issuing warp per dz, each with its own accumulator: a warp's waits
    // and commits run beside the others' MMAs.  Warp dz meets plane j of a
    // column (of n steps here, n + 2 planes) at step j - dz, and releases the
    // planes it does not use as they arrive.  The loop is the whole warp's and
    // uniform, one elected lane issues (see k_conv).
    constexpr uint32_t idesc = idesc_bf16(N, true, true);
    const int nkk = a.KBp / 16, dz = warp - 1;
    const uint32_t dacc = tbase + (uint32_t)dz * ACC;
    // MN-major, no swizzle: SBO = stride of 8-element MN groups (one
    // chunk), LBO = stride of 8-row K groups (128 B); 16 positions are
    // 256 bytes on, 16 in the address field
    const uint64_t ad0 = sdesc(saddr(smem), 128, chunk), bd0 = sdesc(saddr(gs), 128, chunk);
    const uint32_t h_u = a.h_bytes >> 4, g_u = a.g_bytes >> 4;
    int sl = 0, ph = 0, g0 = 0;  // slot and phase of the next plane, steps of the columns before
    bool ok = true, any = false;
    for (int s = s0; ok && s < s1;) {
      const int n = min(s1 - s, a.Do - s % a.Do);
      for (int j = 0; j < n + 2; j++) {
        ok = warp_wait(&hfull[sl], ph, a.wait_limit, abort_flag);
        if (!ok) break;
        if (j < dz || j - dz >= n) {
          if (elect_one()) mb_arrive(&hempty[sl]);
        } else {
          const int gi = g0 + j - dz, st = gi % WG_GRADS;
          ok = warp_wait(&gfull[st], (gi / WG_GRADS) & 1, a.wait_limit, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            uint64_t ad = ad0 + (uint64_t)(sl * h_u), bd = bd0 + (uint64_t)(st * g_u);
            for (int kk = 0; kk < nkk; kk++, ad += 16, bd += 16)
              mma_bf16(dacc, ad, bd, idesc, any || kk != 0);
            mma_commit(&gempty[st]);
            mma_commit(&hempty[sl]);
          }
          any = true;
        }
        __syncwarp();
        if (++sl == WG_PLANES) sl = 0, ph ^= 1;
      }
      s += n;
      g0 += n;
    }
    if (!ok && lane == 0) {
      *abort_flag = 1;
      atomicExch(a.err, DEVERR_CNN_TIMEOUT);
    }
    if (elect_one()) {
      if (any) mma_commit(done);
      else mb_arrive(done);
    }
  } else {
    const int q = warp & 3;
    const int m = q * 32 + lane;
    // while the MMAs run, a warp per chunk sums g over the positions of its
    // unshifted copy: the bias gradient (a row of ones among h's rows gave it
    // before, in the shared memory that the third plane of g takes now)
    float2 sum[4] = {both(0.f), both(0.f), both(0.f), both(0.f)};
    bool ok = true;
    for (int gi = 0; ok && gi < s1 - s0; gi++) {
      const int st = gi % WG_GRADS;
      ok = warp_wait(&gfull[st], (gi / WG_GRADS) & 1, a.wait_limit, abort_flag);
      if (!ok) break;
      if (q < CO) {
        const uint4 *p = reinterpret_cast<const uint4 *>(gs + st * a.g_bytes + q * chunk);
        for (int i = lane; i < a.KB; i += 32) {
          const uint4 g = p[i];
          const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
          for (int k = 0; k < 4; k++) sum[k] = add2(sum[k], unpack2(gw[k]));
        }
      }
      __syncwarp();
      if (lane == 0) mb_arrive(&gempty[st]);
    }
    if (q < CO) {
#pragma unroll
      for (int k = 0; k < 4; k++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          sum[k] = add2(sum[k], make_float2(__shfl_xor_sync(0xffffffffu, sum[k].x, o),
                                            __shfl_xor_sync(0xffffffffu, sum[k].y, o)));
      if (lane == 0) {  // the partial row after dz = 0's
        float4 *dst = reinterpret_cast<float4 *>(a.partial) + ((long long)split * 3 * (N / 4) + 2 * q) * 128 + 24 * CI;
        dst[0] = make_float4(sum[0].x, sum[0].y, sum[1].x, sum[1].y);
        dst[128] = make_float4(sum[2].x, sum[2].y, sum[3].x, sum[3].y);
      }
    }
    const bool all = mb_wait(done, 0, a.wait_limit, abort_flag);
    ok = ok && all && !*abort_flag;
    if (!ok) {
      *abort_flag = 1;
      atomicExch(a.err, DEVERR_CNN_TIMEOUT);
    }
    tc_fence_after();
    const bool none = s1 <= s0 || !ok;
    constexpr int W = N % 32 == 0 ? 32 : 16;
    for (int dz = 0; dz < 3; dz++) {
      float4 *dst = reinterpret_cast<float4 *>(a.partial) + ((long long)split * 3 + dz) * (N / 4) * 128 + m;
#pragma unroll 1
      for (int c0 = 0; c0 < N; c0 += W) {
        float v[W];
        tmem_ld<W>(tbase + ((uint32_t)(q * 32) << 16) + dz * ACC + c0, v);
        if (m < 3 * 8 * CI)  // rows beyond: whatever follows in shared memory, nothing reads them
#pragma unroll
          for (int c = 0; c < W; c += 4)
            dst[(c0 + c) / 4 * 128] =
                none ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        __syncwarp();  // the next tensor-memory load is of the whole warp
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_free(tbase, NCOLS);
  }
}

}  // namespace cnn
}  // namespace dnsb
