// One PPO minibatch (racer/ppo.mojo:259-337: forward, clipped loss, backward,
// gradient norm, Adam) in three launches, for policies of at most 128 inputs:
//
//   k_update_tiles   per tile of 128 samples, everything from the inputs to
//                    the weight gradients, which stay in tensor memory
//   k_update_reduce  the CTAs' partial gradients summed in a fixed order
//   k_update_adam    the gradient norm, Adam, and theta's BF16 operand images
//
// What bounds the tile kernel: a sample needs 2 IN bytes of input, 20 bytes of
// loss scalars and 72 kflop, so neither memory nor the tensor pipe; the seven
// products of a tile (three layers, d1, three weight gradients) depend on one
// another through the epilogues (128 tanh, the loss, 128 tanh derivatives a
// sample). Two tiles, each with a group of eight
// warps (two threads a sample, 32 units each), share an SM so that one's
// epilogue covers the other's products: 57 us at 262144 samples x 113 inputs
// (64 with four warps a tile and one region for X; 67 with a warp of its own
// issuing the products, whose registers the epilogues then lacked).
// Separate kernels instead moved h1, h2 in 32 and 16 bits, d1, d2 in 16, and x
// twice: 2.7 KB a sample and minibatch, 275 us.
//
// Operands: X arrives by TMA as [feature][64 samples] rows of 128 bytes. The
// same bytes are layer 1's A (MN-major: samples x features) and, K-major, the A
// of the layer-0 weight gradient (features x samples). The threads
// write h1, h2, d2 and d1 as [sample][64 units] rows: K-major A of the
// next product, MN-major operand of a weight gradient. A constant tile whose
// first unit is 1 stands for the bias input of layers 2 and 3 and gives their
// bias gradients.
//
// The results are those of the separate kernels (mlp_tc.cu, ppo.cu,
// policy_tc.cu), bit for bit: the operands' BF16 values, the FP32 arithmetic
// between the products and the order of every FP32 sum are theirs. (The FP64
// sums, of the log-std gradients, the KL and the gradient norm, run in trees of
// their own and are rounded to FP32.) So the batch is cut
// into the ranges that the separate weight-gradient GEMMs split it into (whole
// 64-sample k-blocks, at most 296 ranges, here one for each of the 304 groups
// of an otherwise empty GPU), each accumulated on its own, and the ranges'
// partials are added in the order of their reduction. A range of an odd number
// of k-blocks ends in half a tile.
//
// Built with --fmad=false for the loss; the backward's multiply-adds are
// written out.
#include <cuda_bf16.h>

#include <algorithm>
#include <string>

#include "common.cuh"
#include "loss.cuh"
#include "policy_tc.h"
#include "tc.cuh"
#include "update_tc.h"

using bf16 = __nv_bfloat16;

namespace racer {
namespace {

constexpr int TB = 128;               // samples per tile
constexpr int TILE_BYTES = TB * 128;  // 128 rows of 64 BF16
constexpr int W_BYTES = 64 * 128;     // 64 rows of 64 BF16
constexpr int CTXS = 2;               // tiles in flight per CTA
constexpr int GROUP = 256;            // threads of a tile
constexpr int UNITS = 64 * TB / GROUP;  // units of its sample a thread takes

struct UpdateCfg {
  static constexpr int THREADS = CTXS * GROUP;
  // per context: two regions of two tiles, which hold X and [h1, h2 (then d2)] and change roles with every tile, and
  // E: d3, then d1
  static constexpr int REGION = 2 * TILE_BYTES, E = 2 * REGION, CTX = E + TILE_BYTES;
  static constexpr int ONE = CTXS * CTX;  // behind every context: MN strides are positive
  static constexpr int W0 = ONE + TILE_BYTES;
  static constexpr int W1 = W0 + 2 * W_BYTES;
  static constexpr int W2 = W1 + 2 * W_BYTES;
  static constexpr int W1T = W2 + 2 * 16 * 128;
  static constexpr int W2F = W1T + W_BYTES;  // FP32 W2 by unit: float4 (w0, w1, w2, 0)
  static constexpr int BAR = W2F + 1024;
  static constexpr int SMEM = BAR + 512 + 1024;  // + alignment slack
  // tensor memory columns per context: accumulator, then the three weight gradients
  static constexpr int ACC = 0, DW0 = 64, DW1 = 128, DW2 = 192, COLS = 256;
};
static_assert(UpdateCfg::SMEM <= 227 * 1024, "one CTA per SM");
static_assert(H * 16 <= 1024, "W2 fits its block");

struct TileArgs {
  const float* samples;  // this minibatch's [5][batch]
  int in, batch;
  int range, ranges;  // samples per range (a multiple of 64), ranges
  const float* theta;
  const uint8_t *pack, *w1t;
  const float* moments;  // sums of the advantages and their squares
  float* part;
  double* sums;
  UpdateDump dump;
  int* err;
};

// xfull: the tile's inputs landed. acc: a product of the chain is complete
// (four times a tile). e, f, w: layer 2's, 1's and 0's weight gradient.
struct CtxBars {
  uint64_t xfull, acc, e, f, w, drain;
};

// The tiles of a context in order: range after range, whole tiles and the rest of each.
struct TileWalk {
  int range, start, end, tile;
  __device__ __forceinline__ TileWalk(const TileArgs& a, int first) { enter(a, first); }
  __device__ __forceinline__ void enter(const TileArgs& a, int r) {
    range = r;
    start = tile = r * a.range;
    end = min(a.batch, start + a.range);
  }
  __device__ __forceinline__ bool live(const TileArgs& a) const { return range < a.ranges; }
  __device__ __forceinline__ bool last() const { return tile + TB >= end; }
  __device__ __forceinline__ void next(const TileArgs& a, int stride) {
    if (last())
      enter(a, range + stride);
    else
      tile += TB;
  }
};

__global__ void __launch_bounds__(UpdateCfg::THREADS, 1)
    k_update_tiles(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ TileArgs a) {
  using C = UpdateCfg;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = tc::smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  CtxBars* bars = reinterpret_cast<CtxBars*>(smem + C::BAR);
  double* sh_sums = reinterpret_cast<double*>(bars + CTXS);  // [CTXS][4 warps][3]
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sh_sums + 8 * 3);
  volatile int* abort = reinterpret_cast<volatile int*>(tslot + 1);  // set by a timed-out wait
  static_assert(CTXS * sizeof(CtxBars) + 8 * 3 * 8 + 16 <= 512, "barriers and sums fit their block");
  float4* w2f = reinterpret_cast<float4*>(smem + C::W2F);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ctx = tid / GROUP;
  const bool leader = tid % GROUP == 0;  // issues the context's copies and products
  const int r = tid & (TB - 1);          // sample of the tile and TMEM lane
  const int half = (tid / TB) % (GROUP / TB);  // units UNITS half .. UNITS half + UNITS - 1
  CtxBars& bar = bars[ctx];
  uint8_t* mine = smem + ctx * C::CTX;
  const int in = a.in, batch = a.batch;
  const int w1 = H * in, w2 = w1 + H * HA, logstd = w2 + OUT * HA;

  if (tid == 0) {
    for (int c = 0; c < CTXS; ++c)
      for (uint64_t* b : {&bars[c].xfull, &bars[c].acc, &bars[c].e, &bars[c].f, &bars[c].w, &bars[c].drain})
        tc::mbar_init(b, 1);
    *abort = 0;
    tc::fence_barrier_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, CTXS * C::COLS);
    tc::tmem_relinquish();
  }
  {
    auto copy = [&](int off, const uint8_t* src, int bytes) {
      const uint4* s = reinterpret_cast<const uint4*>(src);
      for (int e = tid; e < bytes / 16; e += C::THREADS) reinterpret_cast<uint4*>(smem + off)[e] = __ldcg(s + e);
    };
    const int w0_bytes = (in + 63) / 64 * W_BYTES;
    for (int e = tid; e < TILE_BYTES / 16; e += C::THREADS)  // unit 0 of every sample is 1
      reinterpret_cast<uint4*>(smem + C::ONE)[e] =
          make_uint4((e & 7) == ((e >> 3) & 7) ? tc::pack_bf16(1.0f, 0.0f) : 0u, 0u, 0u, 0u);
    early_wait();  // theta and its images are the last minibatch's
    copy(C::W0, a.pack, w0_bytes);
    copy(C::W1, a.pack + w0_bytes, 2 * W_BYTES);
    copy(C::W2, a.pack + w0_bytes + 2 * W_BYTES, 2 * 16 * 128);
    copy(C::W1T, a.w1t, W_BYTES);
    if (tid < H) {
      const float* w = a.theta + w2 + tid;
      w2f[tid] = make_float4(__ldcg(w), __ldcg(w + HA), __ldcg(w + 2 * HA), 0.0f);
    }
  }
  tc::fence_proxy_async_smem();
  tc::tc_fence_before();
  __syncthreads();
  early_next();  // not before the TMEM is allocated: a CTA that waits for this kernel must not hold what this one needs
  tc::tc_fence_after();
  const uint32_t tmem = *tslot + ctx * C::COLS;
  const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  bool ok = true, issued = false;
  float ls[2], invvar[2], adv_mean, adv_scale;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    ls[k] = __ldcg(a.theta + logstd + k);
    invvar[k] = rmath::expf_(-2.0f * ls[k]);
  }
  advantage_moments(a.moments, batch, &adv_mean, &adv_scale);
  const float fbatch = (float)batch;
  double sum[3] = {0.0, 0.0, 0.0};

  const uint32_t region0 = tc::smem_u32(mine), one = tc::smem_u32(smem + C::ONE), acc = tmem + C::ACC;
  const uint32_t id64 = tc::idesc_bf16(TB, 64), id16 = tc::idesc_bf16(TB, 16);
  const uint64_t e_mn = tc::sdesc_mn_sw128(tc::smem_u32(mine + C::E), 0);
  const int ksteps = 4 * ((in + 63) / 64);
  uint32_t loads = 0;
  auto wait = [&](uint64_t* b, uint32_t parity) {
    if (!tc::mbar_wait_abort(b, parity, abort)) ok = false;
    __syncwarp();
    tc::tc_fence_after();
  };
  auto dead = [&] { return __any_sync(0xffffffffu, *abort != 0); };
  // This thread's units of its accumulator row, once the product behind `acc` is done.
  auto read = [&](uint32_t parity, float* v) {
    wait(&bar.acc, parity);
    if (!dead()) {
#pragma unroll
      for (int q = 0; q < UNITS / 16; ++q) tc::tmem_ld16(trow + C::ACC + UNITS * half + 16 * q, v + 16 * q);
      tc::tmem_wait_ld();
    } else {
#pragma unroll
      for (int q = 0; q < UNITS; ++q) v[q] = 0.0f;
    }
  };
  auto store = [&](uint32_t tile, const float* v) {  // as BF16 into this sample's swizzled row
#pragma unroll
    for (int q = 0; q < UNITS / 8; ++q)
      *reinterpret_cast<uint4*>(mine + tile + r * 128 + (((UNITS / 8 * half + q) ^ (r & 7)) << 4)) =
          make_uint4(tc::pack_bf16(v[8 * q], v[8 * q + 1]), tc::pack_bf16(v[8 * q + 2], v[8 * q + 3]),
                     tc::pack_bf16(v[8 * q + 4], v[8 * q + 5]), tc::pack_bf16(v[8 * q + 6], v[8 * q + 7]));
  };
  // Every thread's stores and accumulator reads, before the products the leader issues next.
  auto publish = [&] {
    tc::fence_proxy_async_smem();
    tc::tc_fence_before();
    tc::named_sync(1 + ctx, GROUP);
    tc::tc_fence_after();
  };
  auto load = [&](int tile, uint32_t t) {
    uint8_t* x = mine + (t & 1) * C::REGION;
    tc::mbar_arrive_expect_tx(&bar.xfull, 2 * TILE_BYTES);
    tc::tma_load_2d(x, &xmap, tile, 0, &bar.xfull);
    tc::tma_load_2d(x + TILE_BYTES, &xmap, tile + 64, 0, &bar.xfull);
    ++loads;
  };
  // A descriptor's start address is in units of 16 bytes: a K step of 16 adds 2 (K-major) or 128 (MN-major).
  // [h | 1] . W^T of a layer of 65 inputs: 64 units, then the constant's k step.
  auto layer = [&](uint32_t h, int woff, uint32_t wstride, uint32_t idesc) {
    const uint64_t hd = tc::sdesc_sw128(h), w = tc::sdesc_sw128(tc::smem_u32(smem + woff));
#pragma unroll
    for (int k = 0; k < 4; ++k) tc::mma_bf16(acc, hd + 2 * k, w + 2 * k, idesc, k ? 1u : 0u);
    tc::mma_bf16(acc, tc::sdesc_sw128(one), w + wstride / 16, idesc, 1u);
    tc::mma_commit(&bar.acc);
  };
  // D += [h | 1]^T d over ks times 16 of the tile's samples (M = 65 of 128 units, N = 64).
  auto grad = [&](uint32_t col, uint32_t h, uint64_t d, int ks, bool fresh) {
    const uint64_t hd = tc::sdesc_mn_sw128(h, one - h);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < ks)
        tc::mma_bf16(tmem + col, hd + 128 * k, d + 128 * k, id64 | tc::A_MN | tc::B_MN, fresh && k == 0 ? 0u : 1u);
  };

  TileWalk at(a, blockIdx.x + gridDim.x * ctx);
  if (leader && at.live(a)) load(at.tile, 0);
  uint32_t t = 0;  // tiles this context has run
  for (; at.live(a); ++t) {
    const int j = at.tile + r, range = at.range, ks = at.start + a.range - at.tile <= 64 ? 4 : 8;
    const bool live = j < at.end, last = at.last(), fresh = at.tile == at.start;
    at.next(a, gridDim.x * CTXS);
    const uint32_t off_h1 = (~t & 1) * C::REGION, off_h2 = off_h1 + TILE_BYTES;
    const uint32_t x = region0 + (t & 1) * C::REGION, h1a = region0 + off_h1, h2a = region0 + off_h2;
    if (leader) {
      if (!tc::mbar_wait_abort(&bar.xfull, t & 1, abort)) ok = false;
      if (!*abort) {
        issued = true;
        tc::tc_fence_after();
        const uint64_t x_mn = tc::sdesc_mn_sw128(x, TILE_BYTES), w0 = tc::sdesc_sw128(tc::smem_u32(smem + C::W0));
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < ksteps)
            tc::mma_bf16(acc, x_mn + 128 * k, w0 + (k >> 2) * (W_BYTES / 16) + 2 * (k & 3), id64 | tc::A_MN,
                         k ? 1u : 0u);
        tc::mma_commit(&bar.acc);
        if (at.live(a)) {  // the next tile's inputs, into L2 while this one computes
          tc::tma_prefetch_2d(&xmap, at.tile, 0);
          tc::tma_prefetch_2d(&xmap, at.tile + 64, 0);
        }
      }
    }
    float s[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) s[k] = live ? __ldcg(a.samples + (long)k * batch + j) : 0.0f;

    float h1[UNITS], v[UNITS];
    read(0, h1);  // (the last tile's products, its weight gradients among them, were issued before and are done too)
#pragma unroll
    for (int k = 0; k < UNITS; ++k) h1[k] = tc::tanh_fast(h1[k]);
    store(off_h1, h1);
    publish();
    if (leader && !*abort) layer(h1a, C::W1, W_BYTES, id64);
    if (a.dump.h1 && live) {
#pragma unroll
      for (int k = 0; k < UNITS; ++k) a.dump.h1[(long)(UNITS * half + k) * batch + j] = h1[k];
    }
    read(1, v);
#pragma unroll
    for (int k = 0; k < UNITS; ++k) v[k] = tc::tanh_fast(v[k]);
    store(off_h2, v);
    publish();
    if (leader && !*abort) layer(h2a, C::W2, 16 * 128, id16);
    if (a.dump.h2 && live) {
#pragma unroll
      for (int k = 0; k < UNITS; ++k) a.dump.h2[(long)(UNITS * half + k) * batch + j] = v[k];
    }
    float o[4] = {0.0f, 0.0f, 0.0f, 0.0f}, d[6];
    wait(&bar.acc, 0);
    if (!dead()) {
      tc::tmem_ld4(trow + C::ACC, o);
      tc::tmem_wait_ld();
    }
    ppo_loss(s[0], s[1], s[2], s[3], s[4], o[0], o[1], o[2], ls, invvar, adv_mean, adv_scale, fbatch, d);
    if (!live) d[0] = d[1] = d[2] = 0.0f;
    if (half == 0)  // units 3 to 63 of the tile meet no weight: whatever d1 left there stays
      *reinterpret_cast<uint4*>(mine + C::E + r * 128 + ((r & 7) << 4)) =
          make_uint4(tc::pack_bf16(d[0], d[1]), tc::pack_bf16(d[2], 0.0f), 0u, 0u);
    publish();
    if (leader && !*abort) {
      grad(C::DW2, h2a, e_mn, ks, fresh);
      tc::mma_commit(&bar.e);
    }
    if (live && half == 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k) sum[k] += (double)d[OUT + k];
      if (a.dump.o)
        for (int k = 0; k < OUT; ++k) a.dump.o[(long)k * batch + j] = o[k];
      if (a.dump.d3)
        for (int k = 0; k < 6; ++k) a.dump.d3[(long)k * batch + j] = d[k];
    }
    // d2 = (W2^T d3) (1 - h2^2)
#pragma unroll
    for (int k = 0; k < UNITS; ++k) {
      const float4 w = w2f[UNITS * half + k];
      v[k] = tanh_grad(output_grad(w.x, w.y, w.z, d[0], d[1], d[2]), v[k]);
    }
    wait(&bar.e, t & 1);  // layer 2's weight gradient has read h2 and d3
    store(off_h2, v);
    publish();
    if (leader && !*abort) {  // d1's product, then layer 1's weight gradient behind it
      const uint64_t d2 = tc::sdesc_sw128(h2a), w1t = tc::sdesc_sw128(tc::smem_u32(smem + C::W1T));
#pragma unroll
      for (int k = 0; k < 4; ++k) tc::mma_bf16(acc, d2 + 2 * k, w1t + 2 * k, id64, k ? 1u : 0u);
      tc::mma_commit(&bar.acc);
      grad(C::DW1, h1a, tc::sdesc_mn_sw128(h2a, 0), ks, fresh);
      tc::mma_commit(&bar.f);
    }
    read(1, v);
#pragma unroll
    for (int k = 0; k < UNITS; ++k) v[k] = tanh_grad(v[k], h1[k]);
    store(C::E, v);
    publish();
    if (leader && !*abort) {
      if (at.live(a)) {  // the region of h1 and d2 takes the next tile's inputs: no product reads it any more
        if (!tc::mbar_wait_abort(&bar.f, t & 1, abort)) ok = false;
        if (!*abort) load(at.tile, t + 1);
      }
      const uint64_t x_k = tc::sdesc_sw128(x);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < ks)
          tc::mma_bf16(tmem + C::DW0, x_k + (k >> 2) * (TILE_BYTES / 16) + 2 * (k & 3), e_mn + 128 * k, id64 | tc::B_MN,
                       fresh && k == 0 ? 0u : 1u);
      tc::mma_commit(&bar.w);
    }
    if (!last) continue;
    // the range's gradients, UNITS columns a thread: accumulator row r is an input of the layer
    wait(&bar.w, t & 1);
    if (dead()) continue;
    float* part = a.part + (long)range * logstd;
#pragma unroll 1
    for (int q = UNITS / 16 * half; q < UNITS / 16 * (half + 1); ++q) {
      tc::tmem_ld16(trow + C::DW0 + 16 * q, v);
      tc::tmem_wait_ld();
      if (r < in)
#pragma unroll
        for (int k = 0; k < 16; ++k) part[(16 * q + k) * in + r] = v[k];
      tc::tmem_ld16(trow + C::DW1 + 16 * q, v);
      tc::tmem_wait_ld();
      if (r < HA)
#pragma unroll
        for (int k = 0; k < 16; ++k) part[w1 + (16 * q + k) * HA + r] = v[k];
    }
    if (half == 0) {
      tc::tmem_ld4(trow + C::DW2, v);
      tc::tmem_wait_ld();
      if (r < HA)
#pragma unroll
        for (int k = 0; k < OUT; ++k) part[w2 + k * HA + r] = v[k];
    }
    tc::tc_fence_before();  // the next range's products follow a barrier of this group
  }
  if (half == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      for (int o = 16; o; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
      if (lane == 0) sh_sums[(ctx * 4 + (warp & 3)) * 3 + k] = sum[k];
    }
  }
  // Nothing of the leader's is in flight when the CTA exits: the last copy's phase, then the products issued.
  if (leader && loads && !tc::mbar_wait(&bar.xfull, (loads - 1) & 1)) ok = false;
  if (leader && issued) {
    tc::mma_commit(&bar.drain);
    if (!tc::mbar_wait(&bar.drain, 0)) ok = false;
  }
  __syncwarp();
  tc::tc_fence_before();
  __syncthreads();
  if (tid < 3 && !*abort) {
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += sh_sums[w * 3 + tid];
    a.sums[blockIdx.x * 3 + tid] = s;
  }
  if (warp == 0) tc::tmem_dealloc(*tslot, CTXS * C::COLS);
  if (!ok) atomicExch(a.err, 1);
}

// grad[p] = the ranges' partials of weight p, added as k_wgrad_reduce adds its
// splits (thread l every 32nd range from l in order, then a butterfly over the
// 32): 32 weights a block, so the partials are read in rows of 128 bytes.
// squares[block] = the block's sum of grad^2. The last block takes the log-std
// gradients and the KL from the CTAs' sums.
constexpr int RED_W = 32;
__global__ void __launch_bounds__(RED_W * 32) k_update_reduce(const float* part, int ranges, const double* sums,
                                                             int ctas, int weights, float* grad, double* squares,
                                                             float* stats) {
  __shared__ float sh[32][RED_W + 1];
  __shared__ double sq[32];
  early_start();
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  float g = 0.0f;
  if (blockIdx.x + 1 < gridDim.x) {
    int p = blockIdx.x * RED_W + lane;  // this thread's weight while reading, range slice `row`
    float acc = 0.0f;
    if (p < weights)
#pragma unroll 5
      for (int z = row; z < ranges; z += 32) acc += __ldcg(part + (long)z * weights + p);
    sh[row][lane] = acc;
    __syncthreads();
    g = sh[lane][row];  // now weight `row` of the block, slice `lane`
#pragma unroll
    for (int o = 16; o; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
    p = blockIdx.x * RED_W + row;
    if (lane == 0 && p < weights) grad[p] = g;
    if (lane == 0) sq[row] = p < weights ? (double)g * (double)g : 0.0;
    __syncthreads();
    if (row) return;
    double q = sq[lane];
    for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    if (lane == 0) squares[blockIdx.x] = q;
    return;
  }
  if (row) return;
  double s[3] = {0.0, 0.0, 0.0};
  for (int c = lane; c < ctas; c += 32)
    for (int k = 0; k < 3; ++k) s[k] += __ldcg(sums + c * 3 + k);
#pragma unroll
  for (int k = 0; k < 3; ++k)
    for (int o = 16; o; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
  if (lane == 0) {
    const float g0 = (float)s[0], g1 = (float)s[1];
    grad[weights] = g0, grad[weights + 1] = g1;
    stats[ST_KL] = (float)s[2];
    squares[blockIdx.x] = (double)g0 * (double)g0 + (double)g1 * (double)g1;
  }
}

// racer/ppo.mojo:306-337: the gradient's norm (every block adds the partial
// sums in the same order), Adam, and the new theta's BF16 operand images
// (layouts of k_pack_weights and k_pack_w1t).
__global__ void __launch_bounds__(256) k_update_adam(int in, int parts, const double* squares, const float* c12,
                                                     float* stats, float* theta, const float* grad, float* first,
                                                     float* second, uint8_t* pack, bf16* w1t) {
  __shared__ double sh[256];
  early_start();
  double q = 0.0;
  for (int k = threadIdx.x; k < parts; k += 256) q += __ldcg(squares + k);
  sh[threadIdx.x] = q;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  const float norm = (float)sh[0];
  if (blockIdx.x == 0 && threadIdx.x == 0) stats[ST_NORM] = norm;
  const int w1 = H * in, w2 = w1 + H * HA, logstd = w2 + OUT * HA;
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= logstd + 2) return;
  const float c1 = c12[0], c2 = c12[1];
  float scale = fminf(1.0f, MAX_NORM / (sqrtf(norm) + 1e-8f));
  float g = __ldcg(grad + i) * scale;
  float m = 0.9f * first[i] + 0.1f * g;
  float v = 0.999f * second[i] + (0.001f * g) * g;
  first[i] = m;
  second[i] = v;
  float m_hat = m / c1, v_hat = v / c2;
  float value = theta[i] - (LR * m_hat) / (sqrtf(v_hat) + 1e-5f);
  if (i >= logstd) value = fminf(fmaxf(value, -2.0f), 0.0f);
  theta[i] = value;
  if (i >= logstd) return;
  const bf16 b = __float2bfloat16_rn(value);
  const int kblocks = (in + 63) / 64;
  auto at = [&](int base, int rows, int row, int k) {
    return reinterpret_cast<bf16*>(pack + base + (k >> 6) * rows * 128 + tc::sw128_offset(row, k & 63));
  };
  if (i < w1) {
    *at(0, 64, i / in, i % in) = b;
  } else if (i < w2) {
    const int row = (i - w1) / HA, k = (i - w1) % HA;
    *at(kblocks * W_BYTES, 64, row, k) = b;
    if (k < H) w1t[tc::sw128_offset(k, row) / 2] = b;
  } else {
    *at((kblocks + 2) * W_BYTES, 16, (i - w2) / HA, (i - w2) % HA) = b;
  }
}

// samples[m][5][batch] of the rollout's sample order s = 4 b + m (racer/ppo.mojo:259-268).
__global__ void k_update_samples(int n, int batch, const float* __restrict__ actions, const float* __restrict__ logp,
                                 const float* __restrict__ value, const float* __restrict__ advantage,
                                 float* __restrict__ samples) {
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= 4L * batch) return;
  const long t = s / n, i = s % n;
  float* out = samples + (s & 3) * 5L * batch + (s >> 2);
  out[0] = actions[t * 2 * n + i];
  out[batch] = actions[(t * 2 + 1) * n + i];
  out[2L * batch] = logp[s];
  out[3L * batch] = value[s];
  out[4L * batch] = advantage[s];
}

// W1^T as a swizzled K-major image: row j (input unit) holds W1[0..63][j].
__global__ void k_pack_w1t(const float* __restrict__ theta, int in, bf16* w1t) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= H * H) return;
  const int j = e / H, r = e % H;
  w1t[tc::sw128_offset(j, r) / 2] = __float2bfloat16_rn(theta[H * in + r * HA + j]);
}

int reduce_blocks(int weights) { return (weights + RED_W - 1) / RED_W + 1; }

}  // namespace

int update_work_new(int in, int batch, UpdateWork* w) {
  const int weights = H * in + H * HA + OUT * HA;
  const int kblocks = (batch + 63) / 64, per = (kblocks + WGRAD_SPLITS - 1) / WGRAD_SPLITS;
  w->in = in, w->batch = batch;
  w->range = 64 * per;
  w->ranges = (kblocks + per - 1) / per;
  w->ctas = std::min(device_sms(), w->ranges);
  RACER_TRY(cudaMalloc((void**)&w->part, sizeof(float) * (size_t)w->ranges * weights));
  RACER_TRY(cudaMalloc((void**)&w->sums, sizeof(double) * 3 * w->ctas));
  RACER_TRY(cudaMalloc((void**)&w->squares, sizeof(double) * reduce_blocks(weights)));
  RACER_TRY(cudaMalloc((void**)&w->samples, sizeof(float) * MINIBATCHES * 5 * (size_t)batch));
  RACER_TRY(cudaMalloc((void**)&w->w1t, W_BYTES));
  RACER_TRY(cudaFuncSetAttribute(k_update_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, UpdateCfg::SMEM));
  return 0;
}

void update_work_delete(UpdateWork* w) {
  cudaFree(w->part);
  cudaFree(w->sums);
  cudaFree(w->squares);
  cudaFree(w->samples);
  cudaFree(w->w1t);
  *w = UpdateWork();
}

cudaError_t launch_update_begin(UpdateWork* w, int n, const float* actions, const float* logp, const float* value,
                                const float* advantage, const float* theta, cudaStream_t st) {
  const long samples = 4L * w->batch;
  k_update_samples<<<(unsigned)((samples + 255) / 256), 256, 0, st>>>(n, w->batch, actions, logp, value, advantage,
                                                                       w->samples);
  k_pack_w1t<<<(H * H + 255) / 256, 256, 0, st>>>(theta, w->in, reinterpret_cast<bf16*>(w->w1t));
  return cudaGetLastError();
}

cudaError_t launch_update_minibatch(UpdateWork* w, int m, const CUtensorMap& xmap, float* theta, uint8_t* pack,
                                    float* grad, float* first, float* second, const float* c12, float* stats,
                                    const UpdateDump& dump, int* err, cudaStream_t st) {
  const int weights = H * w->in + H * HA + OUT * HA, blocks = reduce_blocks(weights);
  const TileArgs a{w->samples + (size_t)m * 5 * w->batch, w->in,   w->batch, w->range, w->ranges, theta, pack, w->w1t,
                   stats + ST_ADV,                        w->part, w->sums,  dump,     err};
  // Early, each behind the kernel before it: an update (16 minibatches of 262144 samples x 113 inputs) takes 1.296 ms
  // against 1.310.
  launch_early(k_update_tiles, dim3(w->ctas), UpdateCfg::THREADS, UpdateCfg::SMEM, st, xmap, a);
  launch_early(k_update_reduce, dim3(blocks), RED_W * 32, 0, st, w->part, w->ranges, w->sums, w->ctas, weights, grad,
               w->squares, stats);
  launch_early(k_update_adam, dim3((weights + 2 + 255) / 256), 256, 0, st, w->in, blocks, w->squares, c12, stats, theta,
               grad, first, second, pack, reinterpret_cast<bf16*>(w->w1t));
  return cudaGetLastError();
}

}  // namespace racer
