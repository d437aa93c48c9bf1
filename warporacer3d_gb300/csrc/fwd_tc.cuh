// The policy forward's tcgen05 epilogue (racer/ppo.mojo:40-44,108-111 layers 2
// and 3, and the sampling of racer/sim.mojo:337-346), shared by the forward
// kernels (mlp_tc.cu) and the fused rollout kernel (sim.cu): both translation
// units are built with --fmad=false, so either gives the same bits.
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"
#include "mlp_tc.h"
#include "sample.cuh"
#include "tc.cuh"

namespace racer {
namespace {

constexpr int TILE = 128;
constexpr int A_BYTES = TILE * 128;  // 128 rows x 64 bf16
constexpr int B_BYTES = 64 * 128;    // 64 rows x 64 bf16

// Epilogues of the forward (PARTS groups of four warps, each over TMEM lanes
// 0-127 = sample rows and its share of the 64 units), once
// layer 1's accumulator is complete (`done`, completion p0): tanh, H = [h | 1 | 0]
// as the next layer's A in stages 0-1 (the layer-1 stages, free by then),
// layers 2 and 3 issued by thread 0, the outputs and the fused sampling.
// After a timed-out wait (*abort set) thread 0 issues no more MMAs, the
// waits return at once and no warp reads the accumulator (which no MMA may
// have written); the results are then undefined and the error word set.
// *issued records whether this thread issued an MMA (the drain commits only then).
// With w1s, W1 is not resident: thread 0 copies it to OFF_W1 once layer 1 is done (w1bar).
// A row's 64 tanh and their packing stand in the way of the next layer, so two
// groups share them where eight warps are at hand: 100 fused steps of 1024
// cars take 1.81 ms against 2.00 with one (1.80 once warps without a row of
// the batch skip theirs).
template <int PARTS>
__device__ bool fwd_epilogue(uint8_t* smem, int OFF_A, int OFF_W1, int OFF_W2, uint32_t tmem, uint64_t* done,
                             uint32_t p0, int r, bool live, int c, int cols, float* h1g, float* h2g, float* og,
                             int write_hidden, const SampleArgs& sa, volatile int* abort, uint32_t limit,
                             bool* issued, const uint4* w1s = nullptr, uint64_t* w1bar = nullptr) {
  constexpr int UNITS = 64 / PARTS;  // of each thread's row
  const int tid = threadIdx.x, warp = tid >> 5, part = warp >> 2;
  bool ok = true;
  const uint32_t id64 = tc::idesc_bf16(TILE, 64), id16 = tc::idesc_bf16(TILE, 16);
  {
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    uint8_t* Hs = smem + OFF_A;
    if (!tc::mbar_wait_abort(done, p0 & 1, abort, limit)) ok = false;
    __syncwarp();  // the TMEM loads are warp-collective
    tc::tc_fence_after();
    const bool fetch = w1s && tid == 0 && !*abort;
    if (fetch) {  // layer 1 no longer reads W0's stages
      tc::mbar_arrive_expect_tx(w1bar, 2 * B_BYTES);
      tc::bulk_load(smem + OFF_W1, w1s, 2 * B_BYTES, w1bar);
    }
    float acc[UNITS];
    const bool busy = __any_sync(0xffffffffu, live);  // a warp of rows past the batch has nothing to hand on
    for (int layer = 0; layer < 2; ++layer) {
      if (busy) {
        if (!__any_sync(0xffffffffu, *abort != 0)) {  // warp-uniform: the loads are warp-collective
#pragma unroll
          for (int q = 0; q < UNITS / 16; ++q) tc::tmem_ld16(trow + UNITS * part + 16 * q, acc + 16 * q);
          tc::tmem_wait_ld();
        } else {
#pragma unroll
          for (int q = 0; q < UNITS; ++q) acc[q] = 0.0f;
        }
#pragma unroll
        for (int q = 0; q < UNITS; ++q) acc[q] = tc::tanh_fast(acc[q]);
#pragma unroll
        for (int q = 0; q < UNITS / 8; ++q) {
          uint4 pk = make_uint4(tc::pack_bf16(acc[8 * q], acc[8 * q + 1]),
                                tc::pack_bf16(acc[8 * q + 2], acc[8 * q + 3]),
                                tc::pack_bf16(acc[8 * q + 4], acc[8 * q + 5]),
                                tc::pack_bf16(acc[8 * q + 6], acc[8 * q + 7]));
          *reinterpret_cast<uint4*>(Hs + r * 128 + (((UNITS / 8 * part + q) ^ (r & 7)) << 4)) = pk;
          if (q < 2 && part == 0) {  // the bias's one and 15 zeros: the only step of 16 k's past h
            const uint4 hi = make_uint4(q == 0 ? tc::pack_bf16(1.0f, 0.0f) : 0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4*>(Hs + A_BYTES + r * 128 + ((q ^ (r & 7)) << 4)) = hi;
          }
        }
        if (write_hidden && live) {
          float* hg = layer == 0 ? h1g : h2g;
#pragma unroll
          for (int q = 0; q < UNITS; ++q) hg[(long)(UNITS * part + q) * cols + c] = acc[q];
        }
      }
      tc::fence_proxy_async_smem();
      tc::tc_fence_before();
      tc::named_sync(1, TILE * PARTS);
      if (layer == 0 && fetch && !tc::mbar_wait(w1bar, 0)) ok = false;
      if (tid == 0 && !*abort) {
        *issued = true;
        tc::tc_fence_after();
        const uint64_t h = tc::sdesc_sw128(tc::smem_u32(Hs));
        const uint64_t w = tc::sdesc_sw128(tc::smem_u32(smem + (layer == 0 ? OFF_W1 : OFF_W2)));
        const uint32_t wstride = layer == 0 ? B_BYTES : 16 * 128;
        const uint32_t id = layer == 0 ? id64 : id16;
#pragma unroll
        for (int k = 0; k < 4; ++k) tc::mma_bf16(tmem, h + 2 * k, w + 2 * k, id, k ? 1u : 0u);
        tc::mma_bf16(tmem, h + (A_BYTES >> 4), w + (wstride >> 4), id, 1u);
        tc::mma_commit(done);
      }
      if (!tc::mbar_wait_abort(done, (p0 + 1 + layer) & 1, abort, limit)) ok = false;
      __syncwarp();
      tc::tc_fence_after();
    }
    float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (part == 0 && !__any_sync(0xffffffffu, *abort != 0)) {  // warp-uniform
      tc::tmem_ld4(trow, o);
      tc::tmem_wait_ld();
    }
    if (part == 0 && live) {
      og[c] = o[0];
      og[(long)cols + c] = o[1];
      og[2L * cols + c] = o[2];
      if (sa.actions) {
        int64_t step = (sa.step_base ? *sa.step_base : 0) + sa.step_add;
        sample_car(cols, c, sa.seed, o[0], o[1], o[2], sa.log_std, sa.actions, sa.logp, sa.value, sa.deterministic,
                   step);
      }
    }
  }
  return ok;
}

}  // namespace
}  // namespace racer
