// Policy MLP in FP32 on the CUDA cores (racer/ppo.mojo:108-138), the precision
// of comparison runs: the forward's three layers in one kernel per block of
// samples, both data gradients in one, and the weight gradients as split-K
// products over the batch with a reduction in a fixed order.
//
// Every output is one chain of fused multiply-adds over k in ascending order
// (per split for the weight gradients), whatever the tile, so a tile is chosen
// for the parallelism: 64 outputs by 32 or 64 samples and 128 threads. The
// multiply-adds go two at a time (fma.rn.f32x2, each half rounded as fmaf), so
// the issue slots of a k step are 8 of them, two 16-byte shared loads and four
// register copies for 16 outputs a thread. With one 64 x 64 tile per 256 threads
// and nothing loaded ahead, 4096 samples of 1086 inputs kept 64 of 152 SMs
// busy: forward 333 us, data gradients 53, weight gradients 330; now 38, 13 and
// 47 (a block has one warp a scheduler, so a step costs its loads' latency).
#include "common.cuh"
#include "kernels.h"
#include "policy_tc.h"

namespace racer {
namespace {

constexpr int THREADS = 128;  // 16 rows of threads, four outputs each, by 8 columns of threads
constexpr int BM = 64, BK = 32, LDA = BM + 4;
constexpr int STAGES = 4;  // chunks of BK in flight: a block has an SM almost to itself, so its loads' latency counts

// One word into shared memory, asynchronously; zero where not valid (src is then not read).
__device__ __forceinline__ void copy4(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(valid ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void copies_end() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// This thread's copies of all but the newest STAGES - 2 groups have landed.
__device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
}

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n .reg .b64 a, b, c;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n mov.b64 c, {%6, %7};\n"
      " fma.rn.f32x2 c, a, b, c;\n mov.b64 {%0, %1}, c;\n}\n"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

// acc[r][c] += A[k][m] B[k][n] for one k: m = 4 ty + r; n = 4 tx + c, and for TN = 8 32 + 4 tx + c - 4. The shared
// loads set the pace: two rows a thread instead of four (eight warps a block) took 10% longer, A held twice (its pairs
// then need no copies) 35%.
template <int TN>
struct Acc {
  float2 v[4][TN / 2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < TN / 2; ++c) v[r][c] = make_float2(0.0f, 0.0f);
  }
  __device__ __forceinline__ float at(int r, int c) const { return c & 1 ? v[r][c >> 1].y : v[r][c >> 1].x; }
  template <int LDB>
  __device__ __forceinline__ void step(const float* A, const float* B, int k, int tx, int ty) {
    const float4 a = *reinterpret_cast<const float4*>(A + k * LDA + 4 * ty);
    const float2 m[4] = {make_float2(a.x, a.x), make_float2(a.y, a.y), make_float2(a.z, a.z), make_float2(a.w, a.w)};
#pragma unroll
    for (int h = 0; h < TN / 4; ++h) {
      const float4 b = *reinterpret_cast<const float4*>(B + k * LDB + 32 * h + 4 * tx);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        v[r][2 * h] = fma2(m[r], make_float2(b.x, b.y), v[r][2 * h]);
        v[r][2 * h + 1] = fma2(m[r], make_float2(b.z, b.w), v[r][2 * h + 1]);
      }
    }
  }
};
__device__ __forceinline__ int column(int tx, int c) { return (c >> 2) * 32 + 4 * tx + (c & 3); }

// Forward: x [in, cols] -> h1, h2 [65, cols] (rows < 64), o [3, cols], 8 TN samples a block. The row 64 of h1 and h2
// (the bias input) is read from their buffers.
template <int TN>
__global__ void __launch_bounds__(THREADS) k_fwd_f32(int in, const float* __restrict__ theta,
                                                     const float* __restrict__ x, int cols, float* h1, float* h2,
                                                     float* o) {
  constexpr int BN = 8 * TN, WELEMS = BM * BK / THREADS, XELEMS = BN * BK / THREADS;
  extern __shared__ __align__(16) float smem_f32[];
  float* As = smem_f32;                  // [STAGES][BK][LDA]; then W1 [65][LDA]
  float* Bs = As + STAGES * BK * LDA;    // [STAGES][BK][BN]
  float* Hs = Bs + STAGES * BK * BN;     // [65][BN]
  float* W2s = Hs + HA * BN;             // [3][65]
  static_assert(STAGES * BK >= HA, "W1 takes the place of the stages");
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3, n0 = blockIdx.x * BN;
  const float *w0 = theta, *w1 = theta + H * in, *w2 = w1 + H * HA;
  for (int e = tid; e < OUT * HA; e += THREADS) W2s[e] = __ldg(w2 + e);
  // W0 by 8 k's of 4 rows a warp (32-byte pieces of the rows), x by its rows
  const int wk = tid & 7, wm = 4 * (tid >> 5) + ((tid >> 3) & 3), chunks = (in + BK - 1) / BK;
  const float* wp = w0 + (long)wm * in + wk;                                        // chunk 0's first
  const float* xp = x + (long)(tid / BN) * cols + min(n0 + tid % BN, cols - 1);
  const bool n_ok = n0 + tid % BN < cols;
  auto fetch = [&](int c) {  // chunk c into stage c % STAGES; an empty group past the last
    float *A = As + c % STAGES * BK * LDA + wk * LDA + wm, *B = Bs + c % STAGES * BK * BN + tid;
    const int left = in - c * BK;  // k's of the chunk
    const float *w = wp + c * BK, *v = xp + (long)c * BK * cols;
    if (left > 0) {
#pragma unroll
      for (int i = 0; i < WELEMS; ++i) {
        const int kk = 8 * (i & 3);
        const bool ok = kk + wk < left;
        copy4(A + kk * LDA + 16 * (i >> 2), ok ? w + (long)(16 * (i >> 2)) * in + kk : w0, ok);
      }
#pragma unroll
      for (int i = 0; i < XELEMS; ++i) {
        const int kk = i * (THREADS / BN);
        const bool ok = n_ok && kk + tid / BN < left;
        copy4(B + i * THREADS, ok ? v + (long)kk * cols : x, ok);
      }
    }
    copies_end();
  };
  Acc<TN> acc;
  acc.zero();
  for (int c = 0; c < STAGES - 1; ++c) fetch(c);
  for (int c = 0; c < chunks; ++c) {
    copies_wait();
    __syncthreads();  // chunk c is everyone's, and chunk c - 1's stage is free
    fetch(c + STAGES - 1);
    const float *A = As + c % STAGES * BK * LDA, *B = Bs + c % STAGES * BK * BN;
#pragma unroll
    for (int k = 0; k < BK; ++k) acc.template step<BN>(A, B, k, tx, ty);
  }
  __syncthreads();
  for (int layer = 0; layer < 2; ++layer) {
    float* h = layer ? h2 : h1;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < TN; ++c) {
        const float v = tanhf(acc.at(r, c));
        const int m = 4 * ty + r, n = column(tx, c);
        Hs[m * BN + n] = v;
        if (n0 + n < cols) h[(long)m * cols + n0 + n] = v;
      }
    for (int n = tid; n < BN; n += THREADS) Hs[H * BN + n] = n0 + n < cols ? h[(long)H * cols + n0 + n] : 0.0f;
    if (layer == 0)
      for (int e = tid; e < H * HA; e += THREADS) As[(e % HA) * LDA + e / HA] = __ldg(w1 + e);
    __syncthreads();
    if (layer == 0) {
      acc.zero();
#pragma unroll 5
      for (int k = 0; k < HA; ++k) acc.template step<BN>(As, Hs, k, tx, ty);
      __syncthreads();
    }
  }
  for (int e = tid; e < OUT * BN; e += THREADS) {
    const int m = e / BN, n = e % BN;
    float v = 0.0f;
    for (int k = 0; k < HA; ++k) v = fmaf(W2s[m * HA + k], Hs[k * BN + n], v);
    if (n0 + n < cols) o[(long)m * cols + n0 + n] = v;
  }
}

// Data gradients of 32 samples a block: d2 = (W2^T d3) (1 - h2^2), d1 = (W1^T d2[:64]) (1 - h1^2), all 65 rows.
__global__ void __launch_bounds__(THREADS) k_dgrad_f32(int in, const float* __restrict__ theta,
                                                       const float* __restrict__ d3, const float* __restrict__ h1,
                                                       const float* __restrict__ h2, float* __restrict__ d2,
                                                       float* __restrict__ d1, int cols) {
  constexpr int BN = 32;
  __shared__ __align__(16) float As[H * LDA];  // W1 [r][j]: the product's k is r, its row j
  __shared__ __align__(16) float Ds[H * BN];
  __shared__ float W2s[OUT * HA];
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3, n0 = blockIdx.x * BN;
  const float *w1 = theta + H * in, *w2 = w1 + H * HA;
  for (int e = tid; e < OUT * HA; e += THREADS) W2s[e] = __ldg(w2 + e);
  for (int e = tid; e < H * HA; e += THREADS) As[e / HA * LDA + e % HA] = __ldg(w1 + e);
  const int n = tid & 31, j = n0 + n;
  const bool live = j < cols;
  float e[OUT];
#pragma unroll
  for (int k = 0; k < OUT; ++k) e[k] = live ? __ldg(d3 + (long)k * cols + j) : 0.0f;
  __syncthreads();
#pragma unroll 4
  for (int k = tid >> 5; k < HA; k += THREADS / 32) {
    const float h = live ? __ldg(h2 + (long)k * cols + j) : 0.0f;
    const float v = tanh_grad(output_grad(W2s[k], W2s[HA + k], W2s[2 * HA + k], e[0], e[1], e[2]), h);
    if (k < H) Ds[k * BN + n] = v;
    if (live) d2[(long)k * cols + j] = v;
  }
  __syncthreads();
  Acc<4> acc;
  acc.zero();
#pragma unroll 8
  for (int k = 0; k < H; ++k) acc.step<BN>(As, Ds, k, tx, ty);
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int m = 4 * ty + r, col = n0 + column(tx, c);
      if (col < cols) d1[(long)m * cols + col] = tanh_grad(acc.at(r, c), __ldg(h1 + (long)m * cols + col));
    }
  if (tid < BN && live) {  // the bias input's row
    float v = 0.0f;
    for (int k = 0; k < H; ++k) v = fmaf(As[k * LDA + H], Ds[k * BN + n], v);
    d1[(long)H * cols + j] = tanh_grad(v, __ldg(h1 + (long)H * cols + j));
  }
}

// A weight gradient C[M, N] = A[M, K] B[N, K]^T over the batch (K = cols, contiguous in both): M <= 64 rows a block,
// 32 columns, split z the K range [z kper, (z + 1) kper) into P[z][M][N].
struct WgradArgs {
  const float *A, *B;
  float* P;
  int M, N, kper, tiles, splits;  // tiles of 32 columns
};

__global__ void __launch_bounds__(THREADS) k_wgrad_f32(const WgradArgs first, const WgradArgs second, int K) {
  constexpr int BN = 32, LDB = BN + 4, AELEMS = BM * BK / THREADS, BELEMS = BN * BK / THREADS;
  extern __shared__ __align__(16) float smem_f32[];
  float *As = smem_f32, *Bs = As + STAGES * BK * LDA;
  int b = blockIdx.x;
  const bool own = b < first.tiles * first.splits;
  const WgradArgs& g = own ? first : second;
  if (!own) b -= first.tiles * first.splits;
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3, n0 = b % g.tiles * BN, z = b / g.tiles;
  const int k0 = z * g.kper, k1 = min(K, k0 + g.kper);
  const int lk = tid & 7, lm = 4 * (tid >> 5) + ((tid >> 3) & 3);  // loads: 8 k's of 4 rows a warp, as the forward's W0
  const int chunks = (k1 - k0 + BK - 1) / BK;
  const float *ap = g.A + (long)lm * K + k0 + lk, *bp = g.B + (long)(n0 + lm) * K + k0 + lk;
  auto fetch = [&](int c) {
    float *A = As + c % STAGES * BK * LDA + lk * LDA + lm, *B = Bs + c % STAGES * BK * LDB + lk * LDB + lm;
    const int left = k1 - k0 - c * BK;
    const float *pa = ap + c * BK, *pb = bp + c * BK;
    if (left > 0) {
#pragma unroll
      for (int i = 0; i < AELEMS; ++i) {
        const int kk = 8 * (i & 3), m = 16 * (i >> 2);
        const bool ok = kk + lk < left && m + lm < g.M;
        copy4(A + kk * LDA + m, ok ? pa + (long)m * K + kk : g.A, ok);
      }
#pragma unroll
      for (int i = 0; i < BELEMS; ++i) {
        const int kk = 8 * (i & 3), n = 16 * (i >> 2);
        const bool ok = kk + lk < left && n0 + n + lm < g.N;
        copy4(B + kk * LDB + n, ok ? pb + (long)n * K + kk : g.B, ok);
      }
    }
    copies_end();
  };
  Acc<4> acc;
  acc.zero();
  for (int c = 0; c < STAGES - 1; ++c) fetch(c);
  for (int c = 0; c < chunks; ++c) {
    copies_wait();
    __syncthreads();
    fetch(c + STAGES - 1);
    const float *A = As + c % STAGES * BK * LDA, *B = Bs + c % STAGES * BK * LDB;
#pragma unroll
    for (int k = 0; k < BK; ++k) acc.step<LDB>(A, B, k, tx, ty);
  }
  float* P = g.P + (long)z * g.M * g.N;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int m = 4 * ty + r, n = n0 + column(tx, c);
      if (m < g.M && n < g.N) P[(long)m * g.N + n] = acc.at(r, c);
    }
}

// C[e] = sum over splits of P[z][e] in order; elements [0, count) of the first product, then the second's.
__global__ void k_split_reduce(const float* P, int splits, long count, float* C, const float* P2, int splits2,
                               long count2, float* C2) {
  long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= count) {
    e -= count;
    if (e >= count2) return;
    P = P2, splits = splits2, count = count2, C = C2;
  }
  float acc = 0.0f;
#pragma unroll 8
  for (int z = 0; z < splits; ++z) acc += P[(long)z * count + e];
  C[e] = acc;
}

int splits_for(int K, int tiles) {
  // enough blocks to fill the GPU, at least 512 K per split
  int want = std::max(1, SPLIT_CTAS / std::max(1, tiles));
  int most = std::max(1, K / 512);
  return std::min(want, most);
}

// The split plan of a product [M, N] over K, the same on every device: K ranges of whole 16s, counted over 64 x 64
// tiles.
void split_plan(int M, int N, int K, int* kper, int* splits) {
  *splits = splits_for(K, ((N + 63) / 64) * ((M + 63) / 64));
  *kper = K;
  if (*splits > 1) {
    *kper = ((K + *splits - 1) / *splits + 15) / 16 * 16;
    *splits = (K + *kper - 1) / *kper;
  }
}

// Floats of split-K partials a product uses (0 when unsplit).
size_t split_need(int M, int N, int K) {
  int kper, splits;
  split_plan(M, N, K, &kper, &splits);
  return splits > 1 ? (size_t)splits * M * N : 0;
}

// A product into C (unsplit) or its partials at P.
WgradArgs wgrad_args(const float* A, const float* B, float* C, float* P, int M, int N, int K) {
  WgradArgs g{A, B, C, M, N, 0, (N + 31) / 32, 0};
  split_plan(M, N, K, &g.kper, &g.splits);
  if (g.splits > 1) g.P = P;
  return g;
}

}  // namespace

void launch_fwd_f32(int in, const float* theta, const float* x, int cols, float* h1, float* h2, float* o,
                    cudaStream_t st) {
  auto smem = [](int bn) { return (int)sizeof(float) * (STAGES * BK * (LDA + bn) + HA * bn + OUT * HA + 1); };
  // 64 samples a block once that still gives every SM two blocks: half the shared loads of W0 per multiply-add
  if ((cols + 63) / 64 >= 2 * device_sms()) {
    static unsigned long long configured = 0;  // per device
    once_per_device(&configured, [&] {
      return cudaFuncSetAttribute(k_fwd_f32<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem(64));
    });
    k_fwd_f32<8><<<(cols + 63) / 64, THREADS, smem(64), st>>>(in, theta, x, cols, h1, h2, o);
  } else {
    static unsigned long long configured = 0;
    once_per_device(&configured, [&] {
      return cudaFuncSetAttribute(k_fwd_f32<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem(32));
    });
    k_fwd_f32<4><<<(cols + 31) / 32, THREADS, smem(32), st>>>(in, theta, x, cols, h1, h2, o);
  }
}

// Split-K partials: splits * tiles <= SPLIT_CTAS and every tile is at most 64 x 64.
size_t backward_scratch_floats(int in, int cols) {
  (void)in;
  (void)cols;
  return BACKWARD_SCRATCH_FLOATS;
}

// W0's product uses the scratch alone, then W1's and W2's together.
size_t backward_scratch_needed(int in, int cols) {
  return std::max(split_need(H, in, cols), split_need(H, HA, cols) + split_need(OUT, HA, cols));
}
static_assert((size_t)(SPLIT_CTAS / 2) * (H + OUT) * HA <= BACKWARD_SCRATCH_FLOATS, "W1's and W2's partials together");

// racer/ppo.mojo:113-138: d3 [3, cols] -> d2, d1 [HA, cols], grad[W0|W1|W2].
void launch_backward(int in, const float* theta, const float* x, int cols, const float* h1, const float* h2,
                     const float* d3, float* d2, float* d1, float* grad, float* scratch, cudaStream_t st) {
  const int w1 = H * in, w2 = w1 + H * HA;
  k_dgrad_f32<<<(cols + 31) / 32, THREADS, 0, st>>>(in, theta, d3, h1, h2, d2, d1, cols);
  constexpr int smem = sizeof(float) * STAGES * BK * (LDA + 32 + 4);
  static unsigned long long configured = 0;  // per device
  once_per_device(&configured, [&] {
    return cudaFuncSetAttribute(k_wgrad_f32, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  auto run = [&](const WgradArgs& a, const WgradArgs& b, float* ca, float* cb) {
    k_wgrad_f32<<<a.tiles * a.splits + b.tiles * b.splits, THREADS, smem, st>>>(a, b, cols);
    const long na = a.splits > 1 ? (long)a.M * a.N : 0, nb = b.splits > 1 ? (long)b.M * b.N : 0;
    if (na + nb)
      k_split_reduce<<<(unsigned)((na + nb + 127) / 128), 128, 0, st>>>(a.P, a.splits, na, ca, b.P, b.splits, nb, cb);
  };
  run(wgrad_args(d1, x, grad, scratch, H, in, cols), WgradArgs{}, grad, nullptr);
  const WgradArgs g1 = wgrad_args(d2, h1, grad + w1, scratch, H, HA, cols);
  run(g1, wgrad_args(d3, h2, grad + w2, scratch + split_need(H, HA, cols), OUT, HA, cols), grad + w1, grad + w2);
}

}  // namespace racer
