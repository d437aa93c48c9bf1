// Track compilation on the GPU: the per-cell work of the reference's track
// compiler (racer/track.py:54-125) as CUDA kernels, in binary64 without
// contraction, so the packed grids equal the reference's bit for bit.
//
//   k_cells        racer/track.py:73-86, 89, 56  passes of the route over
//                  each cell (ball query of radius half_width + 0.5), the
//                  nearest waypoint of each pass, their reduction to layers,
//                  and the nearest waypoint overall
//   k_fill         racer/track.py:94-104         clearance, height, waypoint
//   k_ramps        racer/track.py:111-118        ramp boxes onto the heights
//   k_ft_columns,  racer/track.py:119-120        feature transform (nearest
//   k_ft_rows                                    road cell of every cell)
//   k_blur_*       racer/track.py:121            Gaussian blur, sigma 1.5
//   k_image_clear  racer/track.py:57             signed distance of an image
//
// Nearest-waypoint searches are exact brute force over a candidate list: a
// block of 16 x 16 cells keeps, in ascending index order, every waypoint
// whose distance to the block's bounding box could make it the nearest of
// some cell or put it inside the ball of one (bounds in 32 bits with a margin
// above their rounding), so each cell scans a few waypoints in the order the
// full scan would. Ties go to the lower index, as the reference's arrays show.
//
// The feature transform is the separable exact Euclidean one: per column the
// nearest feature row (ties to the lower row), then per row the nearest of
// those candidates (ties to the lower column), found by halving the row: the
// nearest candidate's column is monotone along it. The blur is the 13-tap correlation of sigma 1.5 with
// reflected edges, axis 0 then axis 1, each output summed as its centre tap
// and then symmetric pairs from the outermost inward.
#include <cuda_runtime.h>

#include <climits>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"

namespace {

constexpr int TILE = 16;  // cells per block edge in k_cells
constexpr int MAX_PASSES = 8;
constexpr int CAND_MAX = 2048;

struct RampRow {
  double cx, cy, c, s, length, width, height, rise;
};

struct Blur {
  double w[13];
};

struct CellArgs {
  const double* route;  // [W][3]
  int W;
  double x0, y0, cell;
  int nx, ny;
  double r2;             // ball radius squared; negative: nearest waypoint only
  int* nearest;          // [cells]
  int* count;            // [cells] layers kept (ball query only)
  int* pw;               // [cells][MAX_PASSES]
  unsigned char* upper;  // [W]
  int* error;
};

__device__ __forceinline__ double cell_x(double x0, double cell, int ix) { return x0 + cell * (double)ix; }

// A waypoint's place from the corner of a block's box, in 32 bits.
__device__ __forceinline__ float2 place(const CellArgs& a, int w, double2 corner) {
  return make_float2((float)(a.route[3 * w] - corner.x), (float)(a.route[3 * w + 1] - corner.y));
}

// A block's candidate waypoints: their indices, ascending, and places. `margin` is above twice what rounding can do to
// a difference of two squared distances: what differs by more is ordered as in
// 64 bits, also after the square root. Infinite or NaN where a place is out of
// range, so that 64 bits decide.
struct Candidates {
  const int* w;
  const float2* at;
  int n;
  double2 corner;
  float margin;
};

// One cell's nearest waypoint (*nearest) and, for a ball query, its passes
// and the nearest waypoint of each (racer/track.py:73-86 and 89). (fx, fy) is
// the cell's place from the corner of the block's box. Distances are compared
// in 32 bits and again in 64 where those leave it open: 64-bit arithmetic runs
// at 1/64 of the 32-bit rate, and comparing every candidate in it, with a
// square root for each within the ball, took 257 us for 721 x 441 cells and
// 285 waypoints against 55.
template <bool ALL>
__device__ int cell_passes(const CellArgs& a, const Candidates& cand, double x, double y, float fx, float fy, int* out,
                           int* nearest) {
  auto square = [&](int w) {
    const double dx = a.route[3 * w] - x, dy = a.route[3 * w + 1] - y;
    return dx * dx + dy * dy;
  };
  auto farther = [&](int u, int w) { return sqrt(square(w)) < sqrt(square(u)); };  // w is nearer than u
  const bool ball = a.r2 >= 0.0;
  const float r2 = (float)a.r2, margin = cand.margin;
  int pbest[MAX_PASSES];
  int np = 0, first = -1, last = -10, best = -1, pass = 0;  // pass: the nearest of the last one
  float bd = INFINITY, pd = 0.0f;                           // squared
  for (int i = 0; i < cand.n; ++i) {
    const int w = ALL ? i : cand.w[i];
    const float2 at = ALL ? place(a, w, cand.corner) : cand.at[i];
    const float dx = at.x - fx, dy = at.y - fy, d2 = dx * dx + dy * dy;
    if (d2 < bd - margin) {
      bd = d2, best = w;
    } else if (!(d2 > bd + margin)) {
      const double q = square(w);
      if (q < (best < 0 ? INFINITY : square(best))) bd = d2, best = w;
    }
    if (!ball || d2 > r2 + margin) continue;
    if (!(d2 < r2 - margin) && !(square(w) <= a.r2)) continue;
    if (np == 0 || w - last > 2) {  // a gap of more than 2 starts a new pass
      if (np == MAX_PASSES) return -1;
      if (np) pbest[np - 1] = pass;
      pass = w, pd = d2, ++np;
    } else if (d2 < pd - margin || (!(d2 > pd + margin) && farther(pass, w))) {
      pass = w, pd = d2;
    }
    if (first < 0) first = w;
    last = w;
  }
  *nearest = best < 0 ? 0 : best;
  if (np == 0) return 0;
  pbest[np - 1] = pass;
  if (np > 1 && first == 0 && last == a.W - 1) {  // the pass through the seam: its end, then its start
    if (farther(pbest[np - 1], pbest[0])) pbest[np - 1] = pbest[0];
    pbest[0] = pbest[np - 1], --np;
  }
  for (int i = 1; i < np; ++i) {  // stable sort by height
    const int w = pbest[i];
    const double z = a.route[3 * w + 2];
    int j = i;
    while (j > 0 && a.route[3 * pbest[j - 1] + 2] > z) pbest[j] = pbest[j - 1], --j;
    pbest[j] = w;
  }
  if (a.route[3 * pbest[np - 1] + 2] - a.route[3 * pbest[0] + 2] < 0.3) {  // one level: the nearest pass
    int bw = pbest[0];
    for (int i = 1; i < np; ++i)
      if (farther(bw, pbest[i])) bw = pbest[i];
    out[0] = bw;
    return 1;
  }
  for (int i = 0; i < np; ++i) out[i] = pbest[i];
  return np;
}

__global__ void __launch_bounds__(TILE * TILE) k_cells(CellArgs a) {
  __shared__ float2 s_at[CAND_MAX];
  __shared__ int s_w[CAND_MAX];
  __shared__ float s_min[TILE * TILE / 32];
  __shared__ int s_warp[TILE * TILE / 32];
  __shared__ int s_total;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ix0 = blockIdx.x * TILE, iy0 = blockIdx.y * TILE;
  const double bx0 = cell_x(a.x0, a.cell, ix0), bx1 = cell_x(a.x0, a.cell, min(ix0 + TILE - 1, a.nx - 1));
  const double by0 = cell_x(a.y0, a.cell, iy0), by1 = cell_x(a.y0, a.cell, min(iy0 + TILE - 1, a.ny - 1));

  const double2 corner = make_double2(bx0, by0);
  const float ex = (float)(bx1 - bx0), ey = (float)(by1 - by0);

  // the smallest, over waypoints, of the distance to the box's farthest point
  float m = INFINITY;
  for (int w = tid; w < a.W; w += blockDim.x) {
    const float2 p = place(a, w, corner);
    const float fx = fmaxf(fabsf(p.x), fabsf(p.x - ex)), fy = fmaxf(fabsf(p.y), fabsf(p.y - ey));
    m = fminf(m, fx * fx + fy * fy);
  }
  for (int o = 16; o; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) s_min[warp] = m;
  if (tid == 0) s_total = 0;
  __syncthreads();
  m = s_min[0];
  for (int i = 1; i < TILE * TILE / 32; ++i) m = fminf(m, s_min[i]);
  // Places within sqrt(thr) of the box are at most `reach` long, which is off by 2^-24 of it; so are a cell's. A squared
  // distance between the two is off by 20 x 2^-24 reach^2 at most.
  float thr = fmaxf(m, (float)a.r2) * (1.0f + 1e-5f) + 1e-36f;
  const float reach = sqrtf(thr) + fmaxf(ex, ey), margin = reach * reach * 0x1p-16f + 1e-36f;
  thr += margin;

  // candidates: waypoints whose distance to the box is within thr, in index order
  bool overflow = false;
  for (int base = 0; base < a.W; base += blockDim.x) {
    const int w = base + tid;
    bool take = false;
    float2 p = make_float2(0.0f, 0.0f);
    if (w < a.W) {
      p = place(a, w, corner);
      const float dx = fmaxf(fmaxf(-p.x, p.x - ex), 0.0f), dy = fmaxf(fmaxf(-p.y, p.y - ey), 0.0f);
      take = dx * dx + dy * dy <= thr;
    }
    const unsigned ballot = __ballot_sync(0xffffffffu, take);
    if (lane == 0) s_warp[warp] = __popc(ballot);
    __syncthreads();
    int offset = s_total;
    for (int i = 0; i < warp; ++i) offset += s_warp[i];
    offset += __popc(ballot & ((1u << lane) - 1u));
    if (take && offset < CAND_MAX) s_w[offset] = w, s_at[offset] = p;
    __syncthreads();
    if (tid == 0)
      for (int i = 0; i < TILE * TILE / 32; ++i) s_total += s_warp[i];
    __syncthreads();
  }
  const int total = s_total;
  overflow = total > CAND_MAX;  // scan every waypoint from global memory instead

  const int ix = ix0 + (tid % TILE), iy = iy0 + (tid / TILE);
  if (ix >= a.nx || iy >= a.ny) return;
  const double x = cell_x(a.x0, a.cell, ix), y = cell_x(a.y0, a.cell, iy);
  const long k = (long)iy * a.nx + ix;
  const Candidates cand{s_w, s_at, overflow ? a.W : total, corner, margin};
  int out[MAX_PASSES], best = 0;
  const float fx = (float)(x - corner.x), fy = (float)(y - corner.y);
  const int got = overflow ? cell_passes<true>(a, cand, x, y, fx, fy, out, &best)
                           : cell_passes<false>(a, cand, x, y, fx, fy, out, &best);
  a.nearest[k] = best;
  if (a.r2 < 0.0) return;
  if (got < 0) {
    atomicExch(a.error, 4);
    a.count[k] = 0;
    return;
  }
  a.count[k] = got;
  for (int i = 0; i < got; ++i) {
    a.pw[k * MAX_PASSES + i] = out[i];
    if (i > 0) a.upper[out[i]] = 1;
  }
}

// Bit 1: some pass lies on the lower layer; bit 2: some on the upper.
__global__ void k_layer_flags(const int* count, const int* pw, const unsigned char* upper, long cells, int* flags) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  int f = 0;
  if (k < cells)
    for (int i = 0; i < count[k]; ++i) f |= upper[pw[k * MAX_PASSES + i]] ? 2 : 1;
  f = __reduce_or_sync(0xffffffffu, f);
  if ((threadIdx.x & 31) == 0 && f) atomicOr(flags, f);
}

struct FillArgs {
  const double *route, *cos_h, *sin_h, *grade;
  const int *nearest, *count, *pw;
  const unsigned char* upper;
  double half_width, bank, x0, y0, cell;
  int nx, layers, layer_lo, layer_hi;
  long cells;
  double *clearance, *height;  // [layers][cells]
  int* waypoint;               // [layers][cells]
};

// racer/track.py:94-104: off the road clearance -10, height 0 and the nearest
// waypoint; on it, each pass's clearance, height and waypoint (a later pass
// of the same layer overwrites an earlier one).
__global__ void k_fill(FillArgs a) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= a.cells) return;
  for (int l = 0; l < a.layers; ++l) {
    a.clearance[l * a.cells + k] = -10.0;
    a.height[l * a.cells + k] = 0.0;
    a.waypoint[l * a.cells + k] = a.nearest[k];
  }
  const double x = cell_x(a.x0, a.cell, (int)(k % a.nx)), y = cell_x(a.y0, a.cell, (int)(k / a.nx));
  for (int i = 0; i < a.count[k]; ++i) {
    const int w = a.pw[k * MAX_PASSES + i];
    const int l = a.upper[w] ? a.layer_hi : a.layer_lo;
    const double dx = x - a.route[3 * w], dy = y - a.route[3 * w + 1];
    const double c = a.cos_h[w], s = a.sin_h[w];
    const double along = dx * c + dy * s, left = -dx * s + dy * c;
    a.clearance[l * a.cells + k] = a.half_width - fabs(left);
    a.height[l * a.cells + k] = a.route[3 * w + 2] + a.grade[w] * along - a.bank * left;
    a.waypoint[l * a.cells + k] = w;
  }
}

// racer/track.py:111-117: each ramp's sloped top added to every layer's height.
__global__ void k_ramps(const RampRow* ramps, int n, double x0, double y0, double cell, int nx, long cells, int layers,
                        double* height) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= cells) return;
  const double x = cell_x(x0, cell, (int)(k % nx)), y = cell_x(y0, cell, (int)(k / nx));
  for (int r = 0; r < n; ++r) {
    const RampRow p = ramps[r];
    const double rx = x - p.cx, ry = y - p.cy;
    const double v = -rx * p.s + ry * p.c;
    double add = 0.0;  // outside the box the reference adds +0.0 too
    if (fabs(v) < p.width / 2) {
      const double u = rx * p.c + ry * p.s + p.length / 2;
      const double q = fmin(u, p.length - u) / p.rise;
      add = p.height * fmin(fmax(q, 0.0), 1.0);
    }
    for (int l = 0; l < layers; ++l) height[l * cells + k] += add;
  }
}

__global__ void k_mask_road(const double* clearance, long cells, unsigned char* feature) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k < cells) feature[k] = clearance[k] > 0.0;
}

__global__ void k_mask_image(const unsigned char* free_, long cells, unsigned char* wall, unsigned char* open) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k < cells) wall[k] = free_[k] == 0, open[k] = free_[k] != 0;
}

// Per column, the nearest feature row (ties to the lower row), -1 if none: a
// block per 32 columns, a lane each, a warp per stretch of the rows. Each warp
// finds the first and last feature of its stretch, from which every stretch
// gets the last one above it and the first below; then it walks its rows down
// and up. Rows of 32 cells are read and written together (a warp per column,
// its lanes down the rows, took 22.5 us for 721 x 441 cells; this takes 11.2).
constexpr int FT_WARPS = 32;
__global__ void __launch_bounds__(FT_WARPS * 32) k_ft_columns(const unsigned char* __restrict__ feature, int ny, int nx,
                                                              int* fy) {
  __shared__ int s_first[FT_WARPS][32], s_last[FT_WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, x = blockIdx.x * 32 + lane;
  const int rows = (ny + FT_WARPS - 1) / FT_WARPS, y0 = min(warp * rows, ny), y1 = min(y0 + rows, ny);
  int first = INT_MAX, last = -1;
  if (x < nx) {
#pragma unroll 8
    for (int y = y0; y < y1; ++y)
      if (feature[(long)y * nx + x]) first = min(first, y), last = y;
  }
  s_first[warp][lane] = first, s_last[warp][lane] = last;
  __syncthreads();
  int above = -1, below = INT_MAX;
  for (int i = 0; i < warp; ++i) above = max(above, s_last[i][lane]);
  for (int i = warp + 1; i < FT_WARPS; ++i) below = min(below, s_first[i][lane]);
  if (x >= nx) return;
#pragma unroll 8
  for (int y = y0; y < y1; ++y) {
    if (feature[(long)y * nx + x]) above = y;
    fy[(long)y * nx + x] = above;
  }
#pragma unroll 8
  for (int y = y1 - 1; y >= y0; --y) {
    const int p = fy[(long)y * nx + x];
    if (p == y) below = y;
    if (below != INT_MAX && (p < 0 || below - y < y - p)) fy[(long)y * nx + x] = below;
  }
}

// Per row, the flat index of every cell's nearest feature (-1 when the grid
// has none); of equally near ones, the lowest column's. That column never
// falls from one cell of a row to the next, so a cell halfway between two
// solved ones searches only the columns from the one's answer to the other's:
// a warp per cell down to every 32nd cell, then a lane per cell over the
// columns that the 31 cells between share, nx (1 + log2(nx / 32) / 32) warp
// steps a row at most. D holds a squared distance. A block per row; the row is
// staged in shared memory when STAGED. Bound by the few steps in turn that the
// last segments take: 441 rows of 721 cells take 17 us (a thread per row,
// walking its lower envelope: 210 us).
constexpr int FT_ROW_WARPS = 8;
template <class D, bool STAGED>
__global__ void __launch_bounds__(FT_ROW_WARPS * 32) k_ft_rows(const int* __restrict__ fy, int nx, int* src) {
  extern __shared__ int ft_smem[];
  const int y = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int* row = fy + (long)y * nx;
  int* out = src + (long)y * nx;  // solved cells are read back by the other warps of the block
  if (STAGED) {
    for (int x = threadIdx.x; x < nx; x += FT_ROW_WARPS * 32) ft_smem[x] = row[x];
    __syncthreads();
    row = ft_smem;
  }
  constexpr D FAR = sizeof(D) == 4 ? (D)INT_MAX : (D)LLONG_MAX;
  auto distance = [&](int f, int column, int x) {
    const D dy = f - y, dx = column - x;
    return f < 0 ? FAR : dx * dx + dy * dy;
  };
  auto column_of = [&](int x, int none) { return x < 0 || x >= nx || out[x] < 0 ? none : out[x] % nx; };
  int top = 32;
  while (top < nx) top *= 2;
  for (int step = top; step >= 32; step >>= 1) {  // cells 0, then the odd multiples of each step
    for (long i = warp;; i += FT_ROW_WARPS) {
      const long at = step == top ? i * step : (2 * i + 1) * step;
      if (at >= nx) break;
      const int x = (int)at;
      const int lo = step == top ? 0 : column_of(x - step, 0);
      const int hi = step == top ? nx - 1 : column_of(at + step < nx ? x + step : -1, nx - 1);
      D best = FAR;
      int column = -1;
      for (int c = lo + lane; c <= hi; c += 32) {
        const D d = distance(row[c], c, x);
        if (d < best) best = d, column = c;
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        const D d = __shfl_xor_sync(0xffffffffu, best, o);
        const int c = __shfl_xor_sync(0xffffffffu, column, o);
        if (d < best || (d == best && (unsigned)c < (unsigned)column)) best = d, column = c;
      }
      if (lane == 0) out[x] = column < 0 ? -1 : row[column] * nx + column;
    }
    __syncthreads();
  }
  for (int x0 = warp * 32; x0 < nx; x0 += FT_ROW_WARPS * 32) {
    const int lo = column_of(x0, 0), hi = column_of(nx - x0 > 32 ? x0 + 32 : -1, nx - 1);
    const int x = min(x0 + lane, nx - 1);
    D best = FAR;
    int column = -1;
#pragma unroll 4
    for (int c = lo; c <= hi; ++c) {
      const D d = distance(row[c], c, x);
      if (d < best) best = d, column = c;
    }
    if (lane && x0 + lane < nx) out[x] = column < 0 ? -1 : row[column] * nx + column;
  }
}

__global__ void k_gather(const double* height, const int* src, long cells, double* filled) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k < cells) filled[k] = height[src[k]];
}

__device__ __forceinline__ int reflect(int i, int n) {
  int m = i % (2 * n);
  if (m < 0) m += 2 * n;
  return m >= n ? 2 * n - 1 - m : m;
}

__global__ void k_blur_rows(const double* in, int ny, int nx, Blur b, double* out) {  // along axis 0
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= (long)nx * ny) return;
  const int x = (int)(k % nx), y = (int)(k / nx);
  double s = in[k] * b.w[6];
#pragma unroll
  for (int j = 6; j >= 1; --j)
    s += (in[(long)reflect(y - j, ny) * nx + x] + in[(long)reflect(y + j, ny) * nx + x]) * b.w[6 - j];
  out[k] = s;
}

__global__ void k_blur_cols(const double* in, int ny, int nx, Blur b, float* out) {  // along axis 1, to float32
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= (long)nx * ny) return;
  const int x = (int)(k % nx);
  const double* r = in + (k - x);
  double s = r[x] * b.w[6];
#pragma unroll
  for (int j = 6; j >= 1; --j) s += (r[reflect(x - j, nx)] + r[reflect(x + j, nx)]) * b.w[6 - j];
  out[k] = (float)s;
}

__global__ void k_write_layer(const double* clearance, const int* waypoint, long cells, float* out) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= cells) return;
  out[k] = (float)clearance[k];
  out[2 * cells + k] = (float)waypoint[k];
}

// racer/track.py:57: (distance to the nearest wall - distance to the nearest
// free cell - 0.5) * cell, distances from the feature transforms.
__global__ void k_image_clear(const unsigned char* free_, const int* to_wall, const int* to_open, int nx, long cells,
                              double cell, double* clearance) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= cells) return;
  const int f = free_[k] ? to_wall[k] : to_open[k];
  const double dy = (double)(f / nx) - (double)(k / nx), dx = (double)(f % nx) - (double)(k % nx);
  const double d = sqrt(dy * dy + dx * dx);
  const double a = free_[k] ? d : 0.0, b = free_[k] ? 0.0 : d;
  clearance[k] = (a - b - 0.5) * cell;
}

Blur blur_weights() {  // sigma 1.5, radius 6
  const double sigma = 1.5;
  double phi[13];
  for (int i = 0; i < 13; ++i) {
    const double x = i - 6;
    phi[i] = std::exp(-0.5 / (sigma * sigma) * (x * x));
  }
  // the sum in pairwise order: eight leading terms as a tree, then the rest in turn
  double sum = ((phi[0] + phi[1]) + (phi[2] + phi[3])) + ((phi[4] + phi[5]) + (phi[6] + phi[7]));
  for (int i = 8; i < 13; ++i) sum += phi[i];
  Blur b;
  for (int i = 0; i < 13; ++i) b.w[i] = phi[i] / sum;
  return b;
}

// Device buffers of one compilation, freed on every exit path: `get` names the
// ones that `take` then lays out in one allocation (an allocation and its
// release cost 20 us or more of host time each, and a ribbon has 19 buffers).
struct Scratch {
  struct Buffer {
    void** p;
    size_t bytes;
  };
  std::vector<Buffer> wanted;
  std::vector<void*> ptrs;
  ~Scratch() {
    for (void* p : ptrs) cudaFree(p);
  }
  template <class T>
  void get(T** p, size_t count) {
    wanted.push_back({(void**)p, (count * sizeof(T) + 255) / 256 * 256});
  }
  cudaError_t take() {
    size_t total = 0;
    for (const Buffer& b : wanted) total += b.bytes;
    char* at = nullptr;
    if (cudaError_t e = cudaMalloc((void**)&at, total); e != cudaSuccess) return e;
    ptrs.push_back(at);
    for (const Buffer& b : wanted) *b.p = at, at += b.bytes;
    wanted.clear();
    return cudaSuccess;
  }
};

// What `pack` needs besides its grids.
struct PackScratch {
  unsigned char* feature;
  int *fy, *src;
  double *filled, *tmp;
  void get(Scratch& s, size_t cells) {
    s.get(&feature, cells);
    s.get(&fy, cells);
    s.get(&src, cells);
    s.get(&filled, cells);
    s.get(&tmp, cells);
  }
};

inline unsigned blocks(long n, int t) { return (unsigned)((n + t - 1) / t); }

// The feature transform of `feature` into `src` (flat index of each cell's
// nearest feature); fy is [cells] scratch.
template <class D>
void feature_rows(const int* fy, int ny, int nx, int* src, cudaStream_t st) {
  const size_t smem = sizeof(int) * (size_t)nx;
  if (smem <= 48 * 1024)
    k_ft_rows<D, true><<<ny, FT_ROW_WARPS * 32, smem, st>>>(fy, nx, src);
  else
    k_ft_rows<D, false><<<ny, FT_ROW_WARPS * 32, 0, st>>>(fy, nx, src);
}

cudaError_t feature_transform(const unsigned char* feature, int ny, int nx, int* fy, int* src, cudaStream_t st) {
  k_ft_columns<<<blocks(nx, 32), FT_WARPS * 32, 0, st>>>(feature, ny, nx, fy);
  if ((nx > ny ? nx : ny) <= 32767)  // a squared distance fits 32 bits
    feature_rows<int>(fy, ny, nx, src, st);
  else
    feature_rows<long long>(fy, ny, nx, src, st);
  return cudaGetLastError();
}

#define TRACK_LAUNCH()                                                                            \
  do {                                                                                            \
    cudaError_t e_ = cudaGetLastError();                                                          \
    if (e_ != cudaSuccess) {                                                                      \
      racer_host::set_error(std::string("track kernel launch: ") + cudaGetErrorString(e_));       \
      return 2;                                                                                   \
    }                                                                                             \
  } while (0)

// racer/track.py:108-125 from the device grids: ramps, off-road fill, blur,
// float32 grids [layers][3][cells] into `grids` (device).
int pack(const PackScratch& s, int layers, double* clearance, double* height, const int* waypoint, const RampRow* ramps_dev,
         int n_ramps, double x0, double y0, double cell, int nx, int ny, float* grids, cudaStream_t st) {
  const long cells = (long)nx * ny;
  const int T = 256;
  if (n_ramps) {
    k_ramps<<<blocks(cells, T), T, 0, st>>>(ramps_dev, n_ramps, x0, y0, cell, nx, cells, layers, height);
    TRACK_LAUNCH();
  }
  const Blur b = blur_weights();
  for (int l = 0; l < layers; ++l) {
    k_mask_road<<<blocks(cells, T), T, 0, st>>>(clearance + l * cells, cells, s.feature);
    RACER_TRY(feature_transform(s.feature, ny, nx, s.fy, s.src, st));
    TRACK_LAUNCH();
    int first = 0;
    RACER_TRY(cudaMemcpyAsync(&first, s.src, sizeof(int), cudaMemcpyDeviceToHost, st));
    RACER_TRY(cudaStreamSynchronize(st));
    if (first < 0) {
      racer_host::set_error("track: a layer has no road cell (clearance > 0)");
      return 3;
    }
    float* out = grids + (long)l * 3 * cells;
    k_gather<<<blocks(cells, T), T, 0, st>>>(height + l * cells, s.src, cells, s.filled);
    k_blur_rows<<<blocks(cells, T), T, 0, st>>>(s.filled, ny, nx, b, s.tmp);
    k_blur_cols<<<blocks(cells, T), T, 0, st>>>(s.tmp, ny, nx, b, out + cells);
    k_write_layer<<<blocks(cells, T), T, 0, st>>>(clearance + l * cells, waypoint + l * cells, cells, out);
    TRACK_LAUNCH();
  }
  return 0;
}

struct Stream {
  cudaStream_t s = nullptr;
  ~Stream() {
    if (s) cudaStreamDestroy(s);
  }
};

bool grid_ok(int nx, int ny) { return nx >= 2 && ny >= 2 && (long)nx * ny <= (1L << 30) / 8; }

}  // namespace

extern "C" {

int racer_track_ribbon(const double* route, const double* cos_h, const double* sin_h, const double* grade, int W,
                       double half_width, double bank, double x0, double y0, double cell, int nx, int ny,
                       const double* ramps, int n_ramps, float* grids, int64_t grids_len, int* layers_out) {
  if (!route || !cos_h || !sin_h || !grade || !grids || !layers_out || W < 2 || !grid_ok(nx, ny) || !(cell > 0) ||
      n_ramps < 0 || (n_ramps && !ramps)) {
    racer_host::set_error("racer_track_ribbon: invalid arguments");
    return 1;
  }
  const long cells = (long)nx * ny;
  if (grids_len < 6 * cells) {
    racer_host::set_error("racer_track_ribbon: grids needs 6 * nx * ny floats");
    return 1;
  }
  Stream st;
  RACER_TRY(cudaStreamCreateWithFlags(&st.s, cudaStreamNonBlocking));
  Scratch s;
  double *d_route, *d_cos, *d_sin, *d_grade;
  int *nearest, *count, *pw, *flags;
  unsigned char* upper;
  s.get(&d_route, 3 * (size_t)W);
  s.get(&d_cos, W);
  s.get(&d_sin, W);
  s.get(&d_grade, W);
  s.get(&nearest, cells);
  s.get(&count, cells);
  s.get(&pw, cells * MAX_PASSES);
  s.get(&flags, 2);
  s.get(&upper, W);
  PackScratch ps;
  ps.get(s, cells);
  RACER_TRY(s.take());
  RACER_TRY(cudaMemcpyAsync(d_route, route, 3 * sizeof(double) * W, cudaMemcpyHostToDevice, st.s));
  RACER_TRY(cudaMemcpyAsync(d_cos, cos_h, sizeof(double) * W, cudaMemcpyHostToDevice, st.s));
  RACER_TRY(cudaMemcpyAsync(d_sin, sin_h, sizeof(double) * W, cudaMemcpyHostToDevice, st.s));
  RACER_TRY(cudaMemcpyAsync(d_grade, grade, sizeof(double) * W, cudaMemcpyHostToDevice, st.s));
  RACER_TRY(cudaMemsetAsync(flags, 0, 2 * sizeof(int), st.s));
  RACER_TRY(cudaMemsetAsync(upper, 0, W, st.s));

  const double r = half_width + 0.5;
  CellArgs ca{d_route, W, x0, y0, cell, nx, ny, r * r, nearest, count, pw, upper, flags + 1};
  k_cells<<<dim3(blocks(nx, TILE), blocks(ny, TILE)), TILE * TILE, 0, st.s>>>(ca);
  TRACK_LAUNCH();

  // racer/track.py:88-93: the upper layer grows along the route while it stays raised
  std::vector<unsigned char> up(W), grown(W);
  int err = 0;
  RACER_TRY(cudaMemcpyAsync(up.data(), upper, W, cudaMemcpyDeviceToHost, st.s));
  RACER_TRY(cudaMemcpyAsync(&err, flags + 1, sizeof(int), cudaMemcpyDeviceToHost, st.s));
  RACER_TRY(cudaStreamSynchronize(st.s));
  if (err) {
    racer_host::set_error("racer_track_ribbon: a cell lies under more than 8 passes of the route");
    return 4;
  }
  double zmin = route[2];
  for (int w = 1; w < W; ++w) zmin = std::fmin(zmin, route[3 * w + 2]);
  for (;;) {
    bool same = true;
    for (int w = 0; w < W; ++w) {
      const unsigned char high = route[3 * w + 2] > zmin + 0.1;
      grown[w] = up[w] | ((up[(w + W - 1) % W] | up[(w + 1) % W]) & high);
      same = same && grown[w] == up[w];
    }
    if (same) break;
    up.swap(grown);
  }
  RACER_TRY(cudaMemcpyAsync(upper, up.data(), W, cudaMemcpyHostToDevice, st.s));
  k_layer_flags<<<blocks(cells, 256), 256, 0, st.s>>>(count, pw, upper, cells, flags);
  TRACK_LAUNCH();
  int f = 0;
  RACER_TRY(cudaMemcpyAsync(&f, flags, sizeof(int), cudaMemcpyDeviceToHost, st.s));
  RACER_TRY(cudaStreamSynchronize(st.s));
  const int layers = (f & 1) + ((f >> 1) & 1);
  if (layers == 0) {
    racer_host::set_error("racer_track_ribbon: no cell lies on the road");
    return 3;
  }
  double *clearance, *height;
  int* waypoint;
  float* d_grids;
  RampRow* d_ramps = nullptr;
  s.get(&clearance, layers * cells);
  s.get(&height, layers * cells);
  s.get(&waypoint, layers * cells);
  s.get(&d_grids, 3 * layers * cells);
  if (n_ramps) s.get(&d_ramps, n_ramps);
  RACER_TRY(s.take());
  if (n_ramps)
    RACER_TRY(cudaMemcpyAsync(d_ramps, ramps, sizeof(RampRow) * n_ramps, cudaMemcpyHostToDevice, st.s));
  FillArgs fa{d_route, d_cos, d_sin, d_grade, nearest, count, pw, upper, half_width, bank, x0, y0, cell,
              nx, layers, 0, (f & 1) ? 1 : 0, cells, clearance, height, waypoint};
  k_fill<<<blocks(cells, 256), 256, 0, st.s>>>(fa);
  TRACK_LAUNCH();
  int rc = pack(ps, layers, clearance, height, waypoint, d_ramps, n_ramps, x0, y0, cell, nx, ny, d_grids, st.s);
  if (rc) return rc;
  RACER_TRY(cudaMemcpyAsync(grids, d_grids, sizeof(float) * 3 * layers * cells, cudaMemcpyDeviceToHost, st.s));
  RACER_TRY(cudaStreamSynchronize(st.s));
  *layers_out = layers;
  return 0;
}

int racer_track_image(const uint8_t* free_, const double* route, int W, double x0, double y0, double cell, int nx,
                      int ny, const double* ramps, int n_ramps, float* grids, int64_t grids_len) {
  if (!free_ || !route || !grids || W < 1 || !grid_ok(nx, ny) || !(cell > 0) || n_ramps < 0 ||
      (n_ramps && !ramps)) {
    racer_host::set_error("racer_track_image: invalid arguments");
    return 1;
  }
  const long cells = (long)nx * ny;
  if (grids_len < 3 * cells) {
    racer_host::set_error("racer_track_image: grids needs 3 * nx * ny floats");
    return 1;
  }
  Stream st;
  RACER_TRY(cudaStreamCreateWithFlags(&st.s, cudaStreamNonBlocking));
  Scratch s;
  double *d_route, *clearance, *height;
  unsigned char *d_free, *wall, *open;
  int *nearest, *to_wall, *to_open, *flags;
  float* d_grids;
  RampRow* d_ramps = nullptr;
  s.get(&d_route, 3 * (size_t)W);
  s.get(&d_free, cells);
  s.get(&wall, cells);
  s.get(&open, cells);
  s.get(&nearest, cells);
  s.get(&to_wall, cells);
  s.get(&to_open, cells);
  s.get(&flags, 2);
  s.get(&clearance, cells);
  s.get(&height, cells);
  s.get(&d_grids, 3 * cells);
  if (n_ramps) s.get(&d_ramps, n_ramps);
  PackScratch ps;
  ps.get(s, cells);
  RACER_TRY(s.take());
  RACER_TRY(cudaMemcpyAsync(d_route, route, 3 * sizeof(double) * W, cudaMemcpyHostToDevice, st.s));
  RACER_TRY(cudaMemcpyAsync(d_free, free_, cells, cudaMemcpyHostToDevice, st.s));
  RACER_TRY(cudaMemsetAsync(flags, 0, 2 * sizeof(int), st.s));
  RACER_TRY(cudaMemsetAsync(height, 0, sizeof(double) * cells, st.s));
  if (n_ramps)
    RACER_TRY(cudaMemcpyAsync(d_ramps, ramps, sizeof(RampRow) * n_ramps, cudaMemcpyHostToDevice, st.s));
  CellArgs ca{d_route, W, x0, y0, cell, nx, ny, -1.0, nearest, nullptr, nullptr, nullptr, flags + 1};
  k_cells<<<dim3(blocks(nx, TILE), blocks(ny, TILE)), TILE * TILE, 0, st.s>>>(ca);
  k_mask_image<<<blocks(cells, 256), 256, 0, st.s>>>(d_free, cells, wall, open);
  TRACK_LAUNCH();
  RACER_TRY(feature_transform(wall, ny, nx, ps.fy, to_wall, st.s));
  RACER_TRY(feature_transform(open, ny, nx, ps.fy, to_open, st.s));
  int first[2] = {0, 0};
  RACER_TRY(cudaMemcpyAsync(&first[0], to_wall, sizeof(int), cudaMemcpyDeviceToHost, st.s));
  RACER_TRY(cudaMemcpyAsync(&first[1], to_open, sizeof(int), cudaMemcpyDeviceToHost, st.s));
  RACER_TRY(cudaStreamSynchronize(st.s));
  if (first[0] < 0 || first[1] < 0) {
    racer_host::set_error("racer_track_image: the image needs both free and occupied cells");
    return 3;
  }
  k_image_clear<<<blocks(cells, 256), 256, 0, st.s>>>(d_free, to_wall, to_open, nx, cells, cell, clearance);
  TRACK_LAUNCH();
  int rc = pack(ps, 1, clearance, height, nearest, d_ramps, n_ramps, x0, y0, cell, nx, ny, d_grids, st.s);
  if (rc) return rc;
  RACER_TRY(cudaMemcpyAsync(grids, d_grids, sizeof(float) * 3 * cells, cudaMemcpyDeviceToHost, st.s));
  RACER_TRY(cudaStreamSynchronize(st.s));
  return 0;
}

}  // extern "C"
