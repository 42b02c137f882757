// rudy.cu — continuous RUDY routing demand on the GPU
// (`continuous_routing_demand`, crates/texo-pnr/src/eplace.rs:856-937).
//
// A net's bounding box (min_x, max_x, min_y, max_y), widened by half a tile on
// every side, spreads the densities dx / area (horizontal) and dy / area
// (vertical), area = (dx + 1)(dy + 1), over the tiles it overlaps, each tile
// weighted by overlap_x * overlap_y. Along one axis the overlap is exactly 1
// for every tile whose unit interval lies inside the widened box and
// fractional for at most one tile on each side, so a box is at most 3 x 3
// rectangles of constant value. Their corners go into a 2-D difference
// array as int64 2^-40 fixed-point updates (order-independent, so the map is
// deterministic); a row scan and a column scan then give the map.
// The per-rectangle values are the reference's FP64 expressions
// (density * (overlap_x * overlap_y)); the fixed-point rounding (2^-41 per
// rectangle and tile) is the difference from the reference's FP64 sums.
#include <cmath>
#include <cstring>
#include <limits>
#include <string>

#include "common.cuh"
#include "call.h"
#include "engine.h"
#include "kernels.cuh"

namespace tgp {
namespace {

// 2^40: a box adds at most 1 to a tile, so up to 2^22 boxes keep every
// partial sum of the difference array inside int64
constexpr double kRudyFix = 1099511627776.0;
constexpr uint64_t kRudyMaxBoxes = 1ull << 22;

// One axis of a widened box: the tile of its left edge, the run of tiles whose
// unit interval lies inside (overlap 1) and the tile of its right edge, each
// beginning where the one before ends; a piece outside [0, extent) or without
// overlap has the value zero.
struct Pieces {
  int c[4];      // where the pieces begin, and the last one's end
  double v[3];   // their overlaps, eplace.rs:885-906's expressions
};

__device__ __forceinline__ Pieces axis_pieces(double lo, double hi, int extent) {
  const double rlo = lo - 0.5, rhi = hi + 0.5;
  const double ia = ceil(lo), ib = floor(hi);
  auto overlap = [&](double t) {
    return t >= 0.0 && t < extent ? fmax(fmin(t + 0.5, rhi) - fmax(t - 0.5, rlo), 0.0) : 0.0;
  };
  auto at = [&](double t) { return (int)fmin(fmax(t, 0.0), (double)extent); };
  Pieces p;
  p.c[0] = at(ia - 1.0);
  p.c[1] = at(ia);
  p.c[2] = at(ib + 1.0);
  p.c[3] = at(ib + 2.0);
  p.v[0] = overlap(ia - 1.0);
  p.v[1] = p.c[1] < p.c[2] ? 1.0 : 0.0;
  p.v[2] = overlap(ib + 1.0);
  return p;
}
// Pieces without overlap given no tile.
__device__ __forceinline__ void drop_empty(Pieces& p) {
  if (p.v[0] == 0.0) p.c[0] = p.c[1];
  if (p.v[2] == 0.0) p.c[3] = p.c[2];
}

// diff: [2][(H + 1) x (W + 1)] int64, zeroed. The nine rectangles of a box share
// their corners: their rounded values are differenced in registers along both
// axes, and the 16 corners of a plane take one atomic each where four for each
// rectangle made 36 (300,000 boxes, with the copies, 264 -> 241 us, 1.2 million
// 822 -> 789; 50,000 are bound by the copies, 105).
__global__ void k_rudy_boxes(const double* boxes, long long nbox, int W, int H, unsigned long long* diff) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nbox) return;
  const double x0 = boxes[4 * i], x1 = boxes[4 * i + 1], y0 = boxes[4 * i + 2], y1 = boxes[4 * i + 3];
  const double dx = x1 - x0, dy = y1 - y0;
  const double area = (dx + 1.0) * (dy + 1.0);
  const double hd = dx / area, vd = dy / area;
  Pieces px = axis_pieces(x0, x1, W), py = axis_pieces(y0, y1, H);
  if (__double2hiint(dx) == 0x7ff00000 || __double2hiint(dy) == 0x7ff00000) {
    // wider than FP64: its density is no number, nor is zero times that
    drop_empty(px);
    drop_empty(py);
  }
  const size_t plane = (size_t)(W + 1) * (H + 1);
  long long above_h[3] = {0, 0, 0}, above_v[3] = {0, 0, 0};   // the row of rectangles before
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    unsigned long long* row = diff + (size_t)py.c[a] * (W + 1);
    long long left_h = 0, left_v = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      long long h = 0, v = 0, step_h = 0, step_v = 0;   // the rectangle's values, and their step from the row before
      if (b < 3) {
        if (a < 3) {
          const double overlap = px.v[b] * py.v[a];
          h = __double2ll_rn(hd * overlap * kRudyFix);
          v = __double2ll_rn(vd * overlap * kRudyFix);
        }
        step_h = h - above_h[b];
        step_v = v - above_v[b];
        above_h[b] = h;
        above_v[b] = v;
      }
      if (step_h != left_h) atomicAdd(row + px.c[b], (unsigned long long)(step_h - left_h));
      if (step_v != left_v) atomicAdd(row + plane + px.c[b], (unsigned long long)(step_v - left_v));
      left_h = step_h;
      left_v = step_v;
    }
  }
}

// Inclusive scan along each row of both planes: a warp per row, 32 columns
// a step (a shuffle scan plus the carry of the previous step). The sums are
// exact integers, so any order gives the same values.
__global__ void k_rudy_rows(unsigned long long* __restrict__ diff, int W, int H) {
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = (int)(threadIdx.x & 31);
  if (warp >= 2 * H) return;   // uniform across the warp
  const int plane = warp / H, y = warp % H;
  unsigned long long* row = diff + (size_t)plane * (W + 1) * (H + 1) + (size_t)y * (W + 1);
  unsigned long long carry = 0;
  for (int x0 = 0; x0 < W; x0 += 32) {
    const int x = x0 + lane;
    unsigned long long v = x < W ? row[x] : 0ull;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
    }
    v += carry;
    if (x < W) row[x] = v;
    carry = __shfl_sync(0xffffffffu, v, 31);
  }
}

// Inclusive scan along each column, written out as FP64 demand: a block per
// strip of 32 columns of one plane; its warps take consecutive row segments,
// sum them, add the totals of the segments above and scan their own (the
// loads of a segment do not depend on one another).
constexpr int kColWarps = 8;
__global__ void __launch_bounds__(32 * kColWarps) k_rudy_cols(const unsigned long long* __restrict__ diff, int W,
                                                              int H, double* __restrict__ horizontal,
                                                              double* __restrict__ vertical) {
  __shared__ unsigned long long seg[kColWarps][32];
  const int lane = (int)(threadIdx.x & 31), w = (int)(threadIdx.x >> 5);
  const int strips = (W + 31) / 32;
  const int plane = (int)blockIdx.x / strips, x = ((int)blockIdx.x % strips) * 32 + lane;
  const unsigned long long* col = diff + (size_t)plane * (W + 1) * (H + 1) + x;
  double* out = plane ? vertical : horizontal;
  const int per = (H + kColWarps - 1) / kColWarps, y0 = min(H, w * per), y1 = min(H, y0 + per);
  unsigned long long s = 0;
  if (x < W)
    for (int y = y0; y < y1; ++y) s += col[(size_t)y * (W + 1)];
  seg[w][lane] = s;
  __syncthreads();
  unsigned long long c = 0;
  for (int k = 0; k < w; ++k) c += seg[k][lane];
  if (x < W)
    for (int y = y0; y < y1; ++y) {
      c += col[(size_t)y * (W + 1)];
      out[(size_t)y * W + x] = (double)(long long)c / kRudyFix;
    }
}

}  // namespace
}  // namespace tgp

using namespace tgp;

extern "C" int32_t texo_gp_routing_demand(int32_t device, uint32_t width, uint32_t height, uint64_t num_boxes,
                                          const double* boxes, double* horizontal, double* vertical,
                                          double* elapsed_ms) {
  if (elapsed_ms) *elapsed_ms = 0.0;
  if (!horizontal || !vertical || (num_boxes && !boxes)) return TEXO_GP_ERR_INVALID_ARGUMENT;
  if (width == 0 || height == 0 || (uint64_t)width * height > (1ull << 26)) return TEXO_GP_ERR_INVALID_NORMALIZATION;
  unsigned wrong = 0;   // no early way out: this loop is vectorized
  constexpr double kMax = std::numeric_limits<double>::max();
  for (uint64_t i = 0; i < num_boxes; ++i) {
    const double* b = boxes + 4 * i;
    wrong |= !(b[0] <= b[1]) | !(b[2] <= b[3]) | !(b[0] >= -kMax) | !(b[1] <= kMax) | !(b[2] >= -kMax) | !(b[3] <= kMax);
  }
  for (uint64_t i = 0; wrong && i < num_boxes; ++i) {
    const double* b = boxes + 4 * i;
    if (!(std::isfinite(b[0]) && std::isfinite(b[1]) && std::isfinite(b[2]) && std::isfinite(b[3])) ||
        b[0] > b[1] || b[2] > b[3]) {
      set_last_error("routing demand: box " + std::to_string(i) + " is not finite or not ordered");
      return TEXO_GP_ERR_INVALID_NORMALIZATION;
    }
  }
  if (num_boxes > kRudyMaxBoxes) return TEXO_GP_ERR_FIXED_POINT_RANGE;
  if (cudaSetDevice(device) != cudaSuccess) return TEXO_GP_ERR_CUDA;
  const int W = (int)width, H = (int)height;
  const size_t tiles = (size_t)W * H, plane = (size_t)(W + 1) * (H + 1);
  Call call(device);
  if (!call.ok()) return TEXO_GP_ERR_CUDA;
  const cudaStream_t s = call.stream();
  const size_t b_bytes = ((std::max<uint64_t>(num_boxes, 1) * 32) + 255) & ~(size_t)255;
  const size_t d_bytes = ((2 * plane * 8) + 255) & ~(size_t)255;
  const size_t o_bytes = ((tiles * 8) + 255) & ~(size_t)255;
  char* base = call.memory(b_bytes + d_bytes + 2 * o_bytes);
  if (!base) return TEXO_GP_ERR_OUT_OF_MEMORY;
  double* dbox = (double*)base;
  unsigned long long* diff = (unsigned long long*)(base + b_bytes);
  double* dh = (double*)(base + b_bytes + d_bytes);
  double* dv = (double*)(base + b_bytes + d_bytes + o_bytes);
  call.start();
  bool ok = (!num_boxes || cudaMemcpyAsync(dbox, boxes, num_boxes * 32, cudaMemcpyHostToDevice, s) == cudaSuccess) &&
            cudaMemsetAsync(diff, 0, 2 * plane * 8, s) == cudaSuccess;
  if (ok && num_boxes) {
    k_rudy_boxes<<<(unsigned)((num_boxes + kThreads - 1) / kThreads), kThreads, 0, s>>>(dbox, (long long)num_boxes,
                                                                                       W, H, diff);
    note_launch();
  }
  if (ok) {
    k_rudy_rows<<<(unsigned)((2 * (size_t)H * 32 + kThreads - 1) / kThreads), kThreads, 0, s>>>(diff, W, H);
    k_rudy_cols<<<(unsigned)(2 * ((W + 31) / 32)), 32 * kColWarps, 0, s>>>(diff, W, H, dh, dv);
    note_launch();
    note_launch();
    ok = cudaGetLastError() == cudaSuccess &&
         cudaMemcpyAsync(horizontal, dh, tiles * 8, cudaMemcpyDeviceToHost, s) == cudaSuccess &&
         cudaMemcpyAsync(vertical, dv, tiles * 8, cudaMemcpyDeviceToHost, s) == cudaSuccess;
  }
  float ms = 0.f;
  if (!call.finish(&ms)) ok = false;
  if (elapsed_ms) *elapsed_ms = ms;
  if (!ok) {
    set_last_error(std::string("routing demand: ") + cudaGetErrorString(cudaGetLastError()));
    return TEXO_GP_ERR_CUDA;
  }
  return TEXO_GP_OK;
}
