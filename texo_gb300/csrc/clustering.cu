// clustering.cu — elfPlace's register-clustering area estimate on the GPU
// (`clustering_areas`, crates/texo-pnr/src/register_clustering.rs:17-80).
//
// For each register, the expected number of registers of its control set
// (clock, LSR) inside its window, split by clock enable, is a sum over the
// other registers of the set of Gaussian window probabilities, x times y:
// all-pairs work within a control set, which the reference spreads over
// rayon threads. Here one thread owns one focal register and walks its
// control set; the registers are sorted stably by (clock, LSR, clock
// enable) on the host, so a clock enable's sum runs in input order and the
// per-enable totals in ascending enable order, as in the reference's
// BTreeMaps. Sums and soft ceilings use explicitly rounded FP64 operations
// (no fused multiply-add, which the reference never uses).
//
// The window probability of a register at distance x from the focal one,
// (erf((x + w) / s) - erf((x - w) / s)) / 2 with w = 2.5 sigma and
// s = sigma sqrt(2), depends on u = |x| / s alone, so it is one even function
// of u for every call. It is evaluated as a Taylor polynomial of degree 8 on
// intervals of 1/32 (Window), whose remainder stays below 1e-18: 13 FP64
// operations an axis in place of two divisions and two erfs. FP64 runs at a
// sixty-fourth of the FP32 rate here and bounded the kernel (pipe 85 % busy):
// 42,000 registers in 8 control sets, device time with the copies, 10.8 ms
// with the erfs and 0.90 ms with the table; the areas are 3e-16 off the exact
// ones where those were 1.8e-15 off (the window's edges x + w were rounded at
// the coordinates' magnitude). Beyond u = w / s + 6 the two erfs are both one
// and the probability is an exact zero; such pairs are skipped after a
// conservative FP32 test.
//
// Threads take the registers of a control set in blocks of about 32 near one
// another, so a warp's focal registers agree on which others are far: the
// warp tests 32 of them at a time against its bounding box and visits only
// the ones inside, in order (a register that is far from all the warp's adds
// an exact zero to sums and ceilings alike).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "call.h"
#include "engine.h"

namespace tgp {
namespace {

constexpr int kClusterThreads = 128;

// Taylor coefficients of the window probability about the middles of the
// intervals [k / 32, (k + 1) / 32) of u, and the middles.
constexpr int kTerms = 9;
constexpr int kPerUnit = 32;
constexpr double kHalfWindow = 1.7677669529663688;   // 2.5 / sqrt(2)
constexpr double kReach = kHalfWindow + 6.0;         // erf(6) rounds to one
constexpr int kIntervals = (int)(kReach * kPerUnit) + 1;
struct Window {
  double middle, c[kTerms];
};

// The table, formed once in extended precision (erf' = 2 / sqrt(pi)
// exp(-x^2), and its n-th derivative times (-1)^n H_n(x), the Hermite
// polynomials' three-term recurrence).
std::vector<Window> form_table() {
  std::vector<Window> t(kIntervals);
  const long double h = 2.5L / sqrtl(2.0L), two_over_sqrt_pi = 2.0L / sqrtl(3.14159265358979323846264338327950288L);
  for (int k = 0; k < kIntervals; ++k) {
    const long double m = (k + 0.5L) / kPerUnit;
    t[k].middle = (double)m;
    long double c[kTerms] = {0.5L * (erfcl(m - h) - erfcl(m + h))};
    for (int side = 0; side < 2; ++side) {
      const long double x = side ? m - h : m + h, e = (side ? -0.5L : 0.5L) * two_over_sqrt_pi * expl(-x * x);
      long double h0 = 1.0L, h1 = 2.0L * x, sign = 1.0L, factorial = 1.0L;
      for (int n = 0; n + 1 < kTerms; ++n) {   // c[n + 1]: the n-th derivative of erf' over (n + 1)!
        factorial *= n + 1;
        c[n + 1] += sign * h0 * e / factorial;
        const long double h2 = 2.0L * x * h1 - 2.0L * (n + 1) * h0;
        h0 = h1;
        h1 = h2;
        sign = -sign;
      }
    }
    for (int n = 0; n < kTerms; ++n) t[k].c[n] = (double)c[n];
  }
  return t;
}
// The table on a device: sent by its first call, on that call's stream, and
// published once it has arrived (sent with each call's inputs it cost 2 to 9 us
// of a call). nullptr where it could not be.
const Window* window_table(int device, cudaStream_t s) {
  static std::mutex mu;
  static std::map<int, const Window*> on_device;
  std::lock_guard<std::mutex> lk(mu);
  const auto it = on_device.find(device);
  if (it != on_device.end()) return it->second;
  const std::vector<Window> t = form_table();
  Window* d = nullptr;
  if (cudaMallocAsync((void**)&d, t.size() * sizeof(Window), s) != cudaSuccess) return nullptr;
  if (cudaMemcpyAsync(d, t.data(), t.size() * sizeof(Window), cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess) {
    cudaFreeAsync(d, s);
    return nullptr;
  }
  return on_device[device] = d;
}

// soft_division_ceiling (register_clustering.rs:89-97); the divisors are
// powers of two, so the quotients are exact products
__device__ __forceinline__ double soft_ceiling(double value, double divisor, double inverse) {
  const double quotient = __dmul_rn(value, inverse);
  const double fl = floor(quotient);
  if (__dsub_rn(quotient, fl) < inverse) return __dadd_rn(value, __dmul_rn(1.0 - divisor, fl));
  return ceil(quotient);
}

// gaussian_interval_probability (register_clustering.rs:84-87) at distance x
__device__ __forceinline__ double window_probability(double x, double inv_scale, const Window* table) {
  const double u = __dmul_rn(fabs(x), inv_scale);
  const int k = min((int)(__double2float_rn(u) * (float)kPerUnit), kIntervals - 1);   // a neighbour's interval serves too
  const Window& w = table[k];
  const double t = __dsub_rn(u, w.middle);
  double p = w.c[kTerms - 1];
#pragma unroll
  for (int n = kTerms - 2; n >= 0; --n) p = __fma_rn(p, t, w.c[n]);
  return fmax(p, 0.0);   // a NaN distance counts zero
}

struct ClusterDev {
  unsigned n;
  const double2* xy;                   // sorted by (clock, lsr, ce), stable
  const float2* xy32;                  // the same positions in FP32, for the far-pair test
  const unsigned long long* ce;
  const unsigned* focal;               // thread -> sorted position: near registers share a warp
  const unsigned *group_begin, *group_end;   // per sorted register: its control set's range
  const unsigned* order;               // sorted position -> input index
  const Window* table;
  double half_window, inv_scale, cutoff;
  float cutoff32;                      // cutoff plus a margin that covers the FP32 rounding
  double* areas;                       // by input index
  int* bad;
};

__global__ void __launch_bounds__(kClusterThreads) k_clustering(ClusterDev d) {
  __shared__ Window table[kIntervals];
  {
    const double* src = reinterpret_cast<const double*>(d.table);
    double* dst = reinterpret_cast<double*>(table);
    for (int i = threadIdx.x; i < (int)(sizeof(table) / 8); i += kClusterThreads) dst[i] = __ldg(src + i);
  }
  __syncthreads();
  const unsigned all = 0xffffffffu;
  const unsigned t = blockIdx.x * kClusterThreads + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool active = t < d.n;
  const unsigned p = __ldg(d.focal + (active ? t : d.n - 1));
  const float2 fi = __ldg(d.xy32 + p);
  const unsigned gb = __ldg(d.group_begin + p), ge = __ldg(d.group_end + p);
  const double2 at = __ldg(d.xy + p);
  const unsigned long long focal_ce = __ldg(d.ce + p);
  double total = 0.0, focal = 0.0, sum = 0.0;
  unsigned long long cur = 0;
  // the warp's control sets in turn (one but where two meet)
  for (unsigned todo = __ballot_sync(all, active); todo;) {
    const int lead = __ffs(todo) - 1;
    const unsigned b = __shfl_sync(all, gb, lead), e = __shfl_sync(all, ge, lead);
    const bool mine = active && gb == b;
    todo &= ~__ballot_sync(all, mine);
    // the box within which a register may be near one of the warp's
    float x0 = mine ? fi.x : INFINITY, x1 = mine ? fi.x : -INFINITY, y0 = mine ? fi.y : INFINITY,
          y1 = mine ? fi.y : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      x0 = fminf(x0, __shfl_xor_sync(all, x0, o));
      x1 = fmaxf(x1, __shfl_xor_sync(all, x1, o));
      y0 = fminf(y0, __shfl_xor_sync(all, y0, o));
      y1 = fmaxf(y1, __shfl_xor_sync(all, y1, o));
    }
    if (mine) {
      cur = __ldg(d.ce + b);
    }
    float2 fj = b + lane < e ? __ldg(d.xy32 + b + lane) : make_float2(NAN, NAN);
    for (unsigned j0 = b; j0 < e; j0 += 32) {
      const float2 f = fj;
      if (j0 + 32 + lane < e) fj = __ldg(d.xy32 + j0 + 32 + lane);
      const bool in = j0 + lane < e && f.x - x1 <= d.cutoff32 && x0 - f.x <= d.cutoff32 && f.y - y1 <= d.cutoff32 &&
                      y0 - f.y <= d.cutoff32;
      for (unsigned m = __ballot_sync(all, in); m; m &= m - 1) {
        const int q = __ffs(m) - 1;
        const float2 g = make_float2(__shfl_sync(all, f.x, q), __shfl_sync(all, f.y, q));
        if (!mine) continue;
        // far in FP32 (with margin) implies far in FP64: skip without FP64 work
        const bool near = !(fabsf(fi.x - g.x) > d.cutoff32 || fabsf(fi.y - g.y) > d.cutoff32);
        const unsigned long long cj = __ldg(d.ce + j0 + q);
        if (cj != cur) {   // one clock enable's expectation is complete
          total = __dadd_rn(total, soft_ceiling(sum, 2.0, 0.5));
          if (cur == focal_ce) focal = sum;
          sum = 0.0;
          cur = cj;
        }
        if (!near) continue;
        const double2 c = __ldg(d.xy + j0 + q);
        const double dx = __dsub_rn(at.x, c.x), dy = __dsub_rn(at.y, c.y);
        if (fabs(dx) > d.cutoff || fabs(dy) > d.cutoff) continue;
        const double px = window_probability(dx, d.inv_scale, table), py = window_probability(dy, d.inv_scale, table);
        sum = __dadd_rn(sum, __dmul_rn(px, py));
      }
    }
  }
  if (!active) return;
  total = __dadd_rn(total, soft_ceiling(sum, 2.0, 0.5));
  if (cur == focal_ce) focal = sum;
  const unsigned out = __ldg(d.order + p);
  // so far out that the window's edges round to the register's own place
  auto no_window = [&](double v) { return __dadd_rn(v, d.half_window) == __dsub_rn(v, d.half_window); };
  if (!(isfinite(focal) && focal > 0.0) || no_window(at.x) || no_window(at.y)) {
    atomicExch(d.bad, 1);
    d.areas[out] = 0.0;
    return;
  }
  // 8 / E_focal * ceil2(E_focal) / total * ceil4(total), left to right
  const double area =
      __dmul_rn(__ddiv_rn(__dmul_rn(__ddiv_rn(8.0, focal), soft_ceiling(focal, 2.0, 0.5)), total),
                soft_ceiling(total, 4.0, 0.25));
  if (!(isfinite(area) && area >= 0.0)) atomicExch(d.bad, 1);
  d.areas[out] = area;
}

// Puts `order` into stable order of its members' keys, least significant digit
// first; digits that all keys share are passed over. Indirect comparisons took
// 8.4 ms for the two orders of 42,000 registers, this takes
// 0.5 ms.
template <class Key>
void radix_order(std::vector<uint32_t>& order, std::vector<uint32_t>& scratch, Key key_of, std::vector<uint64_t>& key) {
  constexpr int kDigit = 12;
  const size_t n = order.size();
  uint64_t differ = 0;
  for (size_t r = 0; r < n; ++r) {
    key[r] = key_of((uint32_t)r);
    differ |= key[r] ^ key[0];
  }
  for (int shift = 0; shift < 64; shift += kDigit) {
    const uint64_t mask = (1ull << kDigit) - 1;
    if (!(differ >> shift & mask)) continue;
    uint32_t at[1u << kDigit] = {};
    for (size_t r = 0; r < n; ++r) ++at[key[r] >> shift & mask];
    uint32_t sum = 0;
    for (uint32_t& a : at) {
      const uint32_t c = a;
      a = sum;
      sum += c;
    }
    for (size_t i = 0; i < n; ++i) scratch[at[key[order[i]] >> shift & mask]++] = order[i];
    order.swap(scratch);
  }
}

}  // namespace
}  // namespace tgp

using namespace tgp;

extern "C" int32_t texo_gp_register_clustering_areas(int32_t device, uint64_t num_registers, const double* xy,
                                                     const uint64_t* clock_lsr, const uint64_t* ce,
                                                     uint64_t movable_instance_count, double* areas,
                                                     double* elapsed_ms) {
  if (elapsed_ms) *elapsed_ms = 0.0;
  const uint64_t n = num_registers;
  if (n == 0) return TEXO_GP_OK;
  if (!xy || !clock_lsr || !ce || !areas) {
    set_last_error("register clustering: null argument");
    return TEXO_GP_ERR_INVALID_ARGUMENT;
  }
  if (movable_instance_count == 0) {   // the reference's empty map: no clustering area
    for (uint64_t r = 0; r < n; ++r) areas[r] = 0.0;
    return TEXO_GP_OK;
  }
  if (movable_instance_count > 0xffffffffull || n > (1ull << 31)) {
    set_last_error("register clustering: count out of range");
    return TEXO_GP_ERR_INVALID_NORMALIZATION;
  }
  const double sigma = std::sqrt(1.0e-5 * (double)(uint32_t)movable_instance_count);
  if (!std::isfinite(sigma) || sigma <= 0.0) return TEXO_GP_ERR_INVALID_NORMALIZATION;
  const double half_window = 2.5 * sigma, scale = sigma * 1.4142135623730951;   // sigma sqrt(2)
  const double cutoff = half_window + 6.0 * scale;   // kReach in units of scale

  // sort by (clock, lsr, ce), stable: input order within a clock enable
  std::vector<uint32_t> order(n), scratch(n);
  std::vector<uint64_t> key(n);
  std::iota(order.begin(), order.end(), 0u);
  {
    // the three keys side by side, without the leading bits that all share,
    // where that fits 64 bits
    uint64_t differ[3] = {0, 0, 0};
    for (uint64_t r = 0; r < n; ++r) {
      differ[0] |= ce[r] ^ ce[0];
      differ[1] |= clock_lsr[2 * r + 1] ^ clock_lsr[1];
      differ[2] |= clock_lsr[2 * r] ^ clock_lsr[0];
    }
    int bits[3];
    for (int k = 0; k < 3; ++k)
      for (bits[k] = 0; bits[k] < 64 && differ[k] >> bits[k]; ++bits[k]) {
      }
    auto low = [&](uint64_t v, int k) { return bits[k] < 64 ? v & ((1ull << bits[k]) - 1) : v; };
    if (bits[0] + bits[1] + bits[2] < 64) {
      radix_order(order, scratch,
                  [&](uint32_t r) {
                    return (low(clock_lsr[2 * (size_t)r], 2) << bits[1] | low(clock_lsr[2 * (size_t)r + 1], 1)) << bits[0] |
                           low(ce[r], 0);
                  },
                  key);
    } else {
      radix_order(order, scratch, [&](uint32_t r) { return ce[r]; }, key);
      radix_order(order, scratch, [&](uint32_t r) { return clock_lsr[2 * (size_t)r + 1]; }, key);
      radix_order(order, scratch, [&](uint32_t r) { return clock_lsr[2 * (size_t)r]; }, key);
    }
  }
  std::vector<double> sxy(2 * n);
  std::vector<float> s32(2 * n);
  std::vector<unsigned long long> sce(n);
  std::vector<uint32_t> gb(n), ge(n), focal(n);
  // the threads of a control set take its registers block by block, the
  // blocks of a size that holds about a warp's 32 of them
  std::vector<uint64_t> block(n);
  std::vector<uint32_t> set_of(n);
  uint64_t blocks = 1;
  uint32_t sets = 0;
  double extent = 0.0;
  for (uint64_t p = 0; p < n; ++p) {
    for (int k = 0; k < 2; ++k) {
      const double v = xy[2 * (size_t)order[p] + k];
      sxy[2 * p + k] = v;
      s32[2 * p + k] = (float)v;
      if (std::isfinite(v)) extent = std::max(extent, std::fabs(v));
    }
    sce[p] = ce[order[p]];
  }
  for (uint64_t p = 0; p < n;) {
    uint64_t q = p + 1;
    const uint32_t a = order[p];
    while (q < n && clock_lsr[2 * (size_t)order[q]] == clock_lsr[2 * (size_t)a] &&
           clock_lsr[2 * (size_t)order[q] + 1] == clock_lsr[2 * (size_t)a + 1])
      ++q;
    for (uint64_t r = p; r < q; ++r) {
      gb[r] = (uint32_t)p;
      ge[r] = (uint32_t)q;
    }
    double lo[2] = {1e300, 1e300}, hi[2] = {-1e300, -1e300};
    for (uint64_t r = p; r < q; ++r)
      for (int k = 0; k < 2; ++k)
        if (std::isfinite(sxy[2 * r + k])) {
          lo[k] = std::min(lo[k], sxy[2 * r + k]);
          hi[k] = std::max(hi[k], sxy[2 * r + k]);
        }
    const double side = std::max(1.0, std::sqrt(32.0 * std::max(hi[0] - lo[0], 1.0) * std::max(hi[1] - lo[1], 1.0) /
                                                (double)(q - p)));
    auto cell = [&](double distance) -> uint64_t {   // 0 where it is not a number
      const double c = distance / side;
      return c >= 1.0e9 ? 1000000000u : c > 0.0 ? (uint32_t)c : 0u;
    };
    const uint64_t columns = cell(hi[0] - lo[0]) + 1;
    for (uint64_t r = p; r < q; ++r) {
      block[r] = cell(sxy[2 * r + 1] - lo[1]) * columns + cell(sxy[2 * r] - lo[0]);
      blocks = std::max(blocks, block[r] + 1);
      set_of[r] = sets;
    }
    ++sets;
    p = q;
  }
  std::iota(focal.begin(), focal.end(), 0u);
  if (blocks < (1ull << 62) / sets) {
    radix_order(focal, scratch, [&](uint32_t r) { return set_of[r] * blocks + block[r]; }, key);
  } else {
    radix_order(focal, scratch, [&](uint32_t r) { return block[r]; }, key);
    radix_order(focal, scratch, [&](uint32_t r) { return (uint64_t)set_of[r]; }, key);
  }
  // FP32 positions are within 2^-24 |coordinate| of the FP64 ones; a margin of
  // 2^-20 (extent + cutoff) keeps the FP32 far test conservative
  const float cutoff32 = (float)(cutoff + std::ldexp(extent + cutoff + 1.0, -20));

  if (cudaSetDevice(device) != cudaSuccess) return TEXO_GP_ERR_CUDA;
  Call call(device);
  if (!call.ok()) return TEXO_GP_ERR_CUDA;
  const cudaStream_t s = call.stream();
  auto round = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t s8 = round(n * 8), s4 = round(n * 4);
  char* base = call.memory(5 * s8 + 4 * s4 + 256);
  ClusterDev d{};
  if (!base || !(d.table = window_table(device, s))) return TEXO_GP_ERR_OUT_OF_MEMORY;
  d.n = (unsigned)n;
  d.half_window = half_window;
  d.inv_scale = 1.0 / scale;
  d.cutoff = cutoff;
  double2* dxy = (double2*)base;
  unsigned long long* dce = (unsigned long long*)(base + 2 * s8);
  d.areas = (double*)(base + 3 * s8);
  unsigned* dgb = (unsigned*)(base + 4 * s8);
  unsigned* dge = (unsigned*)(base + 4 * s8 + s4);
  unsigned* dord = (unsigned*)(base + 4 * s8 + 2 * s4);
  float2* d32 = (float2*)(base + 4 * s8 + 3 * s4);
  unsigned* dfoc = (unsigned*)(base + 5 * s8 + 3 * s4);
  d.bad = (int*)(base + 5 * s8 + 4 * s4);
  d.xy32 = d32;
  d.focal = dfoc;
  d.cutoff32 = cutoff32;
  d.xy = dxy;
  d.ce = dce;
  d.group_begin = dgb;
  d.group_end = dge;
  d.order = dord;
  call.start();
  bool ok = cudaMemcpyAsync(dxy, sxy.data(), n * 16, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemcpyAsync(dce, sce.data(), n * 8, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemcpyAsync(dgb, gb.data(), n * 4, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemcpyAsync(dge, ge.data(), n * 4, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemcpyAsync(dord, order.data(), n * 4, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemcpyAsync(d32, s32.data(), n * 8, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemcpyAsync(dfoc, focal.data(), n * 4, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemsetAsync(d.bad, 0, sizeof(int), s) == cudaSuccess;
  if (ok) {
    k_clustering<<<(unsigned)((n + kClusterThreads - 1) / kClusterThreads), kClusterThreads, 0, s>>>(d);
    ok = cudaGetLastError() == cudaSuccess;
    if (ok) note_launch();
  }
  int bad = 0;
  ok = ok && cudaMemcpyAsync(areas, d.areas, n * 8, cudaMemcpyDeviceToHost, s) == cudaSuccess &&
       cudaMemcpyAsync(&bad, d.bad, sizeof(int), cudaMemcpyDeviceToHost, s) == cudaSuccess;
  float ms = 0.f;
  if (!call.finish(&ms)) ok = false;
  if (elapsed_ms) *elapsed_ms = ms;
  if (!ok) {
    set_last_error(std::string("register clustering: ") + cudaGetErrorString(cudaGetLastError()));
    return TEXO_GP_ERR_CUDA;
  }
  if (bad) {
    set_last_error("register clustering: a register's expectation is not positive and finite");
    return TEXO_GP_ERR_INVALID_NORMALIZATION;
  }
  return TEXO_GP_OK;
}
