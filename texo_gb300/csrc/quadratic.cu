// quadratic.cu — the coarse quadratic seed's linear solve on the GPU:
// Jacobi-preconditioned conjugate gradients for (D - W) x = b
// (`solve_quadratic`, crates/texo-pnr/src/lib.rs:4586-4752), FP64.
//
// One cooperative persistent kernel runs the whole solve, two grid barriers a
// CG step:
//   product: p = z + beta p_old and q = (D - W) p (`multiply_quadratic`,
//     lib.rs:4767-4782) with the partial of <p, q>. The new direction is formed
//     where it is read, from the pair (z, p_old) that one 16-byte load brings,
//     by one fused operation that gives every reader the same bits;
//   update: x += alpha p, r -= alpha q, z = r / D with the partials of <r, r>
//     and <r, z>, and the pairs (z, p) of the next product, into the other of
//     two buffers.
//
// FP64 issue bounds it: two lanes a cycle on a multiprocessor, whether or not
// a warp's lanes are all at work. So the matrix is laid out once, by each
// block for the rows it owns, so that a warp's lanes stay busy: rows are cut
// into segments of at most 16 entries, a thread takes a segment, and the
// segments of a tile (the rows of up to 512 of them) are dealt to the warps in
// order of length, entry k of a warp's 32 segments side by side. That is two
// FP64 instructions a 32 entries, where eight lanes a row, the rows as they
// come, spend 18 on four rows. At 42,000 unknowns and 565,000 entries (31
// steps, about half of whose 14 us is the two barriers with their reductions):
// 0.43 ms; eight lanes a row 1.00 ms; one thread a row, with a third barrier
// for the direction, 1.2 ms. Segments of 8 entries took 0.07 ms more, eight
// entries' loads in flight instead of four the same, a direct divide by the
// diagonal 0.04 ms more, two blocks of half the registers (which spilled)
// 0.04 ms more.
//
// Sums run in fixed orders (segments, trees, one warp per partial), so the
// solve is deterministic; against the reference's left-to-right sums they
// agree to rounding, not bit for bit. Partials alternate between two sets so a
// block that leaves a barrier early never overwrites a set another block still
// reads. Every wait is the bounded grid barrier of the placement engine.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <new>
#include <string>
#include <vector>

#include "call.h"
#include "engine.h"
#include "persistent_body.cuh"

namespace tgp {
namespace {

enum PcgSlot { PS_A = 0, PS_B, kPcgSlots };   // two dot products a phase at most
constexpr int kMaxPcgBlocks = 2048;
constexpr double kPcgTolerance = 1e-8;      // on squared residuals: 1e-4 on the norm (lib.rs:4592-4594)

struct PcgResult {
  unsigned iterations, restarts;
  int stop;             // 0 residual, 1 breakdown, 2 dimension
  int converged;
  int wrong_entry;      // an entry's index or weight is refused
  double initial_rr, target, final_rr;
};

// A tile: the rows of one pass of a block, cut into at most kPcgThreads
// segments of at most `segment` entries (kSegment, or what makes a longer row
// fit); `base`: where its entries start in the dealt arrays.
constexpr int kPcgThreads = 512;
constexpr unsigned kSegment = 16;
constexpr int kPcgWarps = kPcgThreads / 32;
constexpr unsigned kAhead = 4;   // entries whose loads are in flight together
struct PcgTile {
  unsigned row0, rows, segment;
  unsigned long long base;
};

struct PcgDev {
  int n, tiles;
  const double *diag, *w, *b;
  const unsigned *ptr, *idx;
  const PcgTile* tile;
  double* dealt_w;           // a tile's warps in turn: entry k of its 32 segments side by side
  unsigned* dealt_i;
  uint2* warp;               // [tiles][kPcgWarps] where a warp's entries start in its tile, and how many a lane
  unsigned short* place;     // [tiles][kPcgThreads] a thread's segment, by position in row order
  unsigned* row_segments;    // [n] a row's first segment in its tile | their count << 16
  double *x, *r, *p, *q, *inv;
  double2* zp[2];            // (z, p) of the last update
  double* part;              // [2 sets][kPcgSlots][kMaxPcgBlocks]
  GridBarrier* bar;
  PcgResult* out;
};

struct PcgShared {
  union {
    struct {                       // while the tiles are laid out
      unsigned first[kPcgThreads];       // a segment's first entry, from the tile's first
      unsigned length[kPcgThreads];
      unsigned short seg[kPcgThreads];   // by place
      unsigned total[kPcgWarps];
    } lay;
    double sums[2][kPcgThreads];   // the segments' sums, of alternate tiles
  };
  double part[2][kPcgThreads];
  double quarter[8];
  FoldValue fv[kPcgSlots];
  unsigned gen;
  int failed;
  // controller state, identical in every block (thread 0 writes it)
  double rr, rho, alpha, beta, target;
  unsigned iterations, restarts;
  int stop, action;
};

// a / b from b's rounded reciprocal and one correction by the remainder
// (Markstein 1990). The corrected value is within 1.5 * 2^-53 units in the last
// place of a / b before it is rounded, so the result is the rounded quotient but
// where a / b lies that close to the middle of two numbers, and then the other
// of the two (0.04 ms of a 42,000-cell solve's 0.43 against the divide). A
// diagonal near the ends of the range of exponents has no such reciprocal
// (zero) and is divided by; a quotient beyond FP64 may be no number instead of
// infinite, and either is a breakdown.
__device__ __forceinline__ double reciprocal(double b) { return b > 1e-200 && b < 1e200 ? __drcp_rn(b) : 0.0; }
__device__ __forceinline__ double quotient(double a, double b, double inverse) {
  if (__double2hiint(inverse) == 0) return __ddiv_rn(a, b);
  const double q = __dmul_rn(a, inverse);
  return __fma_rn(__fma_rn(-q, b, a), inverse, q);
}

// Deals a tile's entries to the block's warps.
__device__ void lay_out(const PcgDev& d, int t, PcgShared& S) {
  const PcgTile tile = d.tile[t];
  const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned e0 = d.ptr[tile.row0];
  unsigned b = 0, len = 0, count = 0;
  if (tid < tile.rows) {
    b = d.ptr[tile.row0 + tid];
    len = d.ptr[tile.row0 + tid + 1] - b;
    count = len / tile.segment + (len % tile.segment != 0);
  }
  unsigned at = count;   // the sum up to this row
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, at, o);
    if (lane >= (unsigned)o) at += v;
  }
  if (lane == 31) S.lay.total[warp] = at;
  __syncthreads();
  unsigned before = 0, segments = 0;
  for (int k = 0; k < kPcgWarps; ++k) {
    if (k < (int)warp) before += S.lay.total[k];
    segments += S.lay.total[k];
  }
  at += before - count;
  if (tid < tile.rows) {
    d.row_segments[tile.row0 + tid] = at | count << 16;
    for (unsigned j = 0; j < count; ++j) {
      S.lay.first[at + j] = b - e0 + j * tile.segment;
      S.lay.length[at + j] = min(tile.segment, len - j * tile.segment);
    }
  }
  __syncthreads();
  // the longest first, equal ones in row order
  if (tid < segments) {
    const unsigned mine = S.lay.length[tid];
    unsigned rank = 0;
    for (unsigned j = 0; j < segments; ++j) {
      const unsigned v = S.lay.length[j];
      rank += v > mine || (v == mine && j < tid);
    }
    S.lay.seg[rank] = (unsigned short)tid;
  }
  __syncthreads();
  // the four schedulers take the warps' loads in turn, then in reverse
  const unsigned load = (warp & 4) ? warp ^ 3 : warp, place = 32 * load + lane;
  unsigned start = 0, width = 0;
  for (unsigned k = 0; k <= load; ++k) {
    start += 32 * width;
    width = 32 * k < segments ? S.lay.length[S.lay.seg[32 * k]] : 0;
  }
  if (lane == 0) d.warp[(size_t)t * kPcgWarps + warp] = make_uint2(start, width);
  const bool some = place < segments;
  const unsigned seg = some ? S.lay.seg[place] : place;   // a thread without one: a place of its own
  d.place[(size_t)t * kPcgThreads + tid] = (unsigned short)seg;
  const unsigned have = some ? S.lay.length[seg] : 0;
  const size_t from = (size_t)e0 + (some ? S.lay.first[seg] : 0), to = tile.base + start + lane;
  bool wrong = false;
  for (unsigned k = 0; k < width; ++k) {   // a lane with fewer entries adds zeros times a row of its tile
    double w = 0.0;
    unsigned idx = tile.row0;
    if (k < have) {
      w = d.w[from + k];
      idx = d.idx[from + k];
      if (idx >= (unsigned)d.n || (__double2hiint(w) & 0x7ff00000) == 0x7ff00000) {   // infinite or not a number
        wrong = true;
        idx = tile.row0;
      }
    }
    d.dealt_w[to + 32 * (size_t)k] = w;
    d.dealt_i[to + 32 * (size_t)k] = idx;
  }
  if (wrong) atomicExch(&d.out->wrong_entry, 1);
  __syncthreads();
}

__global__ void __launch_bounds__(kPcgThreads, 1) k_pcg(PcgDev d) {
  __shared__ PcgShared S;
  const int pb = blockIdx.x, np = gridDim.x, n = d.n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned long long nbar = 0;
  unsigned phase = 0;
  int cur = 0;         // the pair buffer the next product reads
  int most = 0;        // the most rows of a tile of this block
  if (tid == 0) {
    S.gen = 0;   // the barrier is cleared before the launch
    S.iterations = S.restarts = 0;
    S.stop = 2;
    S.beta = 0.0;
  }
  for (int t = pb; t < d.tiles; t += np) {
    lay_out(d, t, S);
    most = max(most, (int)d.tile[t].rows);
  }
  auto slot = [&](int s) { return d.part + ((size_t)(phase & 1u) * kPcgSlots + s) * kMaxPcgBlocks; };
  // the block's partials of the phase: four warps a sum, a quarter of the
  // threads' values each
  auto put = [&](double a, double c, int slots) {
    S.part[0][tid] = a;
    if (slots > 1) S.part[1][tid] = c;
    __syncthreads();
    if (warp < 4 * slots) {
      const double* v = S.part[warp >> 2];
      double s = 0.0;
      for (int i = (warp & 3) * 32 + lane; i < most; i += 128) s = __dadd_rn(s, v[i]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
      if (lane == 0) S.quarter[warp] = s;
    }
    __syncthreads();
    if (tid < slots) {
      const double* v = S.quarter + 4 * tid;
      slot(tid)[pb] = __dadd_rn(__dadd_rn(v[0], v[1]), __dadd_rn(v[2], v[3]));
    }
  };
  // barrier, then fold the slots of the phase that just ended
  auto sync_fold = [&](int nslots) -> bool {
    if (!grid_sync(d.bar, (unsigned)np, &S.gen, &nbar, nullptr, &S.failed)) return false;
    if (warp < nslots) {
      const double v = warp_fold(slot(warp), np, 0.0, OpAdd());
      if (lane == 0) S.fv[warp].d = v;
    }
    __syncthreads();
    ++phase;
    return true;
  };
  // what this thread needs to know of a tile; the first one's is kept
  struct Work {
    unsigned row0, rows, segment, segments, width, j[kAhead];
    const double* w;
    const unsigned* idx;
  };
  auto work = [&](int t) {
    const PcgTile tile = d.tile[t];
    const uint2 mine = d.warp[(size_t)t * kPcgWarps + warp];
    Work k;
    k.row0 = tile.row0;
    k.rows = tile.rows;
    k.segment = d.place[(size_t)t * kPcgThreads + tid];
    k.segments = tid < (int)tile.rows ? d.row_segments[tile.row0 + tid] : 0;
    k.width = mine.y;
    k.w = d.dealt_w + tile.base + mine.x + lane;
    k.idx = d.dealt_i + tile.base + mine.x + lane;
#pragma unroll
    for (unsigned u = 0; u < kAhead; ++u) k.j[u] = u < k.width ? k.idx[32 * u] : tile.row0;
    return k;
  };
  const Work first = work(pb);
  // For every row of the block's tiles: the sum of W's row times the vector
  // that `load` and `value` give, handed to `row`.
  auto product = [&](auto load, auto value, auto row) {
    int odd = 0;
    Work k = first;
    for (int t = pb; t < d.tiles; t += np, odd ^= 1) {
      Work next = k;
      if (t + np < d.tiles) next = work(t + np);
      double s = 0.0;
      for (unsigned at = 0; at < k.width; at += kAhead) {
        decltype(load(0u)) v[kAhead];
        double w[kAhead];
#pragma unroll
        for (unsigned u = 0; u < kAhead; ++u) {
          v[u] = load(k.j[u]);
          w[u] = at + u < k.width ? k.w[32 * (size_t)(at + u)] : 0.0;
        }
#pragma unroll
        for (unsigned u = 0; u < kAhead; ++u)
          if (at + kAhead + u < k.width) k.j[u] = k.idx[32 * (size_t)(at + kAhead + u)];
#pragma unroll
        for (unsigned u = 0; u < kAhead; ++u)
          if (at + u < k.width) s = __fma_rn(w[u], value(v[u]), s);
      }
      S.sums[odd][k.segment] = s;
      __syncthreads();
      if (tid < (int)k.rows) {
        double total = 0.0;
        const unsigned from = k.segments & 0xffffu, count = k.segments >> 16;
        for (unsigned j = 0; j < count; ++j) total = j ? __dadd_rn(total, S.sums[odd][from + j]) : S.sums[odd][from];
        row((int)k.row0 + tid, total);
      }
      k = next;
    }
  };
  // r = b - (D - W) x with <r, r>; with `pairs` also z = r / D, the pairs
  // (z, 0) and <r, z>
  auto residual = [&](bool pairs) {
    double a = 0.0, c = 0.0;
    const double* x = d.x;
    product([&](unsigned j) { return x[j]; }, [](double v) { return v; },
            [&](int i, double s) {
              const double ri = __dsub_rn(d.b[i], __dsub_rn(__dmul_rn(d.diag[i], d.x[i]), s));
              d.r[i] = ri;
              a = __dadd_rn(a, __dmul_rn(ri, ri));
              if (pairs) {
                const double zi = __ddiv_rn(ri, d.diag[i]);
                d.inv[i] = reciprocal(d.diag[i]);
                d.zp[cur][i] = make_double2(zi, 0.0);
                c = __dadd_rn(c, __dmul_rn(ri, zi));
              }
            });
    put(a, c, pairs ? 2 : 1);
  };

  residual(true);
  if (!sync_fold(2)) return;
  if (__ldcg(&d.out->wrong_entry)) return;   // set before the barrier: every block leaves
  if (tid == 0) {
    S.rr = S.fv[PS_A].d;
    if (pb == 0) d.out->initial_rr = S.rr;
    S.target = fmax(S.rr, 2.220446049250313e-16) * kPcgTolerance;
    S.rho = S.fv[PS_B].d;
  }
  __syncthreads();

  for (int loop = 0; loop < n; ++loop) {
    if (S.rr <= S.target) break;
    // p = z + beta p, q = (D - W) p and <p, q>
    {
      const double2* zp = d.zp[cur];
      const double bt = S.beta;
      double a = 0.0;
      auto direction = [&](double2 v) { return __fma_rn(bt, v.y, v.x); };
      product([&](unsigned j) { return zp[j]; }, direction, [&](int i, double s) {
        const double pi = direction(zp[i]);
        const double qi = __dsub_rn(__dmul_rn(d.diag[i], pi), s);
        d.p[i] = pi;
        d.q[i] = qi;
        a = __dadd_rn(a, __dmul_rn(pi, qi));
      });
      put(a, 0.0, 1);
    }
    if (!sync_fold(1)) return;
    if (tid == 0) {
      const double den = S.fv[PS_A].d;
      S.action = 0;
      if (!isfinite(den) || den <= 0.0 || !isfinite(S.rho) || S.rho <= 0.0) {
        S.action = 1;
      } else {
        S.alpha = __ddiv_rn(S.rho, den);
        if (!isfinite(S.alpha)) S.action = 1;
      }
      if (S.action) S.stop = 1;
    }
    __syncthreads();
    if (S.action) break;
    // x += alpha p, r -= alpha q; |r|^2, z = r / D, <r, z>
    cur ^= 1;
    {
      double a = 0.0, c = 0.0;
      const double al = S.alpha;
      for (int t = pb; t < d.tiles; t += np) {
        const PcgTile tile = d.tile[t];
        if (tid >= (int)tile.rows) continue;
        const int i = (int)tile.row0 + tid;
        const double pi = d.p[i];
        d.x[i] = __dadd_rn(d.x[i], __dmul_rn(al, pi));
        const double ri = __dsub_rn(d.r[i], __dmul_rn(al, d.q[i]));
        const double zi = quotient(ri, d.diag[i], d.inv[i]);
        d.r[i] = ri;
        d.zp[cur][i] = make_double2(zi, pi);
        a = __dadd_rn(a, __dmul_rn(ri, ri));
        c = __dadd_rn(c, __dmul_rn(ri, zi));
      }
      put(a, c, 2);
    }
    if (!sync_fold(2)) return;
    if (tid == 0) {
      S.iterations++;
      S.rr = S.fv[PS_A].d;
      S.action = S.rr <= S.target ? 2 : 0;
      if (!S.action) {
        const double next = S.fv[PS_B].d;
        if (!isfinite(next) || next <= 0.0) {
          S.stop = 1;
          S.action = 1;
        } else {
          S.beta = __ddiv_rn(next, S.rho);
          S.rho = next;
        }
      }
    }
    __syncthreads();
    if (S.action == 1) break;
    if (S.action == 2) {
      // the recursive residual says converged: recompute the true one
      // (lib.rs:4656-4677) and restart from it when it is not small enough
      // (p = z: the pairs' second parts are zero)
      residual(true);
      if (!sync_fold(2)) return;
      if (tid == 0) {
        S.rr = S.fv[PS_A].d;
        S.action = 0;
        if (S.rr > S.target) {
          const double next = S.fv[PS_B].d;
          S.restarts++;
          S.beta = 0.0;
          if (!isfinite(next) || next <= 0.0) {
            S.stop = 1;
            S.action = 1;
          } else {
            S.rho = next;
          }
        }
      }
      __syncthreads();
      if (S.action == 1) break;
    }
  }

  // the true final residual (finish_quadratic_solve, lib.rs:4702-4752)
  residual(false);
  if (!sync_fold(1)) return;
  if (pb == 0 && tid == 0) {
    PcgResult& o = *d.out;
    o.final_rr = S.fv[PS_A].d;
    o.target = S.target;
    o.iterations = S.iterations;
    o.restarts = S.restarts;
    o.converged = o.final_rr <= S.target ? 1 : 0;
    o.stop = o.converged ? 0 : S.stop;
  }
}

__global__ void k_quotient_selftest(unsigned n, const double* a, const double* b, double* out) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = quotient(a[i], b[i], reciprocal(b[i]));
}

// Cuts the rows into tiles of about equal work, at most kPcgThreads segments
// each, and as many on each multiprocessor; a small system into tiles of 64
// segments or more (fewer blocks meet sooner at the barriers). `padded`: the
// entries with what fills the warps up, which is less than 32 of a tile's
// longest segment.
std::vector<PcgTile> cut_tiles(uint32_t n, const uint32_t* ptr, int sms, int* blocks, uint64_t* padded) {
  uint64_t segments = 0;
  for (uint32_t i = 0; i < n; ++i)
    segments += std::min<uint64_t>(std::max<uint64_t>(1, ((uint64_t)ptr[i + 1] - ptr[i] + kSegment - 1) / kSegment),
                                   kPcgThreads);
  const uint64_t fit = kPcgThreads - kPcgThreads / 8;   // boundaries fall up to a row late
  uint64_t want = std::max<uint64_t>(1, segments / 64);
  if (want > (uint64_t)sms) want = (segments + fit * sms - 1) / (fit * sms) * sms;
  constexpr uint64_t kRowCost = 16;   // a row's own operations, in entries
  const uint64_t cost = ptr[n] + kRowCost * n;
  std::vector<PcgTile> tiles;
  uint64_t base = 0, done = 0, in_tile = 0;
  for (uint32_t i = 0; i < n; ++i) {
    const uint64_t len = (uint64_t)ptr[i + 1] - ptr[i];
    uint64_t segs = std::max<uint64_t>(1, (len + kSegment - 1) / kSegment);
    const bool alone = segs > kPcgThreads;   // a long row is its own tile, of longer segments
    const bool due = done * want >= (uint64_t)tiles.size() * cost;
    if (tiles.empty() || due || in_tile + segs > kPcgThreads) {
      if (!tiles.empty()) base += (uint64_t)ptr[i] - ptr[tiles.back().row0] + 32ull * tiles.back().segment;
      tiles.push_back({i, 0, alone ? (unsigned)((len + kPcgThreads - 1) / kPcgThreads) : kSegment, base});
      in_tile = 0;
    }
    tiles.back().rows++;
    in_tile += alone ? (uint64_t)kPcgThreads : segs;
    done += len + kRowCost;
  }
  *padded = base + ((uint64_t)ptr[n] - ptr[tiles.back().row0]) + 32ull * tiles.back().segment;
  *blocks = (int)std::min<uint64_t>((uint64_t)sms, tiles.size());
  return tiles;
}

}  // namespace
}  // namespace tgp

using namespace tgp;

extern "C" int32_t texo_gp_quadratic_solve(int32_t device, uint32_t n, const double* diagonal,
                                           const uint32_t* adjacency_ptr, const uint32_t* adjacency_index,
                                           const double* adjacency_weight, const double* rhs, double* solution,
                                           texo_gp_pcg_stats* stats) {
  if (stats) std::memset(stats, 0, sizeof(*stats));
  auto fail = [&](int32_t s, const std::string& why) {
    if (!why.empty()) set_last_error(why);
    if (stats) stats->status = s;
    return s;
  };
  if (!diagonal || !adjacency_ptr || !rhs || !solution) return fail(TEXO_GP_ERR_INVALID_ARGUMENT, "null argument");
  if (n == 0) return fail(TEXO_GP_OK, "");
  if (n > (1u << 30)) return fail(TEXO_GP_ERR_INVALID_ARGUMENT, "system too large");
  const uint64_t nnz = adjacency_ptr[n];
  if (adjacency_ptr[0] != 0 || (nnz && (!adjacency_index || !adjacency_weight)))
    return fail(TEXO_GP_ERR_INVALID_ARGUMENT, "adjacency_ptr must start at 0");
  // no early way out: these loops are vectorized
  constexpr double kMax = std::numeric_limits<double>::max();
  unsigned decreases = 0, diagonals = 0, vectors = 0;
  for (uint32_t i = 0; i < n; ++i) decreases |= adjacency_ptr[i + 1] < adjacency_ptr[i];
  for (uint32_t i = 0; i < n; ++i) diagonals |= !(diagonal[i] > 0.0) | !(diagonal[i] <= kMax);
  for (uint32_t i = 0; i < n; ++i) vectors |= !(std::fabs(rhs[i]) <= kMax) | !(std::fabs(solution[i]) <= kMax);
  if (decreases) return fail(TEXO_GP_ERR_INVALID_ARGUMENT, "adjacency_ptr decreases");
  if (diagonals) return fail(TEXO_GP_ERR_INVALID_ARGUMENT, "diagonal entries must be finite and positive");
  if (vectors) return fail(TEXO_GP_ERR_INVALID_ARGUMENT, "non-finite right-hand side or initial solution");
  // The entries are checked where the kernel deals them; without a device,
  // here, so that a wrong system is refused as such.
  const char* const kWrongEntry = "adjacency index out of range or non-finite weight";
  auto no_device = [&](int32_t st, const std::string& why) {
    for (uint64_t k = 0; k < nnz; ++k)
      if (adjacency_index[k] >= n || !std::isfinite(adjacency_weight[k]))
        return fail(TEXO_GP_ERR_INVALID_ARGUMENT, kWrongEntry);
    return fail(st, why);
  };

  if (cudaSetDevice(device) != cudaSuccess) return no_device(TEXO_GP_ERR_CUDA, "cudaSetDevice failed");
  static const int per_sm = [] {   // thread-safe one-time initialisation
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_pcg, kPcgThreads, 0) != cudaSuccess) b = 0;
    return b;
  }();
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (per_sm <= 0 || sms <= 0) return no_device(TEXO_GP_ERR_CUDA, "k_pcg cannot be resident");
  int blocks = 0;
  uint64_t padded = 0;
  std::vector<PcgTile> tiles;
  try {
    tiles = cut_tiles(n, adjacency_ptr, std::min(sms, kMaxPcgBlocks), &blocks, &padded);
  } catch (const std::bad_alloc&) {
    return no_device(TEXO_GP_ERR_OUT_OF_MEMORY, "no memory for the tiles");
  }

  // one allocation: vectors, matrix, partials, barrier, result
  auto round = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t vec = round((size_t)n * 8), nz8 = round(std::max<uint64_t>(nnz, 1) * 8),
               nz4 = round(std::max<uint64_t>(nnz, 1) * 4), p4 = round(((size_t)n + 1) * 4);
  const size_t part = round((size_t)2 * kPcgSlots * kMaxPcgBlocks * 8);
  const size_t pad8 = round(padded * 8), pad4 = round(padded * 4), rows4 = round((size_t)n * 4),
               tile_bytes = round(tiles.size() * sizeof(PcgTile)),
               warp_bytes = round(tiles.size() * kPcgWarps * sizeof(uint2)),
               place_bytes = round(tiles.size() * kPcgThreads * sizeof(unsigned short));
  const size_t total = 11 * vec + nz8 + nz4 + p4 + part + pad8 + pad4 + rows4 + tile_bytes + warp_bytes + place_bytes +
                       round(sizeof(GridBarrier)) + round(sizeof(PcgResult));
  Call call(device);
  if (!call.ok()) return no_device(TEXO_GP_ERR_CUDA, "stream");
  const cudaStream_t s = call.stream();
  char* base = call.memory(total);
  if (!base) return no_device(TEXO_GP_ERR_OUT_OF_MEMORY, "cudaMallocAsync failed");
  char* at = base;
  auto take = [&](size_t b) {
    char* r = at;
    at += b;
    return r;
  };
  PcgDev d{};
  d.n = (int)n;
  double* diag = (double*)take(vec);
  double* b = (double*)take(vec);
  d.x = (double*)take(vec);
  d.r = (double*)take(vec);
  d.p = (double*)take(vec);
  d.q = (double*)take(vec);
  d.inv = (double*)take(vec);
  d.zp[0] = (double2*)take(2 * vec);
  d.zp[1] = (double2*)take(2 * vec);
  double* w = (double*)take(nz8);
  unsigned* idx = (unsigned*)take(nz4);
  unsigned* ptr = (unsigned*)take(p4);
  d.dealt_w = (double*)take(pad8);
  d.dealt_i = (unsigned*)take(pad4);
  d.row_segments = (unsigned*)take(rows4);
  PcgTile* tile = (PcgTile*)take(tile_bytes);
  d.warp = (uint2*)take(warp_bytes);
  d.place = (unsigned short*)take(place_bytes);
  d.tile = tile;
  d.tiles = (int)tiles.size();
  d.part = (double*)take(part);
  d.bar = (GridBarrier*)take(round(sizeof(GridBarrier)));
  d.out = (PcgResult*)take(round(sizeof(PcgResult)));
  d.diag = diag;
  d.b = b;
  d.w = w;
  d.idx = idx;
  d.ptr = ptr;

  int32_t st = TEXO_GP_OK;
  PcgResult res{};
  call.start();
  bool ok = cudaMemcpyAsync(diag, diagonal, (size_t)n * 8, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemcpyAsync(b, rhs, (size_t)n * 8, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemcpyAsync(d.x, solution, (size_t)n * 8, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemcpyAsync(ptr, adjacency_ptr, ((size_t)n + 1) * 4, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            (!nnz || (cudaMemcpyAsync(idx, adjacency_index, nnz * 4, cudaMemcpyHostToDevice, s) == cudaSuccess &&
                      cudaMemcpyAsync(w, adjacency_weight, nnz * 8, cudaMemcpyHostToDevice, s) == cudaSuccess)) &&
            cudaMemcpyAsync(tile, tiles.data(), tiles.size() * sizeof(PcgTile), cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemsetAsync(d.bar, 0, sizeof(GridBarrier), s) == cudaSuccess &&
            cudaMemsetAsync(d.out, 0, sizeof(PcgResult), s) == cudaSuccess;
  if (ok) {
    void* args[] = {&d};
    ok = cudaLaunchCooperativeKernel((const void*)k_pcg, dim3(blocks), dim3(kPcgThreads), args, 0, s) == cudaSuccess;
    if (ok) note_launch();
  }
  GridBarrier hb{};
  ok = ok && cudaMemcpyAsync(solution, d.x, (size_t)n * 8, cudaMemcpyDeviceToHost, s) == cudaSuccess &&
       cudaMemcpyAsync(&res, d.out, sizeof(PcgResult), cudaMemcpyDeviceToHost, s) == cudaSuccess &&
       cudaMemcpyAsync(&hb, d.bar, sizeof(GridBarrier), cudaMemcpyDeviceToHost, s) == cudaSuccess;
  float ms = 0.f;
  if (!call.finish(&ms)) ok = false;
  if (!ok) {
    st = TEXO_GP_ERR_CUDA;
    set_last_error(std::string("quadratic solve: ") + cudaGetErrorString(cudaGetLastError()));
  } else if (hb.error) {
    st = TEXO_GP_ERR_DEVICE_TIMEOUT;
    set_last_error("quadratic solve: a grid barrier wait ran out");
  } else if (res.wrong_entry) {   // the solution came back as it was
    return fail(TEXO_GP_ERR_INVALID_ARGUMENT, kWrongEntry);
  } else if (!res.converged) {
    st = TEXO_GP_ERR_PCG_NOT_CONVERGED;
    set_last_error(std::string("analytical PCG ") + (res.stop == 1 ? "breakdown" : "dimension") + " after " +
                   std::to_string(res.iterations) + "/" + std::to_string(n) + " iterations");
  }
  if (stats) {
    stats->status = st;
    stats->iterations = res.iterations;
    stats->restarts = res.restarts;
    stats->stop = res.stop;
    stats->initial_residual_squared = res.initial_rr;
    stats->target_squared = res.target;
    stats->final_residual_squared = res.final_rr;
    stats->elapsed_ms = ms;
    stats->kernel_launches = 1;
  }
  return st;
}

extern "C" int32_t texo_gp_selftest_quotient(int32_t device, uint32_t n, const double* a, const double* b, double* out) {
  if (n == 0 || n > (1u << 26) || !a || !b || !out) return TEXO_GP_ERR_INVALID_ARGUMENT;
  Call call(device);
  if (!call.ok()) return TEXO_GP_ERR_CUDA;
  const size_t bytes = (size_t)n * 8;
  double* d = (double*)call.memory(3 * bytes);
  if (!d) return TEXO_GP_ERR_OUT_OF_MEMORY;
  const cudaStream_t s = call.stream();
  call.start();
  bool ok = cudaMemcpyAsync(d, a, bytes, cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaMemcpyAsync(d + n, b, bytes, cudaMemcpyHostToDevice, s) == cudaSuccess;
  if (ok) {
    k_quotient_selftest<<<(n + kPcgThreads - 1) / kPcgThreads, kPcgThreads, 0, s>>>(n, d, d + n, d + 2 * (size_t)n);
    ok = cudaGetLastError() == cudaSuccess &&
         cudaMemcpyAsync(out, d + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost, s) == cudaSuccess;
  }
  float ms = 0.f;
  if (!call.finish(&ms)) ok = false;
  return ok ? TEXO_GP_OK : TEXO_GP_ERR_CUDA;
}
