// kernels.cu — standalone kernels (one stage each) and their launchers.
#include "dct_fft.cuh"
#include "dct_tc.cuh"
#include "kernels.cuh"
#include "scatter_tiles.cuh"

namespace tgp {

// The kernels of an evaluation follow one another within microseconds. Launched
// with `follow` a kernel is set up while its predecessor in the stream still
// runs, and its blocks wait here until that kernel has completed and its writes
// can be seen (so no kernel that is launched so reads its predecessors' results
// through the read-only cache). The wait covers the kernel before it in its
// own stream and nothing else: the kernel after a cudaStreamWaitEvent is launched
// plainly (`launch_finalize_joined`), as is k_wa, whose predecessor is in
// another stream, and as are the kernels after a stream-ordered allocation, which
// may make the stream wait for the one that freed the memory. An evaluation at 250,000 cells with the tensor-core transforms,
// 19 launches, 245 -> 215 us; a whole evaluate call at 2,000 cells 166 -> 148.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
void follow(void (*kernel)(P...), int blocks, int threads, size_t shared, cudaStream_t s, A... a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)blocks);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = shared;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(a)...);
}

// The FFT form's three passes (dct_fft.cuh), NB = 2 for 1024 points. Four blocks
// an SM for the row passes (1024^2 rows inverse: 39 us with 118 registers and
// two blocks, 33 with 64 and four).
// PREP: the density preparation folded in (k_prep's rho and overflow sums bit
// for bit, one pass over the grids less: 11 us of 38 at 1024^2), each block
// with groups folding the scatter's totals for the means.
template <int NB, bool PREP>
__global__ void __launch_bounds__(kThreads, 4) k_fft_rows_fwd(Dev d, Partials p) {
  after_previous();
  __shared__ fft::Smem sm;
  __shared__ Shared sh;
  __shared__ long long mean[kMaxFields];
  if (PREP) {
    for (int f = 0; f < d.K; ++f) {
      const long long tot = block_reduce_array(islot(p, IS_GRID_SUM + f), (int)gridDim.x, 0ll, OpAdd(), sh.l);
      if (threadIdx.x == 0) mean[f] = (tot - d.capsum[f]) / d.B;
    }
    __syncthreads();
  }
  fft::rows_fwd<NB, false>(whole_block(), d, p, blockIdx.x, gridDim.x, sm.buf, sh, PREP ? mean : nullptr, false, 0,
                           fft::Inlined());
}
template <int NB>
__global__ void __launch_bounds__(kThreads, NB == 2 ? 4 : 1) k_fft_cols(Dev d) {
  after_previous();
  __shared__ fft::Smem sm;
  fft::cols<NB>(whole_block(), d, blockIdx.x, gridDim.x, sm.buf, false, 0, fft::Inlined());
}
template <int NB>
__global__ void __launch_bounds__(kThreads, 4) k_fft_rows_inv(Dev d, Partials p) {
  after_previous();
  __shared__ fft::Smem sm;
  __shared__ Shared sh;
  fft::rows_inv<NB>(whole_block(), d, p, blockIdx.x, gridDim.x, sm.buf, sh, false, fft::Inlined());
}

// The slice phase before tensor-core pass `step` (memory-bound, every block).
// Before pass 3, whose `energies` blocks write the energy partials, the other
// blocks' are zeroed.
__global__ void __launch_bounds__(kThreads) k_tc_slice(Dev d, Partials p, int step, int energies) {
  after_previous();
  if (step == 3 && (int)blockIdx.x >= energies && (int)threadIdx.x < d.K)
    pslot(p, SLOT_ENERGY + (int)threadIdx.x)[blockIdx.x] = 0.0;
  tc::slice_phase(d, step, blockIdx.x, gridDim.x);
}

// One DCT pass on tcgen05 tensor cores, one 128 x 64 tile per block
// iteration; gridDim.x <= the pass's tiles. The energy partials of pass 3 are
// those of the blocks launched; the slice phase before it zeroes the rest.
template <int STEP>
__global__ void __launch_bounds__(kThreads, 1) k_dct_tc(Dev d, Partials p, unsigned long long* err,
                                                       const __grid_constant__ tc::TcMaps maps) {
  after_previous();
  extern __shared__ __align__(128) unsigned char tc_dyn[];
  tc::Smem& sm = *reinterpret_cast<tc::Smem*>(tc_dyn);
  double eacc[kMaxFields] = {0.0, 0.0, 0.0, 0.0};
  tc::setup(sm);
  tc::dct_pass<STEP>(d, maps, blockIdx.x, gridDim.x, sm, eacc, err);
  tc::teardown(sm);
  if constexpr (STEP == 3) {
    __shared__ Shared sh;
    for (int f = 0; f < d.K; ++f) write_partial(eacc[f], pslot(p, SLOT_ENERGY + f), (int)blockIdx.x, sh.d);
  }
}
template <int STEP>
void launch_dct_tc(const Dev& d, const Reduce& r, int gb, cudaStream_t s, const tc::TcMaps& maps) {
  static const bool attr = cudaFuncSetAttribute(k_dct_tc<STEP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)sizeof(tc::Smem)) == cudaSuccess;
  (void)attr;
  follow(k_dct_tc<STEP>, gb, kThreads, sizeof(tc::Smem), s, d, r.p, (unsigned long long*)(r.iscal + SI_TC_FAIL), maps);
}

__global__ void __launch_bounds__(kThreads) k_init(Dev d, bool grids, bool wa) {
  after_previous();
  stage_init(whole_block(), d, blockIdx.x, gridDim.x, grids, wa);
}
__global__ void __launch_bounds__(kThreads) k_scatter(Dev d, Partials p, const float2* pos) {
  after_previous();
  __shared__ Shared sh;
  stage_scatter(whole_block(), d, pos, p, blockIdx.x, gridDim.x, sh);
}
// The tiled scatter's four passes (scatter_tiles.cuh).
__global__ void __launch_bounds__(kThreads) k_tile_count(Dev d, const float2* pos) {
  tiles::count(d, pos, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(kThreads) k_tile_scan(Dev d) { tiles::scan(d); }
__global__ void __launch_bounds__(kThreads) k_tile_place(Dev d) { tiles::place(d, blockIdx.x, gridDim.x); }
__global__ void __launch_bounds__(kThreads) k_tile_scatter(Dev d, Partials p, const float2* pos) {
  __shared__ tiles::Smem sm;
  __shared__ Shared sh;
  tiles::scatter(d, pos, p, blockIdx.x, gridDim.x, sm, sh);
}
// Every object uniform in its bounds from a fixed hash (the autotuner's
// stand-in for a spread placement).
__global__ void __launch_bounds__(kThreads) k_spread_positions(Dev d, float2* out) {
  for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < d.nobj; o += gridDim.x * blockDim.x) {
    unsigned h = (unsigned)o * 2654435761u + 12345u;
    h ^= h >> 15;
    h *= 2246822519u;
    h ^= h >> 13;
    const float fx = (float)(h & 0xffffu) * (1.0f / 65536.0f), fy = (float)(h >> 16) * (1.0f / 65536.0f);
    const float2 lo = d.lo[o], hi = d.hi[o];
    out[o] = make_float2(fmaf(hi.x - lo.x, fx, lo.x), fmaf(hi.y - lo.y, fy, lo.y));
  }
}
// 4 blocks an SM: the stage waits on memory (72 registers and 3 blocks: 85 us at 1M cells, 79 with 64)
__global__ void __launch_bounds__(kThreads, 4) k_wa(Dev d, Partials p, const float2* pos, double gamma) {
  __shared__ Shared sh;
  stage_wa(whole_block(), d, pos, gamma, p, blockIdx.x, gridDim.x, sh.d);
}
__global__ void __launch_bounds__(kThreads) k_prep(Dev d, Partials p) {
  after_previous();
  __shared__ Shared sh;
  stage_prep(whole_block(), d, p, gridDim.x, blockIdx.x, gridDim.x, sh);
}
template <bool LARGE>
__global__ void __launch_bounds__(kThreads) k_dct(Dev d, Partials p, int step) {
  after_previous();
  __shared__ GemmShared sm;
  __shared__ Shared sh;
  stage_dct_t<LARGE>(whole_block(), d, step, p, blockIdx.x, gridDim.x, sm, sh);
}
__global__ void __launch_bounds__(kThreads) k_gather(Dev d, Partials p, const float2* pos) {
  after_previous();
  __shared__ Shared sh;
  stage_gather(whole_block(), d, pos, p, blockIdx.x, gridDim.x, sh);
}
__global__ void __launch_bounds__(kThreads) k_combine(Dev d, Partials p, const double* coef, float2* gout,
                                                     const float2* kkt_pos) {
  after_previous();
  __shared__ Shared sh;
  __shared__ double buf[(kMaxFields + 1) * (kThreads + 4)];
  stage_combine(whole_block(), d, coef, gout, p, blockIdx.x, gridDim.x, sh, buf, kMaxFields + 1, kkt_pos);
}
// The next point, and (reset) the accumulators cleared for its evaluation.
__global__ void __launch_bounds__(kThreads) k_extrapolate(Dev d, Partials p, const float2* x, const float2* xp,
                                                         float e, float2* y, bool reset) {
  after_previous();
  __shared__ Shared sh;
  if (reset) stage_init(whole_block(), d, blockIdx.x, gridDim.x, true, true);
  stage_extrapolate(whole_block(), d, x, xp, e, y, p, blockIdx.x, gridDim.x, sh);
}
__global__ void __launch_bounds__(kThreads) k_candidate(Dev d, Partials p, const float2* y, const float2* gy,
                                                       float invL, float2* c, bool reset) {
  after_previous();
  __shared__ Shared sh;
  __shared__ double buf[2 * (kThreads + 4)];
  if (reset) stage_init(whole_block(), d, blockIdx.x, gridDim.x, true, true);
  stage_candidate(whole_block(), d, y, gy, invL, c, p, blockIdx.x, gridDim.x, sh, buf);
}
__global__ void __launch_bounds__(kThreads) k_kkt(Dev d, Partials p, const float2* x, const float2* g) {
  after_previous();
  __shared__ Shared sh;
  stage_kkt(whole_block(), d, x, g, p, blockIdx.x, gridDim.x, sh);
}
__global__ void __launch_bounds__(kThreads) k_precond(Dev d, Partials p, const double* lambda) {
  after_previous();
  __shared__ Shared sh;
  stage_precond(whole_block(), d, lambda, p, blockIdx.x, gridDim.x, sh);
}
__global__ void __launch_bounds__(kThreads) k_hpwl(Dev d, Partials p, const float2* pos) {
  __shared__ Shared sh;
  stage_hpwl(d, pos, p, blockIdx.x, gridDim.x, sh);
}

// Reduces the partials selected by `mask` in a fixed order and derives the
// objective scalars (combined_objective / augmented_density_value_and_coefficient,
// eplace.rs:1022-1044, 1111-1124). Each slot is folded by 128 threads (four
// warps, one per SM sub-partition) in block_reduce_array's order, eight slots
// side by side: a slot is a round trip to memory and a chain of FP64 adds of
// 64 cycles each; the nine slots of an evaluation took 14.6 us one after
// another at 1M cells and take 7.5 this way (two rounds of eight).
constexpr int kFinThreads = 1024;
constexpr int kMaxFinJobs = 6 * kMaxFields + 16;
struct FinJob {
  const void* a;
  int op;    // 0 FP64 sum, 1 integer sum, 2 integer minimum, 3 FP64 maximum, 4 FP64 minimum
};
__device__ __forceinline__ unsigned long long fin_fold(const FinJob& j, int n, unsigned long long* warps, int t) {
  auto fold = [&](auto zero, auto op) {
    using T = decltype(zero);
    const T* a = reinterpret_cast<const T*>(j.a);
    T v = t < n ? a[t] : zero;
#pragma unroll 4
    for (int i = t + 128; i < n; i += 128) v = op(v, a[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    T* w = reinterpret_cast<T*>(warps);
    if ((t & 31) == 0) w[t >> 5] = v;
    asm volatile("bar.sync %0, 128;" ::"r"(1 + (int)(threadIdx.x >> 7)) : "memory");
    const T r = op(op(op(w[0], w[1]), w[2]), w[3]);
    asm volatile("bar.sync %0, 128;" ::"r"(1 + (int)(threadIdx.x >> 7)) : "memory");
    unsigned long long bits;
    memcpy(&bits, &r, 8);
    return bits;
  };
  switch (j.op) {
    case 0: return fold(0.0, OpAdd());
    case 1: return fold(0ll, OpAdd());
    case 2: return fold(0x7fffffffffffffffll, OpMin());
    case 3: return fold(0.0, OpMax());
    default: return fold((double)INFINITY, OpMin());
  }
}
__global__ void __launch_bounds__(kFinThreads) k_finalize(Dev d, Reduce r, int nvb, int mask) {
  after_previous();
  __shared__ FinJob jobs[kMaxFinJobs];
  __shared__ int to[kMaxFinJobs];               // output: scalar slot, or kScalars + integer slot
  __shared__ int count;
  __shared__ unsigned long long warps[kFinThreads / 128][4];
  __shared__ double sc[kScalars];
  const Partials& p = r.p;
  if (threadIdx.x < kScalars) sc[threadIdx.x] = r.scal[threadIdx.x];
  if (threadIdx.x == 0) {
    int n = 0;
    auto add = [&](const void* a, int op, int out) {
      jobs[n] = FinJob{a, op};
      to[n++] = out;
    };
    if (mask & (FIN_ENERGY | FIN_WA)) add(pslot(p, SLOT_WA_VALUE), 0, SC_WA);
    if (mask & FIN_ENERGY)
      for (int f = 0; f < d.K; ++f) {
        add(pslot(p, SLOT_ENERGY + f), 0, SC_ENERGY + f);
        add(islot(p, IS_OVERFLOW + f), 1, kScalars + SI_OVERFLOW_FIXED + f);
        add(islot(p, IS_OVER_BINS + f), 1, kScalars + SI_OVER_BINS + f);
        add(islot(p, IS_GRID_SUM + f), 1, kScalars + SI_GRID_SUM + f);
      }
    if (mask & FIN_COMBINE) {
      for (int f = 0; f < d.K; ++f) {
        add(pslot(p, SLOT_RAWL1 + f), 0, SC_RAWL1 + f);
        add(pslot(p, SLOT_FORCE + f), 0, SC_FORCE + f);
      }
      add(pslot(p, SLOT_WAL1), 0, SC_WAL1);
      add(islot(p, IS_BAD), 2, kScalars + SI_BAD);
    }
    if (mask & (FIN_CAND | FIN_DIFF)) add(islot(p, IS_DIFF), 1, kScalars + SI_DIFF);
    if (mask & FIN_CAND) {
      add(pslot(p, SLOT_DOT), 0, SC_DOT);
      add(pslot(p, SLOT_MSN), 0, SC_MSN);
    }
    if (mask & FIN_KKT) add(mslot(p, MS_KKT), 3, SC_KKT);
    if (mask & FIN_PRECOND) {
      add(mslot(p, MS_PMIN), 4, SC_PMIN);
      add(mslot(p, MS_PMAX), 3, SC_PMAX);
      add(islot(p, IS_PBAD), 1, kScalars + SI_PBAD);
    }
    if (mask & FIN_HPWL) add(pslot(p, SLOT_HPWL), 0, SC_HPWL);
    count = n;
  }
  __syncthreads();
  const int g = threadIdx.x >> 7, t = threadIdx.x & 127;
  for (int j = g; j < count; j += kFinThreads / 128) {
    const unsigned long long v = fin_fold(jobs[j], nvb, warps[g], t);
    if (t == 0) {
      const int o = to[j];
      if (o >= kScalars) {
        r.iscal[o - kScalars] = (long long)v;
        // the derived values of an integer sum, by the thread that has it
        const int s = o - kScalars;
        if (s >= SI_OVERFLOW_FIXED && s < SI_OVERFLOW_FIXED + kMaxFields) {
          const int f = s - SI_OVERFLOW_FIXED;
          r.scal[SC_OVERFLOW + f] = ((double)(long long)v * kInvFix) / sc[SC_REAL_AREA + f];
        } else if (s >= SI_GRID_SUM && s < SI_GRID_SUM + kMaxFields) {
          const int f = s - SI_GRID_SUM;
          r.scal[SC_MEAN + f] = (double)((long long)v - d.capsum[f]) * kInvFix;
        }
      } else {
        double x;
        memcpy(&x, &v, 8);
        if (o >= SC_ENERGY && o < SC_ENERGY + kMaxFields) x *= 0.5;
        sc[o] = x;
        r.scal[o] = x;
      }
    }
  }
  if (!(mask & (FIN_ENERGY | FIN_WA))) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    double value = sc[SC_WA];
    const double beta = sc[SC_BETA];
    for (int f = 0; f < d.K; ++f) {
      const double e0 = sc[SC_E0 + f], lam = sc[SC_LAMBDA + f];
      const double ne = sc[SC_ENERGY + f] / e0;
      value += lam * e0 * (ne + 0.5 * beta * ne * ne);
      r.scal[SC_COEF + f] = lam * (1.0 + beta * ne);
    }
    r.scal[SC_VALUE] = value;
  }
}

// The API's FP64 arrays on the device: the host arrays are copied as they are
// (on this machine a copy from or to pageable memory runs at the pinned rate)
// and narrowed or widened here. On one host core the conversions of a
// million-cell call took 6.5 ms of its 15.
__global__ void __launch_bounds__(kThreads) k_narrow(const double* __restrict__ src, float* __restrict__ dst, size_t n,
                                                     long long* nonfinite, long long mark) {
  bool bad = false;
  for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kThreads) {
    const double v = src[i];
    dst[i] = __double2float_rn(v);
    bad = bad || !isfinite(v);
  }
  if (nonfinite && bad) atomicMax(nonfinite, mark);
}
// rounded_targets_from_coordinates (eplace.rs:954-971) of the checkpoint, and
// the current coordinates; either output may be null.
__global__ void __launch_bounds__(kThreads) k_widen_point(Dev d, const float2* best, const float2* x,
                                                          uint2* __restrict__ targets, double2* __restrict__ coords) {
  const float top_x = (float)(d.g.W - 1), top_y = (float)(d.g.H - 1);
  for (int o = blockIdx.x * kThreads + threadIdx.x; o < d.nobj; o += gridDim.x * kThreads) {
    if (targets && o < d.U) {
      const float2 b = best[o];
      targets[o] = make_uint2((uint32_t)fminf(fmaxf(roundf(b.x), 0.f), top_x),
                              (uint32_t)fminf(fmaxf(roundf(b.y), 0.f), top_y));
    }
    if (coords) {
      const float2 a = x[o];
      coords[o] = make_double2((double)a.x, (double)a.y);
    }
  }
}
// texo_gp_evaluate's arrays; each may be null.
__global__ void __launch_bounds__(kThreads) k_widen_eval(Dev d, double* wa, double2* field, double* density,
                                                         double* potential) {
  const int first = blockIdx.x * kThreads + threadIdx.x, stride = gridDim.x * kThreads;
  if (wa)
    for (int i = first; i < 2 * d.U; i += stride) wa[i] = (double)(long long)d.wa_fix[i] * kInvFix;
  if (field)
    for (int f = 0; f < d.K; ++f)
      for (int o = first; o < d.nobj; o += stride) {
        const bool valid = o < d.U || d.fil_field[o - d.U] == f;
        const float2 v = valid ? d.graw[(size_t)f * d.nobj + o] : make_float2(0.f, 0.f);
        field[(size_t)f * d.nobj + o] = make_double2((double)v.x, (double)v.y);
      }
  if (density)
    for (int i = first; i < d.K * d.B; i += stride) density[i] = (double)(d.phys[i] + d.fill[i]) * kInvFix;
  if (potential)
    for (int i = first; i < d.K * d.B; i += stride) potential[i] = (double)d.phi[i];
}

// rounded_targets_from_coordinates (eplace.rs:954-971) compared with the
// previous stationary targets (stationary_target_is_fixed, :973-985).
__global__ void k_round_compare(Dev d, const float2* x, uint32_t* prev, int W, int H, unsigned long long* mismatch) {
  for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < d.U; u += gridDim.x * blockDim.x) {
    const float2 a = x[u];
    const float rx = fminf(fmaxf(roundf(a.x), 0.f), (float)(W - 1));
    const float ry = fminf(fmaxf(roundf(a.y), 0.f), (float)(H - 1));
    const uint32_t tx = (uint32_t)rx, ty = (uint32_t)ry;
    if (prev[2 * u] != tx || prev[2 * u + 1] != ty) atomicAdd(mismatch, 1ull);
    prev[2 * u] = tx;
    prev[2 * u + 1] = ty;
  }
}

static thread_local unsigned long long t_launches = 0;
unsigned long long launches_issued() { return t_launches; }
void note_launch() { ++t_launches; }
#define COUNT ++t_launches

static inline bool use_large_tiles(const Dev& d) { return d.dct_large != 0; }

void launch_init(const Dev& d, bool grids, bool wa, int nvb, cudaStream_t s) {
  COUNT;
  follow(k_init, nvb, kThreads, 0, s, d, grids, wa);
}
void launch_scatter(const Dev& d, const Reduce& r, const float2* pos, int nvb, cudaStream_t s) {
  if (d.scatter_tiles && d.Mm + d.F > 0) {
    t_launches += 4;
    k_tile_count<<<nvb, kThreads, 0, s>>>(d, pos);
    k_tile_scan<<<1, kThreads, 0, s>>>(d);
    k_tile_place<<<nvb, kThreads, 0, s>>>(d);
    k_tile_scatter<<<nvb, kThreads, 0, s>>>(d, r.p, pos);
    return;
  }
  COUNT;
  follow(k_scatter, nvb, kThreads, 0, s, d, r.p, pos);
}
void launch_spread_positions(const Dev& d, float2* out, int nvb, cudaStream_t s) {
  COUNT;
  k_spread_positions<<<nvb, kThreads, 0, s>>>(d, out);
}
void launch_wa(const Dev& d, const Reduce& r, const float2* pos, double gamma, int nvb, cudaStream_t s) {
  COUNT;
  k_wa<<<nvb, kThreads, 0, s>>>(d, r.p, pos, gamma);
}
void launch_prep(const Dev& d, const Reduce& r, int nvb, cudaStream_t s) {
  COUNT;
  follow(k_prep, nvb, kThreads, 0, s, d, r.p);
}
void launch_dct(const Dev& d, const Reduce& r, int step, int nvb, cudaStream_t s, const tc::TcMaps* maps, bool prep) {
  if (d.fft) {   // rows, columns (forward, scale, inverse), rows: step 2 has no work
    if (step == 2) return;
    COUNT;
    if (step == 0)
      follow(prep ? (d.logW == 10 ? k_fft_rows_fwd<2, true> : k_fft_rows_fwd<1, true>)
                  : (d.logW == 10 ? k_fft_rows_fwd<2, false> : k_fft_rows_fwd<1, false>),
             nvb, kThreads, 0, s, d, r.p);
    else if (step == 1)
      follow(d.logH == 10 ? k_fft_cols<2> : k_fft_cols<1>, nvb, kThreads, 0, s, d);
    else
      follow(d.logW == 10 ? k_fft_rows_inv<2> : k_fft_rows_inv<1>, nvb, kThreads, 0, s, d, r.p);
    return;
  }
  if (d.tc) {
    if (!maps) return;   // the tensor-core form needs the instance's tensor maps
    // one block a tile (at most one resident a multiprocessor: the pipeline
    // holds 192 KB of shared memory and 256 TMEM columns)
    const int gb = std::max(1, std::min(nvb, tc::pass_tiles_host(d)));
    COUNT;
    follow(k_tc_slice, nvb, kThreads, 0, s, d, r.p, step, gb);
    COUNT;
    switch (step) {
      case 0: launch_dct_tc<0>(d, r, gb, s, *maps); break;
      case 1: launch_dct_tc<1>(d, r, gb, s, *maps); break;
      case 2: launch_dct_tc<2>(d, r, gb, s, *maps); break;
      default: launch_dct_tc<3>(d, r, gb, s, *maps); break;
    }
    return;
  }
  COUNT;
  if (use_large_tiles(d))
    follow(k_dct<true>, nvb, kThreads, 0, s, d, r.p, step);
  else
    follow(k_dct<false>, nvb, kThreads, 0, s, d, r.p, step);
}
void launch_gather(const Dev& d, const Reduce& r, const float2* pos, int nvb, cudaStream_t s) {
  COUNT;
  follow(k_gather, nvb, kThreads, 0, s, d, r.p, pos);
}
void launch_combine(const Dev& d, const Reduce& r, float2* gout, int nvb, cudaStream_t s, const float2* kkt_pos) {
  COUNT;
  follow(k_combine, nvb, kThreads, 0, s, d, r.p, r.scal + SC_COEF, gout, kkt_pos);
}
void launch_extrapolate(const Dev& d, const Reduce& r, const float2* x, const float2* xp, float e, float2* y,
                        int nvb, cudaStream_t s, bool reset) {
  COUNT;
  follow(k_extrapolate, nvb, kThreads, 0, s, d, r.p, x, xp, e, y, reset);
}
void launch_candidate(const Dev& d, const Reduce& r, const float2* y, const float2* gy, float invL, float2* c,
                      int nvb, cudaStream_t s, bool reset) {
  COUNT;
  follow(k_candidate, nvb, kThreads, 0, s, d, r.p, y, gy, invL, c, reset);
}
void launch_kkt(const Dev& d, const Reduce& r, const float2* x, const float2* g, int nvb, cudaStream_t s) {
  COUNT;
  follow(k_kkt, nvb, kThreads, 0, s, d, r.p, x, g);
}
void launch_precond(const Dev& d, const Reduce& r, int nvb, cudaStream_t s) {
  COUNT;
  follow(k_precond, nvb, kThreads, 0, s, d, r.p, r.scal + SC_LAMBDA);
}
void launch_hpwl(const Dev& d, const Reduce& r, const float2* pos, int nvb, cudaStream_t s) {
  COUNT;
  k_hpwl<<<nvb, kThreads, 0, s>>>(d, r.p, pos);
}
void launch_finalize(const Dev& d, const Reduce& r, int nvb, int mask, cudaStream_t s) {
  COUNT;
  follow(k_finalize, 1, kFinThreads, 0, s, d, r, nvb, mask);
}
void launch_finalize_joined(const Dev& d, const Reduce& r, int nvb, int mask, cudaStream_t s) {
  COUNT;
  k_finalize<<<1, kFinThreads, 0, s>>>(d, r, nvb, mask);
}
static inline int wide_blocks(size_t n) { return (int)std::min<size_t>((n + kThreads - 1) / kThreads, 2048); }
void launch_narrow(const double* src, float* dst, size_t n, long long* nonfinite, long long mark, cudaStream_t s) {
  if (!n) return;
  COUNT;
  k_narrow<<<wide_blocks(n), kThreads, 0, s>>>(src, dst, n, nonfinite, mark);
}
void launch_widen_point(const Dev& d, const float2* best, const float2* x, uint32_t* targets, double* coords,
                        cudaStream_t s) {
  if (!d.nobj) return;
  COUNT;
  k_widen_point<<<wide_blocks((size_t)d.nobj), kThreads, 0, s>>>(d, best, x, (uint2*)targets, (double2*)coords);
}
void launch_widen_eval(const Dev& d, double* wa, double* field, double* density, double* potential, cudaStream_t s) {
  COUNT;
  k_widen_eval<<<wide_blocks(std::max<size_t>((size_t)d.nobj, (size_t)d.B)), kThreads, 0, s>>>(
      d, wa, (double2*)field, density, potential);
}
void launch_round_compare(const Dev& d, const float2* x, uint32_t* prev, int W, int H, unsigned long long* mismatch,
                          int nvb, cudaStream_t s) {
  COUNT;
  k_round_compare<<<nvb, kThreads, 0, s>>>(d, x, prev, W, H, mismatch);
}

}  // namespace tgp
