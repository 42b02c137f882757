// persistent_body.cuh — the whole placement loop in one cooperative kernel.
//
// The kernel runs `optimize_density_once` (crates/texo-pnr/src/eplace.rs:439-582)
// with `dynamic_nesterov_step` (crates/texo-pnr/src/global_placement.rs:121-335)
// on the device. Phases are separated by a barrier over the instance's
// blocks; after each barrier every block reduces the partials it needs in the
// same fixed order, so all blocks hold bit-identical scalars and take the same
// branch. Thread 0 of each block keeps the controller state in shared memory;
// the instance's first block writes it back when the kernel returns.
//
// Work is split into a fixed number V of virtual blocks per instance; the
// instance's physical blocks loop over them. Partials are indexed by virtual
// block, so an instance computes bit-identical results whether it runs alone
// on every SM or shares one launch with other instances (batched serving).
//
// One iteration, with the usual origin whose density is known (X the origin,
// Y the extrapolated point, C a candidate; "|" a grid barrier; A and B run
// side by side):
//   A: preconditioner, Y, scatter(Y)            B: WA(X) |
//   A: rows(Y)                                  B: combine(X) |
//   A: columns(Y) |a rows inverse(Y)            B: WA(Y) |
//   gather(Y), combine(Y), reset of the grids |
//   A: candidate C, scatter(C) |
//   A: rows(C) |a columns(C) |a rows inverse(C) B: WA(C) |
//   gather(C), combine(C), reset of the grids |
// A point is scattered by the thread that formed it, so it needs no barrier
// of its own; a point's WA runs beside its transforms, and they only meet in
// the gradient's combination.
//
// A launch for one placement alone runs double blocks (SETS = 2): A is the
// first half of the block, B the second (|a is a barrier of the halves A
// alone). What an object's owner reads in every phase and never changes (its
// density member, its box, the tile-to-bin map) and the point being evaluated
// stay in the block's shared memory: behind each grid barrier L1 is cold, and
// a phase's time was the length of its chain of dependent L2 trips. Batched
// launches run single blocks (SETS = 1) that do A's and B's work one after
// the other and read everything from memory: there other instances' blocks
// hide the latency.
//
// Every wait is bounded: a barrier that does not complete within its spin
// budget sets an error word, and the instance's blocks then leave the kernel
// at their next barrier.
//
// run_body is instantiated by four small translation units (one kernel
// each: alone or batched, small or large DCT tiles) so that they compile in
// parallel.
#pragma once
#include <cmath>
#include <cstring>

#include "dct_fft.cuh"
#include "persistent.cuh"

namespace tgp {

constexpr unsigned kSpinLimit = 1u << 25;   // ~seconds of polling before giving up
constexpr unsigned kMaxTrialsPerStep = 8192;

struct ERec {
  double value, wa, wal1, kkt;
  double energy[kMaxFields], overflow[kMaxFields], force[kMaxFields], rawl1[kMaxFields];
  long long ovfix[kMaxFields], bins[kMaxFields];
  long long bad;
};

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// (arrivals, error) of a barrier in one acquire load: every write made
// before a releasing arrival is visible once that arrival is counted
__device__ __forceinline__ unsigned long long load_arrivals_error(const GridBarrier* b) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&b->arrived) : "memory");
  return v;
}

// Barrier over the np physical blocks of one instance, for the one thread a
// block sends to it (its block's writes are ordered before by a block
// barrier). Arrivals are counted up from zero for a whole launch: every
// block adds one with a release reduction, whose result it does not wait
// for, and polls the counter itself with acquire loads until np more
// arrivals than at the last barrier are in. A barrier is then one trip of
// the last arrival to L2 and one poll, where a counter that the last arriver
// resets before it publishes a generation takes an atomic's round trip and a
// second release between the two. The counter cannot wrap into a false
// match: the comparison is on the signed difference. (Wait per barrier as
// block 0 sees it: 152 blocks at 42k cells 2.4 us with the resetting form,
// 1.9 us with this one; 21 blocks at 2k cells 2.0 and 1.4 us.)
__device__ __forceinline__ bool grid_arrive_wait(GridBarrier* b, unsigned np, unsigned* gen, unsigned limit) {
  const unsigned target = *gen + np;
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&b->arrived) : "memory");
  unsigned spins = 0;
  unsigned long long ge;
  for (;;) {
    ge = load_arrivals_error(b);
    if ((int)((unsigned)ge - target) >= 0 || (ge >> 32) != 0ull) break;
    if (++spins > limit) {
      atomicExch(&b->error, 1);
      ge |= 1ull << 32;
      break;
    }
    if (spins > 64) __nanosleep(32);
  }
  *gen = target;
  return (ge >> 32) == 0ull;
}

// grid_arrive_wait for every thread of the block.
__device__ __forceinline__ bool grid_sync(GridBarrier* b, unsigned np, unsigned* gen, unsigned long long* count,
                                          unsigned long long* wait_acc, int* failed, unsigned limit = kSpinLimit) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long t0 = wait_acc ? now_ns() : 0ull;
    *failed = !grid_arrive_wait(b, np, gen, limit);
    ++*count;
    if (wait_acc) *wait_acc += now_ns() - t0;
  }
  __syncthreads();
  // one read of the error word per block, so all its threads agree
  return *failed == 0;
}

// One reduction of the V partials of a slot, folded by one warp in a fixed
// order (lanes stride the partials, then an xor tree over the lanes).
enum FoldOp { FOLD_DSUM, FOLD_ISUM, FOLD_IMIN, FOLD_DMAX, FOLD_DMIN };
struct FoldJob {
  const void* a;
  int op;
};
union FoldValue {
  double d;
  long long l;
};
constexpr int kMaxFoldJobs = 3 * kMaxFields + 3;   // the largest fold (energies, overflows, WA, the origin's KKT)
// The partials a warp folds, loaded ahead of the fold itself (five a lane:
// an instance has at most one virtual block a multiprocessor; more are read
// when they are folded).
constexpr int kFoldAhead = 5;
struct FoldAhead {
  unsigned long long v[kFoldAhead];
};
__device__ __forceinline__ FoldAhead fold_load(const void* a, int n) {
  FoldAhead f;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int u = 0; u < kFoldAhead; ++u) {
    const int i = lane + 32 * u;
    f.v[u] = i < n ? reinterpret_cast<const unsigned long long*>(a)[i] : 0ull;
  }
  return f;
}
template <typename T, typename Op>
__device__ __forceinline__ T fold_loaded(const FoldAhead& f, const T* a, int n, T init, Op op) {
  const int lane = threadIdx.x & 31;
  auto as = [](unsigned long long x) {
    T t;
    memcpy(&t, &x, sizeof(T));
    return t;
  };
  T v = lane < n ? as(f.v[0]) : init;
#pragma unroll
  for (int u = 1; u < kFoldAhead; ++u)
    if (lane + 32 * u < n) v = op(v, as(f.v[u]));
#pragma unroll 1
  for (int i = lane + 32 * kFoldAhead; i < n; i += 32) v = op(v, a[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <typename T, typename Op>
__device__ __forceinline__ T warp_fold(const T* a, int n, T init, Op op) {
  return fold_loaded(fold_load(a, n), a, n, init, op);
}
// One copy for all folds (the values in registers).
static __device__ __noinline__ FoldValue fold_values(unsigned long long v0, unsigned long long v1,
                                                     unsigned long long v2, unsigned long long v3,
                                                     unsigned long long v4, const void* a, int op, int n) {
  const FoldAhead f{{v0, v1, v2, v3, v4}};
  FoldValue out;
  switch (op) {
    case FOLD_DSUM: out.d = fold_loaded(f, (const double*)a, n, 0.0, OpAdd()); break;
    case FOLD_ISUM: out.l = fold_loaded(f, (const long long*)a, n, 0ll, OpAdd()); break;
    case FOLD_IMIN: out.l = fold_loaded(f, (const long long*)a, n, 0x7fffffffffffffffll, OpMin()); break;
    case FOLD_DMAX: out.d = fold_loaded(f, (const double*)a, n, 0.0, OpMax()); break;
    default: out.d = fold_loaded(f, (const double*)a, n, (double)INFINITY, OpMin()); break;
  }
  return out;
}
__device__ __forceinline__ FoldValue fold_ahead(const FoldAhead& f, const FoldJob& jb, int n) {
  static_assert(kFoldAhead == 5, "one argument a value");
  return fold_values(f.v[0], f.v[1], f.v[2], f.v[3], f.v[4], jb.a, jb.op, n);
}

// Block-level scratch of the loop's own reductions.
template <int SETS>
struct LoopShared {
  Shared a;                                   // half A's (the block's) folds
  double pair[2 * (kThreads + 4)];            // two FP64 sums at once (half A)
  double wa[SETS == 2 ? kThreads + 4 : 1];    // half B's WA value
  long long tot[kMaxFields][SETS * kThreads / 32];
  unsigned u[3][SETS * kThreads / 32];
  unsigned x[2][kThreads / 32];               // half B's combination
};

// What stays in a double block's shared memory (dynamic): the first kResident
// objects of the block, in the order (k, thread) of its threads' objects.
constexpr int kResident = 1536;     // 6 a thread: 233 k objects on 152 SMs; further ones are read from memory
constexpr int kResidentMap = 512;   // tiles a side the resident map covers
struct Resident {
  float2 pos[kResident];     // the point being evaluated
  float4 mem[kResident];     // (offset x, offset y, charge, field bits): kNoMember, kManyMembers or a field
  float4 box[kResident];     // (lo.x, lo.y, hi.x, hi.y)
  float2 mapx[kResidentMap], mapy[kResidentMap];
};
constexpr int kNoMember = -1, kManyMembers = -2;

// Shared-memory step bookkeeping that every thread reads after a barrier.
struct StepVars {
  int restart, y_is_origin, may_reduce, has_wL, action, stationary, fresh, deposited, dirty;
  double wL, tL, f_y, y_stat, next_m, pmin, pmax;
  double gamma, growth;                       // of the next iteration
  int st_multipliers, st_growth, st_gamma;
  unsigned ws;                                // phases that wrote an alternating partial set
  float extrapolation, lambda[kMaxFields], inv_L;
  unsigned trials;
  int pending_best, pending_prev;
};
// Everything a block's phases read, in its shared memory: the phases are
// functions of their own (inlined wherever they are called the loop was two
// megabytes of code, and its phases, each run once between two grid barriers,
// were bound by instruction fetches), and what they would otherwise pass on
// the stack would be an L2 trip behind every grid barrier, which leaves L1
// cold.
template <int SETS>
struct LoopState {
  InstDesc inst;
  DevRun S;            // written by thread 0
  ERec eo, ey, ec;     // the origin's, the extrapolated point's and the candidate's evaluation
  StepVars V;
  GemmShared gsm;
  LoopShared<SETS> sh;
  double coef[kMaxFields];
  float coef32[kMaxFields];
  FoldValue fv[kMaxFoldJobs];        // results of the folds after a barrier
  long long fmean[kMaxFields];       // fixed-point density means
  long long capsum[kMaxFields];      // copy of d.capsum
  unsigned long long nbar, clock[10];   // clock: [8] phase accumulators, [8] last mark, [9] barrier wait
  Resident* res;                     // null: nothing is resident
  const float2 *mapx, *mapy;         // tile-to-bin maps (resident, or d's)
  unsigned gen;
  int gen_failed;                    // the barrier's error word as thread 0 last read it
  int pb, np;                        // physical block of the instance, physical block count
  int tables;                        // the FFT tables stay in the work buffer
};
template <int SETS>
__device__ __forceinline__ LoopState<SETS>& loop_state() {
  __shared__ LoopState<SETS> state;
  return state;
}

template <bool LARGE, int SETS>
struct Ctx;
// The phases out of line, one copy each.
#define OUTLINED(type, name) template <bool LARGE, int SETS> static __device__ __noinline__ type name
template <int NB, int SETS> static __device__ __noinline__ void run_rows_fwd();
template <int NB, int SETS> static __device__ __noinline__ void run_cols();
template <int NB, int SETS> static __device__ __noinline__ void run_rows_inv();
OUTLINED(bool, run_sync)();
OUTLINED(void, run_wa)(const float2* pos, double gam);
OUTLINED(void, run_scatter)(const float2* pos);
OUTLINED(void, run_combine_kept)(const float2* pos, float2* g);
OUTLINED(bool, run_transform_first)();
OUTLINED(bool, run_transform_rest)();
OUTLINED(bool, run_density_and_wa)(const float2* pos, double gam, const float2* origin, float2* origin_g);
OUTLINED(bool, run_gradient)(const float2* pos, float2* g, ERec* out, ERec* origin);
OUTLINED(bool, run_eval_initial)(const float2* pos, float2* g, double gam, bool full);
OUTLINED(void, run_precondition)(bool deposits);
OUTLINED(void, run_candidate)(const float2* y, const float2* gy, float2* c);

template <bool LARGE, int SETS>
struct Ctx {
  static constexpr int kBlock = SETS * kThreads;
  static constexpr int kWarps = kBlock / 32;
  using GA = Group<SETS == 2 ? 1 : 0>;
  using GB = Group<SETS == 2 ? 2 : 0>;
  LoopState<SETS>& L;
  const Dev& d;
  const Reduce& r;
  const Buffers& B;
  DevRun& S;
  GemmShared& gsm;
  LoopShared<SETS>& sh;
  FoldValue* fv;
  Resident* res;
  const float2 *mapx, *mapy;
  int pb, np;
  int V;              // virtual blocks of the instance

  __device__ __forceinline__ explicit Ctx(LoopState<SETS>& l)
      : L(l), d(l.inst.d), r(l.inst.r), B(l.inst.B), S(l.S), gsm(l.gsm), sh(l.sh), fv(l.fv), res(l.res), mapx(l.mapx),
        mapy(l.mapy), pb(l.pb), np(l.np), V(l.inst.V) {}

  __device__ bool in_a() const { return SETS == 1 || threadIdx.x < kThreads; }
  __device__ bool in_b() const { return SETS == 1 || threadIdx.x >= kThreads; }
  __device__ GA half_a() const { return GA{(int)threadIdx.x & (kThreads - 1)}; }
  __device__ GB half_b() const { return GB{(int)threadIdx.x & (kThreads - 1)}; }

  __device__ void meet() {   // thread 0's part of a grid barrier
    const unsigned long long t0 = pb == 0 ? now_ns() : 0ull;
    L.gen_failed = !grid_arrive_wait(L.inst.bar, (unsigned)np, &L.gen, kSpinLimit);
    ++L.nbar;
    if (pb == 0) L.clock[9] += now_ns() - t0;
  }
  // Grid barrier, every thread of the block.
  __device__ __forceinline__ bool sync() { return run_sync<LARGE, SETS>(); }
  __device__ __forceinline__ bool sync_body() {
    __syncthreads();
    if (threadIdx.x == 0) meet();
    __syncthreads();
    return L.gen_failed == 0;   // one read of the error word per block, so all its threads agree
  }
  // Grid barrier of half A alone, while half B works on. It orders what the
  // whole block wrote before its last block barrier, and half A since. After
  // a failure half A goes on to the next whole-block barrier, which fails at
  // once, so half B never waits for it.
  __device__ bool sync_a(const GA& g) {
    g.sync();
    if (threadIdx.x == 0) meet();
    g.sync();
    return L.gen_failed == 0;
  }
  // Partials of phases that may follow one another directly (extrapolation,
  // candidates, stationary check) alternate between two sets (V.ws counts
  // them): a block that leaves a barrier early and writes the next phase's
  // partials must not overwrite the ones a slower block of the instance is
  // still reducing. Every other slot is written again only after a barrier
  // that its readers have reached.
  __device__ Partials set() const { return (L.V.ws & 1u) ? r.q : r.p; }

  // Charges the time since the previous mark to phase category `cat` (block 0).
  __device__ void mark(int cat) {
    if (pb == 0 && threadIdx.x == 0) {
      const unsigned long long t = now_ns();
      L.clock[cat] += t - L.clock[8];
      L.clock[8] = t;
    }
  }
  // Several reductions of partials at once, right after a grid barrier: job j
  // is folded by warp j (mod the warp count), so the loads of all jobs are in
  // flight together (one L2 round trip for partials that other SMs wrote,
  // often on the other die) and the FP64 folds of different jobs run on
  // different SM sub-partitions. Every thread reads the results in fv after
  // the final block barrier.
  template <class Job>
  __device__ __forceinline__ void fold(int n, Job job) {
#pragma unroll 1
    for (int j = threadIdx.x >> 5; j < n; j += kWarps) {
      const FoldJob jb = job(j);
      const FoldValue out = fold_ahead(fold_load(jb.a, V), jb, V);
      if ((threadIdx.x & 31) == 0) fv[j] = out;
    }
    __syncthreads();
  }
  __device__ float2* X() const { return B.pos[S.ix]; }
  __device__ float2* Xp() const { return B.pos[S.ixp]; }
  __device__ float2* Y() const { return B.pos[S.iy]; }
  __device__ float2* C() const { return B.pos[S.ic]; }
  __device__ float2* gX() const { return B.grad[S.igx]; }
  __device__ float2* gY() const { return B.grad[S.igy]; }
  __device__ float2* gC() const { return B.grad[S.igc]; }

  __device__ void copy(float2* dst, const float2* src, int n) {
    for (int i = pb * kBlock + threadIdx.x; i < n; i += np * kBlock) dst[i] = src[i];
  }

  // ---- objects ----------------------------------------------------------------
  // Virtual block v owns the objects v * kThreads + t + k * V * kThreads of its
  // threads t; `j` = k * kThreads + t numbers them inside the block.
  __device__ __forceinline__ int object(int v, int j) const {
    return v * kThreads + (j & (kThreads - 1)) + (j / kThreads) * V * kThreads;
  }
  __device__ __forceinline__ bool resident(int j) const { return SETS == 2 && res && j < kResident; }
  // an object's one density member, or kNoMember / kManyMembers
  __device__ __forceinline__ float4 member(int j, int o) const {
    return resident(j) ? res->mem[j] : member_from_memory(o);
  }
  __device__ __forceinline__ float4 member_from_memory(int o) const {
    // a filler deposits at its position itself (a zero offset changes no bit
    // of the taps: an offset of +0 leaves every coordinate but -0 as it is,
    // and the axis clamps -0 like +0)
    if (o >= d.U) return make_float4(0.f, 0.f, d.fil_q[o - d.U], __int_as_float(d.fil_field[o - d.U]));
    const int m = d.unit_mem_ptr[o], n = d.unit_mem_ptr[o + 1] - m;
    if (n != 1) return make_float4(0.f, 0.f, 0.f, __int_as_float(n == 0 ? kNoMember : kManyMembers));
    return member_at(m);
  }
  __device__ __forceinline__ float4 member_at(int m) const {
    const float2 off = d.mem_off[m];
    return make_float4(off.x, off.y, d.mem_q[m], __int_as_float(d.mem_field[m]));
  }
  __device__ __forceinline__ float4 box(int j, int o) const {
    if (resident(j)) return res->box[j];
    const float2 lo = d.lo[o], hi = d.hi[o];
    return make_float4(lo.x, lo.y, hi.x, hi.y);
  }
  __device__ void make_resident() {
    if constexpr (SETS == 2) {
      if (!res) return;
      for (int j = threadIdx.x; j < kResident; j += kBlock) {
        const int o = object(pb, j);
        if (o >= d.nobj) break;
        const float2 lo = d.lo[o], hi = d.hi[o];
        res->mem[j] = member_from_memory(o);
        res->box[j] = make_float4(lo.x, lo.y, hi.x, hi.y);
      }
      if (mapx != d.binmap_x) {
        for (int i = threadIdx.x; i < d.g.W; i += kBlock) res->mapx[i] = d.binmap_x[i];
        for (int i = threadIdx.x; i < d.g.H; i += kBlock) res->mapy[i] = d.binmap_y[i];
      }
    }
  }
  __device__ __forceinline__ AxisTaps tx(float s) const {
    return axis_taps(d.g.Wb, s, mapx, d.g.sx, d.g.identity, d.g.W);
  }
  __device__ __forceinline__ AxisTaps ty(float s) const {
    return axis_taps(d.g.Hb, s, mapy, d.g.sy, d.g.identity, d.g.H);
  }

  // ---- the phases' work on one virtual block ------------------------------

  // Resets of the accumulators, dealt to all threads of the block.
  __device__ void reset_grids(int v, int from = 0) {
    const int n = d.K * d.B, stride = V * kBlock;
#pragma unroll 1
    for (int i = from + v * kBlock + (int)threadIdx.x; i < n; i += stride) {
      d.phys[i] = -d.capfix[i];
      d.fill[i] = 0;
    }
  }
  __device__ void reset_wa(int v) {
#pragma unroll 1
    for (int i = v * kBlock + (int)threadIdx.x; i < 2 * d.U; i += V * kBlock) d.wa_fix[i] = 0ull;
  }

  // Scatters object o at p, into the totals per field.
  __device__ __forceinline__ void deposit(float4 m, int o, float2 p, long long (&tot)[kMaxFields]) {
    int f = __float_as_int(m.w);
    if (f == kNoMember) return;
    int i = 0, left = 1;
    if (f == kManyMembers) {
      i = d.unit_mem_ptr[o];
      left = d.unit_mem_ptr[o + 1] - i;
      m = member_at(i);
      f = __float_as_int(m.w);
    }
    long long* const grids = o < d.U ? d.phys : d.fill;
#pragma unroll 1
    for (;;) {
      const long long s = deposit_taps<kSharedBinLoop>(d, (unsigned long long*)(grids + (size_t)f * d.B), m.z, tx(__fadd_rn(p.x, m.x)),
                                       ty(__fadd_rn(p.y, m.y)));
#pragma unroll
      for (int ff = 0; ff < kMaxFields; ++ff)
        if (ff == f) tot[ff] += s;
      if (--left == 0) break;
      m = member_at(++i);
      f = __float_as_int(m.w);
    }
  }
  // the warps' totals, then (after a barrier, half A) partial v of half A's or
  // all warps' totals
  __device__ __forceinline__ void stage_totals(const long long (&tot)[kMaxFields]) {
#pragma unroll
    for (int f = 0; f < kMaxFields; ++f)
      if (f < d.K) {
        const long long t = warp_sum(tot[f]);
        if ((threadIdx.x & 31) == 0) sh.tot[f][threadIdx.x >> 5] = t;
      }
  }
  template <int WARPS = kThreads / 32>
  __device__ __forceinline__ void write_totals(const GA& g, int v) {
    const int f = g.tid - 128;
    if (f >= 0 && f < d.K) {
      long long t = 0;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) t += sh.tot[f][w];
      islot(r.p, IS_GRID_SUM + f)[v] = t;
    }
  }
  // Half A: the scatter of a point that is in memory.
  __device__ void scatter(const float2* pos, int v) {
    const GA g = half_a();
    long long tot[kMaxFields] = {0, 0, 0, 0};
    for (int j = g.tid, o; (o = object(v, j)) < d.nobj; j += kThreads) {
      const float2 p = pos[o];
      if (resident(j)) res->pos[j] = p;
      deposit(member(j, o), o, p, tot);
    }
    g.sync();   // earlier readers of the scratch are done
    stage_totals(tot);
    g.sync();
    write_totals(g, v);
  }

  // WA by half B (the whole single block).
  __device__ void wa(const float2* pos, double gam) {
    const GB g = half_b();
    for (int v = pb; v < V; v += np) {
      if constexpr (SETS == 2)
        stage_wa(g, d, pos, gam, r.p, v, V, sh.wa);
      else
        stage_wa(g, d, pos, gam, r.p, v, V, sh.a.d);
    }
  }

  // Raw field gradients of an object and what its combination reads besides,
  // all loaded together. (The L1 norms and the density force, which only the
  // two evaluations before the first iteration use, come from stage_gather /
  // stage_combine there.)
  struct Raw {
    float2 f[kMaxFields];
    float2 at;
    ulonglong2 wa;
    float P;
  };
  __device__ __forceinline__ void operands(Raw& a, int o) {
    a.P = d.P[o];
    a.wa = o < d.U ? reinterpret_cast<const ulonglong2*>(d.wa_fix)[o] : make_ulonglong2(0ull, 0ull);
  }
  // gathered at pos (sample_quadratic_bspline_with_gradient and the member and
  // filler loops, electrostatic_placement.rs:338-374, 919-941), and kept
  __device__ __forceinline__ void gathered(Raw& a, const float2* pos, int j, int o) {
#pragma unroll
    for (int f = 0; f < kMaxFields; ++f) a.f[f] = make_float2(0.f, 0.f);
    if (o >= d.nobj) return;
    operands(a, o);
    a.at = resident(j) ? res->pos[j] : pos[o];
    float4 m = member(j, o);
    int f = __float_as_int(m.w), i = 0, left = 1;
    if (f == kManyMembers) {
      i = d.unit_mem_ptr[o];
      left = d.unit_mem_ptr[o + 1] - i;
      m = member_at(i);
      f = __float_as_int(m.w);
    }
    if (f != kNoMember) {
#pragma unroll 1
      for (;;) {
        const float2 s = sample_grad(d, d.phi + (size_t)f * d.B, tx(__fadd_rn(a.at.x, m.x)), ty(__fadd_rn(a.at.y, m.y)));
#pragma unroll
        for (int ff = 0; ff < kMaxFields; ++ff)
          if (ff == f) {
            a.f[ff].x += m.z * s.x;
            a.f[ff].y += m.z * s.y;
          }
        if (--left == 0) break;
        m = member_at(++i);
        f = __float_as_int(m.w);
      }
    }
#pragma unroll
    for (int ff = 0; ff < kMaxFields; ++ff)
      if (ff < d.K && (o < d.U || ff == f)) d.graw[(size_t)ff * d.nobj + o] = a.f[ff];
  }
  // the ones kept from the last density evaluation
  __device__ __forceinline__ void kept(Raw& a, const float2* pos, int o) {
    operands(a, o);
    a.at = pos[o];
    const int only = o < d.U || d.K == 1 ? -1 : d.fil_field[o - d.U];
#pragma unroll
    for (int f = 0; f < kMaxFields; ++f)
      a.f[f] = f < d.K && (only < 0 || only == f) ? d.graw[(size_t)f * d.nobj + o] : make_float2(0.f, 0.f);
  }
  // The combined gradient of an object (combined_objective, eplace.rs:1022-
  // 1044); the WA accumulators it has read are cleared for the next evaluation.
  // The KKT residual and the first non-finite index need no order.
  __device__ __forceinline__ void combine(const Raw& a, int j, int o, float2* g, float& kkt, unsigned& bad) {
    if (o >= d.nobj) return;
    const float4 bx = box(j, o);
    float gx = 0.f, gy = 0.f;
    if (o < d.U) {
      reinterpret_cast<ulonglong2*>(d.wa_fix)[o] = make_ulonglong2(0ull, 0ull);
      gx = __ll2float_rn((long long)a.wa.x) * kInvFixF;
      gy = __ll2float_rn((long long)a.wa.y) * kInvFixF;
    }
    // a filler has one field: the others' gradients are zero and add nothing
#pragma unroll
    for (int f = 0; f < kMaxFields; ++f)
      if (f < d.K) {
        const float c = L.coef32[f];
        gx = fmaf(c, a.f[f].x, gx);
        gy = fmaf(c, a.f[f].y, gy);
      }
    if (!isfinite(gx)) bad = min(bad, 2u * (unsigned)o);
    else if (!isfinite(gy)) bad = min(bad, 2u * (unsigned)o + 1u);
    g[o] = make_float2(gx, gy);
    const float s = rsqrtf(a.P);
    kkt = fmaxf(kkt, kkt_comp(gx, a.at.x, bx.x, bx.z) * s);
    kkt = fmaxf(kkt, kkt_comp(gy, a.at.y, bx.y, bx.w) * s);
  }
  // Warp results of a KKT maximum and a least bad index: the residuals are not
  // negative, so their bits order as integers.
  __device__ __forceinline__ void stage_kkt_warp(float kkt, unsigned bad, unsigned* ks, unsigned* bs, int w) {
    const unsigned k = __reduce_max_sync(0xffffffffu, __float_as_uint(kkt));
    const unsigned b = __reduce_min_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
      ks[w] = k;
      bs[w] = b;
    }
  }
  __device__ __forceinline__ void write_kkt(const Partials& p, const unsigned* ks, const unsigned* bs, int n, int v) {
    unsigned k = 0u, b = 0xffffffffu;
    for (int w = 0; w < n; ++w) {
      k = max(k, ks[w]);
      b = min(b, bs[w]);
    }
    mslot(p, MS_KKT)[v] = (double)__uint_as_float(k);
    islot(p, IS_BAD)[v] = b == 0xffffffffu ? 0x7fffffffffffffffll : (long long)b;
  }
  // Half B: the origin's combined gradient from the kept field gradients; its
  // partials go to the second set (the first holds the evaluated points').
  __device__ void combine_kept(const float2* pos, float2* g, int v) {
    const GB gb = half_b();
    float kkt = 0.f;
    unsigned bad = 0xffffffffu;
    Raw a, b;
    int j = gb.tid, o = object(v, j);
    if (o < d.nobj) kept(a, pos, o);
#pragma unroll 1
    while (o < d.nobj) {   // the next object's loads in flight
      const int o2 = object(v, j + kThreads);
      if (o2 < d.nobj) kept(b, pos, o2);
      combine(a, j, o, g, kkt, bad);
      a = b;
      o = o2;
      j += kThreads;
    }
    gb.sync();   // earlier readers of the scratch are done
    stage_kkt_warp(kkt, bad, sh.x[0], sh.x[1], gb.tid >> 5);
    gb.sync();
    if (gb.tid == 0) write_kkt(r.q, sh.x[0], sh.x[1], kThreads / 32, v);
  }
  __device__ FoldJob kkt_job(const Partials& p, int j) const {
    return j == 0 ? FoldJob{mslot(p, MS_KKT), FOLD_DMAX} : FoldJob{islot(p, IS_BAD), FOLD_IMIN};
  }

  // fixed-point density mean (DC mode) of field f, from its folded grid sum;
  // truncated division, a shift for the power-of-two grids
  __device__ void set_mean(int f, long long sum) {
    const long long t = sum - L.capsum[f];
    const int B_ = d.B;
    L.fmean[f] = (B_ & (B_ - 1)) == 0 ? (t + (long long)((unsigned long long)(t >> 63) & (unsigned long long)(B_ - 1))) >> (31 - __clz(B_))
                                    : t / B_;
  }
  __device__ FoldJob sum_job(int f) const { return FoldJob{islot(r.p, IS_GRID_SUM + f), FOLD_ISUM}; }

  // Half A's side of a density evaluation once the grids are complete, in two
  // parts around the first barrier: the density preparation with the first
  // transform, and the rest to phi and the overflow and energy partials.
  // The first pass of the transforms, and the others (the FFT form's straight
  // away: a call within a call keeps registers in memory twice).
  __device__ __forceinline__ bool first() {
    if (!d.fft) return run_transform_first<LARGE, SETS>();
    d.logW == 10 ? run_rows_fwd<2, SETS>() : run_rows_fwd<1, SETS>();
    return true;
  }
  __device__ __forceinline__ bool rest() {
    if (!d.fft) return run_transform_rest<LARGE, SETS>();
    d.logH == 10 ? run_cols<2, SETS>() : run_cols<1, SETS>();
    if (!sync_a(half_a())) return false;
    d.logW == 10 ? run_rows_inv<2, SETS>() : run_rows_inv<1, SETS>();
    return true;
  }
  __device__ bool transform_first() {
    const GA g = half_a();
    if (LARGE) {
      for (int v = pb; v < V; v += np) stage_prep(g, d, r.p, V, v, V, sh.a);
      if (!sync_a(g)) return false;
      mark(PC_PREP);
      for (int v = pb; v < V; v += np) stage_dct_t<LARGE>(g, d, 0, r.p, v, V, gsm, sh.a);
    } else {
      for (int v = pb; v < V; v += np) stage_prep_dct0(g, d, L.fmean, r.p, v, V, gsm, sh.a);
    }
    return true;
  }
  __device__ bool transform_rest() {
    const GA g = half_a();
    for (int st = 1; st < 4; ++st) {
      for (int v = pb; v < V; v += np) stage_dct_t<LARGE>(g, d, st, r.p, v, V, gsm, sh.a);
      if (st < 3 && !sync_a(g)) return false;
    }
    return true;
  }

  // Energies, overflow and WA value of the last evaluation (density side
  // rebuilt), or the WA value alone, from the folded jobs.
  __device__ FoldJob eval_job(int j, bool full) const {
    if (!full || j == 3 * d.K) return FoldJob{pslot(r.p, SLOT_WA_VALUE), FOLD_DSUM};
    const int f = j / 3, k = j % 3;
    return k == 0   ? FoldJob{pslot(r.p, SLOT_ENERGY + f), FOLD_DSUM}
           : k == 1 ? FoldJob{islot(r.p, IS_OVERFLOW + f), FOLD_ISUM}
                    : FoldJob{islot(r.p, IS_OVER_BINS + f), FOLD_ISUM};
  }
  __device__ int eval_jobs(bool full) const { return full ? 3 * d.K + 1 : 1; }
  // one thread: the fields' coefficients from the jobs at fv[at...]
  __device__ void eval_coefficients(bool full, int at = 0) {
#pragma unroll 1
    for (int f = 0; f < d.K; ++f) {
      const double ne = (full ? 0.5 * fv[at + 3 * f].d : S.cur_energy[f]) * S.inv_e0[f];
      L.coef[f] = S.lambda[f] * (1.0 + S.beta * ne);
      L.coef32[f] = (float)L.coef[f];
    }
  }
  // one thread: the objective
  __device__ void eval_value(ERec& out, bool full, int at = 0) {
    const double wa = fv[at + (full ? 3 * d.K : 0)].d;
    out.wa = wa;
    double value = wa;
#pragma unroll 1
    for (int f = 0; f < d.K; ++f) {
      if (full) {
        const long long ov = fv[at + 3 * f + 1].l;
        out.energy[f] = 0.5 * fv[at + 3 * f].d;
        out.ovfix[f] = ov;
        out.bins[f] = fv[at + 3 * f + 2].l;
        out.overflow[f] = ((double)ov * kInvFix) * S.inv_real_area[f];
      } else {
        out.energy[f] = S.cur_energy[f];
        out.overflow[f] = S.cur_overflow[f];
        out.ovfix[f] = S.cur_overflow_fixed[f];
        out.bins[f] = 0;
      }
      const double ne = out.energy[f] * S.inv_e0[f];
      value += S.lambda[f] * S.e0[f] * (ne + 0.5 * S.beta * ne * ne);
    }
    out.value = value;
  }

  // Objective evaluation with the sums only the initial probes use, after a
  // barrier that left the accumulators reset (ContinuousProblem::evaluate +
  // combined_objective, eplace.rs:137-205, 1022-1044).
  __device__ bool eval_initial(const float2* pos, float2* g, double gam, bool full, ERec& out) {
    if (full) {
      if (in_a()) run_scatter<LARGE, SETS>(pos);
      if (!sync()) return false;
      fold(d.K, [&](int j) { return sum_job(j); });
      if ((int)threadIdx.x < d.K) set_mean(threadIdx.x, fv[threadIdx.x].l);
      __syncthreads();
      if (in_a()) {
        if (first() && sync_a(half_a())) rest();
      }
      __syncthreads();
    }
    if (in_b()) run_wa<LARGE, SETS>(pos, gam);
    if (!sync()) return false;
    mark(full ? PC_DCT : PC_SCATTER_WA);
    fold(eval_jobs(full), [&](int j) { return eval_job(j, full); });
    if (threadIdx.x == 0) {
      eval_coefficients(full);
      eval_value(out, full);
    }
    __syncthreads();
    if (in_a()) {
      const GA ga = half_a();
      for (int v = pb; v < V; v += np) {
        if (full) stage_gather(ga, d, pos, r.p, v, V, sh.a);
        stage_combine(ga, d, L.coef, g, r.p, v, V, sh.a, sh.pair, 2);
      }
    }
    if (!sync()) return false;
    mark(PC_GATHER);
    fold(2 * d.K + 2, [&](int j) {
      return j < d.K       ? FoldJob{pslot(r.p, SLOT_RAWL1 + j), FOLD_DSUM}
             : j < 2 * d.K ? FoldJob{pslot(r.p, SLOT_FORCE + j - d.K), FOLD_DSUM}
             : j == 2 * d.K ? FoldJob{pslot(r.p, SLOT_WAL1), FOLD_DSUM}
                            : FoldJob{islot(r.p, IS_BAD), FOLD_IMIN};
    });
    if (threadIdx.x == 0) {
      for (int f = 0; f < d.K; ++f) {
        out.rawl1[f] = fv[f].d;
        out.force[f] = fv[d.K + f].d;
      }
      out.wal1 = fv[2 * d.K].d;
      out.bad = fv[2 * d.K + 1].l;
      out.kkt = 0.0;
      S.evaluations++;
      if (full) S.density_evaluations++;
    }
    __syncthreads();
    return true;
  }

  // The loop's evaluation at pos, scattered and the means known. With
  // origin_g, half B first combines the origin's gradient, and WA(pos) starts
  // once every block has read the origin's WA accumulators.
  __device__ bool density_and_wa(const float2* pos, double gam, const float2* origin, float2* origin_g) {
    bool ready = true;
    if (SETS == 1 && !origin_g) run_wa<LARGE, SETS>(pos, gam);
    if (in_a()) ready = first();
    if (origin_g) {
      if (in_b()) run_combine_kept<LARGE, SETS>(origin, origin_g);
      ready = sync();
      if (SETS == 1 && ready) run_wa<LARGE, SETS>(pos, gam);
    }
    if (in_a()) {
      if (!origin_g && ready) ready = sync_a(half_a());
      if (ready) rest();
    } else {
      if (ready) run_wa<LARGE, SETS>(pos, gam);
    }
    const bool k = sync();
    mark(PC_DCT);
    return k;
  }
  // The rest of it: the scalars, the gathered field gradients and the
  // combined gradient with its KKT residual, and the grids reset for the next
  // scatter. A double block gathers while the partials are on their way and
  // folded, and needs the coefficients only to combine; the objective's value
  // is formed by a warp of its own meanwhile. With `origin` the origin's
  // deferred KKT residual and index check are folded too.
  __device__ bool gradient(const float2* pos, float2* g, ERec& out, ERec* origin) {
    const int ne = eval_jobs(true), n = ne + (origin ? 2 : 0);
    auto job = [&](int j) { return j < ne ? eval_job(j, true) : kkt_job(r.q, j - ne); };
    auto scalars = [&]() {
      eval_value(out, true);
      if (origin) {
        origin->kkt = fv[ne].d;
        origin->bad = fv[ne + 1].l;
      }
    };
    float kkt = 0.f;
    unsigned bad = 0xffffffffu;
    int v = pb;
    if constexpr (SETS == 2) {
      const int w = threadIdx.x >> 5;
      FoldJob jb{nullptr, FOLD_DSUM};
      FoldAhead fa;
      if (w < n) {
        jb = job(w);
        fa = fold_load(jb.a, V);
      }
      int j = threadIdx.x, o = object(v, j);
      const int bin = v * kBlock + j;   // the first bin this thread resets
      const long long cap = bin < d.K * d.B ? d.capfix[bin] : 0;
      Raw a;
      gathered(a, pos, j, o);
      if (w < n) {
        const FoldValue q = fold_ahead(fa, jb, V);
        if ((threadIdx.x & 31) == 0) fv[w] = q;
      }
      __syncthreads();
      if (threadIdx.x == 0) eval_coefficients(true);
      __syncthreads();
      if (threadIdx.x == kBlock - 32) scalars();
#pragma unroll 1
      while (o < d.nobj) {
        combine(a, j, o, g, kkt, bad);
        j += kBlock;
        o = object(v, j);
        gathered(a, pos, j, o);
      }
      if (bin < d.K * d.B) {
        d.phys[bin] = -cap;
        d.fill[bin] = 0;
      }
      reset_grids(v, V * kBlock);
      stage_kkt_warp(kkt, bad, sh.u[0], sh.u[1], w);
      __syncthreads();
      if (threadIdx.x == 0) write_kkt(r.p, sh.u[0], sh.u[1], kWarps, v);
      v += np;
    } else {
      fold(n, job);
      if (threadIdx.x == 0) {
        eval_coefficients(true);
        scalars();
      }
      __syncthreads();
    }
    for (; v < V; v += np) {
      kkt = 0.f;
      bad = 0xffffffffu;
      Raw a;
#pragma unroll 1
      for (int j = threadIdx.x, o; (o = object(v, j)) < d.nobj; j += kBlock) {
        gathered(a, pos, j, o);
        combine(a, j, o, g, kkt, bad);
      }
      reset_grids(v);
      __syncthreads();   // earlier readers of the scratch are done
      stage_kkt_warp(kkt, bad, sh.u[0], sh.u[1], threadIdx.x >> 5);
      __syncthreads();
      if (threadIdx.x == 0) write_kkt(r.p, sh.u[0], sh.u[1], kWarps, v);
    }
    if (!sync()) return false;
    mark(PC_GATHER);
    fold(2, [&](int j) { return kkt_job(r.p, j); });
    if (threadIdx.x == 0) {
      out.kkt = fv[0].d;
      out.bad = fv[1].l;
      S.evaluations++;
      S.density_evaluations++;
    }
    __syncthreads();
    return true;
  }

  // Half A, before an iteration's evaluations: the preconditioner
  // (diagonal_preconditioner, eplace.rs:1046-1100) and y = clamp(x + e (x -
  // xp)) with the count of coordinates that moved; y is scattered with
  // `deposits`. The next object's loads are in flight.
  __device__ void precondition(const float* lam, const float2* x, const float2* xp, float e, float2* y, bool deposits,
                               int v) {
    const GA g = half_a();
    float lambda[kMaxFields];
#pragma unroll
    for (int f = 0; f < kMaxFields; ++f) lambda[f] = f < d.K ? lam[f] : 0.f;
    float pmin = INFINITY, pmax = 0.f;
    unsigned diff = 0;
    bool badp = false;
    long long tot[kMaxFields] = {0, 0, 0, 0};
    struct In {
      float2 a, b;
      float4 bx, mem;
      float m, q[kMaxFields];
    };
    auto load = [&](int j, int o) {
      In i;
      i.a = x[o];
      i.b = xp[o];
      i.m = d.pre_static[o];
#pragma unroll
      for (int f = 0; f < kMaxFields; ++f) i.q[f] = f < d.K ? d.pre_q[(size_t)f * d.nobj + o] : 0.f;
      i.bx = box(j, o);
      i.mem = member(j, o);
      return i;
    };
    auto step = [&](const In& i, int j, int o) {
      float2 t;
      t.x = fclamp(i.a.x + e * (i.a.x - i.b.x), i.bx.x, i.bx.z);
      t.y = fclamp(i.a.y + e * (i.a.y - i.b.y), i.bx.y, i.bx.w);
      diff += (t.x != i.a.x) + (t.y != i.a.y);
      y[o] = t;
      if (resident(j)) res->pos[j] = t;
      float m = i.m;
#pragma unroll
      for (int f = 0; f < kMaxFields; ++f)
        if (i.q[f] != 0.f) m = fmaf(lambda[f], i.q[f], m);
      if (!isfinite(m) || m < 0.f) badp = true;
      m = fmaxf(m, 1.f);
      d.P[o] = m;
      pmin = fminf(pmin, m);
      pmax = fmaxf(pmax, m);
      return t;
    };
    int j = g.tid, o = object(v, j);
    In cur, next;
    if (o < d.nobj) cur = load(j, o);
#pragma unroll 1
    while (o < d.nobj) {
      const int o2 = object(v, j + kThreads);
      if (o2 < d.nobj) next = load(j + kThreads, o2);
      const float2 t = step(cur, j, o);
      if (deposits) deposit(cur.mem, o, t, tot);
      cur = next;
      j += kThreads;
      o = o2;
    }
    // not negative, so the bits order as integers
    const unsigned lo = __reduce_min_sync(0xffffffffu, __float_as_uint(pmin));
    const unsigned hi = __reduce_max_sync(0xffffffffu, __float_as_uint(pmax));
    const unsigned c = __reduce_add_sync(0xffffffffu, diff) | (__any_sync(0xffffffffu, badp) ? 0x80000000u : 0u);
    g.sync();   // earlier readers of the scratch are done
    stage_totals(tot);
    if ((g.tid & 31) == 0) {
      sh.u[0][g.tid >> 5] = lo;
      sh.u[1][g.tid >> 5] = hi;
      sh.u[2][g.tid >> 5] = c;
    }
    g.sync();
    if (g.tid == 0) {
      unsigned a = 0x7f800000u, b = 0u, bad = 0u;
      long long n = 0;
  #pragma unroll 1
      for (int w = 0; w < kThreads / 32; ++w) {
        a = min(a, sh.u[0][w]);
        b = max(b, sh.u[1][w]);
        bad |= sh.u[2][w] >> 31;
        n += sh.u[2][w] & 0x7fffffffu;
      }
      mslot(r.p, MS_PMIN)[v] = (double)__uint_as_float(a);
      mslot(r.p, MS_PMAX)[v] = (double)__uint_as_float(b);
      islot(r.p, IS_PBAD)[v] = bad;
      islot(set(), IS_DIFF)[v] = n;
    }
    if (deposits) write_totals(g, v);
  }

  // The block: c = clamp(y - g / (L P)) and its scatter; changed count,
  // <g, c - y>, sum P (c - y)^2. Half A forms the points (each thread's objects
  // and the order of its sums are those of the 256-thread stage, the sums are
  // FP32), the next object's loads in flight. Then both halves scatter them,
  // which is most of the phase and integer arithmetic, so of any order: by half
  // A alone, each object as it was formed, the phase and its barrier took 13.9
  // us at 42,000 cells, this takes 12.9 (2,000 cells: 9.3, 8.9).
  __device__ void candidate(const float2* y, const float2* gy, float invL, float2* c, int v) {
    const GA g = half_a();
    const bool a_half = in_a();
    unsigned diff = 0;
    float dot = 0.f, msn = 0.f;
    long long tot[kMaxFields] = {0, 0, 0, 0};
    struct In {
      float2 a, gr;
      float4 bx, mem;
      float m;
    };
    auto load = [&](int j, int o) { return In{y[o], gy[o], box(j, o), member(j, o), d.P[o]}; };
    auto step = [&](const In& i, int j, int o) {
      const float s = invL / i.m;
      float2 t;
      t.x = fclamp(i.a.x - i.gr.x * s, i.bx.x, i.bx.z);
      t.y = fclamp(i.a.y - i.gr.y * s, i.bx.y, i.bx.w);
      diff += (t.x != i.a.x) + (t.y != i.a.y);
      const float dx = t.x - i.a.x, dy = t.y - i.a.y;
      dot = fmaf(i.gr.x, dx, fmaf(i.gr.y, dy, dot));
      msn = fmaf(i.m * dx, dx, fmaf(i.m * dy, dy, msn));
      c[o] = t;
      if (resident(j)) res->pos[j] = t;
      return t;
    };
    int j = g.tid, o = a_half ? object(v, j) : d.nobj;
    In cur, next;
    if (o < d.nobj) cur = load(j, o);
#pragma unroll 1
    while (o < d.nobj) {
      const int o2 = object(v, j + kThreads);
      if (o2 < d.nobj) next = load(j + kThreads, o2);
      const float2 t = step(cur, j, o);
      if constexpr (SETS == 1) deposit(cur.mem, o, t, tot);
      cur = next;
      j += kThreads;
      o = o2;
    }
    __syncthreads();   // the points are there, and earlier readers of the scratch are done
    double *b0 = sh.pair, *b1 = sh.pair + kThreads + 4;
    if (a_half) {
      b0[g.tid] = (double)dot;
      b1[g.tid] = (double)msn;
      const unsigned n = __reduce_add_sync(0xffffffffu, diff);
      if ((g.tid & 31) == 0) sh.u[0][g.tid >> 5] = n;
    }
    if constexpr (SETS == 2) {
#pragma unroll 1
      for (j = threadIdx.x; (o = object(v, j)) < d.nobj; j += kBlock)
        deposit(member(j, o), o, resident(j) ? res->pos[j] : c[o], tot);
    }
    stage_totals(tot);
    __syncthreads();
    if (!a_half) return;
    // both FP64 sums at once, each in block_fold_fp64's order
    if (g.tid == 64) {
      long long t = 0;
      for (int w = 0; w < kThreads / 32; ++w) t += sh.u[0][w];
      islot(set(), IS_DIFF)[v] = t;
    }
    write_totals<kWarps>(g, v);
    {
      const int w = g.tid >> 5, at = (w & 3) * 32 + (g.tid & 31);
      double* b = w < 4 ? b0 : b1;
      double t = b[at] + b[at + 128];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t = t + __shfl_xor_sync(0xffffffffu, t, o);
      if ((g.tid & 31) == 0) b[kThreads + (w & 3)] = t;
    }
    g.sync();
    if (g.tid == 0 || g.tid == 32) {
      const double* b = (g.tid == 0 ? b0 : b1) + kThreads;
      pslot(set(), g.tid == 0 ? SLOT_DOT : SLOT_MSN)[v] = ((b[0] + b[1]) + b[2]) + b[3];
    }
  }
};

// The one copy of the transform in the loop, for both directions and all
// passes. The loop is bound by fetching its instructions: a pass meets them
// cold in the multiprocessor's instruction cache, of whose requests a third
// missed, and a third of those the next level too. With the calls within calls
// and the divisions taken out of the passes, an evaluation's transforms and
// their barriers took 21.9 -> 19.8 us at 64 x 64 bins, 26.8 -> 25.6 at 256.
template <int NB, int SETS>
static __device__ __noinline__ void run_transform(int axis, int direction, int vectors, int src, int dst, float ie0,
                                                  float ie1, float ie2, float ie3) {
  Ctx<false, SETS> c(loop_state<SETS>());
  const auto g = c.half_a();
  const float ie[4] = {ie0, ie1, ie2, ie3};
  float ies[2 * NB];
#pragma unroll
  for (int r = 0; r < 2 * NB; ++r) ies[r] = ie[r];
  const fft::Axis a = fft::stage_tables(g, axis ? fft::axis_y(c.d) : fft::axis_x(c.d), c.gsm.fft, true);
  fft::transform<NB>(g, a, direction, vectors, c.gsm.fft, src, dst, ies);
}
template <int SETS>
struct SharedCopy {
  int axis;
  template <int NB, class G>
  __device__ __forceinline__ void run(const G&, const fft::Axis&, fft::Direction direction, int vectors, float4*,
                                      int src, int dst, const float (&ie)[2 * NB]) const {
    run_transform<NB, SETS>(axis, direction, vectors, src, dst, ie[0], ie[1], ie[NB], ie[2 * NB - 1]);
  }
};
template <int NB, int SETS>
static __device__ __noinline__ void run_rows_fwd() {
  Ctx<false, SETS> c(loop_state<SETS>());
#pragma unroll 1
  for (int v = c.pb; v < c.V; v += c.np)
    fft::rows_fwd<NB, true>(c.half_a(), c.d, c.r.p, v, c.V, c.gsm.fft, c.sh.a, c.L.fmean, c.L.tables,
                            c.np, SharedCopy<SETS>{0});
}
template <int NB, int SETS>
static __device__ __noinline__ void run_cols() {
  Ctx<false, SETS> c(loop_state<SETS>());
#pragma unroll 1
  for (int v = c.pb; v < c.V; v += c.np)
    fft::cols<NB>(c.half_a(), c.d, v, c.V, c.gsm.fft, c.L.tables, c.np, SharedCopy<SETS>{1});
}
template <int NB, int SETS>
static __device__ __noinline__ void run_rows_inv() {
  Ctx<false, SETS> c(loop_state<SETS>());
#pragma unroll 1
  for (int v = c.pb; v < c.V; v += c.np)
    fft::rows_inv<NB>(c.half_a(), c.d, c.r.p, v, c.V, c.gsm.fft, c.sh.a, c.L.tables, SharedCopy<SETS>{0});
}
OUTLINED(bool, run_sync)() { return Ctx<LARGE, SETS>(loop_state<SETS>()).sync_body(); }
OUTLINED(void, run_wa)(const float2* pos, double gam) { Ctx<LARGE, SETS>(loop_state<SETS>()).wa(pos, gam); }
OUTLINED(void, run_scatter)(const float2* pos) {
  Ctx<LARGE, SETS> c(loop_state<SETS>());
#pragma unroll 1
  for (int v = c.pb; v < c.V; v += c.np) c.scatter(pos, v);
}
OUTLINED(void, run_combine_kept)(const float2* pos, float2* g) {
  Ctx<LARGE, SETS> c(loop_state<SETS>());
#pragma unroll 1
  for (int v = c.pb; v < c.V; v += c.np) c.combine_kept(pos, g, v);
}
OUTLINED(bool, run_transform_first)() { return Ctx<LARGE, SETS>(loop_state<SETS>()).transform_first(); }
OUTLINED(bool, run_transform_rest)() { return Ctx<LARGE, SETS>(loop_state<SETS>()).transform_rest(); }
OUTLINED(bool, run_density_and_wa)(const float2* pos, double gam, const float2* origin, float2* origin_g) {
  return Ctx<LARGE, SETS>(loop_state<SETS>()).density_and_wa(pos, gam, origin, origin_g);
}
OUTLINED(bool, run_gradient)(const float2* pos, float2* g, ERec* out, ERec* origin) {
  return Ctx<LARGE, SETS>(loop_state<SETS>()).gradient(pos, g, *out, origin);
}
OUTLINED(bool, run_eval_initial)(const float2* pos, float2* g, double gam, bool full) {
  Ctx<LARGE, SETS> c(loop_state<SETS>());
  return c.eval_initial(pos, g, gam, full, c.L.eo);
}
OUTLINED(void, run_precondition)(bool deposits) {
  Ctx<LARGE, SETS> c(loop_state<SETS>());
  const StepVars& V = c.L.V;
#pragma unroll 1
  for (int v = c.pb; v < c.V; v += c.np)
    c.precondition(V.lambda, c.X(), V.pending_prev ? c.X() : c.Xp(), V.extrapolation, c.Y(), deposits, v);
}
OUTLINED(void, run_candidate)(const float2* y, const float2* gy, float2* to) {
  Ctx<LARGE, SETS> c(loop_state<SETS>());
#pragma unroll 1
  for (int v = c.pb; v < c.V; v += c.np) c.candidate(y, gy, c.L.V.inv_L, to, v);
}
#undef OUTLINED

// ---- scalar rules (eplace.rs:1300-1415), evaluated by thread 0 ------------
static __device__ int field_gamma_dev(double overflow, double target, double slope, double base, double& g) {
  if (!isfinite(overflow) || overflow < 0.0 || !(target >= 0.0 && target < 1.0) || !(base > 0.0))
    return TEXO_GP_ERR_INVALID_NORMALIZATION;
  const double intercept = 1.0 - slope;   // slope = 2 / (1 - target), from the host
  // 10^t as exp(t ln 10): a fraction of pow's cost on the device, within a
  // few ulps for the exponents this rule produces
  constexpr double kLn10 = 2.302585092994045684;
  g = base * exp(kLn10 * (slope * overflow + intercept));
  return (isfinite(g) && g > 0.0) ? TEXO_GP_OK : TEXO_GP_ERR_INVALID_NORMALIZATION;
}
static __device__ int adaptive_gamma_dev(const DevRun& S, const double* overflow, double& out) {
  double ws = 0.0, wsum = 0.0;
  for (int f = 0; f < S.K; ++f) {
    double g;
    const int st = field_gamma_dev(overflow[f], S.target[f], S.gamma_slope[f], S.gamma_base, g);
    if (st) return st;
    ws += g * S.gamma_weight[f];
    wsum += S.gamma_weight[f];
  }
  out = wsum == 0.0 ? S.gamma_base : ws * S.inv_gamma_weight_sum;
  return (isfinite(out) && out > 0.0) ? TEXO_GP_OK : TEXO_GP_ERR_INVALID_NORMALIZATION;
}
// density_stop_reached (eplace.rs:1397-1415): Final, or AreaAdjustmentReady
// (LUT and register fields at 0.15, AREA_ADJUSTMENT_OVERFLOW_TARGET)
static __device__ bool stop_dev(const DevRun& S, const double* overflow) {
  for (int f = 0; f < S.K; ++f) {
    if (S.stop_mode == 1) {
      if (S.area_field[f] && !(overflow[f] <= 0.15)) return false;
    } else if (!(overflow[f] <= S.target[f])) {
      return false;
    }
  }
  return true;
}
// area_adjusted_density_multipliers and area_adjusted_multiplier_step
// (eplace.rs:1183-1232), elfPlace eqs. (27)-(28)
static __device__ int area_multipliers_dev(DevRun& S, const ERec& e) {
  double sg[kMaxFields], dens = 0.0;
  for (int f = 0; f < S.K; ++f) {
    const double ne = e.energy[f] * S.inv_e0[f];
    sg[f] = ne + 0.5 * S.beta * ne * ne;
    if (!isfinite(sg[f]) || sg[f] < 0.0) return TEXO_GP_ERR_INVALID_NORMALIZATION;
    dens += e.force[f] * sg[f];
  }
  if (!isfinite(e.wal1) || e.wal1 <= 0.0 || !isfinite(dens) || dens <= 0.0) return TEXO_GP_ERR_INVALID_NORMALIZATION;
  const double scale = 0.1 * e.wal1 / dens;
  bool any = false;
  double nn = 0.0;
  for (int f = 0; f < S.K; ++f) {
    S.lambda[f] = scale * sg[f];
    if (!isfinite(S.lambda[f]) || S.lambda[f] < 0.0) return TEXO_GP_ERR_INVALID_NORMALIZATION;
    any = any || S.lambda[f] > 0.0;
    nn += S.lambda[f] * S.lambda[f];
  }
  if (!any) return TEXO_GP_ERR_INVALID_NORMALIZATION;
  S.mstep = (S.alpha_high - 1.0) * sqrt(nn);
  return (isfinite(S.mstep) && S.mstep > 0.0) ? TEXO_GP_OK : TEXO_GP_ERR_INVALID_NORMALIZATION;
}
static __device__ void excess_dev(const DevRun& S, const double* overflow, double& mx, double& tot) {
  mx = 0.0;
  tot = 0.0;
  for (int f = 0; f < S.K; ++f) {
    const double x = fmax(overflow[f] - S.target[f], 0.0);
    mx = fmax(mx, x);
    tot += x;
  }
}
static __device__ int validate_initial_dev(const DevRun& S, const ERec& e) {
  bool ok = isfinite(e.wa) && e.bad == 0x7fffffffffffffffll;
  for (int f = 0; f < S.K && ok; ++f)
    ok = isfinite(e.energy[f]) && e.energy[f] >= 0.0 && isfinite(e.overflow[f]) && isfinite(e.force[f]) &&
         e.force[f] >= 0.0;
  return ok ? TEXO_GP_OK : TEXO_GP_ERR_INVALID_NORMALIZATION;
}
static __device__ int checked_dev(const ERec& e) {
  if (!isfinite(e.value)) return TEXO_GP_ERR_INVALID_OBJECTIVE;
  if (e.bad != 0x7fffffffffffffffll) return TEXO_GP_ERR_NONFINITE_GRADIENT;
  return TEXO_GP_OK;
}
// update_density_multipliers (eplace.rs:1234-1260), with the step of this
// iteration; growth_dev gives the next step's factor (next_multiplier_step,
// :1261-1298), which depends on the energies alone
static __device__ int update_multipliers_dev(DevRun& S) {
  for (int f = 0; f < S.K; ++f)
    if (!isfinite(S.cur_energy[f]) || !(S.e0[f] > 0.0)) return TEXO_GP_ERR_DENSITY_FIELD_CHANGED;
  double sg[kMaxFields], nn = 0.0;
#pragma unroll
  for (int f = 0; f < kMaxFields; ++f)
    if (f < S.K) {
      const double ne = S.cur_energy[f] * S.inv_e0[f];
      sg[f] = ne + 0.5 * S.beta * ne * ne;
      if (!isfinite(sg[f]) || sg[f] < 0.0) return TEXO_GP_ERR_INVALID_NORMALIZATION;
      nn += sg[f] * sg[f];
    }
  const double norm = sqrt(nn);
  if (norm != 0.0) {
    if (!isfinite(norm) || !isfinite(S.mstep) || S.mstep <= 0.0) return TEXO_GP_ERR_INVALID_NORMALIZATION;
#pragma unroll
    for (int f = 0; f < kMaxFields; ++f)
      if (f < S.K) {
        S.lambda[f] += S.mstep * sg[f] / norm;
        if (!isfinite(S.lambda[f]) || S.lambda[f] < 0.0) return TEXO_GP_ERR_INVALID_NORMALIZATION;
      }
  }
  return TEXO_GP_OK;
}
static __device__ int growth_dev(const DevRun& S, double& growth) {
  double en = 0.0;
  for (int f = 0; f < S.K; ++f) {
    const double ne = S.cur_energy[f] * S.inv_e0[f];
    en += ne * ne;
  }
  const double lg = log(S.beta * sqrt(en) + 1.0);
  if (!isfinite(lg) || lg < 0.0) return TEXO_GP_ERR_INVALID_NORMALIZATION;
  growth = S.alpha_low + (1.0 - 1.0 / (1.0 + lg)) * (S.alpha_high - S.alpha_low);
  return (growth >= S.alpha_low && growth <= S.alpha_high) ? TEXO_GP_OK : TEXO_GP_ERR_INVALID_NORMALIZATION;
}
// f64::midpoint(1, sqrt(1 + 4 m^2))
__device__ __forceinline__ double next_momentum_dev(double m) {
  const double s = sqrt(1.0 + 4.0 * m * m);
  return fabs(s) <= 8.0e307 ? (1.0 + s) / 2.0 : 0.5 + s / 2.0;
}
__device__ __forceinline__ double half_nonzero_dev(double v) {
  const double h = v * 0.5;
  return h == 0.0 ? v : h;
}
__device__ __forceinline__ double margin_dev(const DevRun& S, double x, double y) {
  return S.margin_eps * (1.0 + fabs(x) + fabs(y));
}
static __device__ void adopt_density(DevRun& S, const ERec& e) {
  for (int f = 0; f < S.K; ++f) {
    S.cur_overflow[f] = e.overflow[f];
    S.cur_energy[f] = e.energy[f];
    S.cur_overflow_fixed[f] = e.ovfix[f];
  }
}

enum { ACT_NONE = 0, ACT_RESTART, ACT_CONTINUE, ACT_ACCEPT, ACT_STATIONARY };

// Copies *src to *dst one 8-byte word per thread of the block (a struct copy
// by one thread waits for each load in turn). The caller synchronizes.
template <class T>
__device__ __forceinline__ void copy_words(T* dst, const T* src) {
  static_assert(sizeof(T) % 8 == 0 && alignof(T) >= 8, "copied as 8-byte words");
  for (int i = threadIdx.x; i < (int)(sizeof(T) / 8); i += blockDim.x)
    reinterpret_cast<unsigned long long*>(dst)[i] = reinterpret_cast<const unsigned long long*>(src)[i];
}

// The placement loop of one instance, run by its np physical blocks of SETS *
// kThreads threads; the caller has the instance's descriptor in
// loop_state<SETS>().inst. `resident` is a double block's dynamic shared
// memory.
template <bool LARGE, int SETS>
static __device__ void run_body(int pb, int np, Resident* resident) {
  LoopState<SETS>& L = loop_state<SETS>();
  DevRun& S = L.S;
  ERec &eo = L.eo, &ey = L.ey, &ec = L.ec;
  StepVars& V = L.V;
  FoldValue* const fvals = L.fv;
  const Dev& d = L.inst.d;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 10; ++i) L.clock[i] = 0;
    L.clock[8] = now_ns();
    L.nbar = 0;
    L.gen = 0;   // the barrier is cleared with the state copy before every launch
    L.pb = pb;
    L.np = np;
    // one virtual block a physical one: its objects can stay in shared memory
    L.res = SETS == 2 && np == L.inst.V ? resident : nullptr;
    const bool maps = L.res && !d.g.identity && d.g.W <= kResidentMap && d.g.H <= kResidentMap;
    L.mapx = maps ? L.res->mapx : d.binmap_x;
    L.mapy = maps ? L.res->mapy : d.binmap_y;
    L.tables = fft::tables_stay(d);
    V.ws = 0;
    V.pending_best = 0;
    V.pending_prev = 0;
    V.dirty = 0;
  }
  if ((int)threadIdx.x < d.K) L.capsum[threadIdx.x] = d.capsum[threadIdx.x];
  copy_words(&S, L.inst.run);
  __syncthreads();
  Ctx<LARGE, SETS> c(L);
  const Reduce& r = c.r;
  const Buffers& B = c.B;
  c.make_resident();
  __syncthreads();
  if (L.tables && c.in_a())
    fft::stage_tables(c.half_a(), fft::axis_x(d), reinterpret_cast<fft::Smem*>(L.gsm.fft)->buf, false);
  const int n = d.nobj;
  unsigned done = 0;
  bool ok = true;

// Thread 0 updates the block's shared controller state. The leading
// __syncthreads keeps it from overwriting a field (S, V) that a slower warp
// of the block is still reading from the previous update.
#define T0            \
  __syncthreads();    \
  if (threadIdx.x == 0)
#define VLOOP _Pragma("unroll 1") for (int v = c.pb; v < c.V; v += c.np)
#define LEAVE   \
  {             \
    ok = false; \
    goto out;   \
  }
#define SYNC_OR_EXIT(cat) \
  if (!c.sync()) LEAVE    \
  c.mark(cat);
#define FAIL(code)            \
  {                           \
    T0 {                      \
      S.status = (code);      \
      S.phase = 2;            \
    }                         \
    __syncthreads();          \
    goto out;                 \
  }

  if (S.phase == 2) goto out;
  if (S.phase == 0) {
    // initial probe at the ePlace gamma base, then at the adaptive gamma with
    // the density side reused (same coordinates), eplace.rs:455-471
    VLOOP {
      c.reset_grids(v);
      c.reset_wa(v);
    }
    SYNC_OR_EXIT(PC_PRECOND)
    if (!run_eval_initial<LARGE, SETS>(c.X(), c.gX(), S.gamma_base, true)) LEAVE
    {
      T0 {
        double g0 = 0.0;
        int st = validate_initial_dev(S, eo);
        if (!st) st = adaptive_gamma_dev(S, eo.overflow, g0);
        S.status = st;
        S.gamma = g0;
        adopt_density(S, eo);
      }
      __syncthreads();
      if (S.status) FAIL(S.status)
    }
    VLOOP c.reset_wa(v);
    SYNC_OR_EXIT(PC_PRECOND)
    if (!run_eval_initial<LARGE, SETS>(c.X(), c.gX(), S.gamma, false)) LEAVE
    T0 {
      int st = validate_initial_dev(S, eo);
      for (int f = 0; f < S.K; ++f) {
        if (!S.fixed_e0) S.e0[f] = fmax(eo.energy[f], 1.0);
        if (!st && !(isfinite(S.e0[f]) && S.e0[f] > 0.0)) st = TEXO_GP_ERR_DENSITY_FIELD_CHANGED;
        S.inv_e0[f] = 1.0 / S.e0[f];
      }
      S.status = st;
      excess_dev(S, eo.overflow, S.best_max, S.best_tot);
      S.density_at_x = 1;
      S.phase = 1;
      S.a = 1.0;
      S.has_L = 0;
      if (!st && stop_dev(S, eo.overflow)) {
        S.phase = 2;
        S.converged = 1;
      } else if (!st && S.reset_mult) {
        S.status = area_multipliers_dev(S, eo);
      } else if (!st) {
        // initial_density_multiplier (eplace.rs:1126-1148)
        double dens = 0.0;
        for (int f = 0; f < S.K; ++f) dens += eo.rawl1[f];
        const double m0 = (eo.wal1 == 0.0 || dens == 0.0) ? 1.0 : S.init_weight * eo.wal1 / dens;
        if (!(isfinite(m0) && m0 > 0.0)) S.status = TEXO_GP_ERR_INVALID_NORMALIZATION;
        for (int f = 0; f < S.K; ++f) S.lambda[f] = m0;
        S.mstep = S.alpha_high - 1.0;
      }
      V.pending_best = 1;
      V.pending_prev = 1;
    }
    __syncthreads();
    if (S.status) FAIL(S.status)
    if (S.phase == 2) goto out;
  }
  // the loop's evaluations leave the accumulators reset; whatever ran before
  // this launch, or the probes above, may have left them dirty
  VLOOP {
    c.reset_grids(v);
    c.reset_wa(v);
  }
  SYNC_OR_EXIT(PC_PRECOND)

  // ---- outer loop -------------------------------------------------------
  for (bool update = false;; update = true) {
    // The scalar rules between two iterations (FP64 functions of a thousand
    // cycles and more each on this part) are independent of one another: the
    // multipliers, their step's growth, gamma and the momentum run in a warp
    // each.
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
      switch (threadIdx.x >> 5) {
        case 0:
          if (update) V.st_multipliers = update_multipliers_dev(S);
          break;
        case 1:
          if (update) V.st_growth = growth_dev(S, V.growth);
          break;
        case 2: V.st_gamma = adaptive_gamma_dev(S, S.cur_overflow, V.gamma); break;
        case 3:
          V.next_m = next_momentum_dev(S.a);
          V.extrapolation = (float)((S.a - 1.0) / V.next_m);
          break;
        default: break;
      }
    }
    T0 {
      V.action = ACT_NONE;
      if (update) {
        int st = V.st_multipliers;
        if (!st) st = V.st_growth;
        if (!st) {
          S.mstep *= V.growth;
          if (!(isfinite(S.mstep) && S.mstep > 0.0)) st = TEXO_GP_ERR_INVALID_NORMALIZATION;
        }
        if (st) {
          S.status = st;
          S.phase = 2;
        }
      }
      if (S.phase == 2) {
      } else if (stop_dev(S, S.cur_overflow)) {
        S.converged = 1;
        S.phase = 2;
      } else if (S.completed >= S.max_iterations) {
        S.exhausted = 1;
        S.phase = 2;
        S.status = S.best_effort ? TEXO_GP_OK : TEXO_GP_ERR_DID_NOT_CONVERGE;
      } else if (S.budget && done >= S.budget) {
        V.action = ACT_CONTINUE;   // leave with the loop still running
      } else {
        if (V.st_gamma) {
          S.status = V.st_gamma;
          S.phase = 2;
        }
        S.gamma = V.gamma;
        S.completed++;
        if (!isfinite(S.a) || S.a < 1.0) {
          S.status = TEXO_GP_ERR_INVALID_MOMENTUM_PARAMETER;
          S.phase = 2;
        }
        if (S.has_L && (!isfinite(S.L) || S.L <= 0.0)) {
          S.status = TEXO_GP_ERR_INVALID_LIPSCHITZ_ESTIMATE;
          S.phase = 2;
        }
        V.restart = 0;
        V.has_wL = S.has_L;
        V.wL = S.L;
        V.trials = 0;
        V.fresh = !S.density_at_x;
        V.deposited = !V.fresh && V.extrapolation != 0.f;   // without momentum y is the origin
        for (int f = 0; f < S.K; ++f) V.lambda[f] = (float)S.lambda[f];
      }
    }
    __syncthreads();
    if (S.phase == 2 || V.action == ACT_CONTINUE) break;
    ++done;

    // Phase 1: the preconditioner (eplace.rs:1046-1100), the extrapolated
    // point (it needs the positions and the momentum alone) and its scatter,
    // pending copies, and the origin's WA. The origin is re-evaluated
    // (eplace's closure changes with gamma and the multipliers); its density
    // side is reused when the device already holds it for these coordinates.
    const bool fresh = V.fresh != 0, deposited = V.deposited != 0;
    {
      if (c.in_a()) run_precondition<LARGE, SETS>(deposited);
      if (V.pending_best) c.copy(B.best, c.X(), d.U);
      if (V.pending_prev) c.copy(c.Xp(), c.X(), n);
      if (!fresh && c.in_b()) run_wa<LARGE, SETS>(c.X(), S.gamma);
      SYNC_OR_EXIT(PC_PRECOND)
      const Partials q = c.set();
      const int nj = (fresh ? 4 : 5), ns = deposited ? d.K : 0;
      c.fold(nj + ns, [&](int j) {
        return j == 0   ? FoldJob{mslot(r.p, MS_PMIN), FOLD_DMIN}
               : j == 1 ? FoldJob{mslot(r.p, MS_PMAX), FOLD_DMAX}
               : j == 2 ? FoldJob{islot(r.p, IS_PBAD), FOLD_ISUM}
               : j == 3 ? FoldJob{islot(q, IS_DIFF), FOLD_ISUM}
               : j < nj ? FoldJob{pslot(r.p, SLOT_WA_VALUE), FOLD_DSUM}
                        : c.sum_job(j - nj);
      });
      if (threadIdx.x == 0) {
        ++V.ws;
        V.pmin = fvals[0].d;
        V.pmax = fvals[1].d;
        V.y_is_origin = fvals[3].l == 0;
        V.dirty = deposited && fvals[3].l == 0;
        V.pending_best = 0;
        V.pending_prev = 0;
        if (fvals[2].l) S.status = TEXO_GP_ERR_INVALID_NORMALIZATION;
        else if (!fresh) c.eval_coefficients(false);
      }
      if (threadIdx.x == 32 && !fresh) c.eval_value(eo, false, 4);
      if ((int)threadIdx.x >= 64 && (int)threadIdx.x < 64 + ns) c.set_mean(threadIdx.x - 64, fvals[nj + threadIdx.x - 64].l);
      __syncthreads();
      if (S.status) FAIL(S.status)
      if (!fresh) {
        T0 {
          S.evaluations++;
          if (!isfinite(eo.value)) S.status = TEXO_GP_ERR_INVALID_OBJECTIVE;
        }
        __syncthreads();
        if (S.status) FAIL(S.status)
      }
    }
    if (fresh) {
      if (c.in_a()) run_scatter<LARGE, SETS>(c.X());
      SYNC_OR_EXIT(PC_SCATTER_WA)
      c.fold(d.K, [&](int j) { return c.sum_job(j); });
      if ((int)threadIdx.x < d.K) c.set_mean(threadIdx.x, fvals[threadIdx.x].l);
      __syncthreads();
      if (!run_density_and_wa<LARGE, SETS>(c.X(), S.gamma, nullptr, nullptr)) LEAVE
      if (!run_gradient<LARGE, SETS>(c.X(), c.gX(), &eo, nullptr)) LEAVE
      T0 {
        S.status = checked_dev(eo);
        adopt_density(S, eo);
        S.density_at_x = 1;
      }
      __syncthreads();
      if (S.status) FAIL(S.status)
      if (!V.y_is_origin) {
        if (c.in_a()) run_scatter<LARGE, SETS>(c.Y());
        SYNC_OR_EXIT(PC_EXTRAP)
        c.fold(d.K, [&](int j) { return c.sum_job(j); });
        if ((int)threadIdx.x < d.K) c.set_mean(threadIdx.x, fvals[threadIdx.x].l);
        __syncthreads();
      }
    } else if (V.y_is_origin) {
      // the origin's gradient in a phase of its own
      if (c.in_b()) run_combine_kept<LARGE, SETS>(c.X(), c.gX());
      if (V.dirty) VLOOP c.reset_grids(v);
      SYNC_OR_EXIT(PC_SCATTER_WA)
      c.fold(2, [&](int j) { return c.kkt_job(r.q, j); });
      T0 {
        eo.kkt = fvals[0].d;
        eo.bad = fvals[1].l;
        V.dirty = 0;
        S.status = checked_dev(eo);
      }
      __syncthreads();
      if (S.status) FAIL(S.status)
    }

    // Phase 2: the dynamic Nesterov step (global_placement.rs:152-335)
    for (;;) {  // 'step
      T0 {
        if (V.restart) {
          V.next_m = next_momentum_dev(1.0);
          V.y_is_origin = 1;
        }
        if (!isfinite(V.next_m)) S.status = TEXO_GP_ERR_ITERATION_OVERFLOW;
        V.f_y = eo.value;
        V.y_stat = eo.kkt;
      }
      __syncthreads();
      if (S.status) FAIL(S.status)
      if (!V.y_is_origin) {
        if (!run_density_and_wa<LARGE, SETS>(c.Y(), S.gamma, fresh ? nullptr : c.X(), fresh ? nullptr : c.gX())) LEAVE
        if (!run_gradient<LARGE, SETS>(c.Y(), c.gY(), &ey, fresh ? nullptr : &eo)) LEAVE
      }
      T0 {
        if (!V.y_is_origin) {
          if (!fresh) S.status = checked_dev(eo);   // the origin's own check, folded with y's
          if (!S.status) {
            S.density_at_x = 0;
            S.status = checked_dev(ey);
          }
          V.f_y = ey.value;
          V.y_stat = ey.kkt;
        }
        V.action = ACT_NONE;
        if (S.status) {
        } else if (!isfinite(V.y_stat)) {
          S.status = TEXO_GP_ERR_LINE_SEARCH_OVERFLOW;
        } else if (V.y_stat == 0.0) {
          V.action = V.y_is_origin ? ACT_STATIONARY : ACT_RESTART;
          if (!V.y_is_origin) V.restart = 1;
        } else {
          V.tL = half_nonzero_dev(V.has_wL ? V.wL : V.y_stat);
          V.may_reduce = 1;
        }
      }
      __syncthreads();
      if (S.status) FAIL(S.status)
      if (V.action == ACT_RESTART) continue;
      if (V.action == ACT_NONE) {
        const float2* ybuf = V.y_is_origin ? c.X() : c.Y();
        const float2* gy = V.y_is_origin ? c.gX() : c.gY();
        for (;;) {  // line search
          T0 {
            V.action = ACT_NONE;
            V.trials++;
            if (V.trials > kMaxTrialsPerStep) {
              S.status = TEXO_GP_ERR_ITERATION_OVERFLOW;
            } else if (!isfinite(V.tL * V.pmax)) {
              S.status = TEXO_GP_ERR_LINE_SEARCH_OVERFLOW;
            } else if (V.tL * V.pmin == 0.0) {
              V.tL *= 2.0;
              V.may_reduce = 0;
              if (!isfinite(V.tL)) S.status = TEXO_GP_ERR_LINE_SEARCH_OVERFLOW;
              V.action = ACT_CONTINUE;
            } else {
              // 1/L saturates at FLT_MAX: a huge step clamps to the box as it
              // does in FP64, where an infinite one would turn 0 * inf into NaN
              V.inv_L = (float)fmin(1.0 / V.tL, 3.0e38);
            }
          }
          __syncthreads();
          if (S.status) FAIL(S.status)
          if (V.action == ACT_CONTINUE) continue;
          if (V.dirty) {   // a rejected scatter is in the grids
            VLOOP c.reset_grids(v);
            SYNC_OR_EXIT(PC_EXTRAP)
          }
          run_candidate<LARGE, SETS>(ybuf, gy, c.C());
          SYNC_OR_EXIT(PC_CANDIDATE)
          {
            const Partials q = c.set();
            c.fold(3 + d.K, [&](int j) {
              return j == 0   ? FoldJob{islot(q, IS_DIFF), FOLD_ISUM}
                     : j == 1 ? FoldJob{pslot(q, SLOT_DOT), FOLD_DSUM}
                     : j == 2 ? FoldJob{pslot(q, SLOT_MSN), FOLD_DSUM}
                              : c.sum_job(j - 3);
            });
          }
          const long long changed = fvals[0].l;
          const double dot = fvals[1].d, msn = fvals[2].d;
          if ((int)threadIdx.x >= 64 && (int)threadIdx.x < 64 + d.K) c.set_mean(threadIdx.x - 64, fvals[3 + threadIdx.x - 64].l);
          T0 {
            ++V.ws;
            V.action = ACT_NONE;
            V.dirty = changed == 0;
            if (changed == 0) {
              const double smaller = half_nonzero_dev(V.tL);
              if (V.may_reduce && smaller < V.tL) {
                V.tL = smaller;
                V.action = ACT_CONTINUE;
              } else if (!V.y_is_origin) {
                V.restart = 1;
                V.has_wL = 1;
                V.wL = V.tL;
                V.action = ACT_RESTART;
              } else {
                V.action = ACT_STATIONARY;
                S.has_L = 1;
                S.L = V.tL;
              }
            }
          }
          __syncthreads();
          if (V.action == ACT_CONTINUE) continue;
          if (V.action != ACT_NONE) break;
          if (!run_density_and_wa<LARGE, SETS>(c.C(), S.gamma, nullptr, nullptr)) LEAVE
          if (!run_gradient<LARGE, SETS>(c.C(), c.gC(), &ec, nullptr)) LEAVE
          T0 {
            S.density_at_x = 0;
            S.status = checked_dev(ec);
            const double upper = V.f_y + dot + 0.5 * V.tL * msn;
            if (!S.status && !isfinite(upper)) S.status = TEXO_GP_ERR_LINE_SEARCH_OVERFLOW;
            const bool smooth = ec.value <= upper + margin_dev(S, ec.value, upper);
            const bool mono = ec.value <= eo.value + margin_dev(S, ec.value, eo.value);
            if (smooth && mono) {
              V.action = ACT_ACCEPT;
              if (!isfinite(ec.kkt)) S.status = TEXO_GP_ERR_LINE_SEARCH_OVERFLOW;
              S.last_objective = ec.value;
            } else if (smooth && !V.restart) {
              V.restart = 1;
              V.has_wL = 1;
              V.wL = V.tL;
              V.action = ACT_RESTART;
            } else {
              V.tL *= 2.0;
              V.may_reduce = 0;
              if (!isfinite(V.tL)) S.status = TEXO_GP_ERR_LINE_SEARCH_OVERFLOW;
              V.action = ACT_CONTINUE;
            }
          }
          __syncthreads();
          if (S.status) FAIL(S.status)
          if (V.action != ACT_CONTINUE) break;
        }
      }
      if (V.action == ACT_RESTART) continue;
      // leave the step: accepted or numerically stationary; then the
      // checkpoint and the stop rules (eplace.rs:550-573)
      T0 {
        S.trials += V.trials;
        if (V.action == ACT_ACCEPT) {
          const int oxp = S.ixp;
          S.ixp = S.ix;
          S.ix = S.ic;
          S.ic = oxp;
          const int og = S.igx;
          S.igx = S.igc;
          S.igc = og;
          S.a = V.next_m;
          S.has_L = 1;
          S.L = V.tL;
          S.density_at_x = 1;
          adopt_density(S, ec);
          V.stationary = 0;
        } else {
          S.a = 1.0;
          S.last_objective = eo.value;
          adopt_density(S, eo);
          V.pending_prev = 1;
          V.stationary = 1;
        }
        double mx, tot;
        excess_dev(S, S.cur_overflow, mx, tot);
        if (mx < S.best_max || (mx == S.best_max && tot < S.best_tot)) {
          S.best_max = mx;
          S.best_tot = tot;
          V.pending_best = 1;
        }
        if (stop_dev(S, S.cur_overflow)) {
          S.converged = 1;
          S.phase = 2;
        } else if (!V.stationary) {
          S.have_prev_stationary = 0;
        }
      }
      __syncthreads();
      break;
    }
    if (S.phase == 2) break;
    if (V.stationary) {
      // stationary_target_is_fixed (eplace.rs:973-985): compare rounded targets
      const float2* x = c.X();
      if (c.in_a()) VLOOP {
        const auto g = c.half_a();
        long long mism = 0;
        for (int u = v * kThreads + g.tid; u < d.U; u += c.V * kThreads) {
          const float2 a = x[u];
          const uint32_t tx = (uint32_t)fminf(fmaxf(roundf(a.x), 0.f), (float)(S.W - 1));
          const uint32_t ty = (uint32_t)fminf(fmaxf(roundf(a.y), 0.f), (float)(S.H - 1));
          mism += (B.prev_targets[2 * u] != tx) + (B.prev_targets[2 * u + 1] != ty);
          B.prev_targets[2 * u] = tx;
          B.prev_targets[2 * u + 1] = ty;
        }
        write_partial(g, mism, islot(c.set(), IS_DIFF), v, L.sh.a.l);
      }
      if (V.dirty) VLOOP c.reset_grids(v);   // the next iteration scatters at once
      SYNC_OR_EXIT(PC_OTHER)
      const Partials q = c.set();
      c.fold(1, [&](int) { return FoldJob{islot(q, IS_DIFF), FOLD_ISUM}; });
      const long long total = fvals[0].l;
      T0 {
        ++V.ws;
        const bool fixed = S.have_prev_stationary && total == 0;
        S.have_prev_stationary = 1;
        V.dirty = 0;
        if (fixed) {
          S.exhausted = 1;
          S.phase = 2;
          S.status = S.best_effort ? TEXO_GP_OK : TEXO_GP_ERR_DID_NOT_CONVERGE;
        }
      }
      __syncthreads();
      if (S.phase == 2) break;
    }
  }

out:
  // flush pending copies so the host sees the checkpoint and the state
  if (ok && (V.pending_best || V.pending_prev)) {
    if (V.pending_best) c.copy(B.best, c.X(), d.U);
    if (V.pending_prev) c.copy(c.Xp(), c.X(), n);
    ok = c.sync();
  }
  c.mark(PC_OTHER);
  __syncthreads();
  if (pb == 0) {
    if (threadIdx.x == 0) {
      S.barriers += L.nbar;
      for (int i = 0; i < 8; ++i) S.phase_ns[i] += L.clock[i];
      S.barrier_wait_ns += L.clock[9];
    }
    __syncthreads();
    copy_words(L.inst.run, &S);
  }
#undef T0
#undef VLOOP
#undef SYNC_OR_EXIT
#undef LEAVE
#undef FAIL
}

}  // namespace tgp
