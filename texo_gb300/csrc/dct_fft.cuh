// dct_fft.cuh — the spectral Poisson solve as FFT-based DCTs, for
// power-of-two bin grids up to 1024, in double-float arithmetic.
//
// The orthonormal DCT-II of a real vector x of length n is computed with
// Makhoul's reordering (IEEE TASSP 28(1), 1980): v = (x0, x2, x4, ...,
// x5, x3, x1), V = FFT_n(v), X_k = s_k Re(exp(-i pi k / 2n) V_k) with
// s_0 = sqrt(1/n), s_k = sqrt(2/n). The inverse (DCT-III) forms
// W_k = exp(-i pi k / 2n) (X_k / s_k + i X_{n-k} / s_{n-k}) (X_n = 0), takes
// F = FFT_n(W) and reads x_{2j} = Re F_j / n, x_{2j+1} = Re F_{n-1-j} / n.
// The FFT is a radix-2 decimation-in-time transform over a group of vectors,
// each thread keeping the two points of its butterfly in registers from
// stage to stage.
//
// Every value inside a transform is a double-float: an unevaluated sum
// hi + lo of two FP32 numbers, added with Knuth's two-sum and multiplied with
// the exact FMA product (the double-double arithmetic of Dekker 1971 and of
// Hida, Li and Bailey 2001, in single precision: about 2^-44 relative). The
// twiddle and scaling tables are FP64 values split into such pairs. Plain
// FP32 butterflies lose about log2(n) roundings of the vector norm, which the
// 1/lambda scaling and the field gather amplify (potential 2.6e-6 and field
// gradient 1.3e-5 normwise at 256 x 256); with double-float butterflies the
// transforms are exact to FP32 and the only roundings left are the FP32
// stores between the passes, as in the compensated GEMM form. The arithmetic
// runs on the FP32 pipes: an FP64 butterfly would occupy this part's FP64
// pipe for hundreds of cycles.
//
// The 2-D solve t1 = rows-DCT(rho), t2 = cols-IDCT(cols-DCT(t1) / lambda),
// phi = rows-IDCT(t2) takes three passes: the column pass owns whole
// columns, so the forward transform, the inverse-eigenvalue scaling and the
// inverse transform run back to back in shared memory. The intermediate
// grids t1 and t2 are stored as double-float pairs (float2 per bin), so the
// only FP32 roundings are the density entering (exact from fixed point when
// the preparation is folded in) and the potential leaving.
#pragma once
#include "stages.cuh"

namespace tgp {
namespace fft {

// Work buffer, in 16-byte slots: [0, exch) the butterflies' points crossing
// between warps (two buffers), then the staged vectors (float2 a point), then
// the tables of one axis up to 256 points. Lengths up to 512 take 512 points
// a group, 1024 takes 1024 (two butterflies a thread).
constexpr int kBuf = 2048;
constexpr int kLogPoints = 9;                    // log2 of the points of a group
static_assert(1 << kLogPoints == 2 * kThreads, "one butterfly a thread");
constexpr int kStage = 640;                      // float2 slots of one staged copy, padding included (512 points)
constexpr int kTables = 512 + kStage;            // the tables' first slot

struct Smem {
  float4 buf[kBuf];
};

// ---- double-float arithmetic ---------------------------------------------
// The _rn intrinsics keep the compiler from contracting a product into a
// following add, which would break the error-free transformations.
struct DF {
  float hi, lo;
};
__device__ __forceinline__ DF two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return DF{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ DF quick_two_sum(float a, float b) {   // |a| >= |b| or a == 0
  const float s = __fadd_rn(a, b);
  return DF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ DF df_add(DF a, DF b) {
  const DF s = two_sum(a.hi, b.hi);
  return quick_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ DF df_neg(DF a) { return DF{-a.hi, -a.lo}; }
__device__ __forceinline__ DF df_sub(DF a, DF b) { return df_add(a, df_neg(b)); }
__device__ __forceinline__ DF df_mul(DF a, DF b) {
  const float p = __fmul_rn(a.hi, b.hi);
  const float e = __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.hi, -p)));
  return quick_two_sum(p, e);
}
__device__ __forceinline__ DF df_scale(DF a, float s) {   // s a power of two: exact
  return DF{__fmul_rn(a.hi, s), __fmul_rn(a.lo, s)};
}
__device__ __forceinline__ float df_float(DF a) { return __fadd_rn(a.hi, a.lo); }
// an int64 as a double-float (exact for |v| < 2^48)
__device__ __forceinline__ DF df_from_ll(long long v) {
  const float hi = __ll2float_rn(v);
  return DF{hi, __ll2float_rn(v - __float2ll_rn(hi))};
}

struct CDF {
  DF re, im;
};
__device__ __forceinline__ CDF cdf_load(const float4& v) { return CDF{{v.x, v.z}, {v.y, v.w}}; }
__device__ __forceinline__ float4 cdf_store(const CDF& c) { return make_float4(c.re.hi, c.im.hi, c.re.lo, c.im.lo); }
__device__ __forceinline__ CDF cdf_mul(const CDF& a, const CDF& b) {
  return CDF{df_sub(df_mul(a.re, b.re), df_mul(a.im, b.im)), df_add(df_mul(a.re, b.im), df_mul(a.im, b.re))};
}

// Tables of one transform length n (a power of two), FP64 values as
// double-float pairs: complex tables (re.hi, im.hi, re.lo, im.lo), real
// (hi, lo).
struct Axis {
  const float4* tw;      // [n/2] exp(-2 pi i j / n)
  const float4* post;    // [n]   s_k exp(-i pi k / 2n)
  const float4* pre;     // [n]   exp(-i pi k / 2n)
  const float2* inv_s;   // [n]   1 / s_k
  int n, logn;
};

__device__ __forceinline__ Axis axis_x(const Dev& d) {
  return Axis{d.fx_tw, d.fx_post, d.fx_pre, d.fx_inv_s, d.g.Wb, d.logW};
}
__device__ __forceinline__ Axis axis_y(const Dev& d) {
  return Axis{d.fy_tw, d.fy_post, d.fy_pre, d.fy_inv_s, d.g.Hb, d.logH};
}

// Up to 256 points the tables (n/2 twiddles, n post and n pre factors, n
// 1/s_k) fit in the work buffer beside the data and are copied there: the
// stages then read their twiddles from shared memory instead of making an L2
// round trip per stage (the persistent kernel's grid barriers leave L1 cold).
// With `there` they are in place already: the persistent kernel copies the
// tables of a square grid once, both axes sharing them.
constexpr int kTableLog = 8;
template <class G>
__device__ __forceinline__ Axis stage_tables(const G& g, const Axis& a, float4* buf, bool there) {
  if (a.logn > kTableLog) return a;
  float4* tw = buf + kTables;
  float4* post = tw + (a.n >> 1);
  float4* pre = post + a.n;
  float2* inv_s = reinterpret_cast<float2*>(pre + a.n);
  if (!there) {
    g.sync();   // earlier readers of the buffer are done
#pragma unroll 1
    for (int i = g.tid; i < a.n; i += kThreads) {
      if (i < (a.n >> 1)) tw[i] = a.tw[i];
      post[i] = a.post[i];
      pre[i] = a.pre[i];
      inv_s[i] = a.inv_s[i];
    }
    g.sync();
  }
  return Axis{tw, post, pre, inv_s, a.n, a.logn};
}
__device__ __forceinline__ bool tables_stay(const Dev& d) {
  return d.fft && d.logW == d.logH && d.logW <= kTableLog;
}

// Vectors transformed together: one butterfly per thread per stage (n/2
// butterflies per vector), at least one vector, and no more than spreads the
// groups over `blocks` blocks (the warps of the absent vectors then leave the
// multiprocessor to the others: 64 x 64 bins on 21 blocks took 8 vectors on 8
// of them, 4 on 16 save 0.8 us of an evaluation's 20). 0 blocks: as many as
// fit. Lengths and groups are powers of two, so a group's field and first
// vector are found by shifts.
struct Groups {
  int log_vectors, log_per_field;   // vectors a group, groups a field
  __device__ __forceinline__ Groups(int logn, int log_count, int fields, int blocks) {
    log_vectors = min(max(kLogPoints - logn, 0), log_count);
    while (log_vectors > 0 && fields << (log_count - log_vectors + 1) <= blocks) --log_vectors;
    log_per_field = log_count - log_vectors;
  }
  __device__ __forceinline__ int vectors() const { return 1 << log_vectors; }
  __device__ __forceinline__ int count(int fields) const { return fields << log_per_field; }
  __device__ __forceinline__ int field(int t) const { return t >> log_per_field; }
  __device__ __forceinline__ int first(int t) const { return (t & ((1 << log_per_field) - 1)) << log_vectors; }
};

__device__ __forceinline__ int brev(int m, int logn) {
  return logn ? (int)(__brev((unsigned)m) >> (32 - logn)) : 0;
}
// position of sample i in Makhoul's order (and, for the inverse, the FFT
// output index that holds sample i), and the sample at a position
__device__ __forceinline__ int mak(int i, int n) { return (i & 1) ? n - 1 - (i >> 1) : (i >> 1); }
__device__ __forceinline__ int unmak(int m, int n) { return m < (n >> 1) ? 2 * m : 2 * (n - 1 - m) + 1; }
// staged slots, padded so that the strided accesses of the butterflies'
// outputs meet different banks
__device__ __forceinline__ int pad_k(int k) { return k + (k >> 2); }   // coefficients, four apart a lane
__device__ __forceinline__ int pad_i(int i) { return i + (i >> 3); }   // samples, eight apart a lane

// The radix-2 network. Positions are the bit-reversed input order: stage s
// pairs the positions that differ in bit s. A thread holds, at stage s, the
// two points whose positions agree with its thread index in every other bit,
// and between the stages s - 1 and s it hands one of them to the thread whose
// index differs in the bit that stands for position bit s; that index bit
// then stands for bit s - 1. Lane bits stand for the high position bits (low
// bits of the sample index, so that the staged samples are read without
// conflicts) and trade with shuffles; the warp bits, if a vector spans
// several warps, stand for the low ones and trade through shared memory, one
// block barrier each: two exchanges of 256 points' seven. A transform is bound
// by the latency of its chain on 8 warps; a block barrier and two trips
// through shared memory for every stage were half of it. The butterflies'
// values are the same, operation for operation. Measured: the three passes
// of a 256 x 256 solve in the persistent loop, its three grid barriers
// included, 28.8 -> 25.3 us; a 1024 x 1024 solve in the host engine (rows
// forward / columns / rows inverse) 37 / 80 / 55 -> 24 / 60 / 30 us.
// NB = 2 (1024 points): a thread runs two butterflies, whose points differ in
// position bit 1 at stage 0.
template <int NB>
struct Place {
  int L, n;      // log2 length, length
  int vec;       // vector of the group
  int p;         // position of the thread's first point at stage 0 (butterfly 0)
  int lanes;     // index bits of a vector inside a warp
  __device__ __forceinline__ Place(int tid, int logn) {
    L = logn;
    n = 1 << logn;
    const int bits = logn - NB;                   // index bits of a vector
    const int t = tid & ((1 << max(bits, 0)) - 1);
    vec = tid >> max(bits, 0);
    lanes = min(bits, 5);
    p = brev(t & ((1 << max(lanes, 0)) - 1), logn) | ((t >> max(lanes, 0)) << NB);
  }
};
struct Pair {
  CDF a, b;
};

__device__ __forceinline__ void butterfly(Pair& x, const CDF& w) {
  const CDF t = cdf_mul(x.b, w);
  x.b = CDF{df_sub(x.a.re, t.re), df_sub(x.a.im, t.im)};
  x.a = CDF{df_add(x.a.re, t.re), df_add(x.a.im, t.im)};
}

// Whether the exchange before stage s is between warps (a barrier of the group).
template <int NB>
__device__ __forceinline__ bool crosses_warps(const Place<NB>& at, int s) {
  return s >= NB && s - NB < at.L - NB - at.lanes;
}
// Brings position bit s into the pairs (s >= 1).
template <int NB, class G>
__device__ __forceinline__ void exchange(const G& g, const Place<NB>& at, int s, Pair (&x)[NB], float4* exch) {
  if (NB == 2 && s == 1) {   // between the thread's own butterflies
    const CDF t = x[0].b;
    x[0].b = x[NB - 1].a;
    x[NB - 1].a = t;
    return;
  }
  const bool up = (at.p >> s) & 1;
  if (crosses_warps<NB>(at, s)) {                // through shared memory, the two buffers in turn
    const int w = s - NB;                        // warp bit
    float4* e = exch + (w & 1) * NB * kThreads;
#pragma unroll
    for (int r = 0; r < NB; ++r) e[r * kThreads + g.tid] = cdf_store(up ? x[r].a : x[r].b);
    g.sync();
    const int from = g.tid ^ (32 << w);
#pragma unroll
    for (int r = 0; r < NB; ++r) {
      const CDF v = cdf_load(e[r * kThreads + from]);
      if (up)
        x[r].a = v;
      else
        x[r].b = v;
    }
  } else {
    const int m = 1 << (at.L - 1 - s);
#pragma unroll
    for (int r = 0; r < NB; ++r) {
      const CDF q = up ? x[r].a : x[r].b;
      CDF v;
      v.re.hi = __shfl_xor_sync(0xffffffffu, q.re.hi, m);
      v.re.lo = __shfl_xor_sync(0xffffffffu, q.re.lo, m);
      v.im.hi = __shfl_xor_sync(0xffffffffu, q.im.hi, m);
      v.im.lo = __shfl_xor_sync(0xffffffffu, q.im.lo, m);
      if (up)
        x[r].a = v;
      else
        x[r].b = v;
    }
  }
}

// Stages [from, L); on return pair r holds the outputs of frequencies (or
// sample positions) out_index(at, r) and out_index(at, r) + n / 2.
template <int NB, class G>
__device__ __forceinline__ void stages(const G& g, const Place<NB>& at, int from, Pair (&x)[NB], const Axis& a,
                                       float4* exch) {
#pragma unroll 1
  for (int s = from; s < at.L; ++s) {
    exchange(g, at, s, x, exch);
#pragma unroll
    for (int r = 0; r < NB; ++r) {
      const int j = ((at.p >> 1) | r) & ((1 << s) - 1);
      butterfly(x[r], cdf_load(a.tw[j << (at.L - 1 - s)]));
    }
  }
}
template <int NB>
__device__ __forceinline__ int out_index(const Place<NB>& at, int r) {
  return (at.p >> 1) | r;
}

// Stages 0 and 1 of a forward transform: the vectors' real samples staged in Makhoul's order (st[vec * n +
// m], conflict-free). The inputs are real and stage 0's twiddle is one,
// so stage 0 is two real sums, formed from four staged samples by each of the
// two threads that would trade them (no exchange before stage 1); the
// products by one and the sums with zero that are left out change no value.
template <int NB>
__device__ __forceinline__ void forward_start(const Place<NB>& at, const float2* st, const Axis& a, Pair (&x)[NB]) {
  const DF zero{0.f, 0.f};
  auto sample = [&](int m) {
    const float2 v = st[(at.vec << at.L) + m];
    return DF{v.x, v.y};
  };
  const int m = brev(at.p, at.L), h = at.n >> 1, q = at.n >> 2;
  if (NB == 1 && at.L == 1) {
    const DF u = sample(0), v = sample(1);
    x[0] = Pair{{df_add(u, v), zero}, {df_sub(u, v), zero}};
    return;
  }
  const int m0 = NB == 1 ? m & ~q : m;
  const DF u0 = sample(m0), u1 = sample(m0 + h), v0 = sample(m0 + q), v1 = sample(m0 + h + q);
#pragma unroll
  for (int r = 0; r < NB; ++r) {
    const bool odd = NB == 2 ? r == 1 : (at.p >> 1) & 1;   // position bit 0 after stage 0
    const DF u = odd ? df_sub(u0, u1) : df_add(u0, u1), v = odd ? df_sub(v0, v1) : df_add(v0, v1);
    const CDF w = cdf_load(a.tw[odd ? q : 0]);
    const CDF t{df_mul(v, w.re), df_mul(v, w.im)};
    x[r].a = CDF{df_add(u, t.re), t.im};
    x[r].b = CDF{df_sub(u, t.re), df_neg(t.im)};
  }
}
// X_k = Re(post_k V_k)
__device__ __forceinline__ DF coef(const Axis& a, const CDF& v, int k) {
  const CDF p = cdf_load(a.post[k]);
  return df_sub(df_mul(p.re, v.re), df_mul(p.im, v.im));
}

// Stage 0 of an inverse transform: the coefficients X_k / s_k staged (st[vec *
// stride + pad_k(k)]); at the end sample unmak(m) of the vector is Re F_m / n.
template <int NB>
__device__ __forceinline__ void inverse_start(const Place<NB>& at, const float2* st, int stride, const Axis& a,
                                              Pair (&x)[NB]) {
  const float2* v = st + at.vec * stride;
  auto w = [&](int k) {
    const float2 c = v[pad_k(k)];
    DF cn{0.f, 0.f};
    if (k) {
      const float2 r = v[pad_k(at.n - k)];
      cn = DF{r.x, r.y};
    }
    return cdf_mul(cdf_load(a.pre[k]), CDF{DF{c.x, c.y}, cn});
  };
  const int m = brev(at.p, at.L);
#pragma unroll
  for (int r = 0; r < NB; ++r) {
    const int k = m + r * (at.n >> 2);
    const CDF u = w(k), t = w(k + (at.n >> 1));
    x[r].a = CDF{df_add(u.re, t.re), df_add(u.im, t.im)};   // stage 0: twiddle one
    x[r].b = CDF{df_sub(u.re, t.re), df_sub(u.im, t.im)};
  }
}
// an inverse output times 1/n (a power of two)
__device__ __forceinline__ DF out_sample(const CDF& v, float inv_n) { return df_scale(v.re, inv_n); }
// t1 / t2 as double-float grids
__device__ __forceinline__ float2* df_grid(float* g) { return reinterpret_cast<float2*>(g); }
__device__ __forceinline__ DF df_at(const float* g, size_t i) {
  const float2 v = reinterpret_cast<const float2*>(g)[i];
  return DF{v.x, v.y};
}
// the staged copies: NB = 1 has two (one filled while the other may still be
// read by a vector of one or two warps, whose transforms cross no block
// barrier), NB = 2 one (its exchanges' barriers lie between)
template <int NB>
constexpr int kStageIn = 2 * (NB == 1 ? 512 : 1024);         // first float2 slot
template <int NB>
constexpr int kStageOut = kStageIn<NB> + (NB == 1 ? kStage : 0);
__device__ __forceinline__ float2* staged(float4* buf, int slot) { return reinterpret_cast<float2*>(buf) + slot; }

// The transform of a group's `vectors` staged vectors, from slot `src` to slot
// `dst` of the buffer:
//   FORWARD  samples (Makhoul's order) -> coefficients (four apart)
//   SCALED   the same, the coefficients times `ie` (1 / eigenvalue) and 1 / s_k
//   INVERSE  coefficients over s_k -> samples (eight apart), times 1/n
enum Direction { FORWARD, SCALED, INVERSE };
template <int NB, class G>
__device__ __forceinline__ void transform(const G& g, const Axis& a, int direction, int vectors, float4* buf, int src,
                                          int dst, const float (&ie)[2 * NB]) {
  const Place<NB> at(g.tid, a.logn);
  const bool mine = at.vec < vectors;   // fewer vectors than a group holds
  const int from = direction == INVERSE ? 1 : 2;   // the first stage after an exchange
  if (!__any_sync(0xffffffffu, mine)) {   // only the barriers of the exchanges between warps
#pragma unroll 1
    for (int s = from; s < at.L; ++s)
      if (crosses_warps<NB>(at, s)) g.sync();
    return;
  }
  Place<NB> pl = at;
  if (!mine) pl.vec = 0;                // idle threads of a warp that works trade what is not kept
  const int stride = pad_k(a.n), h = a.n >> 1;
  const float2* in = staged(buf, src);
  float2* out = staged(buf, dst);
  Pair x[NB];
  if (direction == INVERSE)
    inverse_start(pl, in, stride, a, x);
  else
    forward_start(pl, in, a, x);
  stages(g, pl, from, x, a, buf);
  if (!mine) return;
  if (direction == INVERSE) {
    const int ostride = pad_i(a.n);
    const float inv_n = __int_as_float((127 - a.logn) << 23);   // 2^-logn
#pragma unroll
    for (int r = 0; r < NB; ++r) {
      const int m = out_index(at, r);
      const DF v0 = out_sample(x[r].a, inv_n), v1 = out_sample(x[r].b, inv_n);
      out[at.vec * ostride + pad_i(unmak(m, a.n))] = make_float2(v0.hi, v0.lo);
      out[at.vec * ostride + pad_i(unmak(m + h, a.n))] = make_float2(v1.hi, v1.lo);
    }
  } else {
#pragma unroll
    for (int r = 0; r < NB; ++r) {
      const int k = out_index(at, r);
      DF c0 = coef(a, x[r].a, k), c1 = coef(a, x[r].b, k + h);
      if (direction == SCALED) {
        const float2 s0 = a.inv_s[k], s1 = a.inv_s[k + h];
        c0 = df_mul(df_mul(c0, DF{ie[2 * r], 0.f}), DF{s0.x, s0.y});
        c1 = df_mul(df_mul(c1, DF{ie[2 * r + 1], 0.f}), DF{s1.x, s1.y});
      }
      out[at.vec * stride + pad_k(k)] = make_float2(c0.hi, c0.lo);
      out[at.vec * stride + pad_k(k + h)] = make_float2(c1.hi, c1.lo);
    }
  }
}
// The passes take the transform as a callable, `run(g, axis, direction,
// vectors, buf, src, dst, ie)`: the standalone kernels have it inlined, with
// its direction known; the persistent loop shares one copy among its passes.
struct Inlined {
  template <int NB, class G>
  __device__ __forceinline__ void run(const G& g, const Axis& a, Direction direction, int vectors, float4* buf, int src,
                                      int dst, const float (&ie)[2 * NB]) const {
    transform<NB>(g, a, direction, vectors, buf, src, dst, ie);
  }
};

// Pass 1: t1 = rows-DCT(rho). With `mean` (fixed-point mean per field) the
// density preparation is folded in: rho = (phys + fill - mean) 2^-32 enters
// the transform exactly (EXACT, as a double-float) or as the FP32 value that
// is stored, and the physical overflow is counted into the IS_OVERFLOW /
// IS_OVER_BINS partials.
template <int NB, bool EXACT, class G, class T>
static __device__ __forceinline__ void rows_fwd(const G& g, const Dev& d, Partials p, int vb, int nvb, float4* buf,
                                                Shared& sh, const long long* mean, bool tables, int spread, const T& dct) {
  const int W = d.g.Wb, L = d.logW;
  const Groups grp(L, d.logH, d.K, spread);
  const int GV = grp.vectors(), per = GV << L, groups = grp.count(d.K);
  const Axis a = vb < groups ? stage_tables(g, axis_x(d), buf, tables) : axis_x(d);
  const int stride = pad_k(W);
  float2 *in = staged(buf, kStageIn<NB>), *out = staged(buf, kStageOut<NB>);
  long long ov[kMaxFields], cnt[kMaxFields];
#pragma unroll
  for (int f = 0; f < kMaxFields; ++f) ov[f] = cnt[f] = 0;
#pragma unroll 1
  for (int t = vb; t < groups; t += nvb) {
    const int f = grp.field(t), y0 = grp.first(t);
    const size_t base = (size_t)f * d.B + (size_t)y0 * W;
    g.sync();   // earlier readers of the buffer are done
    long long o = 0, c = 0;
#pragma unroll
    for (int q = 0; q < 2 * NB; ++q) {
      const int e = g.tid + q * kThreads;
      if (e < per) {
        DF x;
        if (!mean) {
          x = DF{d.rho[base + e], 0.f};
        } else {
          const long long ph = d.phys[base + e];
          const long long v = ph + d.fill[base + e] - mean[f];
          const float rho = __ll2float_rn(v) * kInvFixF;
          d.rho[base + e] = rho;
          if (ph > 0) {
            o += ph;
            c += 1;
          }
          x = EXACT ? df_scale(df_from_ll(v), kInvFixF) : DF{rho, 0.f};
        }
        in[(e & ~(W - 1)) + mak(e & (W - 1), W)] = make_float2(x.hi, x.lo);
      }
    }
#pragma unroll
    for (int ff = 0; ff < kMaxFields; ++ff)
      if (ff == f) {
        ov[ff] += o;
        cnt[ff] += c;
      }
    g.sync();
    const float none[2 * NB] = {};
    dct.template run<NB>(g, a, FORWARD, GV, buf, kStageIn<NB>, kStageOut<NB>, none);
    g.sync();
#pragma unroll
    for (int q = 0; q < 2 * NB; ++q) {
      const int e = g.tid + q * kThreads;
      if (e < per) df_grid(d.t1)[base + e] = out[(e >> L) * stride + pad_k(e & (W - 1))];
    }
  }
  if (mean)
#pragma unroll
    for (int f = 0; f < kMaxFields; ++f)
      if (f < d.K) {
        write_partial(g, ov[f], islot(p, IS_OVERFLOW + f), vb, sh.l);
        write_partial(g, cnt[f], islot(p, IS_OVER_BINS + f), vb, sh.l);
      }
}

// Pass 2: t2 = cols-IDCT(cols-DCT(t1) * inv_eig), whole columns per group;
// the scaled coefficients stay double-floats between the two transforms.
template <int NB, class G, class T>
static __device__ __forceinline__ void cols(const G& g, const Dev& d, int vb, int nvb, float4* buf, bool tables, int spread,
                                            const T& dct) {
  const int W = d.g.Wb, H = d.g.Hb, L = d.logH;
  const Groups grp(L, d.logW, d.K, spread);
  const int GV = grp.vectors(), per = GV << L, groups = grp.count(d.K);
  const Axis a = vb < groups ? stage_tables(g, axis_y(d), buf, tables) : axis_y(d);
  const Place<NB> at(g.tid, L);
  const int logG = grp.log_vectors;
  float2* in = staged(buf, kStageIn<NB>);
#pragma unroll 1
  for (int t = vb; t < groups; t += nvb) {
    const int f = grp.field(t), x0 = grp.first(t);
    const size_t base = (size_t)f * d.B + x0;
    g.sync();   // earlier readers of the buffer are done
#pragma unroll
    for (int q = 0; q < 2 * NB; ++q) {   // neighbouring columns read together
      const int e = g.tid + q * kThreads, v = e & (GV - 1), y = e >> logG;
      if (e < per) in[(v << L) + mak(y, H)] = df_grid(d.t1)[base + (size_t)y * W + v];
    }
    const int column = x0 + (at.vec < GV ? at.vec : 0);
    float ie[2 * NB];   // in flight while the samples are staged
#pragma unroll
    for (int r = 0; r < NB; ++r) {
      const int k = out_index(at, r);
      ie[2 * r] = d.inv_eig[(size_t)k * W + column];
      ie[2 * r + 1] = d.inv_eig[(size_t)(k + (H >> 1)) * W + column];
    }
    g.sync();
    dct.template run<NB>(g, a, SCALED, GV, buf, kStageIn<NB>, kStageOut<NB>, ie);
    g.sync();
    dct.template run<NB>(g, a, INVERSE, GV, buf, kStageOut<NB>, kStageIn<NB>, ie);
    const int ostride = pad_i(H);
    g.sync();
#pragma unroll
    for (int q = 0; q < 2 * NB; ++q) {
      const int e = g.tid + q * kThreads, v = e & (GV - 1), y = e >> logG;
      if (e < per) df_grid(d.t2)[base + (size_t)y * W + v] = in[v * ostride + pad_i(y)];
    }
  }
}

// Pass 3: phi = rows-IDCT(t2) and the energy partials <rho, phi>.
template <int NB, class G, class T>
static __device__ __forceinline__ void rows_inv(const G& g, const Dev& d, Partials p, int vb, int nvb, float4* buf,
                                                Shared& sh, bool tables, const T& dct) {
  const int W = d.g.Wb, L = d.logW;
  const Groups grp(L, d.logH, d.K, 0);   // fixed: the energy's partials are a group's sums
  const int GV = grp.vectors(), per = GV << L, groups = grp.count(d.K);
  const Axis a = vb < groups ? stage_tables(g, axis_x(d), buf, tables) : axis_x(d);
  const int stride = pad_k(W), ostride = pad_i(W);
  float2 *mid = staged(buf, kStageIn<NB>), *out = staged(buf, kStageOut<NB>);
  double eacc[kMaxFields] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
  for (int t = vb; t < groups; t += nvb) {
    const int f = grp.field(t), y0 = grp.first(t);
    const size_t base = (size_t)f * d.B + (size_t)y0 * W;
    float rho[2 * NB];
    g.sync();   // earlier readers of the buffer are done
#pragma unroll
    for (int q = 0; q < 2 * NB; ++q) {
      const int e = g.tid + q * kThreads;
      if (e < per) {
        const int k = e & (W - 1);
        const float2 s = a.inv_s[k];
        const DF c = df_mul(df_at(d.t2, base + e), DF{s.x, s.y});
        mid[(e >> L) * stride + pad_k(k)] = make_float2(c.hi, c.lo);
        rho[q] = d.rho[base + e];
      }
    }
    g.sync();
    const float none[2 * NB] = {};
    dct.template run<NB>(g, a, INVERSE, GV, buf, kStageIn<NB>, kStageOut<NB>, none);
    g.sync();
#pragma unroll
    for (int q = 0; q < 2 * NB; ++q) {
      const int e = g.tid + q * kThreads;
      if (e < per) {
        const float2 c = out[(e >> L) * ostride + pad_i(e & (W - 1))];
        const float v = df_float(DF{c.x, c.y});
        d.phi[base + e] = v;
#pragma unroll
        for (int ff = 0; ff < kMaxFields; ++ff)
          if (ff == f) eacc[ff] += (double)(rho[q] * v);
      }
    }
  }
#pragma unroll
  for (int f = 0; f < kMaxFields; ++f)
    if (f < d.K) write_partial(g, eacc[f], pslot(p, SLOT_ENERGY + f), vb, sh.d);
}

}  // namespace fft
}  // namespace tgp
