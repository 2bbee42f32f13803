// Weighted sum of materialised integrand values: acc[s] += sum_i w_i f[i][s]
// over a range of a tensor-product grid's nodes (or plain sums, for Monte
// Carlo).  It replaces the weight multiply of base_integrator.py:77-89 and
// the per-dimension collapse of grid_integrator.py:57-91, and the sum of
// monte_carlo.py:77.
//
// One value per node of a grid: the nodes are walked as rows (the last m
// dimensions joined, so that a row has at least 32 nodes; the other
// dimensions' weights are one factor per row).  A warp takes segments of
// rows; its lanes read consecutive values, sum them with the row's inner
// weights and fold the outer weight in once per segment.  On GB300 an FP64
// warp instruction holds a sub-partition's FP64 unit for about 64 cycles,
// longer than the loads and all other work of a value, so:
//   fp64 values   pairs of a lane's values added in fp64, the sums of pairs as
//                 double-floats (one weight a lane), or one FP64 fused
//                 multiply-add a value (Gauss weights, joined rows), groups of
//                 up to 32 values of a lane then added exactly
//   fp32 values   a compensated fp32 sum per segment and a double-float sum
//                 of the segments, no FP64 instruction per value
// Monte Carlo, and several values per node (vector integrands): sums that
// keep every bit of the terms, in each lane, without FP64 additions:
//   fp64 terms    added as 128-bit integers (FixAcc: about 35 integer
//                 instructions; a compensated fp64 sum has 8 FP64 ones)
//   fp32 terms    an exact product with the double-float weight, into three
//                 floats (F3Acc)
// For vector integrands a lane belongs to one component, a warp reads 32
// consecutive components (or as many nodes as fit), and a second launch adds
// the CTAs' partials, one warp per component.  The lanes' sums are added
// exactly (fixed point, tq_common.cuh).
//
// Measured (GB300), before and after: 301^3 fp64 values 96 us (double-floats
// split from each value, 75 instructions a value) and 58 us (3.7 TB/s); 301^3
// fp32 77 and 43 us; 15^6 fp64 475 and 45 us (outer weights per value strip);
// 10001 nodes x 200 components fp32 969 and 26 us (one component per thread
// and node group: uncoalesced, eight FP64 operations a value); 10^6 Monte
// Carlo values fp64 96 and 14 us.

#include <type_traits>

#include "tq_grid_common.cuh"
#include "tq_ranges.cuh"

namespace tq {

constexpr int kJoin = 2048;   // inner weights a CTA keeps when several dimensions are joined
constexpr int kPairMax = 2048;  // longest row of the double-float sums of fp64 values
constexpr int kComps = 32;    // components per warp of the vector kernel

struct WsumArgs {
  int rule, dim;
  int m;                  // joined inner dimensions
  int64_t n, n_values;
  RowWalk w;              // the range; a row has n^m nodes (Monte Carlo: all of them)
  int chunk;              // components per CTA (vector kernel)
  const void* domain;
  const double* gl_weights;
  const void* f;
  double* acc;   // running sums [n_values][2] (out == nullptr)
  void* out;     // or the results themselves, of out_dtype
  int out_dtype;
  Acc* partials;
  unsigned* ticket;
};

// Sum t of component s into the running sum, or as the result: times the
// domain's volume over the samples (monte_carlo.py:72-77, the volume in the
// domain's type) for Monte Carlo.
template <typename D>
__device__ __forceinline__ void wsum_store(const WsumArgs& a, int64_t s, Acc t) {
  if (!a.out) {
    Acc run{a.acc[2 * s], a.acc[2 * s + 1]};
    acc_merge(run, t);
    a.acc[2 * s] = run.s;
    a.acc[2 * s + 1] = run.c;
    return;
  }
  double v = t.s + t.c;
  if (a.rule == TQ_RULE_MC) {
    const D* dom = (const D*)a.domain;
    D vol = (D)1;
    for (int k = 0; k < a.dim; ++k) vol = vol * (D)(dom[2 * k + 1] - dom[2 * k]);
    v *= (double)vol / (double)a.w.count;
  }
  if (a.out_dtype == TQ_F64)
    ((double*)a.out)[s] = v;
  else
    ((float*)a.out)[s] = (float)v;
}

// Inner weights.  One dimension: a lane's nodes keep their place modulo four
// as it strides over a segment, so a Newton-Cotes lane has one interior and
// one end weight; Gauss weights are read from their table.  Joined
// dimensions: a table of the products, made by the CTA.
template <typename F>
__device__ __forceinline__ F wsum_weight(int rule, int j, bool end) {
  if (rule == TQ_RULE_MC) return (F)1;
  if (rule == TQ_RULE_TRAPEZOID) return end ? (F)1 : (F)2;
  if (rule == TQ_RULE_SIMPSON) return end ? (F)1 : ((j & 1) ? (F)4 : (F)2);
  return end ? (F)7 : ((j & 1) ? (F)32 : ((j & 3) == 2 ? (F)12 : (F)14));
}
// 2^e, -1022 <= e <= 1023.
__device__ __forceinline__ double exp2i(int e) { return __hiloint2double((1023 + e) << 20, 0); }
// Joined whole-number weights are held 2^join_exp down, no larger than one
// dimension's.
__device__ __forceinline__ int join_exp(const WsumArgs& a) {
  const int bits = a.rule == TQ_RULE_TRAPEZOID ? 1 : a.rule == TQ_RULE_SIMPSON ? 2 : a.rule == TQ_RULE_BOOLE ? 5 : 0;
  return bits * (a.m - 1);
}
template <bool GL>
__device__ void wsum_join_table(const WsumArgs& a, double* tab) {
  const uint32_t n = (uint32_t)a.n;
  const double down = exp2i(-join_exp(a));
  for (int j = threadIdx.x; j < (int)a.w.R; j += blockDim.x) {
    uint32_t r = (uint32_t)j;
    double w = down;
    for (int k = 0; k < a.m; ++k) {
      const uint32_t q = r / n, digit = r - q * n;
      r = q;
      w *= GL ? __ldg(a.gl_weights + digit)
              : wsum_weight<double>(a.rule, (int)digit, digit == 0 || digit == n - 1);
    }
    tab[j] = w;
  }
}
// Outer weight of a row: the remaining dimensions' unscaled weights (whole
// numbers for the Newton-Cotes rules, exact as double-floats too).
template <bool GL>
__device__ __forceinline__ double wsum_outer(const WsumArgs& a, const FastDiv& fd, int64_t row) {
  double w = 1.0;
  const int n32 = (int)a.n;
  if (row <= (int64_t)0xffffffffll) {
    uint32_t r = (uint32_t)row;
    for (int k = a.dim - a.m - 1; k >= 0; --k) {
      const uint32_t q = fdiv(r, fd);
      const int d = (int)(r - q * fd.d);
      r = q;
      w *= GL ? __ldg(a.gl_weights + d) : wsum_weight<double>(a.rule, d, d == 0 || d == n32 - 1);
    }
  } else {
    uint64_t r = (uint64_t)row;
    for (int k = a.dim - a.m - 1; k >= 0; --k) {
      const uint64_t q = r / (uint64_t)a.n;
      const int64_t d = (int64_t)(r - q * (uint64_t)a.n);
      r = q;
      w *= GL ? __ldg(a.gl_weights + d) : wsum_weight<double>(a.rule, (int)(d & 3), d == 0 || d == a.n - 1);
    }
  }
  return w;
}

// A double split into two floats by integer operations alone (no FP64
// instruction; on GB300 conversions also occupy the FP64 unit): hi takes the
// sign, the exponent and the leading 24 significant bits (truncated), lo the
// remaining 29 bits rounded to 23, so |x - (hi + lo)| <= 2^-47 |x|, without
// bias.  lo comes from a float whose exponent is known, 2^(e-1046) + q
// 2^(e-1069) with q the rounded top 23 of the 29 bits, minus 2^(e-1046)
// (exact).  Branch-free.  Only 2^-40 <= |x| < 2^40 is split, so that
// weighted products and long sums of such values stay far inside the float
// range; otherwise hi = lo = 0, and ok is false unless x is a zero: other
// values (small, large, subnormal, infinite, NaN) are the caller's to
// handle in fp64.
struct F2Split {
  F2 v;
  bool ok;
};
__device__ __forceinline__ F2Split f2_split(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const uint32_t bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  const uint32_t em = bh & 0x7ff00000u;  // biased binary exponent e, << 20
  const uint32_t sgn = bh & 0x80000000u;
  F2Split r;
  const bool in = em - (983u << 20) <= (79u << 20) + 0xfffffu;  // 983 <= e <= 1062
  // bits 30..23: the low 8 bits of e, 22..0: fraction bits 51..29; the
  // float exponent e - 896 is those 8 bits with the top one flipped
  const uint32_t fs = __funnelshift_l(bl, bh, 3);
  const float hi = __uint_as_float(((fs ^ 0x40000000u) & 0x7fffffffu) | sgn);
  const uint32_t ex = em * 8u - (919u << 23);
  const uint32_t q = ((bl & 0x1fffffffu) + 32u) >> 6;  // a carry into the exponent stays exact
  const float lo = __fsub_rn(__uint_as_float(ex + q), __uint_as_float(ex));
  r.v.hi = in ? hi : 0.f;
  r.v.lo = in ? __uint_as_float(__float_as_uint(lo) | sgn) : 0.f;
  r.ok = in || ((bh & 0x7fffffffu) | bl) == 0u;
  return r;
}

// The rare terms that the double-float sums leave out, in fp64.  Not inlined
// and called behind votes: an FP64 instruction holds the FP64 unit even where
// its predicate is off in every lane.
__device__ __noinline__ void side_add(double* side, double w, double v) { *side = fma(w, v, *side); }

// A lane's sum of (weight x) value within one unit.
struct UnitSumD {  // fp64, weights that differ from node to node
  double s = 0.0;
  __device__ __forceinline__ void add(double w, double v) { s = fma(w, v, s); }
};
struct UnitSumF {  // fp32: Kahan's sum, the product fused into its first step
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float w, float v) {
    const float y = __fmaf_rn(w, v, -c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  }
};
// fp64 values of one weight, two at a time: they are added in fp64, their sum
// split into a double-float (47 of its 53 bits, rounded) and added on the
// FP32 pipe.  Half an FP64 addition and some 17 other instructions a value:
// both take less time than the value's bytes, where one FP64 operation a
// value (115 us at 301^3) or a split of every value (87 us) takes twice as
// long.  Returns false where the sum is outside the split's range (the
// caller adds it in fp64).
struct UnitSumP {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ bool add(double x) {
    const F2Split f = f2_split(x);
    const F2 t = two_sum(hi, f.v.hi);
    hi = t.hi;
    lo = __fadd_rn(lo, __fadd_rn(t.lo, f.v.lo));
    return f.ok;
  }
};

// A lane's sum over its units, each folded in with its outer weight w: in
// fp64, or as double-floats, with unit sums of 2^60 and more (and infinities
// and NaN) in the fp64 side sum.  In fp64, groups of up to 32 values of a lane
// are added plainly and the groups' sums exactly, by integers (a Neumaier
// pair's seven FP64 operations a group: 8e7 nodes 211 us, plain sums 177).
struct LaneSumD {
  double s = 0.0;
  FixAcc t;
  int k = 0;          // values in s; the same in the whole warp
  bool many = false;  // t holds groups
  __device__ __forceinline__ void fold(const UnitSumD& u, int n, double w, F2, double*) {
    if (k + n > 32) {
      t.add(s);
      many = true;
      s = 0.0;
      k = 0;
    }
    s = fma(u.s, w, s);
    k += n;
  }
  __device__ __forceinline__ Acc value() const {
    if (!many) return Acc{s, 0.0};
    Acc r = t.value();
    acc_add(r, s);
    return r;
  }
};
struct LaneSumF {
  F2 s{0.f, 0.f};
  __device__ __forceinline__ void fold(const UnitSumF& u, int, double w, F2 wf, double* side) {
    const bool in = fabsf(u.s) < 0x1p60f;
    if (in) s = f2_add(s, f2_mul(two_sum(u.s, -u.c), wf));
    if (__any_sync(0xffffffffu, !in)) side_add(side, in ? 0.0 : w, in ? 0.0 : (double)u.s - (double)u.c);
  }
  __device__ __forceinline__ void fold(const UnitSumP& u, int, double, F2 wf, double*) {
    s = f2_add(s, f2_mul(two_sum(u.hi, u.lo), wf));
  }
  __device__ __forceinline__ Acc value() const { return Acc{(double)s.hi, (double)s.lo}; }
};

// Exact running sums of a lane (Monte Carlo and vector integrands): FixAcc
// (tq_common.cuh) for fp64 terms; for fp32 terms
// F3Acc: fp32 terms hi + lo (a product and its rounding error) into three
// floats, every rounding kept down to the third.
struct F3Acc {
  float a = 0.f, b = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float hi) {
    const F2 t = two_sum(a, hi), u = two_sum(b, t.lo);
    a = t.hi;
    b = u.hi;
    c = __fadd_rn(c, u.lo);
  }
  __device__ __forceinline__ void add(float hi, float lo) {
    add(hi);
    const F2 u = two_sum(b, lo);
    b = u.hi;
    c = __fadd_rn(c, u.lo);
  }
  __device__ __forceinline__ void value(Acc& r, double unit) const {  // unit: a power of two
    acc_add(r, (double)a * unit);
    acc_add(r, ((double)b + (double)c) * unit);
  }
};
// A lane's exact sum of weight x value.  fp32: values below 2^-60 go into a
// sum of their own, scaled up (products of theirs would lose their last bits
// below the float range), values of 2^50 and more, infinities and NaN into an
// fp64 sum; the weight is a double-float.
template <typename F>
struct ExactSum;
template <>
struct ExactSum<double> {
  FixAcc s;
  __device__ __forceinline__ void add(double v) { s.add(v); }
  __device__ __forceinline__ void add(double w, F2, double v) { s.add(w * v); }
  __device__ __forceinline__ Acc value() const { return s.value(); }
};
template <>
struct ExactSum<float> {
  F3Acc s, small;
  Acc side{0.0, 0.0};
  __device__ __forceinline__ void add(float v) {
    if (fabsf(v) < 0x1p50f)
      s.add(v);  // sums of values themselves lose nothing below the float range
    else
      acc_add(side, (double)v);
  }
  __device__ __forceinline__ void add(double w, F2 wf, float v) {
    if (fabsf(v) < 0x1p50f) {
      const bool tiny = fabsf(v) < 0x1p-60f;
      const float x = tiny ? v * 0x1p96f : v;
      const float p = __fmul_rn(wf.hi, x);
      const float e = __fmaf_rn(wf.lo, x, __fmaf_rn(wf.hi, x, -p));
      if (tiny)
        small.add(p, e);
      else
        s.add(p, e);
    } else {
      acc_add(side, w * (double)v);
    }
  }
  __device__ __forceinline__ Acc value() const {
    Acc r = side;
    s.value(r, 1.0);
    if (small.a != 0.f || small.b != 0.f || small.c != 0.f) small.value(r, 0x1p-96);
    return r;
  }
};

// Shared set-up of the kernels: the join table, and the product of the
// dimensions' weight scales.  Its power of two (with that of the join table)
// goes into the rows' outer weights of fp64 sums and the lanes' sums of others
// (exact; sums of unscaled terms could leave the range of doubles where the
// integral does not).  The rest, between one and 2^dim, multiplies a CTA's
// sums at the very end, so its rounding is the same for all nodes: a pair, by
// a warp of its own while the others read; visible from the next barrier on.
struct WsumSetup {
  double pow2;
  Acc scale;
  FastDiv fd;
};
// v s for unevaluated pairs
__device__ __forceinline__ Acc wsum_scaled(Acc v, Acc s) {
  const double p = v.s * s.s;
  return Acc{p, fma(v.c, s.s, fma(v.s, s.c, fma(v.s, s.s, -p)))};
}
__device__ __forceinline__ int scale_exp(double w) {
  const int f = exp_field(w);
  return f == 0 || f == 0x7ff ? 0 : min(f - 1023, 1022);
}
template <typename T, typename D, bool GL, bool JOIN>
__device__ __forceinline__ void wsum_setup(const WsumArgs& a, Geo<T>& g, WsumSetup& su, double* tab) {
  geo_setup<T, D>(g, a.rule, a.dim, a.n, (const D*)a.domain);
  if constexpr (JOIN) wsum_join_table<GL>(a, tab);
  if (threadIdx.x < 32) {
    const int e = __reduce_add_sync(0xffffffffu, threadIdx.x < a.dim ? scale_exp(g.wscale[threadIdx.x]) : 0);
    if (threadIdx.x == 0) {
      su.pow2 = exp2i(max(-900, min(900, e)) + (JOIN ? join_exp(a) : 0));
      su.fd = make_fastdiv((uint32_t)a.n);
    }
  }
  __syncthreads();
  if (threadIdx.x == kBlock - 32) {
    Acc s{1.0, 0.0};
    int sum = 0;
    for (int k = 0; k < a.dim; ++k) {
      const int e = scale_exp(g.wscale[k]);
      sum += e;
      s = wsum_scaled(s, Acc{g.wscale[k] * exp2i(-e), 0.0});
    }
    const int left = sum - max(-900, min(900, sum));
    if (left) s = Acc{scalbn(s.s, left), scalbn(s.c, left)};
    su.scale = s;
  }
}

// The CTAs' sums into the running sum or the result, by the last of them.
template <typename D>
__device__ __forceinline__ void wsum_finish(const WsumArgs& a, Acc mine, const Acc& scale) {
  const Acc acc = block_reduce<kBlock>(mine);
  if (threadIdx.x == 0) a.partials[blockIdx.x] = wsum_scaled(acc, scale);
  if (last_block_arrives(a.ticket)) {
    const Acc t = partials_reduce<kBlock>(a.partials, (int)gridDim.x);
    if (threadIdx.x == 0) {
      wsum_store<D>(a, 0, t);
      *a.ticket = 0u;
    }
  }
}

// One value per node of a grid.  PAIR: the double-float sums of fp64 values
// (one-dimensional Newton-Cotes rows).
template <typename T, typename D, bool GL, bool JOIN, typename F, bool PAIR>
__global__ void __launch_bounds__(kBlock, 4) weighted_sum_kernel(WsumArgs a) {
  __shared__ Geo<T> g;
  __shared__ WsumSetup su;
  __shared__ double tab[JOIN ? kJoin : 1];
  wsum_setup<T, D, GL, JOIN>(a, g, su, tab);
  constexpr bool F32 = std::is_same<F, float>::value;
  // one-dimensional Newton-Cotes rows: a segment starts at a multiple of
  // four, so a lane's nodes have one interior weight, which its sum takes at
  // the very end; the rows' end nodes (half of it) are corrected row by row,
  // one row a lane
  constexpr bool ONE = !GL && !JOIN;
  static_assert(!PAIR || (ONE && !F32), "pairs share a weight");
  using Unit = typename std::conditional<F32, UnitSumF, typename std::conditional<PAIR, UnitSumP, UnitSumD>::type>::type;
  typename std::conditional<F32 || PAIR, LaneSumF, LaneSumD>::type sum;
  double side = 0.0, ends = 0.0;  // terms left out of the sum; the end nodes' surplus
  const F* __restrict__ f = (const F*)a.f;
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = (int64_t)gridDim.x * (kBlock / 32);
  const int64_t gw = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const int64_t units = a.w.units, start = a.w.start, end = start + a.w.count;
  const int64_t ub = gw * units / nwarps, ue = (gw + 1) * units / nwarps;
  const double wi = wsum_weight<double>(a.rule, lane, false);
  for (int64_t u0 = ub; u0 < ue; u0 += 32) {
    const int cnt = (int)min((int64_t)32, ue - u0);
    double wu = 0.0, w = 0.0;  // outer weight of unit u0 + lane, without and with the scales' power of two
    if (lane < cnt) {
      const RowPart pt = row_part(a.w, u0 + lane);
      wu = wsum_outer<GL>(a, su.fd, a.w.row0 + pt.row);
      w = wu * su.pow2;
      if (ONE) {
        const int64_t p0 = pt.r0, p1 = p0 + a.w.R - 1;
        double e = 0.0;
        if (pt.j0 == 0 && p0 >= start && p0 < end) e = (double)__ldg(f + (p0 - start));
        if (pt.j0 + a.w.seg >= a.w.R && p1 >= start && p1 < end) e += (double)__ldg(f + (p1 - start));
        ends = fma(-0.5 * wsum_weight<double>(a.rule, 0, false) * e, w, ends);
      }
    }
    F2 wf{0.f, 0.f};
    if (F32 || PAIR) wf = f2_from_double(wu);
    for (int q = 0; q < cnt; ++q) {
      const RowPart pt = row_part(a.w, u0 + q);
      const int64_t j0 = pt.j0;
      const int lo = pt.lo, len = pt.len;
      const F* fr = f + (pt.r0 - start) + j0 + lane;
      const double wq = __shfl_sync(0xffffffffu, w, q);
      Unit us;
      // N values a lane from offset i
      auto batch = [&](int i, auto full, auto count) {
        constexpr bool FULL = decltype(full)::value;
        constexpr int N = decltype(count)::value;
        F v[N];
#pragma unroll
        for (int p = 0; p < N; ++p) {
          const int o = i + 32 * p + lane;
          v[p] = (FULL || (o >= lo && o < len)) ? __ldg(fr + i + 32 * p) : (F)0;
        }
        if constexpr (PAIR) {
          double x[N / 2];
          bool in[N / 2], all = true;
#pragma unroll
          for (int p = 0; p < N / 2; ++p) {
            x[p] = v[2 * p] + v[2 * p + 1];
            in[p] = us.add(x[p]);
            all = all && in[p];
          }
          if (__any_sync(0xffffffffu, !all)) {
#pragma unroll
            for (int p = 0; p < N / 2; ++p) side_add(&side, wq, in[p] ? 0.0 : x[p]);
          }
        } else {
#pragma unroll
          for (int p = 0; p < N; ++p) {
            [[maybe_unused]] const int o = i + 32 * p + lane;
            F wj = (F)1;
            if constexpr (JOIN)
              wj = FULL || o < len ? (F)tab[(int)j0 + o] : (F)0;
            else if constexpr (GL)
              wj = FULL || o < len ? (F)__ldg(a.gl_weights + j0 + o) : (F)0;
            us.add(wj, v[p]);
          }
        }
      };
      int i = 0;
      if (lo == 0)
        for (; i + 256 <= len; i += 256) batch(i, std::true_type{}, std::integral_constant<int, 8>{});
      if (i < len && len - i > 128) {
        batch(i, std::false_type{}, std::integral_constant<int, 8>{});
        i += 256;
      } else if (i < len && len - i > 64) {
        batch(i, std::false_type{}, std::integral_constant<int, 4>{});
        i += 128;
      }
      for (; i < len; i += 64) batch(i, std::false_type{}, std::integral_constant<int, 2>{});
      F2 wqf{0.f, 0.f};
      if (F32 || PAIR) wqf = F2{__shfl_sync(0xffffffffu, wf.hi, q), __shfl_sync(0xffffffffu, wf.lo, q)};
      sum.fold(us, (len - lo + 31) / 32, wq, wqf, &side);  // at most so many values a lane
    }
  }
  Acc r = sum.value();
  if (F32 || PAIR) {
    r.s *= su.pow2;
    r.c *= su.pow2;
  }
  if (side != 0.0) acc_add(r, side);
  if (ONE) {  // the lane's weight (a small integer), then the end nodes
    r.s *= wi;
    r.c *= wi;
    acc_add(r, ends);
  }
  wsum_finish<D>(a, r, su.scale);
}

// Monte Carlo samples of one value: their plain sum.
template <typename D, typename F>
__global__ void __launch_bounds__(kBlock, 4) sample_sum_kernel(WsumArgs a) {
  const F* __restrict__ f = (const F*)a.f;
  const int64_t step = (int64_t)gridDim.x * kBlock;
  ExactSum<F> sum;
  int64_t i = (int64_t)blockIdx.x * kBlock + threadIdx.x;
  for (; i + 7 * step < a.w.count; i += 8 * step) {
    F v[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) v[p] = __ldg(f + i + p * step);
#pragma unroll
    for (int p = 0; p < 8; ++p) sum.add(v[p]);
  }
  for (; i < a.w.count; i += step) sum.add(__ldg(f + i));
  wsum_finish<D>(a, sum.value(), Acc{1.0, 0.0});
}

// Several values per node: lane = component + chunk * node, partials[CTA of
// x][component].  The nodes go in batches of as many as the lanes hold; a
// batch's weights are computed one node per lane and handed round.
template <typename T, typename D, bool GL, bool JOIN, typename F>
__global__ void __launch_bounds__(kBlock, 4) weighted_sum_vec_kernel(WsumArgs a) {
  __shared__ Geo<T> g;
  __shared__ WsumSetup su;
  __shared__ double tab[JOIN ? kJoin : 1];
  __shared__ Acc part[kBlock];
  wsum_setup<T, D, GL, JOIN>(a, g, su, tab);
  constexpr bool F32 = std::is_same<F, float>::value;
  const bool mc = a.rule == TQ_RULE_MC;
  const int64_t S = a.n_values;
  const int64_t s0 = (int64_t)blockIdx.y * a.chunk;
  const int ncomp = (int)min((int64_t)a.chunk, S - s0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = 32 / ncomp;        // nodes a warp reads at once
  const int batch = 32 / per * per;  // nodes of a batch
  const int sub = lane / ncomp, comp = lane - sub * ncomp;
  const F* __restrict__ f = (const F*)a.f + s0 + comp;
  const int64_t nwarps = (int64_t)gridDim.x * (kBlock / 32);
  const int64_t units = a.w.units;
  const double up = F32 ? 1.0 : su.pow2;
  ExactSum<F> sum;
  for (int64_t u = (int64_t)warp * gridDim.x + blockIdx.x; u < units; u += nwarps) {
    const RowPart pt = row_part(a.w, u);
    const int64_t j1 = pt.j0 + pt.len;
    const double wo = mc ? 1.0 : wsum_outer<GL>(a, su.fd, a.w.row0 + pt.row) * up;
    for (int64_t jb = pt.j0 + pt.lo; jb < j1; jb += batch) {
      const int nb = (int)min((int64_t)batch, j1 - jb);
      double w = 0.0;  // weight of the batch's node `lane`
      F2 wf{0.f, 0.f};
      if (!mc) {
        const int64_t j = jb + min(lane, nb - 1);
        w = wo * (JOIN ? tab[j] : GL ? __ldg(a.gl_weights + j)
                                     : wsum_weight<double>(a.rule, (int)(j & 3), j == 0 || j == a.w.R - 1));
        if (F32) wf = f2_from_double(w);
      }
      const F* fr = f + (pt.r0 - a.w.start + jb) * S;
      for (int i = 0; i < nb; i += 8 * per) {
        F v[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          const int o = i + p * per + sub;
          v[p] = (sub < per && o < nb) ? __ldg(fr + (int64_t)o * S) : (F)0;
        }
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          const int o = min(i + p * per + sub, 31);
          if (i + p * per >= nb) break;
          if (mc) {
            sum.add(v[p]);
          } else {
            const double wq = __shfl_sync(0xffffffffu, w, o);
            F2 wqf{0.f, 0.f};
            if (F32) wqf = F2{__shfl_sync(0xffffffffu, wf.hi, o), __shfl_sync(0xffffffffu, wf.lo, o)};
            sum.add(wq, wqf, v[p]);
          }
        }
      }
    }
  }
  Acc r = sum.value();
  if (F32) r = Acc{r.s * su.pow2, r.c * su.pow2};
  part[threadIdx.x] = r;
  __syncthreads();
  const int entries = (kBlock / 32) * per;  // a component's lanes: warp e / per, node e % per
  for (int c = warp; c < ncomp; c += kBlock / 32) {
    const Acc t = warp_sum(entries, [&](int e) { return part[(e / per) * 32 + (e % per) * ncomp + c]; });
    if (lane == 0) a.partials[(int64_t)blockIdx.x * S + s0 + c] = mc ? t : wsum_scaled(t, su.scale);
  }
}

// The partials of component s added up, one warp per component.
template <typename D>
__global__ void __launch_bounds__(kBlock) weighted_sum_combine_kernel(WsumArgs a, int n) {
  const int64_t s = ((int64_t)blockIdx.x * kBlock + threadIdx.x) >> 5;
  if (s >= a.n_values) return;
  const Acc t = warp_sum(n, [&](int e) { return a.partials[(int64_t)e * a.n_values + s]; });
  if ((threadIdx.x & 31) == 0) wsum_store<D>(a, s, t);
}

template <typename D>
__global__ void finalize_kernel(int rule, int dim, const D* __restrict__ dom, int64_t npts,
                                const double* __restrict__ acc, int64_t S, void* out,
                                int out_dtype) {
  double scale = 1.0;
  if (rule == TQ_RULE_MC) {
    // monte_carlo.py:72-77: volume = prod(b - a) in the domain type
    D vol = (D)1;
    for (int k = 0; k < dim; ++k) vol = vol * (D)(dom[2 * k + 1] - dom[2 * k]);
    scale = (double)vol / (double)npts;
  }
  for (int64_t s = blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gridDim.x * blockDim.x) {
    const double v = scale * (acc[2 * s] + acc[2 * s + 1]);
    if (out_dtype == TQ_F64)
      ((double*)out)[s] = v;
    else
      ((float*)out)[s] = (float)v;
  }
}

}  // namespace tq

using namespace tq;

// CTAs over the nodes: up to four an SM, a warp having at least 128 nodes
// (vector integrands: 32).
static int64_t wsum_ctas(int64_t count, int64_t n_values) {
  const int64_t chunks = (n_values + kComps - 1) / kComps;
  const int64_t cap = ((int64_t)sm_count() * 4 + chunks - 1) / chunks;
  const int64_t per = (kBlock / 32) * (n_values == 1 ? 128 : 32);
  const int64_t need = (count + per - 1) / per;
  return need < 1 ? 1 : (need < cap ? need : cap);
}

// Partials that any workspace of this call has always held.
static int64_t wsum_least_slots(int64_t count, int64_t n_values) {
  int64_t need = (count + (int64_t)kBlock * 8 - 1) / ((int64_t)kBlock * 8);
  const int64_t cap = (int64_t)sm_count() * 8;
  need = need < 1 ? 1 : (need < cap ? need : cap);
  return need * ((n_values + 3) / 4) * 4;
}

extern "C" size_t tq_weighted_sum_workspace_size(int64_t count, int64_t n_values) {
  const int64_t a = wsum_least_slots(count, n_values), b = wsum_ctas(count, n_values) * n_values;
  return reduce_ws_bytes(a > b ? a : b);
}

static bool wsum_valid_rule(int rule, int64_t n) {
  switch (rule) {
    case TQ_RULE_TRAPEZOID:
    case TQ_RULE_GAUSS:
      return n >= 2;
    case TQ_RULE_SIMPSON:
      return n >= 3 && (n & 1) == 1;
    case TQ_RULE_BOOLE:
      return n >= 5 && (n - 1) % 4 == 0;
    default:
      return false;
  }
}

static int wsum_launch(int dtype, int rule, int dim, int64_t n_per_dim, const void* domain,
                       const double* gl_weights, int64_t start, int64_t count, const void* f, int f_dtype,
                       int64_t n_values, double* acc, void* out, int out_dtype, void* workspace,
                       size_t workspace_bytes, void* stream) {
  if (!valid_dtype(dtype) || !valid_dtype(f_dtype)) return TQ_ERR_DTYPE;
  if (dim < 1 || dim > kMaxDim) return TQ_ERR_DIM;
  if (rule != TQ_RULE_MC && !wsum_valid_rule(rule, n_per_dim)) return TQ_ERR_RULE;
  if (!domain || !f || (!acc && !out) || !workspace || start < 0 || count < 0 || n_values < 1)
    return TQ_ERR_ARG;
  if (rule == TQ_RULE_GAUSS && !gl_weights) return TQ_ERR_ARG;
  if (rule != TQ_RULE_MC) {
    int64_t total = 1;
    for (int k = 0; k < dim; ++k) {
      if (total > (int64_t(1) << 62) / n_per_dim) return TQ_ERR_TOO_LARGE;
      total *= n_per_dim;
    }
    if (start + count > total) return TQ_ERR_ARG;
  }
  if (count == 0) return TQ_OK;
  if ((n_values + 3) / 4 > 65535) return TQ_ERR_TOO_LARGE;
  if (workspace_bytes < reduce_ws_bytes(wsum_least_slots(count, n_values))) return TQ_ERR_WORKSPACE;
  const int64_t slots = (int64_t)((workspace_bytes - 256) / sizeof(Acc));
  WsumArgs a;
  a.rule = rule;
  a.dim = dim;
  a.n = n_per_dim;
  a.n_values = n_values;
  a.domain = domain;
  a.gl_weights = gl_weights;
  a.f = f;
  a.acc = acc;
  a.out = out;
  a.out_dtype = out_dtype;
  a.ticket = (unsigned*)workspace;
  a.partials = (Acc*)((char*)workspace + 256);
  const bool gl = rule == TQ_RULE_GAUSS, mc = rule == TQ_RULE_MC;
  // rows of at least 32 nodes: join the inner dimensions of short ones (a
  // lane would otherwise fold an outer weight in, in FP64, every few values)
  a.m = mc ? dim : 1;
  int64_t R = mc ? count : n_per_dim;
  if (mc) {  // one row of all the samples
    start = 0;
  } else {
    while (R < 32 && a.m < dim && R * n_per_dim <= kJoin) {
      R *= n_per_dim;
      ++a.m;
    }
  }
  const bool join = !mc && a.m > 1;
  // double-float sums where enough nodes share them that their 2^-47 of a term
  // is below the sum's own last bit; few nodes, and long rows, in fp64
  const bool pair = f_dtype == TQ_F64 && n_values == 1 && !mc && !gl && !join && n_per_dim >= 32 &&
                    n_per_dim <= kPairMax && (dim - 1) * n_per_dim <= kPairMax;
  int64_t gx = wsum_ctas(count, n_values);
  if (gx > slots / n_values) gx = slots / n_values;
  // segments: long (a lane's 32 values where its groups of fp64 values end),
  // unless that leaves warps without work
  const int64_t warps = gx * (kBlock / 32);
  const int64_t least = n_values == 1 ? 128 : 32;
  int64_t seg = f_dtype == TQ_F64 && n_values == 1 && !pair ? 1024 : 2048;
  while (seg / 2 >= least && make_walk(start, count, R, seg).units < warps) seg /= 2;
  a.w = make_walk(start, count, R, seg);
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t chunks = (n_values + kComps - 1) / kComps;
  a.chunk = (int)(n_values < kComps ? n_values : kComps);
  const dim3 grid((unsigned)gx, (unsigned)(n_values == 1 ? 1 : chunks));
  if (mc && n_values == 1) {
    if (dtype == TQ_F64) {
      if (f_dtype == TQ_F64) sample_sum_kernel<double, double><<<grid, kBlock, 0, s>>>(a);
      else sample_sum_kernel<double, float><<<grid, kBlock, 0, s>>>(a);
    } else {
      if (f_dtype == TQ_F64) sample_sum_kernel<float, double><<<grid, kBlock, 0, s>>>(a);
      else sample_sum_kernel<float, float><<<grid, kBlock, 0, s>>>(a);
    }
    return launch_status();
  }
  if (pair) {
    if (dtype == TQ_F64)
      weighted_sum_kernel<double, double, false, false, double, true><<<grid, kBlock, 0, s>>>(a);
    else
      weighted_sum_kernel<float, float, false, false, double, true><<<grid, kBlock, 0, s>>>(a);
    return launch_status();
  }
#define TQ_WSUM_F(T, D, GLB, JOINB, F)                                                   \
  if (n_values == 1)                                                                     \
    weighted_sum_kernel<T, D, GLB, JOINB, F, false><<<grid, kBlock, 0, s>>>(a);          \
  else                                                                                   \
    weighted_sum_vec_kernel<T, D, GLB, JOINB, F><<<grid, kBlock, 0, s>>>(a);
#define TQ_WSUM(T, D, GLB)                                                               \
  if (join) {                                                                            \
    if (f_dtype == TQ_F64) { TQ_WSUM_F(T, D, GLB, true, double) }                        \
    else { TQ_WSUM_F(T, D, GLB, true, float) }                                           \
  } else {                                                                               \
    if (f_dtype == TQ_F64) { TQ_WSUM_F(T, D, GLB, false, double) }                       \
    else { TQ_WSUM_F(T, D, GLB, false, float) }                                          \
  }
  if (gl) {
    if (dtype == TQ_F64) {
      TQ_WSUM(double, double, true)
    } else {
      TQ_WSUM(double, float, true)
    }
  } else if (dtype == TQ_F64) {
    TQ_WSUM(double, double, false)
  } else {
    TQ_WSUM(float, float, false)
  }
#undef TQ_WSUM
#undef TQ_WSUM_F
  if (n_values > 1) {
    const int e = launch_status();
    if (e != TQ_OK) return e;
    const unsigned cb = (unsigned)((n_values * 32 + kBlock - 1) / kBlock);
    if (dtype == TQ_F64)
      weighted_sum_combine_kernel<double><<<cb, kBlock, 0, s>>>(a, (int)gx);
    else
      weighted_sum_combine_kernel<float><<<cb, kBlock, 0, s>>>(a, (int)gx);
  }
  return launch_status();
}

extern "C" int tq_weighted_sum(int dtype, int rule, int dim, int64_t n_per_dim,
                               const void* domain, const double* gl_weights, int64_t start,
                               int64_t count, const void* f, int f_dtype, int64_t n_values,
                               double* acc, void* workspace, size_t workspace_bytes,
                               void* stream) {
  if (!acc && count > 0) return TQ_ERR_ARG;
  return wsum_launch(dtype, rule, dim, n_per_dim, domain, gl_weights, start, count, f, f_dtype, n_values, acc,
                     nullptr, TQ_F64, workspace, workspace_bytes, stream);
}

extern "C" int tq_weighted_result(int dtype, int rule, int dim, int64_t n_per_dim, const void* domain,
                                  const double* gl_weights, int64_t start, int64_t count, const void* f,
                                  int f_dtype, int64_t n_values, void* out, int out_dtype, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  if (!valid_dtype(out_dtype)) return TQ_ERR_DTYPE;
  if (!out || count < 1) return TQ_ERR_ARG;
  return wsum_launch(dtype, rule, dim, n_per_dim, domain, gl_weights, start, count, f, f_dtype, n_values, nullptr,
                     out, out_dtype, workspace, workspace_bytes, stream);
}

extern "C" int tq_finalize_sum(int dtype, int rule, int dim, const void* domain, int64_t n_points,
                               const double* acc, int64_t n_values, void* out, int out_dtype,
                               void* stream) {
  if (!valid_dtype(dtype) || !valid_dtype(out_dtype)) return TQ_ERR_DTYPE;
  if (dim < 1) return TQ_ERR_DIM;
  if (!domain || !acc || !out || n_values < 1 || n_points < 1) return TQ_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const unsigned blocks = (unsigned)((n_values + kBlock - 1) / kBlock);
  if (dtype == TQ_F64)
    finalize_kernel<double><<<blocks, kBlock, 0, s>>>(rule, dim, (const double*)domain, n_points,
                                                      acc, n_values, out, out_dtype);
  else
    finalize_kernel<float><<<blocks, kBlock, 0, s>>>(rule, dim, (const float*)domain, n_points,
                                                     acc, n_values, out, out_dtype);
  return launch_status();
}
