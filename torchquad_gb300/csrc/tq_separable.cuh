// Sum factorisation of the built-in families on tensor-product grids.
//
// A built-in integrand is a function of a separable sum, so its tensor-
// product rule factors into 1-D sums over each dimension's nodes, with the
// same nodes and weights (Orszag's sum factorisation):
//   ExpSum   c prod_k sum_j w_kj exp(a_k x_kj)          (b joins dimension 0)
//   Gaussian c prod_k sum_j w_kj exp(-a_k (x_kj - u_k)^2)
//   Oscill.  c Re prod_k sum_j w_kj exp(i a_k x_kj)     (2 pi b joins dimension 0)
//   SumSin   c sum_k (sum_j w_kj sin(a_k x_kj)) prod_{m != k} (sum_j w_mj)
// and the sums of its adjoint factor likewise with a few more moments per
// dimension.  That is dim * n terms instead of n^dim.  Terms are evaluated
// in fp64 (from the working type's nodes and parameters), weighted exactly,
// summed exactly (fixed-point warp sums) and multiplied as unevaluated
// hi + lo pairs, so the result carries little more than its last rounding.
//
// It holds only where the factors stay inside the floating range although
// the product does: sep_ok decides that from the bounds and the parameters
// alone, equally in every warp; other integrals take the node-by-node path.
#pragma once

#include "tq_grid_common.cuh"

namespace tq {

// Largest one-dimensional grid the per-call kernels sum this way: up to four
// terms a lane of 32 warps (1001 nodes fp64 10.3 us, 14.4 us by the strips);
// longer rows go to the strips, whose terms come by recurrence (fp64) or in
// fp32, over the whole chip.
constexpr int64_t kSepRow = 4096;

template <int FAM, bool GRAD>
struct SepM {  // 1-D moments per dimension
  static constexpr int value = !GRAD ? (FAM == TQ_FN_EXP_SUM || FAM == TQ_FN_GAUSSIAN ? 1 : 2)
                               : FAM == TQ_FN_EXP_SUM  ? 3
                               : FAM == TQ_FN_GAUSSIAN ? 4
                               : FAM == TQ_FN_OSCILLATORY ? 6
                                                          : 5;
};
template <bool GRAD>
constexpr int kSepMaxM = GRAD ? 6 : 2;  // the largest of the families
template <bool GRAD>
constexpr int kSepSlots = kMaxDim * kSepMaxM<GRAD>;  // partials of one CTA (at most kMaxDim units)

// CTAs the factored form of one integral can use: dim * parts units of one
// warp, four to a CTA.
__host__ __device__ inline int sep_parts(int64_t n) { return (int)(n < 32 * 31 ? (n + 31) / 32 : 32); }
__host__ __device__ inline int sep_ctas(int dim, int64_t n) { return (dim * sep_parts(n) + 3) / 4; }

// Whether the factored form is safe (see above), by a whole warp, lane k on
// dimension k; the same in every warp that asks.  D: type of the domain,
// T: type the node-by-node path works in.  Its limits: exponents up to 300
// (80 in fp32, where e^88 overflows in the node-by-node path), angles up to
// 10^6, |c| and the weights' product within 2^+-200 (fp32: no node value
// near overflow), everything finite, no empty dimension.  A Gaussian's
// largest term in a dimension is at most two mean node gaps beyond the
// distance of u to the interval.
template <typename T, typename D>
__device__ __forceinline__ bool sep_ok(int family, int dim, int64_t n, const D* __restrict__ dom,
                                       const double* __restrict__ par) {
  const int k = threadIdx.x & 31;
  constexpr bool F32 = sizeof(T) == 4;
  const double c = par[0];
  const float b = (float)par[1];
  const int ce = exp_field(c) - 1023;
  float m = 0.f;  // the dimension's share of the exponent or angle
  int we = 0;
  bool ok = true;
  if (k < dim) {
    const float lo = (float)dom[2 * k], hi = (float)dom[2 * k + 1], a = (float)par[2 + k];
    const float wid = fabsf(hi - lo);
    we = ((int)(__float_as_uint(wid / (float)n) >> 23) & 0xff) - 127;
    ok = isfinite(lo) && isfinite(hi) && isfinite(a) && wid > 0.f && abs(we) <= 100;
    const float far = fmaxf(fabsf(lo), fabsf(hi));
    if (family == TQ_FN_GAUSSIAN) {
      const float u = (float)par[2 + dim + k];
      ok = ok && isfinite(u) && a >= 0.f;
      const float l = fminf(lo, hi), h = fmaxf(lo, hi);
      const float dist = fmaxf(fmaxf(l - u, u - h), 0.f) + 2.f * wid / (float)n;
      m = a * dist * dist;
    } else {
      m = fabsf(a) * far;
    }
  }
  float sum = m;
  int wsum = we;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
  }
  ok = ok && isfinite(b) && abs(wsum) <= 200;
  if (family == TQ_FN_EXP_SUM || family == TQ_FN_GAUSSIAN) {
    if (family == TQ_FN_EXP_SUM) sum += fabsf(b);
    ok = ok && sum <= (F32 ? 80.f : 300.f);
    if (F32) ok = ok && abs(ce) <= 120 && (float)ce + (family == TQ_FN_EXP_SUM ? 1.45f * sum : 0.f) <= 120.f;
  } else {
    ok = ok && sum + 7.f * fabsf(b) <= 1e6f;
    if (F32) ok = ok && abs(ce) <= 100;
  }
  ok = ok && abs(ce) <= 200;
  return __all_sync(0xffffffffu, ok);  // false with any NaN
}

// a + (p + e) for a compensated pair a (Knuth's TwoSum)
__device__ __forceinline__ void sep_add(Acc& a, double p, double e) {
  const double t = a.s + p, bb = t - a.s;
  a.c += ((a.s - (t - bb)) + (p - bb)) + e;
  a.s = t;
}
// products and sums of unevaluated pairs hi + lo
__device__ __forceinline__ Acc dd_mul(Acc a, Acc b) {
  const double p = a.s * b.s;
  double e = fma(a.s, b.s, -p);
  e = fma(a.s, b.c, e);
  return Acc{p, fma(a.c, b.s, e)};
}
__device__ __forceinline__ Acc dd_mul(Acc a, double b) {
  const double p = a.s * b;
  return Acc{p, fma(a.c, b, fma(a.s, b, -p))};
}
__device__ __forceinline__ Acc dd_add(Acc a, Acc b) {
  sep_add(a, b.s, b.c);
  return a;
}
__device__ __forceinline__ Acc dd_neg(Acc a) { return Acc{-a.s, -a.c}; }
__device__ __forceinline__ Acc dd_shfl_down(Acc a, int o) { return acc_shfl_down(a, o); }

// One warp's share of dimension k: the moments over the nodes [j0, j1).
// Result valid in lane 0.
template <typename T, int FAM, bool GRAD>
__device__ void sep_unit(const Geo<T>& g, const Family<T>& fam, int rule, int64_t n,
                         const double* __restrict__ gln, const double* __restrict__ glw, int k, int64_t j0,
                         int64_t j1, Acc* m) {
  constexpr int M = SepM<FAM, GRAD>::value;
  const bool gl = rule == TQ_RULE_GAUSS;
  const double a = (double)fam.a[k], u = (double)fam.u[k];
  const double phase = k != 0 ? 0.0
                       : FAM == TQ_FN_EXP_SUM       ? (double)fam.b
                       : FAM == TQ_FN_OSCILLATORY   ? (double)((T)(2.0 * CUDART_PI) * fam.b)
                                                    : 0.0;
#pragma unroll
  for (int i = 0; i < M; ++i) m[i] = Acc{0.0, 0.0};
  const T ustep = GRAD ? (T)1 / (T)(n - 1) : (T)0;
  for (int64_t j = j0 + (threadIdx.x & 31); j < j1; j += 32) {
    const double x = gl ? __dadd_rn(__dmul_rn(g.half[k], __ldg(gln + j)), g.mid[k])
                        : (double)linspace_node<T>(g.a[k], g.b[k], g.step[k], n, j);
    const double w = gl ? __ldg(glw + j) : (double)nc_coef_f(rule, (int)j, (int)n);
    double t = 0.0;  // unit node
    if (GRAD) t = gl ? (__ldg(gln + j) + 1.0) * 0.5 : (double)linspace_node<T>((T)0, (T)1, ustep, n, j);
    auto add = [&](int i, double v) {  // w v, exactly
      if constexpr (GRAD && sizeof(T) == 4) {
        // moments of fp32 nodes: plainly, as node by node (256 rows of 1001
        // nodes, cosines: 86 us with the residuals, FP64 bound)
        m[i].s = fma(w, v, m[i].s);
      } else {
        const double p = w * v;
        sep_add(m[i], p, fma(w, v, -p));
      }
    };
    if (FAM == TQ_FN_EXP_SUM) {
      const double e = exp(fma(a, x, phase));
      add(0, e);
      if (GRAD) {
        add(1, e * t);
        add(2, e * x);
      }
    } else if (FAM == TQ_FN_GAUSSIAN) {
      const double d = x - u;
      const double e = exp(-(a * (d * d)));
      add(0, e);
      if (GRAD) {
        const double eg = e * (2.0 * a * d);
        add(1, eg);
        add(2, eg * t);
        add(3, e * (d * d));
      }
    } else if (FAM == TQ_FN_OSCILLATORY) {
      double sn, cs;
      sincos(fma(a, x, phase), &sn, &cs);
      add(0, cs);
      add(1, sn);
      if (GRAD) {
        add(2, cs * t);
        add(3, sn * t);
        add(4, cs * x);
        add(5, sn * x);
      }
    } else {
      double sn, cs = 0.0;
      if (GRAD)
        sincos(a * x, &sn, &cs);
      else
        sn = sin(a * x);
      add(0, 1.0);
      add(1, sn);
      if (GRAD) {
        add(2, a * cs);
        add(3, a * cs * t);
        add(4, x * cs);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < M; ++i) m[i] = warp_reduce(m[i]);
}

// The weighted moments dsum[k][i] (in shared memory) of every dimension.
// CTA bid of nblk; up to dim * 32 units of at most a few terms per lane are
// spread over CTAs, four to a CTA: one warp per sub-partition, since the
// FP64 unit of a sub-partition is the limit.  gpart holds `slots` partials;
// sp: kSepSlots<GRAD> partials in shared memory.  Returns true (in every thread)
// in the one CTA that has the sums; the ticket is left at zero.
template <typename T, int FAM, bool GRAD>
__device__ bool sep_sums(const Geo<T>& g, const Family<T>& fam, int rule, int dim, int64_t n,
                         const double* __restrict__ gln, const double* __restrict__ glw, unsigned bid,
                         unsigned nblk, Acc* gpart, int64_t slots, unsigned* ticket,
                         Acc (*dsum)[kSepMaxM<GRAD>], Acc* sp) {
  constexpr int M = SepM<FAM, GRAD>::value;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  int parts = sep_parts(n);
  unsigned ctas = min(nblk, (unsigned)sep_ctas(dim, n));
  if (ctas > 1 && (int64_t)dim * parts * M > slots) ctas = 1;
  if (ctas == 1) parts = min(parts, max(1, nw / dim));
  if (bid >= ctas) return false;
  Acc* dst = ctas > 1 ? gpart : sp;
  for (int v = (int)bid + warp * (int)ctas; v < dim * parts; v += (int)ctas * nw) {
    const int k = v / parts, q = v - k * parts;
    Acc m[M];
    sep_unit<T, FAM, GRAD>(g, fam, rule, n, gln, glw, k, n * q / parts, n * (q + 1) / parts, m);
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < M; ++i) dst[v * M + i] = m[i];
    }
  }
  if (ctas > 1) {
    if (!last_block_of(ticket, ctas)) return false;
    if (threadIdx.x == 0) *ticket = 0u;
  } else {
    __syncthreads();
  }
  for (int q = warp; q < dim * M; q += nw) {
    const int k = q / M, i = q - k * M;
    Acc v{0.0, 0.0};
    if (lane < parts) {
      const double* e = &dst[(k * parts + lane) * M + i].s;
      v = ctas > 1 ? Acc{__ldcg(e), __ldcg(e + 1)} : Acc{e[0], e[1]};
    }
    if (parts > 1) v = warp_reduce(v);
    if (lane == 0) dsum[k][i] = dd_mul(v, g.wscale[k]);
  }
  __syncthreads();
  return true;
}

// The integral without c from the dimensions' moments, by one warp (products
// in a tree over the dimensions); valid in lane 0.
template <int FAM>
__device__ Acc sep_value(const Acc (*dsum)[kSepMaxM<false>], int dim) {
  const int k = threadIdx.x & 31;
  Acc p = k < dim ? dsum[k][0] : Acc{1.0, 0.0};
  Acc q = (k < dim && (FAM == TQ_FN_OSCILLATORY || FAM == TQ_FN_SUM_SIN)) ? dsum[k][1] : Acc{0.0, 0.0};
  for (int o = 8; o > 0; o >>= 1) {
    if (o >= dim) continue;
    const Acc p2 = dd_shfl_down(p, o);
    if (FAM == TQ_FN_OSCILLATORY) {  // (p + i q) (p2 + i q2)
      const Acc q2 = dd_shfl_down(q, o);
      const Acc re = dd_add(dd_mul(p, p2), dd_neg(dd_mul(q, q2)));
      q = dd_add(dd_mul(p, q2), dd_mul(q, p2));
      p = re;
    } else if (FAM == TQ_FN_SUM_SIN) {  // p: product of the weights, q: the sum
      const Acc q2 = dd_shfl_down(q, o);
      q = dd_add(dd_mul(q, p2), dd_mul(p, q2));
      p = dd_mul(p, p2);
    } else {
      p = dd_mul(p, p2);
    }
  }
  return FAM == TQ_FN_SUM_SIN ? q : p;
}

// The adjoint's accumulators out[0 .. 2 + 4 dim) (sum W F, sum W F', then by
// dimension sum W F' g', W F' g' t, W F' dg/da, W F' dg/du; no factor c)
// from the dimensions' moments, by one warp.
template <int FAM, typename T>
__device__ void sep_adjoint(const Acc (*dsum)[kSepMaxM<true>], const T* av, int dim, double* out) {
  const int k = threadIdx.x & 31;
  auto val = [](Acc v) { return v.s + v.c; };
  if (k < dim) {
    // product over the other dimensions (lane k), complex for oscillations
    Acc pr{1.0, 0.0}, pi{0.0, 0.0};
    Acc so{0.0, 0.0};  // sum of sines: sum over the others of S_m prod W
    for (int m = 0; m < dim; ++m) {
      if (m == k) continue;
      if (FAM == TQ_FN_OSCILLATORY) {
        const Acc zr = dsum[m][0], zi = dsum[m][1];
        const Acc re = dd_add(dd_mul(pr, zr), dd_neg(dd_mul(pi, zi)));
        pi = dd_add(dd_mul(pr, zi), dd_mul(pi, zr));
        pr = re;
      } else {
        if (FAM == TQ_FN_SUM_SIN) so = dd_add(dd_mul(so, dsum[m][0]), dd_mul(pr, dsum[m][1]));
        pr = dd_mul(pr, dsum[m][0]);
      }
    }
    // imaginary part of (pr + i pi)(moment r + i moment i), negated
    auto nim = [&](int r, int i) { return -val(dd_add(dd_mul(pr, dsum[k][i]), dd_mul(pi, dsum[k][r]))); };
    const double a = (double)av[k];
    double F, Fp, sx, st, pa, pu = 0.0;
    if (FAM == TQ_FN_OSCILLATORY) {
      F = val(dd_add(dd_mul(pr, dsum[k][0]), dd_neg(dd_mul(pi, dsum[k][1]))));
      Fp = nim(0, 1);
      sx = a * Fp;
      st = a * nim(2, 3);
      pa = nim(4, 5);
    } else if (FAM == TQ_FN_EXP_SUM) {
      F = Fp = val(dd_mul(pr, dsum[k][0]));
      sx = a * F;
      st = a * val(dd_mul(pr, dsum[k][1]));
      pa = val(dd_mul(pr, dsum[k][2]));
    } else if (FAM == TQ_FN_GAUSSIAN) {
      F = val(dd_mul(pr, dsum[k][0]));
      Fp = -F;
      sx = -val(dd_mul(pr, dsum[k][1]));
      st = -val(dd_mul(pr, dsum[k][2]));
      pa = -val(dd_mul(pr, dsum[k][3]));
      pu = -sx;
    } else {
      F = val(dd_add(dd_mul(so, dsum[k][0]), dd_mul(pr, dsum[k][1])));
      Fp = val(dd_mul(pr, dsum[k][0]));
      sx = val(dd_mul(pr, dsum[k][2]));
      st = val(dd_mul(pr, dsum[k][3]));
      pa = val(dd_mul(pr, dsum[k][4]));
    }
    if (k == 0) {
      out[0] = F;
      out[1] = Fp;
    }
    out[2 + k] = sx;
    out[2 + dim + k] = st;
    out[2 + 2 * dim + k] = pa;
    out[2 + 3 * dim + k] = pu;
  }
}

// ------------------------------------------------ fp64 rows in one dimension
// A one-dimensional Newton-Cotes rule of equally spaced nodes, a thread
// walking a chain of up to kChain nodes in blocks of kBlk from one direct
// evaluation (two or three exp or one sincos) at the chain's start:
//   Gaussian  f(x + i h) = F R^i G_i with F = f(x), R = exp(-2 a h (x - u)),
//             G_i = exp(-a h^2 i^2): a block is F times a polynomial in R
//             whose coefficients (weight times G_i) are the same for every
//             block, by Horner's rule; F and R step to the next block by
//             two factors that are themselves geometric
//   exp sum   f(x + i h) = f(x) exp(a h i): a block is f(x) times a constant
//   cosines   by the addition theorem: a block is cos and sin of the first
//             angle times two constants, the angle rotated block by block.
// So a node costs about 1.2 (Gaussian) or 0.2-0.4 FP64 operations plus the
// chain's start, where stepping node by node from strips of 16 took 3 and a
// start (two exp and the guards, 70 operations) every 16 nodes; the FP64 unit
// bounds both.  Rounding accumulates over at most kChain / kBlk steps of a
// factor, fewer than the 16 of the strips (rms errors of 200 random rows, strips
// and chains of 128: Gaussians 1.2e-15 and 0.9e-15 of the sum of magnitudes,
// exponentials 3.7e-16 and 2.3e-16; compensated sums in the chain: the same to
// two digits).  4096 mixed integrals, a quarter
// of them such rows: 2.0 ms by strips, 0.62 ms by chains (and the
// factored integrals spread over the CTAs by integral).
constexpr int kBlk = 16;    // nodes per block (a multiple of 4: the rules' weight period)
constexpr int kChain = 128;  // nodes per chain at most

struct ChainTab {
  double t[kBlk], t2[kBlk];  // weight times G_i, exp(a h i), or cos / sin(a h i)
  double A, B;               // their sums
  double q[3];               // Gaussian: G_kBlk, steps of R and of the block factor; exp: exp(a h kBlk);
                             // cosines: cos and sin of a h kBlk
};

// Builds the table for chains that start at nodes off + m * kBlk (warp 0 of
// the CTA; the caller puts a barrier before the first use).
template <int FAM>
__device__ void chain_table(ChainTab& tb, const Family<double>& fam, int rule, double h, int64_t off) {
  const int i = threadIdx.x;
  if (i >= 32) return;
  const double a = fam.a[0];
  const int m = (int)((off + i) & 3);
  const double w = i >= kBlk ? 1.0
                   : rule == TQ_RULE_TRAPEZOID ? 2.0
                   : rule == TQ_RULE_SIMPSON ? ((m & 1) ? 4.0 : 2.0)
                                             : ((m & 1) ? 32.0 : (m == 2 ? 12.0 : 14.0));
  double v, v2 = 0.0;
  if (FAM == TQ_FN_GAUSSIAN) {
    const int e = i <= kBlk ? i * i : (i == kBlk + 1 ? 2 * kBlk : 2 * kBlk * kBlk);
    v = w * exp(-(a * h * h) * (double)e);
  } else if (FAM == TQ_FN_EXP_SUM) {
    v = w * exp(a * h * (double)min(i, kBlk));
  } else {
    double sn, cs;
    sincos(a * h * (double)min(i, kBlk), &sn, &cs);
    v = w * cs;
    v2 = w * sn;
  }
  if (i < kBlk) {
    tb.t[i] = v;
    tb.t2[i] = v2;
  } else if (FAM == TQ_FN_GAUSSIAN) {
    if (i < kBlk + 3) tb.q[i - kBlk] = v;
  } else if (i == kBlk) {
    tb.q[0] = v;
    tb.q[1] = v2;
  }
  const Acc A = warp_reduce(Acc{i < kBlk ? v : 0.0, 0.0}), B = warp_reduce(Acc{i < kBlk ? v2 : 0.0, 0.0});
  if (i == 0) {
    tb.A = A.s + A.c;
    tb.B = B.s + B.c;
  }
}

// Sum over the nodes j0 .. j0 + cnt - 1 (x0 the first, x1 the last one's
// coordinate) of the weighted integrand into *out.  Returns false where the
// factors could leave the range of doubles: the exponent has to stay within
// [-600, 600] at both ends (that of a Gaussian, a >= 0, is at most 0) and
// change by at most 300 over a block; the factor c joins the sum at its end,
// as c times the first node's value may leave it.  The rules' end weights are
// half of the interior's at the same place.
template <int FAM>
__device__ __forceinline__ bool chain_sum(const Family<double>& fam, const ChainTab& tb, int rule, double x0,
                                          double x1, double h, int64_t j0, int cnt, int64_t n, double* out) {
  const double a = fam.a[0];
  const double half = rule == TQ_RULE_BOOLE ? 7.0 : 1.0;
  const bool first = j0 == 0, final = j0 + cnt == n;
  double acc = 0.0;
  if (FAM == TQ_FN_GAUSSIAN) {
    const double d0 = x0 - fam.u[0], d1 = x1 - fam.u[0];
    const double e0 = -(a * (d0 * d0)), e1 = -(a * (d1 * d1)), r0 = -(2.0 * a * h * d0);
    if (!(a >= 0.0 && e0 >= -600.0 && e1 >= -600.0 && fabs(r0) <= 15.0 &&
          2.0 * a * h * h * (kBlk * kBlk) <= 200.0 && fabs(2.0 * a * h * d1) <= 15.0))
      return false;
    double F = exp(e0), R = exp(r0), P = exp(r0 * (double)kBlk) * tb.q[0];
    if (first) acc = -half * F;
    int left = cnt;
    for (; left >= kBlk; left -= kBlk) {
      double p = tb.t[kBlk - 1];
#pragma unroll
      for (int i = kBlk - 2; i >= 0; --i) p = fma(p, R, tb.t[i]);
      acc = fma(F, p, acc);
      F *= P;
      P *= tb.q[2];
      R *= tb.q[1];
    }
    if (left > 0) {
      double p = tb.t[left - 1];
      for (int i = left - 2; i >= 0; --i) p = fma(p, R, tb.t[i]);
      acc = fma(F, p, acc);
    }
    if (final) acc = fma(-half, exp(e1), acc);
  } else if (FAM == TQ_FN_EXP_SUM) {
    const double e0 = fma(a, x0, fam.b), e1 = fma(a, x1, fam.b);
    if (!(fabs(e0) <= 600.0 && fabs(e1) <= 600.0 && fabs(a * h) <= 15.0)) return false;
    double f = exp(e0);
    if (first) acc = -half * f;
    int left = cnt;
    for (; left >= kBlk; left -= kBlk) {
      acc = fma(f, tb.A, acc);
      f *= tb.q[0];
    }
    for (int i = 0; i < left; ++i) acc = fma(f, tb.t[i], acc);
    if (final) acc = fma(-half, exp(e1), acc);
  } else {
    // f = cos(angle) (oscillatory) or sin(angle) (sum of sines)
    const double ph = FAM == TQ_FN_OSCILLATORY ? 2.0 * CUDART_PI * fam.b : 0.0;
    double sn, cs;
    sincos(fma(a, x0, ph), &sn, &cs);
    const bool osc = FAM == TQ_FN_OSCILLATORY;
    if (first) acc = -half * (osc ? cs : sn);
    int left = cnt;
    for (; left >= kBlk; left -= kBlk) {
      acc = osc ? fma(cs, tb.A, fma(-sn, tb.B, acc)) : fma(sn, tb.A, fma(cs, tb.B, acc));
      const double c2 = fma(cs, tb.q[0], -(sn * tb.q[1]));
      sn = fma(sn, tb.q[0], cs * tb.q[1]);
      cs = c2;
    }
    for (int i = 0; i < left; ++i)
      acc = osc ? fma(cs, tb.t[i], fma(-sn, tb.t2[i], acc)) : fma(sn, tb.t[i], fma(cs, tb.t2[i], acc));
    if (final) acc = fma(-half, osc ? cos(fma(a, x1, ph)) : sin(a * x1), acc);
  }
  *out = acc * fam.c;
  return true;
}

// Nodes per chain for `count` nodes of a CTA: as few as leave the number of
// its warps with chains what it is with the longest (1001 nodes: one warp of
// 32 chains of 32, not of 8 chains of 128).
__device__ __forceinline__ int chain_len(int64_t count, int longest) {
  const int64_t lanes = (count + 32 * longest - 1) / (32 * longest) * 32;
  return (int)(((count + lanes - 1) / lanes + kBlk - 1) / kBlk * kBlk);
}

// Chains of a round that chain_sum refused.
struct ChainTodo {
  int64_t first[8];         // a warp's chain of lane 0
  unsigned mask[8];         // its lanes whose chains are refused
  unsigned char list[256];  // the CTA's threads whose chains are
};

// The CTA's part of the nodes [begin, end) of a one-dimensional fp64
// Newton-Cotes grid, without the weight scale (each thread's share is
// returned): chains of `len` nodes (a multiple of kBlk), in rounds of one a
// thread, this thread's the chains first, first + step, ... (consecutive over
// a warp; `round` the number of rounds, equal in the whole CTA).  The nodes of
// chains that chain_sum refuses are evaluated one by one, spread over all
// threads of the CTA: left to the chains' own threads, a row of 1001 nodes
// whose chains are all refused kept 8 threads busy (256 narrow Gaussian rows
// 151 us; 45 in strips of 16 nodes a thread, 41 this way).
template <int FAM>
__device__ Acc chain_rows(const Geo<double>& g, const Family<double>& fam, const ChainTab& tb, ChainTodo& todo,
                          int rule, int64_t n, int64_t begin, int64_t end, int len, int64_t first, int64_t step,
                          int64_t rounds) {
  Acc acc{0.0, 0.0};
  const double h = g.step[0];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  for (int64_t r = 0; r < rounds; ++r) {
    const int64_t chain = first + r * step, j0 = begin + chain * len;
    bool refused = false;
    if (j0 < end) {
      const int cnt = (int)min((int64_t)len, end - j0);
      const double x0 = linspace_node<double>(g.a[0], g.b[0], h, n, j0);
      const double x1 = linspace_node<double>(g.a[0], g.b[0], h, n, j0 + cnt - 1);
      double v;
      refused = !chain_sum<FAM>(fam, tb, rule, x0, x1, h, j0, cnt, n, &v);
      if (!refused) acc_add(acc, v);
    }
    const unsigned mask = __ballot_sync(0xffffffffu, refused);
    if (lane == 0) {
      todo.first[warp] = chain;
      todo.mask[warp] = mask;
    }
    if (!__syncthreads_or(refused)) continue;
    int before = 0, all = 0;  // refused chains of the warps before this one, of all
    for (int w = 0; w < nw; ++w) {
      const int k = __popc(todo.mask[w]);
      before += w < warp ? k : 0;
      all += k;
    }
    if (refused) todo.list[before + __popc(mask & ((1u << lane) - 1u))] = (unsigned char)threadIdx.x;
    __syncthreads();
    double sum = 0.0;
    int held = 0;  // values in sum
    for (int e = threadIdx.x; e < all * len; e += blockDim.x) {
      const int q = e / len, t = todo.list[q];
      const int64_t j = begin + (todo.first[t >> 5] + (t & 31)) * len + (e - q * len);
      if (j >= end) continue;
      const double x = linspace_node<double>(g.a[0], g.b[0], h, n, j);
      const int place = j == 0 || j == n - 1 ? 0 : 4 + (int)(j & 3);  // an end, or like the node
      sum = fma((double)nc_coef_f(rule, place, 1 << 30),
                fam_outer<FAM, double>(fam, fam_term<FAM, double>(fam, 0, x)), sum);
      if (++held == 16) {
        acc_add(acc, sum);
        sum = 0.0;
        held = 0;
      }
    }
    acc_add(acc, sum);
    __syncthreads();  // the round's list is rewritten
  }
  return acc;
}

}  // namespace tq
