// Shared device code of the torchquad_gb300 kernels: status plumbing,
// compensated accumulators, Philox4x32-10, node/weight formulas of the grid
// rules and the built-in integrand families.
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "torchquad_gb300.h"

namespace tq {

constexpr int kMaxDim = TQ_MAX_DIM;
constexpr int kBlock = 256;  // threads per CTA of the streaming kernels
// VEGAS control block entry: 1 while cube_start holds prefixes local to each
// kBlock-cube block of get_NH, the block offsets being in the workspace
// (tq_vegas_get_nh_split); the sampler adds them, finish writes them back.
constexpr int kCtlSplit = 14;

// ---------------------------------------------------------------- host side
int set_cuda_error(cudaError_t e);  // records e, returns TQ_ERR_CUDA
int launch_status();                // TQ_OK or TQ_ERR_CUDA for the last launch
int sm_count();                     // SMs of the current device (cached)
int grid_for(const void* kernel, int block, size_t smem, int64_t work_blocks);

// Opt-in for dynamic shared memory: a launch gets 48 KB of shared memory
// (static and dynamic together) unless the kernel's attribute allows more,
// so the attribute is raised whenever the dynamic part alone exceeds 32 KB
// (the static shared memory of the kernels launched this way stays below
// 16 KB).
template <typename K>
inline int opt_in_smem(K kfn, size_t smem) {
  if (smem <= 32 * 1024) return TQ_OK;
  const cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return e == cudaSuccess ? TQ_OK : set_cuda_error(e);
}

inline bool valid_dtype(int d) { return d == TQ_F32 || d == TQ_F64; }
inline size_t dtype_size(int d) { return d == TQ_F64 ? 8 : 4; }

// Workspace layout shared by the reducing kernels: a 16-byte ticket word
// followed by `slots` compensated pairs (2 doubles each).
inline size_t reduce_ws_bytes(int64_t slots) { return 256 + (size_t)slots * 16; }

// ------------------------------------------------- compensated accumulation
// Neumaier's variant of Kahan summation: exact error term of each addition.
struct Acc {
  double s, c;
};
__device__ __forceinline__ void acc_add(Acc& a, double x) {
  double t = a.s + x;
  double e = (fabs(a.s) >= fabs(x)) ? ((a.s - t) + x) : ((x - t) + a.s);
  a.c += e;
  a.s = t;
}
__device__ __forceinline__ void acc_merge(Acc& a, const Acc& b) {
  acc_add(a, b.s);
  a.c += b.c;
}
__device__ __forceinline__ Acc acc_shfl_down(const Acc& a, int off) {
  Acc r;
  r.s = __shfl_down_sync(0xffffffffu, a.s, off);
  r.c = __shfl_down_sync(0xffffffffu, a.c, off);
  return r;
}
// ------------------------------------------------------ exact CTA sums
// Sums of doubles as fixed-point integers.  A compensated fp64 tree over a
// CTA takes about 130 dependent FP64 warp instructions, and on GB300 each
// holds a sub-partition's FP64 unit for about 64 cycles (4 us a reduction,
// more than the work of a small launch).  Here every value is placed in a
// 112-bit window below the CTA's largest binary exponent, as five signed
// limbs of 24 bits (the lowest of 16; integer shifts only), the limbs are
// summed over a warp by redux.sync and over the CTA as 64-bit integers, and
// one thread turns the total into hi + lo doubles by bit moves.  Integer sums
// are exact and do not depend on their order; a value loses only bits below
// 2^-111 of the largest (the pair hi + lo holds 106).  A 101^3 fused Simpson launch by nodes (252 CTAs): 26.4 us with the
// fp64 trees, 18.7 us with these sums and the dimensions set up in parallel; a
// 10001-node rule over 200 components (50 reductions a component group): 969
// and 431 us.
__device__ __forceinline__ int exp_field(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

constexpr int kLimbs = 5;  // limb 0 has weight 1, limb i > 0 weight 2^(24 i - 8)

// L += v in units of 2^(emax - 1134); v finite, its exponent field at most
// emax, emax >= 1.
__device__ __forceinline__ void fix_add(int (&L)[kLimbs], double v, int emax) {
  const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
  const int ef = (int)(hi >> 20) & 0x7ff;
  const uint32_t mh = (hi & 0xfffffu) | (ef ? 0x100000u : 0u);
  const int s = emax - (ef ? ef : 1);
  const uint32_t w3 = (mh << 11) | (lo >> 21), w2 = lo << 11;  // mantissa << 75, 128 bits
  uint32_t a3 = w3 >> (s & 31), a2 = __funnelshift_r(w2, w3, s), a1 = __funnelshift_r(0u, w2, s), a0 = 0u;
  const int q = s >> 5;
  a0 = q == 1 ? a1 : q == 2 ? a2 : q == 3 ? a3 : 0u;
  a1 = q == 0 ? a1 : q == 1 ? a2 : q == 2 ? a3 : 0u;
  a2 = q == 0 ? a2 : q == 1 ? a3 : 0u;
  a3 = q == 0 ? a3 : 0u;
  const int sg = (int)hi >> 31;
  L[0] += ((int)(a0 >> 16) ^ sg) - sg;
  L[1] += ((int)(a1 & 0xffffffu) ^ sg) - sg;
  L[2] += ((int)(__funnelshift_r(a1, a2, 24) & 0xffffffu) ^ sg) - sg;
  L[3] += ((int)(__funnelshift_r(a2, a3, 16) & 0xffffffu) ^ sg) - sg;
  L[4] += ((int)(a3 >> 8) ^ sg) - sg;
}

// The leading 53 bits of A 2^p as a double (truncated); A keeps the rest.
__device__ __forceinline__ double fix_take(unsigned __int128& A, int p) {
  const uint64_t ah = (uint64_t)(A >> 64), al = (uint64_t)A;
  if ((ah | al) == 0) return 0.0;
  const int n = ah ? 127 - __clzll((long long)ah) : 63 - __clzll((long long)al);  // leading bit
  uint64_t top;
  if (n > 52) {
    top = (uint64_t)(A >> (n - 52));
    A -= (unsigned __int128)top << (n - 52);
  } else {
    top = al << (52 - n);
    A = 0;
  }
  const int e = n + p + 1023;
  if (e >= 1 && e <= 2046)
    return __longlong_as_double((long long)(((uint64_t)e << 52) | (top & 0xfffffffffffffull)));
  return scalbn((double)(long long)top, n - 52 + p);  // subnormal or infinite
}
// The total of the limb sums S in units of 2^(emax - 1134) as hi + lo (up to
// 2^14 values stay inside 127 bits).
__device__ __forceinline__ Acc fix_value(const int64_t (&S)[kLimbs], int emax) {
  __int128 t = (__int128)S[0] + ((__int128)S[1] << 16) + ((__int128)S[2] << 40) + ((__int128)S[3] << 64) +
               ((__int128)S[4] << 88);
  const bool neg = t < 0;
  unsigned __int128 A = neg ? (unsigned __int128)(-t) : (unsigned __int128)t;
  Acc r;
  r.s = fix_take(A, emax - 1134);
  r.c = fix_take(A, emax - 1134);
  if (neg) {
    r.s = -r.s;
    r.c = -r.c;
  }
  return r;
}

// Exact running sum of a thread: fp64 terms as 128-bit two's-complement
// integers, about 35 integer instructions a term where a compensated fp64
// sum has 8 on the FP64 unit (64 cycles each).  A term of exponent
// field E has its last bit at 2^58, which leaves room for 2^15 terms of that
// size and loses bits below 2^-110 of it; a larger term, or a sum near the
// top, first shifts the sum down.  Infinities and NaN go to an fp64 side sum.
struct FixAcc {
  uint32_t w0 = 0, w1 = 0, w2 = 0;
  int w3 = 0;
  int top = 6;  // E + 6
  double side = 0.0;
  __device__ __forceinline__ static void shift(uint32_t& a0, uint32_t& a1, uint32_t& a2, int& a3, int t) {  // t < 128
    const int q = t >> 5;
    const uint32_t sg = (uint32_t)(a3 >> 31);
    const uint32_t b0 = q == 0 ? a0 : q == 1 ? a1 : q == 2 ? a2 : (uint32_t)a3;
    const uint32_t b1 = q == 0 ? a1 : q == 1 ? a2 : q == 2 ? (uint32_t)a3 : sg;
    const uint32_t b2 = q == 0 ? a2 : q == 1 ? (uint32_t)a3 : sg;
    const int b3 = q == 0 ? a3 : (int)sg;
    a0 = __funnelshift_r(b0, b1, t);
    a1 = __funnelshift_r(b1, b2, t);
    a2 = __funnelshift_r(b2, (uint32_t)b3, t);
    a3 = b3 >> (t & 31);
  }
  __device__ __forceinline__ void down(int d) {
    if (d < 128)
      shift(w0, w1, w2, w3, d);
    else
      w0 = w1 = w2 = 0, w3 = 0;
    top += d;
  }
  __device__ __forceinline__ void add(double v) {
    const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
    int e = (int)(hi >> 20) & 0x7ff;
    if (e == 0x7ff) {
      side += v;
      return;
    }
    const uint32_t mh = (hi & 0xfffffu) | (e ? 0x100000u : 0u);
    e = e ? e : 1;
    if (e + 6 > top) down(e + 6 - top);
    const int t = top - e;
    if (t >= 128) return;  // below the window
    // the mantissa's two's complement, 64 bits up, then down by t
    const int sg = (int)hi >> 31;
    const uint32_t one = (uint32_t)sg & 1u;
    uint32_t a0 = 0, a1 = 0, a2 = (lo ^ (uint32_t)sg) + one;
    int a3 = ((int)mh ^ sg) + (int)(a2 < one);
    shift(a0, a1, a2, a3, t);
    const uint64_t s0 = (uint64_t)w0 + a0, s1 = (uint64_t)w1 + a1 + (s0 >> 32), s2 = (uint64_t)w2 + a2 + (s1 >> 32);
    w0 = (uint32_t)s0;
    w1 = (uint32_t)s1;
    w2 = (uint32_t)s2;
    w3 += a3 + (int)(s2 >> 32);
    if ((uint32_t)(w3 + (1 << 29)) >> 30) down(8);  // within two bits of the top
  }
  __device__ __forceinline__ Acc value() const {
    const __int128 t = ((__int128)w3 << 96) | ((unsigned __int128)w2 << 64) | ((uint64_t)w1 << 32) | w0;
    const bool neg = t < 0;
    unsigned __int128 A = neg ? (unsigned __int128)(-t) : (unsigned __int128)t;
    Acc r;
    r.s = fix_take(A, top - 1139);
    r.c = fix_take(A, top - 1139);
    if (neg) r = Acc{-r.s, -r.c};
    if (!(side == 0.0)) r.s += side;
    return r;
  }
};
// Sum of get(0) .. get(n - 1) by a whole warp (get is called twice for each);
// result valid in lane 0.
template <typename Get>
__device__ __forceinline__ Acc warp_sum(int n, Get get) {
  const int lane = threadIdx.x & 31;
  int e = 1;
  for (int i = lane; i < n; i += 32) {
    const Acc v = get(i);
    e = max(e, max(exp_field(v.s), exp_field(v.c)));
  }
  const int emax = __reduce_max_sync(0xffffffffu, e);
  if (emax == 0x7ff) {  // infinities or NaN: in the floating format
    Acc a{0.0, 0.0};
    for (int i = lane; i < n; i += 32) acc_merge(a, get(i));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc_merge(a, acc_shfl_down(a, off));
    return a;
  }
  int64_t S[kLimbs] = {0, 0, 0, 0, 0};
  for (int base = 0; base < n; base += 32) {
    int L[kLimbs] = {0, 0, 0, 0, 0};
    if (base + lane < n) {
      const Acc v = get(base + lane);
      fix_add(L, v.s, emax);
      fix_add(L, v.c, emax);
    }
#pragma unroll
    for (int i = 0; i < kLimbs; ++i) S[i] += __reduce_add_sync(0xffffffffu, L[i]);
  }
  return fix_value(S, emax);
}
// Sum of one Acc per lane over a warp; result valid in lane 0.
__device__ __forceinline__ Acc warp_reduce(Acc a) {
  return warp_sum(32, [&](int) { return a; });
}

// Sum of get(0) .. get(n - 1) by the CTA (blockDim.x <= BLOCK, whole warps;
// get(i) is called twice, by thread i mod blockDim.x); result valid in
// thread 0.
template <int BLOCK, typename Get>
__device__ __forceinline__ Acc block_sum(int n, Get get) {
  constexpr int kW = BLOCK / 32;
  __shared__ int wexp[kW];
  __shared__ int64_t wlimb[kW][kLimbs];
  __shared__ Acc part[kW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  int e = 1;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const Acc v = get(i);
    e = max(e, max(exp_field(v.s), exp_field(v.c)));
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if (lane == 0) wexp[warp] = e;
  __syncthreads();
  int emax = 1;
  for (int i = 0; i < nw; ++i) emax = max(emax, wexp[i]);
  Acc a{0.0, 0.0};
  if (emax == 0x7ff) {  // infinities or NaN: in the floating format
    for (int i = threadIdx.x; i < n; i += blockDim.x) acc_merge(a, get(i));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc_merge(a, acc_shfl_down(a, off));
    if (lane == 0) part[warp] = a;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int i = 1; i < nw; ++i) acc_merge(a, part[i]);
    __syncthreads();
    return a;
  }
  int64_t S[kLimbs] = {0, 0, 0, 0, 0};
  for (int base = 0; base < n; base += blockDim.x) {
    int L[kLimbs] = {0, 0, 0, 0, 0};
    const int i = base + (int)threadIdx.x;
    if (i < n) {
      const Acc v = get(i);
      fix_add(L, v.s, emax);
      fix_add(L, v.c, emax);
    }
#pragma unroll
    for (int q = 0; q < kLimbs; ++q) S[q] += __reduce_add_sync(0xffffffffu, L[q]);
  }
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < kLimbs; ++i) wlimb[warp][i] = S[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < nw; ++w) {
#pragma unroll
      for (int i = 0; i < kLimbs; ++i) S[i] += wlimb[w][i];
    }
    a = fix_value(S, emax);
  }
  __syncthreads();
  return a;
}
// Sum of one Acc per thread over the CTA; result valid in thread 0.
template <int BLOCK>
__device__ __forceinline__ Acc block_reduce(Acc a) {
  return block_sum<BLOCK>((int)blockDim.x, [&](int) { return a; });
}
// Sum of the partials [0, n) of a launch's CTAs by the last of them (they
// were written by other CTAs: read past L1); result valid in thread 0.
template <int BLOCK>
__device__ __forceinline__ Acc partials_reduce(const Acc* partials, int n) {
  return block_sum<BLOCK>(n, [&](int i) { return Acc{__ldcg(&partials[i].s), __ldcg(&partials[i].c)}; });
}

// fp32 compensated strip accumulator (cheap on the FP32 pipe).
struct AccF {
  float s, c;
};
__device__ __forceinline__ void accf_add(AccF& a, float x) {
  float t = __fadd_rn(a.s, x);
  float e = (fabsf(a.s) >= fabsf(x)) ? __fadd_rn(__fsub_rn(a.s, t), x)
                                     : __fadd_rn(__fsub_rn(x, t), a.s);
  a.c = __fadd_rn(a.c, e);
  a.s = t;
}

// Double-float (two-float) accumulation on the FP32 pipe: the unevaluated
// sum hi + lo, |lo| <= ulp(hi) / 2, about 48 significant bits.  Additions
// use Knuth's TwoSum and Dekker's Fast2Sum for the renormalisation (the
// accurate variant: two TwoSums per addition, so cancellation between terms
// of either sign keeps the bound).  On GB300 an FP64 warp instruction
// occupies an SM sub-partition's FP64 unit for about 64 cycles; these
// operations keep long reductions off that unit.
struct F2 {
  float hi, lo;
};
__device__ __forceinline__ F2 two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return F2{s, e};
}
__device__ __forceinline__ F2 fast_two_sum(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return F2{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 s = two_sum(a.hi, b.hi);
  const F2 t = two_sum(a.lo, b.lo);
  s = fast_two_sum(s.hi, __fadd_rn(s.lo, t.hi));
  return fast_two_sum(s.hi, __fadd_rn(s.lo, t.lo));
}
__device__ __forceinline__ F2 f2_add(F2 a, float b) {
  const F2 s = two_sum(a.hi, b);
  return fast_two_sum(s.hi, __fadd_rn(s.lo, a.lo));
}
__device__ __forceinline__ F2 f2_shfl_down(F2 a, int off) {
  return F2{__shfl_down_sync(0xffffffffu, a.hi, off), __shfl_down_sync(0xffffffffu, a.lo, off)};
}
__device__ __forceinline__ F2 f2_shfl_up(F2 a, int off) {
  return F2{__shfl_up_sync(0xffffffffu, a.hi, off), __shfl_up_sync(0xffffffffu, a.lo, off)};
}
__device__ __forceinline__ double f2_value(F2 a) { return (double)a.hi + (double)a.lo; }
// Products (Dekker's TwoProduct through an FMA, then one renormalisation):
// about 48 significant bits, FP32 pipe only.
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fmaf_rn(a.hi, b.lo, e);
  e = __fmaf_rn(a.lo, b.hi, e);
  return fast_two_sum(p, e);
}
__device__ __forceinline__ F2 f2_mul(F2 a, float b) {
  const float p = __fmul_rn(a.hi, b);
  float e = __fmaf_rn(a.hi, b, -p);
  e = __fmaf_rn(a.lo, b, e);
  return fast_two_sum(p, e);
}
// A double split into a double-float (two conversions; once per set-up).
__device__ __forceinline__ F2 f2_from_double(double x) {
  const float hi = __double2float_rn(x);
  return F2{hi, __double2float_rn(x - (double)hi)};
}
// The double-float rounded to the nearest float.
__device__ __forceinline__ float f2_round(F2 a) { return __fadd_rn(a.hi, a.lo); }

// "Last CTA finishes" pattern: every CTA writes its partial, fences, takes a
// ticket; the CTA that draws the last ticket reduces all partials in index
// order (deterministic) and resets the ticket for the next launch.  No CTA
// waits on another, so nothing can spin.
// `count` CTAs take part (a kernel whose CTAs play several roles counts
// each role's CTAs on its own ticket).
__device__ __forceinline__ bool last_block_of(unsigned* ticket, unsigned count) {
  __shared__ bool is_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned t = atomicAdd(ticket, 1u);
    is_last = (t == count - 1);
  }
  __syncthreads();
  return is_last;
}
__device__ __forceinline__ bool last_block_arrives(unsigned* ticket) {
  return last_block_of(ticket, gridDim.x * gridDim.y * gridDim.z);
}

// ------------------------------------------------------------ Philox4x32-10
// Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as easy as 1, 2, 3",
// SC'11: 10 rounds of the 4x32 bijection with multipliers 0xD2511F53 /
// 0xCD9E8D57 and Weyl key increments 0x9E3779B9 / 0xBB67AE85.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c.x);
    const uint32_t lo0 = 0xD2511F53u * c.x;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z);
    const uint32_t lo1 = 0xCD9E8D57u * c.z;
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    k.x += 0x9E3779B9u;
    k.y += 0xBB67AE85u;
  }
  return c;
}
__device__ __forceinline__ uint4 philox_block(uint64_t seed, uint64_t stream_id,
                                              uint64_t block) {
  return philox4x32_10(make_uint4((uint32_t)block, (uint32_t)(block >> 32),
                                  (uint32_t)stream_id, (uint32_t)(stream_id >> 32)),
                       make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
}
__device__ __forceinline__ uint32_t lane_of(const uint4& r, int l) {
  return l == 0 ? r.x : l == 1 ? r.y : l == 2 ? r.z : r.w;
}
__device__ __forceinline__ float u32_to_unit_f(uint32_t r) {
  return (float)(r >> 8) * 5.9604644775390625e-08f;  // 2^-24
}
// x 2^-53 for the leading 53 bits x, put together by bit moves: a conversion
// and a multiply would each hold the FP64 unit for 64 cycles a warp (fused
// fp64 Monte Carlo, 10^7 points, d = 6: 1296 us, and 913 us this way with the
// values summed as integers too).
__device__ __forceinline__ double u64_to_unit_d(uint32_t lo, uint32_t hi) {
  const uint64_t x = (((uint64_t)hi << 32) | lo) >> 11;
  const int lz = __clzll((long long)x);
  // the leading bit, moved to bit 52, adds one to the exponent field
  const uint64_t b = ((uint64_t)(1032 - lz) << 52) + (x << (lz - 11));
  return x ? __longlong_as_double((long long)b) : 0.0;
}
__host__ __device__ constexpr int gcd_c(int a, int b) { return b == 0 ? a : gcd_c(b, a % b); }
// Uniform number of flat element e of a request starting at block `offset`.
template <typename T>
struct Uniform;
template <>
struct Uniform<float> {
  static constexpr int per_block = 4;
  __device__ static float at(uint64_t seed, uint64_t sid, uint64_t offset, uint64_t e) {
    const uint4 r = philox_block(seed, sid, offset + (e >> 2));
    return u32_to_unit_f(lane_of(r, (int)(e & 3)));
  }
  __device__ static float from(const uint4& r, int lane) {
    return u32_to_unit_f(lane_of(r, lane));
  }
};
template <>
struct Uniform<double> {
  static constexpr int per_block = 2;
  __device__ static double at(uint64_t seed, uint64_t sid, uint64_t offset, uint64_t e) {
    const uint4 r = philox_block(seed, sid, offset + (e >> 1));
    return (e & 1) ? u64_to_unit_d(r.z, r.w) : u64_to_unit_d(r.x, r.y);
  }
  __device__ static double from(const uint4& r, int lane) {
    return lane ? u64_to_unit_d(r.z, r.w) : u64_to_unit_d(r.x, r.y);
  }
};

// --------------------------------------------- division by an invariant
// Unsigned 32-bit division by a run-time constant d >= 1 with one multiply-
// high, the round-up method of Granlund & Montgomery, "Division by invariant
// integers using multiplication" (PLDI 1994), Fig. 4.1:
//   l = ceil(log2 d), m = floor(2^32 (2^l - d) / d) + 1,
//   q = (t + ((n - t) >> min(l,1))) >> max(l-1,0), t = mulhi(m, n).
struct FastDiv {
  uint32_t d, m, s1, s2;
};
__host__ __device__ inline FastDiv make_fastdiv(uint32_t d) {
  FastDiv f;
  uint32_t l = 0;
  while (l < 32 && (uint64_t(1) << l) < d) ++l;
  f.d = d;
  f.m = (uint32_t)(((uint64_t(1) << 32) * ((uint64_t(1) << l) - d)) / d + 1);
  f.s1 = l < 1 ? l : 1;
  f.s2 = l > 1 ? l - 1 : 0;
  return f;
}
__device__ __forceinline__ uint32_t fdiv(uint32_t n, const FastDiv& f) {
  const uint32_t t = __umulhi(f.m, n);
  return (t + ((n - t) >> f.s1)) >> f.s2;
}

// ------------------------------------------------------------- grid nodes
// torch's CPU linspace, which IntegrationGrid uses through
// _linspace_with_grads (utils.py:24-58): step = (b-a)/(n-1) in the working
// type, the first half of the nodes from a forwards, the rest from b
// backwards, each a single rounding of step*i +- endpoint.
template <typename T>
__device__ __forceinline__ T linspace_node(T a, T b, T step, int64_t n, int64_t i) {
  if (i < n / 2) return fma(step, (T)i, a);
  return fma(-step, (T)(n - 1 - i), b);
}

// 1-D composite weights without the h factor, normalised so that the
// weight of node i is h * nc_coef(rule, i, n) (trapezoid.py:35,
// simpson.py:73-80, boole.py:154-163 collapse to these coefficients).
__device__ __forceinline__ double nc_coef(int rule, int64_t i, int64_t n) {
  if (rule == TQ_RULE_TRAPEZOID) return (i == 0 || i == n - 1) ? 0.5 : 1.0;
  if (rule == TQ_RULE_SIMPSON) {
    if (i == 0 || i == n - 1) return 1.0 / 3.0;
    return (i & 1) ? 4.0 / 3.0 : 2.0 / 3.0;
  }
  // Boole: h/22.5 * (7, 32, 12, 32, 14, 32, 12, 32, ..., 7)
  if (i == 0 || i == n - 1) return 7.0 / 22.5;
  const int64_t m = i & 3;
  if (m == 1 || m == 3) return 32.0 / 22.5;
  if (m == 2) return 12.0 / 22.5;
  return 14.0 / 22.5;
}

// ------------------------------------------------------- integrand families
template <typename T>
struct Family {
  int id, dim;
  T c, b;
  T a[kMaxDim];
  T u[kMaxDim];
};
// One dimension per thread (threads 0 .. kMaxDim - 1 of the CTA; the caller
// puts a barrier before the first use): a conversion from fp64 holds the
// FP64 unit as long for one lane as for a warp.
template <typename T>
__device__ __forceinline__ void load_family(Family<T>& f, int id, int dim,
                                            const double* __restrict__ p, int k = threadIdx.x) {
  if (k < kMaxDim) {
    f.a[k] = k < dim ? (T)p[2 + k] : T(0);
    f.u[k] = (k < dim && id == TQ_FN_GAUSSIAN) ? (T)p[2 + dim + k] : T(0);
  }
  if (k == 0) {
    f.id = id;
    f.dim = dim;
    f.c = (T)p[0];
    f.b = (T)p[1];
  }
}
// g_k(x_k): the per-dimension term of the separable sum.
template <int FAM, typename T>
__device__ __forceinline__ T fam_term(const Family<T>& f, int k, T x) {
  if (FAM == TQ_FN_GAUSSIAN) {
    const T d = x - f.u[k];
    return f.a[k] * (d * d);
  } else if (FAM == TQ_FN_SUM_SIN) {
    return sin(f.a[k] * x);
  } else {
    return f.a[k] * x;
  }
}
// F(s): the outer function of the separable sum.
template <int FAM, typename T>
__device__ __forceinline__ T fam_outer(const Family<T>& f, T s) {
  if (FAM == TQ_FN_EXP_SUM) return f.c * exp(s + f.b);
  if (FAM == TQ_FN_GAUSSIAN) return f.c * exp(-s);
  if (FAM == TQ_FN_OSCILLATORY) return f.c * cos((T)(2.0 * CUDART_PI) * f.b + s);
  return f.c * s;  // TQ_FN_SUM_SIN
}

}  // namespace tq

// Dispatch helpers: expand a runtime family id into a template argument.
#define TQ_DISPATCH_FAMILY(fam, FAMC, ...)                    \
  switch (fam) {                                              \
    case TQ_FN_EXP_SUM: {                                     \
      constexpr int FAMC = TQ_FN_EXP_SUM;                     \
      __VA_ARGS__;                                            \
    } break;                                                  \
    case TQ_FN_GAUSSIAN: {                                    \
      constexpr int FAMC = TQ_FN_GAUSSIAN;                    \
      __VA_ARGS__;                                            \
    } break;                                                  \
    case TQ_FN_OSCILLATORY: {                                 \
      constexpr int FAMC = TQ_FN_OSCILLATORY;                 \
      __VA_ARGS__;                                            \
    } break;                                                  \
    case TQ_FN_SUM_SIN: {                                     \
      constexpr int FAMC = TQ_FN_SUM_SIN;                     \
      __VA_ARGS__;                                            \
    } break;                                                  \
    default:                                                  \
      return TQ_ERR_FAMILY;                                   \
  }
