// Counter-based uniforms and fused Monte Carlo.
//
// The reference draws torch.rand([N, dim]) from the global generator
// (rng.py:120-125), scales it onto the domain (monte_carlo.py:102-106),
// evaluates the integrand and averages (monte_carlo.py:60-82).  Here the
// draws come from Philox4x32-10 keyed by the seed with an explicit block
// offset, so the fused kernel regenerates in registers exactly the values
// tq_uniform writes for the materialised path, and no [N, dim] buffer exists.

#include <type_traits>

#include "tq_common.cuh"

namespace tq {

template <typename T>
__global__ void __launch_bounds__(kBlock)
    uniform_kernel(uint64_t seed, uint64_t sid, uint64_t offset, int64_t numel, T* __restrict__ out) {
  constexpr int PB = Uniform<T>::per_block;
  const int64_t nblk = (numel + PB - 1) / PB;
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nblk;
       b += (int64_t)gridDim.x * blockDim.x) {
    const uint4 r = philox_block(seed, sid, offset + (uint64_t)b);
    const int64_t e0 = b * PB;
#pragma unroll
    for (int l = 0; l < PB; ++l)
      if (e0 + l < numel) out[e0 + l] = Uniform<T>::from(r, l);
  }
}

// Uniform points of a box, in one pass (tq_uniform and two torch operations
// wrote and read the [count, dim] array three times: 10^6 x 3 fp64 35 us on
// the device, 16.5 us here).  Two roundings per coordinate, as u * width + lo
// has them in torch.
template <typename T>
__global__ void __launch_bounds__(kBlock)
    sample_points_kernel(int dim, int64_t numel, const T* __restrict__ dom, uint64_t seed, uint64_t sid,
                         uint64_t offset, T* __restrict__ out) {
  constexpr int PB = Uniform<T>::per_block;
  __shared__ T lo[kMaxDim], width[kMaxDim];
  __shared__ FastDiv fd;
  if (threadIdx.x < dim) {
    lo[threadIdx.x] = dom[2 * threadIdx.x];
    width[threadIdx.x] = dom[2 * threadIdx.x + 1] - dom[2 * threadIdx.x];
  }
  if (threadIdx.x == 0) fd = make_fastdiv((uint32_t)dim);
  __syncthreads();
  const int64_t nblk = (numel + PB - 1) / PB;
  const bool small = numel <= (int64_t)0xffffffffll;
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nblk; b += (int64_t)gridDim.x * blockDim.x) {
    const uint4 r = philox_block(seed, sid, offset + (uint64_t)b);
    const int64_t e0 = b * PB;
    int k = small ? (int)((uint32_t)e0 - fdiv((uint32_t)e0, fd) * fd.d) : (int)(e0 % dim);
    alignas(16) T v[PB];
#pragma unroll
    for (int l = 0; l < PB; ++l) {
      const T u = Uniform<T>::from(r, l);
      if constexpr (sizeof(T) == 4)
        v[l] = __fadd_rn(__fmul_rn(u, width[k]), lo[k]);
      else
        v[l] = __dadd_rn(__dmul_rn(u, width[k]), lo[k]);
      k = k + 1 == dim ? 0 : k + 1;
    }
    if (e0 + PB <= numel && ((uintptr_t)out & 15) == 0) {  // a block's values are 16 bytes
      *(uint4*)(out + e0) = *(const uint4*)v;
    } else {
#pragma unroll
      for (int l = 0; l < PB; ++l)
        if (e0 + l < numel) out[e0 + l] = v[l];
    }
  }
}

struct McArgs {
  int dim, family;
  int64_t n_points;
  uint64_t seed, sid, offset;
  const void* domain;
  const double* params;
  Acc* partials;
  unsigned* ticket;
  void* out;
  double* out64;
  uint32_t key[20];  // the ten rounds' keys (operands from the parameter bank, no key arithmetic)
};

// philox_block with the round keys given.
__device__ __forceinline__ uint4 philox_keyed(const McArgs& a, uint64_t block) {
  uint4 c = make_uint4((uint32_t)block, (uint32_t)(block >> 32), (uint32_t)a.sid, (uint32_t)(a.sid >> 32));
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * c.x, p1 = (uint64_t)0xCD9E8D57u * c.z;
    c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ a.key[2 * r], (uint32_t)p1,
                   (uint32_t)(p0 >> 32) ^ c.w ^ a.key[2 * r + 1], (uint32_t)p0);
  }
  return c;
}

// Parameters and domain, one dimension per thread; ends with a barrier.
template <typename T>
__device__ __forceinline__ void mc_setup(const McArgs& a, Family<T>& fam, T* lo, T* width) {
  const T* dom = (const T*)a.domain;
  load_family<T>(fam, a.family, a.dim, a.params);
  if (threadIdx.x < a.dim) {
    const int k = threadIdx.x;
    lo[k] = dom[2 * k];
    width[k] = dom[2 * k + 1] - dom[2 * k];
  }
  __syncthreads();
}
// The threads' sums into the result, by the last CTA.
template <typename T>
__device__ __forceinline__ void mc_finish(const McArgs& a, Acc mine, const T* width) {
  const Acc acc = block_reduce<kBlock>(mine);
  if (threadIdx.x == 0) a.partials[blockIdx.x] = acc;
  if (last_block_arrives(a.ticket)) {
    const Acc t = partials_reduce<kBlock>(a.partials, (int)gridDim.x);
    if (threadIdx.x == 0) {
      T volume = (T)1;
      for (int k = 0; k < a.dim; ++k) volume = volume * width[k];
      const double v = (double)volume * (t.s + t.c) / (double)a.n_points;
      if (a.out) *(T*)a.out = (T)v;
      if (a.out64) *a.out64 = v;
      *a.ticket = 0u;
    }
  }
}

// Any dimension: fp64, and fp32 beyond ten dimensions.
template <typename T, int FAM, int P>
__global__ void __launch_bounds__(kBlock) mc_fused_kernel(McArgs a) {
  __shared__ Family<T> fam;
  __shared__ T lo[kMaxDim], width[kMaxDim];
  mc_setup<T>(a, fam, lo, width);
  constexpr int PB = Uniform<T>::per_block;
  const int dim = a.dim;
  F2 facc{0.f, 0.f};  // fp32: the strip sums as a double-float on the FP32 pipe
  FixAcc facc64;      // fp64: the values, exactly
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * P; base < a.n_points;
       base += nthreads * P) {
    const int64_t end = min(base + P, a.n_points);
    T inner = T(0), comp = T(0);
    uint64_t cur_blk = ~0ull;
    uint4 r = make_uint4(0, 0, 0, 0);
    for (int64_t p = base; p < end; ++p) {
      T s = T(0);
      for (int k = 0; k < dim; ++k) {
        const uint64_t e = (uint64_t)p * dim + k;
        const uint64_t blk = e / PB;
        if (blk != cur_blk) {
          r = philox_block(a.seed, a.sid, a.offset + blk);
          cur_blk = blk;
        }
        const T u = Uniform<T>::from(r, (int)(e - blk * PB));
        // monte_carlo.py:106: uniform * domain_sizes + domain_starts
        const T x = u * width[k] + lo[k];
        const T g = fam_term<FAM, T>(fam, k, x);
        s = (k == 0) ? g : s + g;
      }
      const T f = fam_outer<FAM, T>(fam, s);
      if constexpr (std::is_same<T, float>::value) {
        // compensated strip sum in the working type
        const T t = inner + f;
        comp += (fabs(inner) >= fabs(f)) ? ((inner - t) + f) : ((f - t) + inner);
        inner = t;
      } else {
        facc64.add(f);
      }
    }
    if constexpr (std::is_same<T, float>::value) facc = f2_add(f2_add(facc, inner), comp);
  }
  mc_finish<T>(a, std::is_same<T, float>::value ? Acc{(double)facc.hi, (double)facc.lo} : facc64.value(), width);
}

// fp32, d = D fixed at compile time: a thread takes groups of G consecutive
// points that use whole Philox blocks (no block is computed twice, no draw
// looks for its block), their terms unrolled with the parameters in
// registers.  Instruction issue bounds it: at d = 6 about 70 instructions of
// Philox and 60 of coordinates, terms and exp a point.  10^7 points, d = 6:
// 125 us with a block test per draw, 70 us here.
template <int FAM, int D>
constexpr int mc_ctas() {  // resident CTAs an SM: registers for parameters and draws without spills
  constexpr int regs = (FAM == TQ_FN_GAUSSIAN ? 4 : 3) * D + 4 * D / gcd_c(D, 4) + 24;
  return regs <= 64 ? 4 : regs <= 85 ? 3 : 2;
}
template <int FAM, int D>
__global__ void __launch_bounds__(kBlock, mc_ctas<FAM, D>()) mc_f32_kernel(McArgs a) {
  constexpr int PB = Uniform<float>::per_block;
  constexpr int GS = gcd_c(D, PB), G = PB / GS, NB = D / GS;
  __shared__ Family<float> fam;
  __shared__ float lo[kMaxDim], width[kMaxDim];
  mc_setup<float>(a, fam, lo, width);
  Family<float> f;  // this thread's copy, in registers
  float l[D], w[D];
  f.c = fam.c;
  f.b = fam.b;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    f.a[k] = fam.a[k];
    f.u[k] = fam.u[k];
    l[k] = lo[k];
    w[k] = width[k];
  }
  F2 sum{0.f, 0.f};
  const int64_t groups = (a.n_points + G - 1) / G;
  for (int64_t g = (int64_t)blockIdx.x * kBlock + threadIdx.x; g < groups; g += (int64_t)gridDim.x * kBlock) {
    uint32_t r[4 * NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const uint4 q = philox_keyed(a, a.offset + (uint64_t)g * NB + b);
      r[4 * b] = q.x;
      r[4 * b + 1] = q.y;
      r[4 * b + 2] = q.z;
      r[4 * b + 3] = q.w;
    }
    const int64_t left = a.n_points - g * G;
#pragma unroll
    for (int p = 0; p < G; ++p) {
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < D; ++k) {
        // monte_carlo.py:106: uniform * domain_sizes + domain_starts
        const float x = u32_to_unit_f(r[p * D + k]) * w[k] + l[k];
        const float t = fam_term<FAM, float>(f, k, x);
        s = k == 0 ? t : s + t;
      }
      sum = f2_add(sum, p < left ? fam_outer<FAM, float>(f, s) : 0.f);
    }
  }
  mc_finish<float>(a, Acc{(double)sum.hi, (double)sum.lo}, width);
}

}  // namespace tq

using namespace tq;

extern "C" int tq_uniform(int dtype, uint64_t seed, uint64_t stream_id, uint64_t offset,
                          int64_t numel, void* out, void* stream) {
  if (!valid_dtype(dtype)) return TQ_ERR_DTYPE;
  if (numel < 0 || (!out && numel > 0)) return TQ_ERR_ARG;
  if (numel == 0) return TQ_OK;
  const int64_t nblk = (numel + (dtype == TQ_F64 ? 1 : 3)) / (dtype == TQ_F64 ? 2 : 4);
  int64_t grid = (nblk + kBlock - 1) / kBlock;
  const int64_t cap = (int64_t)sm_count() * 16;
  if (grid > cap) grid = cap;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == TQ_F64)
    uniform_kernel<double><<<(unsigned)grid, kBlock, 0, s>>>(seed, stream_id, offset, numel,
                                                             (double*)out);
  else
    uniform_kernel<float><<<(unsigned)grid, kBlock, 0, s>>>(seed, stream_id, offset, numel,
                                                            (float*)out);
  return launch_status();
}

extern "C" int tq_sample_points(int dtype, int dim, int64_t count, const void* domain, uint64_t seed,
                                uint64_t stream_id, uint64_t offset, void* points, void* stream) {
  if (!valid_dtype(dtype)) return TQ_ERR_DTYPE;
  if (dim < 1 || dim > kMaxDim) return TQ_ERR_DIM;
  if (count < 0 || !domain || (!points && count > 0)) return TQ_ERR_ARG;
  if (count > (int64_t(1) << 60) / dim) return TQ_ERR_TOO_LARGE;
  if (count == 0) return TQ_OK;
  const int64_t numel = count * dim;
  const int64_t nblk = (numel + (dtype == TQ_F64 ? 1 : 3)) / (dtype == TQ_F64 ? 2 : 4);
  int64_t grid = (nblk + kBlock - 1) / kBlock;
  const int64_t cap = (int64_t)sm_count() * 16;
  if (grid > cap) grid = cap;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == TQ_F64)
    sample_points_kernel<double><<<(unsigned)grid, kBlock, 0, s>>>(dim, numel, (const double*)domain, seed, stream_id,
                                                                   offset, (double*)points);
  else
    sample_points_kernel<float><<<(unsigned)grid, kBlock, 0, s>>>(dim, numel, (const float*)domain, seed, stream_id,
                                                                  offset, (float*)points);
  return launch_status();
}

// Points a thread takes at a time: two, so that an odd number of fp64 draws a
// point uses whole Philox blocks; more would leave small calls on few threads
// (10^4 points, d = 6, fp64: 47 us in strips of eight, 16.5 us in pairs).
static constexpr int kStripMC = 2;

static int64_t mc_blocks(int64_t n, int strip) {
  const int64_t need = (n + (int64_t)kBlock * strip - 1) / ((int64_t)kBlock * strip);
  const int64_t cap = (int64_t)sm_count() * 8;
  return need < 1 ? 1 : (need < cap ? need : cap);
}
// CTAs whose partials any workspace of this call has always held.
static int64_t mc_least(int64_t n) { return mc_blocks(n, 8); }

extern "C" size_t tq_mc_fused_workspace_size(int dim, int64_t n_points) {
  (void)dim;
  return reduce_ws_bytes(mc_blocks(n_points, kStripMC));
}

extern "C" int tq_mc_fused(int dtype, int dim, int64_t n_points, const void* domain, int family,
                           const double* params, uint64_t seed, uint64_t stream_id,
                           uint64_t offset, void* out, double* out64, void* workspace,
                           size_t workspace_bytes, void* stream) {
  if (!valid_dtype(dtype)) return TQ_ERR_DTYPE;
  if (dim < 1 || dim > kMaxDim) return TQ_ERR_DIM;
  if (n_points < 1 || !domain || !params || !workspace || (!out && !out64)) return TQ_ERR_ARG;
  if (n_points > (int64_t(1) << 60) / dim) return TQ_ERR_TOO_LARGE;
  if (workspace_bytes < reduce_ws_bytes(mc_least(n_points))) return TQ_ERR_WORKSPACE;
  int64_t blocks = mc_blocks(n_points, kStripMC);
  const int64_t slots = (int64_t)((workspace_bytes - 256) / sizeof(Acc));
  if (blocks > slots) blocks = slots;
  McArgs a;
  a.dim = dim;
  a.family = family;
  a.n_points = n_points;
  a.seed = seed;
  a.sid = stream_id;
  a.offset = offset;
  a.domain = domain;
  a.params = params;
  a.ticket = (unsigned*)workspace;
  a.partials = (Acc*)((char*)workspace + 256);
  a.out = out;
  a.out64 = out64;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  for (int r = 0; r < 10; ++r, k0 += 0x9E3779B9u, k1 += 0xBB67AE85u) {
    a.key[2 * r] = k0;
    a.key[2 * r + 1] = k1;
  }
  cudaStream_t s = (cudaStream_t)stream;
  // one wave of resident CTAs
  const int64_t sms = sm_count();
#define TQ_MC_DIM(DV)                                                              \
  case DV: {                                                                       \
    const int64_t wave = sms * mc_ctas<FAM, DV>();                                 \
    mc_f32_kernel<FAM, DV><<<(unsigned)(blocks < wave ? blocks : wave), kBlock, 0, s>>>(a); \
  } break;
  TQ_DISPATCH_FAMILY(family, FAM, {
    if (dtype == TQ_F64) {
      mc_fused_kernel<double, FAM, kStripMC><<<(unsigned)blocks, kBlock, 0, s>>>(a);
    } else {
      switch (dim) {
        TQ_MC_DIM(1) TQ_MC_DIM(2) TQ_MC_DIM(3) TQ_MC_DIM(4) TQ_MC_DIM(5) TQ_MC_DIM(6) TQ_MC_DIM(7) TQ_MC_DIM(8)
        TQ_MC_DIM(9) TQ_MC_DIM(10)
        default: mc_fused_kernel<float, FAM, kStripMC><<<(unsigned)blocks, kBlock, 0, s>>>(a);
      }
    }
  });
#undef TQ_MC_DIM
  return launch_status();
}
