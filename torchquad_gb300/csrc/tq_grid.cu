// Tensor-product quadrature on GB300: fused node generation + integrand +
// weighted sum for built-in integrands, and the node / weight / weighted-sum
// kernels of the materialised path used for arbitrary torch integrands.
//
// The reference builds the full [n^d, d] point tensor (integration_grid.py:
// 95-99), evaluates the integrand on it, transposes the values
// (grid_integrator.py:80) and collapses one dimension at a time
// (trapezoid.py:27-37, simpson.py:29-46, boole.py:29-48, gaussian.py:131-144).
// Here a thread walks a strip of consecutive flat node indices (last
// dimension fastest, the reference's meshgrid "ij" order), keeps the
// outer-dimension coordinates and weight product in registers, and sums
// w_i * f(x_i) directly; the per-dimension collapse becomes the product of
// 1-D weights, which is the same quadrature.

#include <type_traits>

#include "tq_separable.cuh"

namespace tq {

// ------------------------------------------------------------------ fused
struct FusedArgs {
  int rule, dim, family;
  int64_t n, total;
  const void* domain;
  const double* gl_nodes;
  const double* gl_weights;
  const double* params;
  Acc* partials;
  int64_t slots;  // partials the workspace holds
  int sms;        // SMs of the device
  unsigned* ticket;
  void* out;
  int out_dtype;
  double* out64;
};

__device__ __forceinline__ void write_result(void* out, int out_dtype, double* out64,
                                             double v) {
  if (out) {
    if (out_dtype == TQ_F64)
      *(double*)out = v;
    else
      *(float*)out = (float)v;
  }
  if (out64) *out64 = v;
}

// Compensated sum of one row segment in the working type: Kahan's original
// four-operation update for fp32, plain accumulation for fp64 (a segment is
// at most n terms of one row).
template <typename T>
struct SegSum;
template <>
struct SegSum<float> {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  }
  __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};
template <>
struct SegSum<double> {
  double s = 0.0;
  __device__ __forceinline__ void add(double x) { s += x; }
  __device__ __forceinline__ double value() const { return s; }
};

// Outer-dimension state of a grid row (flat node index / n): the partial
// separable sum g_0 + ... + g_{d-2} in dimension order and the product of
// the outer 1-D weights.  rstride[k] = n^(dim-2-k).
template <typename T, int RULE, int FAM>
__device__ __forceinline__ void outer_state(const Geo<T>& g, const Family<T>& fam,
                                            const uint64_t* rstride, int dim, int64_t n,
                                            uint64_t row, const double* gl_nodes,
                                            const double* gl_w, bool small, T& s_out,
                                            double& w_out) {
  constexpr bool GL = RULE == TQ_RULE_GAUSS;
  T s = T(0);
  double w = 1.0;
#pragma unroll 1
  for (int k = 0; k < dim - 1; ++k) {
    uint64_t digit;
    if (small) {
      const uint32_t q = (uint32_t)row / (uint32_t)rstride[k];
      digit = q % (uint32_t)n;
    } else {
      digit = (row / rstride[k]) % (uint64_t)n;
    }
    const T x = node_at<T, GL>(g, k, n, (int64_t)digit, gl_nodes);
    const T t = fam_term<FAM, T>(fam, k, x);
    s = (k == 0) ? t : s + t;
    w *= g.wscale[k] *
         (GL ? __ldg(gl_w + digit) : (double)nc_int_t<RULE>((int)digit, (int)n));
  }
  s_out = s;
  w_out = w;
}

template <typename T, typename D, int RULE, int FAM, int P>
__global__ void __launch_bounds__(kBlock, 2) grid_fused_kernel(FusedArgs args) {
  constexpr bool GL = RULE == TQ_RULE_GAUSS;
  __shared__ Geo<T> g;
  __shared__ Family<T> fam;
  __shared__ uint64_t rstride[kMaxDim];
  // the factored form, by the first few CTAs; the others have nothing to do
  const bool sep = (args.dim > 1 || args.n <= kSepRow) &&
                   sep_ok<T, D>(FAM, args.dim, args.n, (const D*)args.domain, args.params);
  if (sep && blockIdx.x >= (unsigned)sep_ctas(args.dim, args.n)) return;
  geo_setup<T, D>(g, RULE, args.dim, args.n, (const D*)args.domain);
  load_family<T>(fam, args.family, args.dim, args.params);
  if (sep) {
    __shared__ Acc dsum[kMaxDim][kSepMaxM<false>];
    __shared__ Acc sp[kSepSlots<false>];
    __syncthreads();
    if (sep_sums<T, FAM, false>(g, fam, RULE, args.dim, args.n, args.gl_nodes, args.gl_weights, blockIdx.x,
                                gridDim.x, args.partials, args.slots, args.ticket, dsum, sp) &&
        threadIdx.x < 32) {
      const Acc v = dd_mul(sep_value<FAM>(dsum, args.dim), (double)fam.c);
      if (threadIdx.x == 0) write_result(args.out, args.out_dtype, args.out64, v.s + v.c);
    }
    return;
  }
  if (threadIdx.x == 0) {
    uint64_t st = 1;
    for (int k = args.dim - 2; k >= 0; --k) {
      rstride[k] = st;
      st *= (uint64_t)args.n;
    }
  }
  __syncthreads();
  const int dim = args.dim, last = dim - 1;
  const int64_t n = args.n, total = args.total;
  const int n32 = (int)n;  // n <= total < 2^62 but a row index fits int for n < 2^31
  const bool small = total < (int64_t(1) << 32);
  const double* gl_nodes = args.gl_nodes;
  const double* gl_w = args.gl_weights;
  const double wlast = g.wscale[last];
  const T a_l = g.a[last], b_l = g.b[last], st_l = g.step[last];
  const int half = n32 / 2;
  // fp64: last-dimension tables (one outer-function evaluation per row)
  bool use_tab = false;
  InnerTab* tab = nullptr;
  if constexpr (std::is_same<T, double>::value) {
    __shared__ InnerTab tab_s;
    tab = &tab_s;
    if (dim >= 2 && n <= kTabMax)
      use_tab = build_inner_tab<FAM>(tab_s, g, fam, last, n32, GL, RULE, gl_nodes, gl_w);
  }

  Acc acc{0.0, 0.0};
  bool rows_done = false;
  if constexpr (std::is_same<T, double>::value) {
    if (use_tab) {
      // a contiguous node range per CTA, rows in groups of 32 per warp
      __shared__ FastDiv fdn;
      __shared__ RowTab rt;
      if (threadIdx.x == 0) fdn = make_fastdiv((uint32_t)n);
      __syncthreads();
      const int64_t b0 = total * (int64_t)blockIdx.x / gridDim.x, b1 = total * ((int64_t)blockIdx.x + 1) / gridDim.x;
      if (b1 > b0) acc = tab_rows_sum<FAM>(g, fam, *tab, rt, dim, args.rule, GL, n, fdn, gl_nodes, gl_w, b0, b1);
      rows_done = true;
    }
  }
  if constexpr (std::is_same<T, double>::value && !GL) {
    if (dim == 1) {
      // chains of a length that gives every sub-partition's FP64 unit one warp
      // (a chain's start costs as much as 60 of its nodes), warps in turn
      // over the CTAs
      __shared__ ChainTab ct;
      __shared__ ChainTodo todo;
      chain_table<FAM>(ct, fam, RULE, st_l, 0);
      __syncthreads();
      const int64_t blk = total / (kBlk * (int64_t)args.sms * 128) + 1;
      const int len = (int)min((int64_t)kChain, blk * kBlk);
      const int64_t chain = ((int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
      const int64_t step = (int64_t)gridDim.x * blockDim.x;
      acc = chain_rows<FAM>(g, fam, ct, todo, RULE, n, 0, total, len, chain, step,
                            ((total + len - 1) / len + step - 1) / step);
      acc.s *= wlast;
      acc.c *= wlast;
      rows_done = true;
    }
  }
  RecurConst rc{1.0, 1.0, 0.0};
  if constexpr (std::is_same<T, double>::value) {
    if (!rows_done && !GL) rc = recur_const<FAM>(fam, last, st_l);
  }
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * P; base < total && !rows_done;
       base += nthreads * P) {
    uint64_t row;
    int jl;
    if (small) {
      const uint32_t q = (uint32_t)base / (uint32_t)n;
      row = q;
      jl = (int)((uint32_t)base - q * (uint32_t)n);
    } else {
      row = (uint64_t)base / (uint64_t)n;
      jl = (int)(base - (int64_t)row * n);
    }
    int64_t left = min((int64_t)P, total - base);
    while (left > 0) {
      T s_outer;
      double w_outer;
      outer_state<T, RULE, FAM>(g, fam, rstride, dim, n, row, gl_nodes, gl_w, small, s_outer,
                                w_outer);
      const int seg_end = (int)min((int64_t)n32, (int64_t)jl + left);
      SegSum<T> seg;
      bool tabbed = false;
      if constexpr (std::is_same<T, double>::value) {
        if (!GL) {
          // rows longer than a table: equally spaced nodes by recurrence
          double v;
          const double x0 = linspace_node<double>(a_l, b_l, st_l, n, jl);
          const double x1 = linspace_node<double>(a_l, b_l, st_l, n, seg_end - 1);
          if (recur_seg<FAM, RULE>(fam, rc, last, s_outer, x0, x1, st_l, jl, seg_end, n32, &v)) {
            seg.add(v);
            tabbed = true;
          }
        }
      }
      if (!tabbed) {
        for (int j = jl; j < seg_end; ++j) {
          T x;
          if (GL)
            x = (T)__dadd_rn(__dmul_rn(g.half[last], __ldg(gl_nodes + j)), g.mid[last]);
          else
            x = (j < half) ? fma(st_l, (T)j, a_l) : fma(-st_l, (T)(n32 - 1 - j), b_l);
          const T f = fam_outer<FAM, T>(fam, s_outer + fam_term<FAM, T>(fam, last, x));
          const T wj = GL ? (T)__ldg(gl_w + j) : (T)nc_int_t<RULE>(j, n32);
          seg.add(wj * f);
        }
      }
      acc_add(acc, seg.value() * (w_outer * wlast));
      left -= seg_end - jl;
      jl = 0;
      ++row;
    }
  }

  acc = block_reduce<kBlock>(acc);
  if (threadIdx.x == 0) args.partials[blockIdx.x] = acc;
  if (last_block_arrives(args.ticket)) {
    const Acc t = partials_reduce<kBlock>(args.partials, (int)gridDim.x);
    if (threadIdx.x == 0) {
      write_result(args.out, args.out_dtype, args.out64, t.s + t.c);
      *args.ticket = 0u;
    }
  }
}

// ------------------------------------------------------ materialised path
struct PointsArgs {
  int rule, dim;
  int64_t n, start, count;
  const void* domain;
  const double* gl_nodes;
  void* points;
};

// One thread per output element (point p, dimension k): coalesced stores of
// the [count, dim] row-major point tensor.
template <typename T, typename D, bool GL>
__global__ void __launch_bounds__(kBlock) grid_points_kernel(PointsArgs args) {
  __shared__ Geo<T> g;
  __shared__ uint64_t stride[kMaxDim];
  geo_setup<T, D>(g, args.rule, args.dim, args.n, (const D*)args.domain);
  if (threadIdx.x == 0) {
    uint64_t s = 1;
    for (int k = args.dim - 1; k >= 0; --k) {
      stride[k] = s;
      s *= (uint64_t)args.n;
    }
  }
  __syncthreads();
  const int dim = args.dim;
  const uint64_t n = (uint64_t)args.n;
  const uint64_t numel = (uint64_t)args.count * dim;
  T* out = (T*)args.points;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < numel;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t p = e / (uint64_t)dim;
    const int k = (int)(e - p * dim);
    const uint64_t digit = ((args.start + p) / stride[k]) % n;
    out[e] = node_at<T, GL>(g, k, (int64_t)n, (int64_t)digit, args.gl_nodes);
  }
}

// Tiled variant (HBM-write bound): a CTA builds a tile of consecutive
// points in shared memory (one thread per point; digits by multiply-high
// division by n; node values from a per-CTA table of every dimension's
// nodes), then one thread hands the tile to the bulk-copy engine
// (cp.async.bulk shared -> global), so the stores are full-line writes
// issued without per-thread store instructions.  Two tile buffers alternate;
// a buffer is rewritten only after its previous copy has been read out
// (cp.async.bulk.wait_group.read 1).  Needs a 16-byte aligned output.
constexpr int kPtsTileBytes = 24 * 1024;  // per buffer (two buffers per CTA)
constexpr int kPtsTab = 2048;             // node-table entries (dim * n) a CTA keeps

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

template <typename T, typename D, bool GL>
__global__ void __launch_bounds__(kBlock) grid_points_tiled_kernel(PointsArgs args, int tile_pts,
                                                                   int64_t n_tiles) {
  extern __shared__ __align__(128) unsigned char pts_smem[];
  __shared__ Geo<T> g;
  __shared__ FastDiv fd_n;
  __shared__ T nodes[kPtsTab];  // nodes[k * n + j], when dim * n fits
  geo_setup<T, D>(g, args.rule, args.dim, args.n, (const D*)args.domain);
  if (threadIdx.x == 0) {
    fd_n = make_fastdiv((uint32_t)args.n);
  }
  __syncthreads();
  const int dim = args.dim;
  const uint64_t n = (uint64_t)args.n;
  const int n32 = (int)args.n;
  // the nodes of every dimension once per CTA (no per-point node arithmetic)
  const bool tab = (int64_t)dim * args.n <= kPtsTab;
  if (tab)
    for (int e = threadIdx.x; e < dim * n32; e += blockDim.x)
      nodes[e] = node_at<T, GL>(g, e / n32, (int64_t)n, (int64_t)(e % n32), args.gl_nodes);
  // point indices below 2^32 (all but huge grids): 32-bit digits
  const bool small = (uint64_t)(args.start + args.count) <= 0xffffffffull;
  int buf = 0;
  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    T* sm = (T*)(pts_smem + (size_t)buf * kPtsTileBytes);
    const int64_t p0 = tile * (int64_t)tile_pts;  // local point index
    const int np = (int)min((int64_t)tile_pts, args.count - p0);
    if (threadIdx.x == 0) {
      // the copy that last read this buffer (two tiles ago) must be done
      asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
    }
    __syncthreads();
    for (int p = threadIdx.x; p < np; p += blockDim.x) {
      const uint64_t idx = (uint64_t)(args.start + p0 + p);
      T* row = sm + (size_t)p * dim;
      if (small && tab) {
        uint32_t r = (uint32_t)idx;
        for (int k = dim - 1; k >= 0; --k) {
          const uint32_t q = fdiv(r, fd_n);
          row[k] = nodes[k * n32 + (int)(r - q * fd_n.d)];
          r = q;
        }
      } else {
        uint64_t r = idx;
        for (int k = dim - 1; k >= 0; --k) {
          const uint64_t q = r / n;
          row[k] = node_at<T, GL>(g, k, (int64_t)n, (int64_t)(r - q * n), args.gl_nodes);
          r = q;
        }
      }
    }
    // generic-proxy writes of the tile -> visible to the bulk copy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    const size_t bytes = (size_t)np * dim * sizeof(T);
    const size_t bulk = bytes & ~(size_t)15;
    unsigned char* dst = (unsigned char*)args.points + (size_t)p0 * dim * sizeof(T);
    if (threadIdx.x == 0 && bulk > 0) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                   "r"(smem_u32(sm)), "r"((uint32_t)bulk)
                   : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    // a tail of 4, 8 or 12 bytes (only in the last tile) by plain stores
    for (size_t b = bulk + threadIdx.x * sizeof(T); b < bytes; b += blockDim.x * sizeof(T))
      *(T*)(dst + b) = *(const T*)((const unsigned char*)sm + b);
    buf ^= 1;
  }
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

struct WeightsArgs {
  int rule, dim;
  int64_t n, start, count;
  const void* domain;
  const double* gl_weights;
  double* weights;
};

template <typename T, typename D, bool GL>
__global__ void __launch_bounds__(kBlock) grid_weights_kernel(WeightsArgs args) {
  __shared__ Geo<T> g;
  geo_setup<T, D>(g, args.rule, args.dim, args.n, (const D*)args.domain);
  __syncthreads();
  const int dim = args.dim;
  const uint64_t n = (uint64_t)args.n;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < (uint64_t)args.count;
       p += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t r = args.start + p;
    double w = 1.0;
    for (int k = dim - 1; k >= 0; --k) {
      const uint64_t q = r / n, digit = r - q * n;
      r = q;
      w *= g.wscale[k] * wunit_at<GL>(args.rule, (int64_t)n, (int64_t)digit, args.gl_weights);
    }
    args.weights[p] = w;
  }
}

}  // namespace tq

using namespace tq;

// --------------------------------------------------------------- C ABI
static bool valid_rule(int rule, int64_t n) {
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

static bool grid_total(int dim, int64_t n, int64_t* total) {
  int64_t t = 1;
  for (int k = 0; k < dim; ++k) {
    if (t > (int64_t(1) << 62) / n) return false;
    t *= n;
  }
  *total = t;
  return true;
}

static constexpr int kStripF = 32, kStripD = 16;

static int64_t fused_blocks(int64_t total, int strip) {
  const int64_t need = (total + (int64_t)kBlock * strip - 1) / ((int64_t)kBlock * strip);
  const int64_t cap = (int64_t)sm_count() * 8;
  return need < 1 ? 1 : (need < cap ? need : cap);
}

extern "C" size_t tq_grid_fused_workspace_size(int rule, int dim, int64_t n_per_dim) {
  (void)rule;
  (void)dim;
  (void)n_per_dim;
  return reduce_ws_bytes((int64_t)sm_count() * 8);
}

extern "C" int tq_grid_fused(int dtype, int rule, int dim, int64_t n_per_dim, const void* domain,
                             const double* gl_nodes, const double* gl_weights, int family,
                             const double* params, void* out, int out_dtype, double* out64,
                             void* workspace, size_t workspace_bytes, void* stream) {
  if (!valid_dtype(dtype) || !valid_dtype(out_dtype)) return TQ_ERR_DTYPE;
  if (dim < 1 || dim > kMaxDim) return TQ_ERR_DIM;
  if (!valid_rule(rule, n_per_dim)) return TQ_ERR_RULE;
  if (!domain || !params || !workspace || (!out && !out64)) return TQ_ERR_ARG;
  if (rule == TQ_RULE_GAUSS && (!gl_nodes || !gl_weights)) return TQ_ERR_ARG;
  int64_t total;
  if (!grid_total(dim, n_per_dim, &total)) return TQ_ERR_TOO_LARGE;
  const bool gl = rule == TQ_RULE_GAUSS;
  const bool f64 = gl || dtype == TQ_F64;
  int64_t blocks = fused_blocks(total, f64 ? kStripD : kStripF);
  if (workspace_bytes < reduce_ws_bytes(blocks)) return TQ_ERR_WORKSPACE;
  // a small grid whose 1-D sums can use more CTAs than its nodes need
  const int64_t sb = sep_ctas(dim, n_per_dim);
  if (blocks < sb && (dim > 1 || n_per_dim <= kSepRow) && workspace_bytes >= reduce_ws_bytes(sb)) blocks = sb;
  FusedArgs a;
  a.rule = rule;
  a.dim = dim;
  a.family = family;
  a.n = n_per_dim;
  a.total = total;
  a.domain = domain;
  a.gl_nodes = gl_nodes;
  a.gl_weights = gl_weights;
  a.params = params;
  a.ticket = (unsigned*)workspace;
  a.partials = (Acc*)((char*)workspace + 256);
  a.slots = (int64_t)((workspace_bytes - 256) / sizeof(Acc));
  a.sms = sm_count();
  a.out = out;
  a.out_dtype = out_dtype;
  a.out64 = out64;
  cudaStream_t s = (cudaStream_t)stream;
  const dim3 grid((unsigned)blocks);
#define TQ_FUSED_RULE(RULEC)                                                              \
  if (dtype == TQ_F64)                                                                     \
    grid_fused_kernel<double, double, RULEC, FAM, kStripD><<<grid, kBlock, 0, s>>>(a);     \
  else                                                                                     \
    grid_fused_kernel<float, float, RULEC, FAM, kStripF><<<grid, kBlock, 0, s>>>(a);
  TQ_DISPATCH_FAMILY(family, FAM, {
    switch (rule) {
      case TQ_RULE_TRAPEZOID: { TQ_FUSED_RULE(TQ_RULE_TRAPEZOID) } break;
      case TQ_RULE_SIMPSON: { TQ_FUSED_RULE(TQ_RULE_SIMPSON) } break;
      case TQ_RULE_BOOLE: { TQ_FUSED_RULE(TQ_RULE_BOOLE) } break;
      default: {  // Gauss: fp64 nodes on the domain of either type
        if (dtype == TQ_F64)
          grid_fused_kernel<double, double, TQ_RULE_GAUSS, FAM, kStripD><<<grid, kBlock, 0, s>>>(a);
        else
          grid_fused_kernel<double, float, TQ_RULE_GAUSS, FAM, kStripD><<<grid, kBlock, 0, s>>>(a);
      }
    }
  });
#undef TQ_FUSED_RULE
  return launch_status();
}

static int64_t stream_blocks(int64_t work) {
  const int64_t need = (work + kBlock - 1) / kBlock;
  const int64_t cap = (int64_t)sm_count() * 16;
  return need < 1 ? 1 : (need < cap ? need : cap);
}

extern "C" int tq_grid_points(int dtype, int rule, int dim, int64_t n_per_dim,
                              const void* domain, const double* gl_nodes, int64_t start,
                              int64_t count, void* points, void* stream) {
  if (!valid_dtype(dtype)) return TQ_ERR_DTYPE;
  if (dim < 1 || dim > kMaxDim) return TQ_ERR_DIM;
  if (!valid_rule(rule, n_per_dim)) return TQ_ERR_RULE;
  if (!domain || !points || start < 0 || count < 0) return TQ_ERR_ARG;
  if (rule == TQ_RULE_GAUSS && !gl_nodes) return TQ_ERR_ARG;
  int64_t total;
  if (!grid_total(dim, n_per_dim, &total)) return TQ_ERR_TOO_LARGE;
  if (start + count > total) return TQ_ERR_ARG;
  if (count == 0) return TQ_OK;
  PointsArgs a{rule, dim, n_per_dim, start, count, domain, gl_nodes, points};
  cudaStream_t s = (cudaStream_t)stream;
  const size_t tsize = (rule == TQ_RULE_GAUSS || dtype == TQ_F64) ? 8 : 4;
  // tiles of a multiple of 16 points that fill a 24 KiB buffer
  const int tile_pts = (int)((kPtsTileBytes / (tsize * (size_t)dim)) & ~(size_t)15);
  if ((((uintptr_t)points) & 15) == 0 && tile_pts >= 16) {
    const int64_t n_tiles = (count + tile_pts - 1) / tile_pts;
    const int64_t cap = (int64_t)sm_count() * 4;
    const dim3 grid((unsigned)(n_tiles < cap ? n_tiles : cap));
    const size_t smem = 2 * (size_t)kPtsTileBytes;
#define TQ_PTS_TILED(T, D, GLB)                                                                     \
  {                                                                                                 \
    auto k = grid_points_tiled_kernel<T, D, GLB>;                                                   \
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (e != cudaSuccess) return set_cuda_error(e);                                                 \
    k<<<grid, kBlock, smem, s>>>(a, tile_pts, n_tiles);                                             \
  }
    if (rule == TQ_RULE_GAUSS) {
      if (dtype == TQ_F64) TQ_PTS_TILED(double, double, true)
      else TQ_PTS_TILED(double, float, true)
    } else if (dtype == TQ_F64) {
      TQ_PTS_TILED(double, double, false)
    } else {
      TQ_PTS_TILED(float, float, false)
    }
#undef TQ_PTS_TILED
    return launch_status();
  }
  // unaligned output: one thread per element
  const dim3 grid((unsigned)stream_blocks(count * dim));
  if (rule == TQ_RULE_GAUSS) {
    if (dtype == TQ_F64)
      grid_points_kernel<double, double, true><<<grid, kBlock, 0, s>>>(a);
    else
      grid_points_kernel<double, float, true><<<grid, kBlock, 0, s>>>(a);
  } else if (dtype == TQ_F64) {
    grid_points_kernel<double, double, false><<<grid, kBlock, 0, s>>>(a);
  } else {
    grid_points_kernel<float, float, false><<<grid, kBlock, 0, s>>>(a);
  }
  return launch_status();
}

extern "C" int tq_grid_weights(int dtype, int rule, int dim, int64_t n_per_dim,
                               const void* domain, const double* gl_weights, int64_t start,
                               int64_t count, double* weights, void* stream) {
  if (!valid_dtype(dtype)) return TQ_ERR_DTYPE;
  if (dim < 1 || dim > kMaxDim) return TQ_ERR_DIM;
  if (!valid_rule(rule, n_per_dim)) return TQ_ERR_RULE;
  if (!domain || !weights || start < 0 || count < 0) return TQ_ERR_ARG;
  if (rule == TQ_RULE_GAUSS && !gl_weights) return TQ_ERR_ARG;
  int64_t total;
  if (!grid_total(dim, n_per_dim, &total)) return TQ_ERR_TOO_LARGE;
  if (start + count > total) return TQ_ERR_ARG;
  if (count == 0) return TQ_OK;
  WeightsArgs a{rule, dim, n_per_dim, start, count, domain, gl_weights, weights};
  cudaStream_t s = (cudaStream_t)stream;
  const dim3 grid((unsigned)stream_blocks(count));
  if (rule == TQ_RULE_GAUSS) {
    if (dtype == TQ_F64)
      grid_weights_kernel<double, double, true><<<grid, kBlock, 0, s>>>(a);
    else
      grid_weights_kernel<double, float, true><<<grid, kBlock, 0, s>>>(a);
  } else if (dtype == TQ_F64) {
    grid_weights_kernel<double, double, false><<<grid, kBlock, 0, s>>>(a);
  } else {
    grid_weights_kernel<float, float, false><<<grid, kBlock, 0, s>>>(a);
  }
  return launch_status();
}

// ------------------------------------------- allocation-free entry point
// For callers that cannot allocate device memory at call time: a plugin
// inside a host application that owns all device memory, code that must not
// allocate once it runs (a fixed-latency loop), or a plain C caller that has
// no allocator to hand.  The CTA partials and the ticket word of the fused
// grid rule live in this file-scope device array instead of a caller-given
// workspace.  Every GPU that loads the library holds it until exit.
#include <mutex>

namespace {

constexpr int kNoAllocSlots = 4096;  // CTA partials the static scratch holds
constexpr size_t kNoAllocBytes = 256 + (size_t)kNoAllocSlots * sizeof(tq::Acc);

__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

std::mutex g_noalloc_mu;
void* g_noalloc_ptr[64] = {};

// Device address of g_noalloc_scratch on the current device, looked up once
// per device (host code only sees a host-side stand-in under the array's
// name, which must never be handed to a kernel).
int noalloc_scratch(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return tq::set_cuda_error(e);
  if (dev < 0 || dev >= 64) return TQ_ERR_ARG;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) return tq::set_cuda_error(e == cudaSuccess ? cudaErrorInvalidSymbol : e);
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return TQ_OK;
}

}  // namespace

extern "C" int tq_grid_fused_noalloc(int dtype, int rule, int dim, int64_t n_per_dim,
                                     const void* domain, const double* gl_nodes,
                                     const double* gl_weights, int family, const double* params,
                                     void* out, int out_dtype, double* out64, void* stream) {
  if (tq_grid_fused_workspace_size(rule, dim, n_per_dim) > kNoAllocBytes) return TQ_ERR_SCRATCH;
  void* scratch = nullptr;
  int rc = noalloc_scratch(&scratch);
  if (rc != TQ_OK) return rc;
  // the ticket word must start at zero; the last CTA leaves it at zero
  const cudaError_t e = cudaMemsetAsync(scratch, 0, 16, (cudaStream_t)stream);
  if (e != cudaSuccess) return tq::set_cuda_error(e);
  return tq_grid_fused(dtype, rule, dim, n_per_dim, domain, gl_nodes, gl_weights, family, params,
                       out, out_dtype, out64, scratch, kNoAllocBytes, stream);
}
