// Elementwise programs with a reduction of one of their results in the same launch.
//
// A reduction behind a program reads again what the program has just written; where the result is wanted for nothing else, as the term
// that a bias gradient sums, it was written for that alone.  Here the column sums of an output are kept in registers, a thread per column or
// four, down a piece of the rows, and only the pieces' sums are written; and a block that has computed a row, up to 8192 columns, goes on to
// its logsumexp while the row is in shared memory.  A program is found as in fused_known.cuh, in a list of its own: each reduction is another
// kernel.
//
// Measured on [4096, 4096], mean of the logsumexp of exp(-x^2) + tanh(x b) + sin(x) / (1 + x^2) and its gradients to x and b in a captured step:
// 204 us with the programs and the reductions apart, 148 us here (201 MB, 31 us at the copy bandwidth): the rows with their logsumexp
// 58 us, the gradient with the column sums 88 us, both bound by instruction issue (125 and 190 slots a warp and element).
#include <algorithm>
#include <vector>

#include "fused_known.cuh"

rt_status rt_sum_axis_internal(rt_ctx* ctx, const float* x, int64_t outer, int64_t len, int64_t inner, float* out, float scale);

namespace {

constexpr int kRowThreads = 256, kLongestRow = 8192;

struct ReducedParams {
  FusedParams f;
  int rows, cols, which;  // the output that is reduced
  int rows_per_block;
  float* out;             // column sums: [piece][cols]; logsumexp: [rows]
};

// Output `which` is added up instead of being written.
template <bool VEC>
struct Sums {
  int which;
  float sum[VEC ? 4 : 1];
  template <int OUT, bool V>
  __device__ __forceinline__ void put(const FusedParams& p, const Quad<VEC>& e, const float (&acc)[4]) {
    if (OUT != which) {
      Store().template put<OUT, VEC>(p, e, acc);
      return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (e.live[VEC ? 0 : i]) sum[VEC ? i : 0] += acc[i];
  }
};
// A warp has 128 columns (VEC: four a lane) or 32 of them (four rows at a time); the four warps of a block take rows in turn.  Eight blocks an
// SM, which is also how many the launch makes: at the 72 registers that the compiler takes otherwise seven fit, and the eighth runs alone
// afterwards (115 us instead of 98).
template <class P, bool VEC>
__global__ void __launch_bounds__(kKnownThreads, 8) sums_kernel(const __grid_constant__ ReducedParams q) {
  RT_PDL_ENTRY();
  constexpr int kWarps = kKnownThreads / 32, kCols = VEC ? 128 : 32, kRows = VEC ? 1 : 4;
  __shared__ float red[kWarps][kCols];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * kCols + (VEC ? 4 * lane : lane);
  const int begin = blockIdx.y * q.rows_per_block, end = min(begin + q.rows_per_block, q.rows);
  Sums<VEC> sink;
  sink.which = q.which;
#pragma unroll
  for (float& v : sink.sum) v = 0.f;
  for (int r = begin + warp * kRows; r < end; r += kWarps * kRows) {
    Quad<VEC> e;
#pragma unroll
    for (int g = 0; g < Quad<VEC>::G; ++g) {
      e.live[g] = c < q.cols && r + g < end;
      e.c0[g] = e.live[g] ? r + g : 0;
      e.c1[g] = e.live[g] ? c : 0;
      e.at[g] = (uint32_t)e.c0[g] * (uint32_t)q.cols + (uint32_t)e.c1[g];
    }
    run<P, VEC>(q.f, e, sink);
  }
#pragma unroll
  for (int i = 0; i < (VEC ? 4 : 1); ++i) red[warp][VEC ? 4 * lane + i : lane] = sink.sum[i];
  __syncthreads();
  for (int i = threadIdx.x; i < kCols; i += kKnownThreads) {
    const int col = blockIdx.x * kCols + i;
    float v = red[0][i];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) v += red[w][i];
    if (col < q.cols) q.out[(int64_t)blockIdx.y * q.cols + col] = v;
  }
}

// Output `which` is written and kept.
template <bool VEC>
struct Keep {
  int which;
  float* row;  // of this block, in shared memory
  float most;
  template <int OUT, bool V>
  __device__ __forceinline__ void put(const FusedParams& p, const Quad<VEC>& e, const float (&acc)[4]) {
    Store().template put<OUT, VEC>(p, e, acc);
    if (OUT != which) return;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (e.live[VEC ? 0 : i]) {
        row[e.c1[VEC ? 0 : i] + (VEC ? i : 0)] = acc[i];
        most = fmaxf(most, acc[i]);
      }
  }
};
template <class F>
__device__ __forceinline__ float over_block(float v, float* red, F f) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = f(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();  // red has been read
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
#pragma unroll
  for (int w = 1; w < kRowThreads / 32; ++w) v = f(v, red[w]);
  return v;
}
// As the stand-alone kernel: the maximum first, then the sum of exp(v - maximum).  A thread reads back what it has put there itself.
template <class P, bool VEC>
__global__ void __launch_bounds__(kRowThreads) logsumexp_kernel(const __grid_constant__ ReducedParams q) {
  RT_PDL_ENTRY();
  extern __shared__ float row[];
  __shared__ float red[kRowThreads / 32];
  for (int r = blockIdx.x; r < q.rows; r += gridDim.x) {
    Keep<VEC> sink{q.which, row, -INFINITY};
    constexpr int kStep = 4 * kRowThreads;
    auto quad = [&](int base, Quad<VEC>& e) {
#pragma unroll
      for (int g = 0; g < Quad<VEC>::G; ++g) {
        const int c = VEC ? base + 4 * (int)threadIdx.x : base + g * kRowThreads + (int)threadIdx.x;
        e.live[g] = c < q.cols;
        e.c0[g] = r;
        e.c1[g] = e.live[g] ? c : 0;
        e.at[g] = (uint32_t)r * (uint32_t)q.cols + (uint32_t)e.c1[g];
      }
    };
    for (int base = 0; base < q.cols; base += kStep) {
      Quad<VEC> e;
      quad(base, e);
      run<P, VEC>(q.f, e, sink);
    }
    const float m = over_block(sink.most, red, [](float a, float b) { return fmaxf(a, b); });
    float s = 0.f;
    for (int base = 0; base < q.cols; base += kStep) {
      Quad<VEC> e;
      quad(base, e);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (e.live[VEC ? 0 : i]) s += expf(row[e.c1[VEC ? 0 : i] + (VEC ? i : 0)] - m);
    }
    s = over_block(s, red, [](float a, float b) { return a + b; });
    if (threadIdx.x == 0) q.out[r] = m + logf(s);
  }
}

struct Reduced {
  const uint32_t* code;
  int n_code, n_preload;
  void (*vector)(const ReducedParams), (*single)(const ReducedParams);
};
template <class P>
constexpr Reduced with_sums{P::code, P::n, P::preload, &sums_kernel<P, true>, &sums_kernel<P, false>};
template <class P>
constexpr Reduced with_logsumexp{P::code, P::n, P::preload, &logsumexp_kernel<P, true>, &logsumexp_kernel<P, false>};

#include "fused_programs_reduced.inc"

// word(i): the i-th instruction as the kernels decode it.
template <int N, class Word>
const Reduced* find(const Reduced (&list)[N], int n_code, int n_preload, const Word& word) {
  for (const Reduced& k : list) {
    bool same = k.n_code == n_code && k.n_preload == n_preload;
    for (int i = 0; i < n_code && same; ++i) same = k.code[i] == word(i);
    if (same) return &k;
  }
  return nullptr;
}
template <int N>
const Reduced* find(const Reduced (&list)[N], const FusedParams& p) {
  return find(list, p.n_code, p.n_preload, [&](int i) { return p.code[i].x; });
}

// The ops of a program as a set; of an op and its reversed form, and of opposite comparisons, the one.
static_assert(RT_F_COUNT <= 64, "a bit an op");
uint64_t one_form(uint64_t ops) {
  auto fold = [&](int from, int to) {
    if (ops >> from & 1) ops = (ops & ~(uint64_t(1) << from)) | uint64_t(1) << to;
  };
  fold(RT_F_LT, RT_F_GT);
  fold(RT_F_LE, RT_F_GE);
  return ops;
}
template <int N>
bool has_ops(const Reduced (&list)[N], uint64_t ops) {
  static const std::vector<uint64_t> sets = [&list] {
    std::vector<uint64_t> v;
    for (const Reduced& k : list) {
      uint64_t set = 0;
      for (int i = 0; i < k.n_code; ++i) {
        const int op = (int)(k.code[i] & 255);
        if (op == RT_F_LOAD || op == RT_F_OUT || op == RT_F_REG || op == RT_F_SELECT) continue;
        set |= uint64_t(1) << (op == kReverseSub ? RT_F_SUB : (op == kReverseDiv ? RT_F_DIV : (op == kReversePow ? RT_F_POWF : op)));
      }
      v.push_back(one_form(set));
    }
    return v;
  }();
  return std::find(sets.begin(), sets.end(), one_form(ops)) != sets.end();
}

}  // namespace

extern "C" {

rt_status rt_fused_reduction_possible(rt_ctx* ctx, int which, uint64_t ops) {
  RT_CHECK_CTX(ctx);
  return (which < 0 ? has_ops(kWithLogsumexp, ops) : has_ops(kWithSums, ops)) ? RT_OK : RT_ERR_UNIMPLEMENTED;
}

rt_status rt_fused_reduction_known(rt_ctx* ctx, const rt_fused_program* f, int which) {
  RT_CHECK_CTX(ctx);
  RT_CHECK_PTR(ctx, f);
  if (f->nd != 2 || f->n_code < 1 || f->n_code > RT_FUSED_MAX_CODE || which < -1 || which >= f->n_outputs)
    RT_FAIL(ctx, RT_ERR_INVALID_OPERATION, "rt_fused_reduction_known: an output of a two-dimensional program, or -1");
  if (f->shape[0] <= 0 || f->shape[1] <= 0 || (which < 0 && f->shape[1] > kLongestRow)) return RT_ERR_UNIMPLEMENTED;
  auto word = [&](int i) { return fused::encode(f->code[i]).x; };
  return (which < 0 ? find(kWithLogsumexp, f->n_code, f->n_preload, word) : find(kWithSums, f->n_code, f->n_preload, word)) ? RT_OK : RT_ERR_UNIMPLEMENTED;
}

rt_status rt_fused_column_sums(rt_ctx* ctx, const rt_fused_program* f, int which, float* sums) {
  ReducedParams q{};
  bool vec;
  int64_t numel;
  rt_status st = fused::prepare(ctx, f, &q.f, &vec, &numel);
  if (st != RT_OK) return st;
  RT_CHECK_PTR(ctx, sums);
  if (f->nd != 2 || which < 0 || which >= f->n_outputs) RT_FAIL(ctx, RT_ERR_INVALID_OPERATION, "rt_fused_column_sums: an output of a two-dimensional program");
  const Reduced* k = numel ? find(kWithSums, q.f) : nullptr;
  if (!k) return RT_ERR_UNIMPLEMENTED;
  q.rows = f->shape[0];
  q.cols = f->shape[1];
  q.which = which;
  // pieces of the rows: so many that the blocks come to eight an SM, of at least 16 rows
  const int tiles = (q.cols + (vec ? 127 : 31)) / (vec ? 128 : 32);
  int pieces = (8 * ctx->sm_count + tiles - 1) / tiles;
  if (pieces > (q.rows + 15) / 16) pieces = (q.rows + 15) / 16;
  q.rows_per_block = (q.rows + pieces - 1) / pieces;
  pieces = (q.rows + q.rows_per_block - 1) / q.rows_per_block;
  RtScratch parts(ctx);
  if (pieces > 1 && (st = parts.alloc(sizeof(float) * (size_t)pieces * q.cols)) != RT_OK) return st;
  q.out = pieces > 1 ? parts.as<float>() : sums;
  ctx->fused_compiled++;
  rt_launch(ctx, vec ? k->vector : k->single, dim3(tiles, pieces), kKnownThreads, 0, q);
  RT_LAUNCHED(ctx);
  return pieces > 1 ? rt_sum_axis_internal(ctx, q.out, 1, pieces, q.cols, sums, 1.f) : RT_OK;
}

rt_status rt_fused_logsumexp(rt_ctx* ctx, const rt_fused_program* f, float* out) {
  ReducedParams q{};
  bool vec;
  int64_t numel;
  rt_status st = fused::prepare(ctx, f, &q.f, &vec, &numel);
  if (st != RT_OK) return st;
  RT_CHECK_PTR(ctx, out);
  if (f->nd != 2) RT_FAIL(ctx, RT_ERR_INVALID_OPERATION, "rt_fused_logsumexp: a two-dimensional program");
  const Reduced* k = numel && f->shape[1] <= kLongestRow ? find(kWithLogsumexp, q.f) : nullptr;
  if (!k) return RT_ERR_UNIMPLEMENTED;
  q.rows = f->shape[0];
  q.cols = f->shape[1];
  q.out = out;
  ctx->fused_compiled++;
  // a block per row: 58 us over 4096 rows; 64 us with eight blocks an SM that take three or four rows each
  const int grid = q.rows < 64 * ctx->sm_count ? q.rows : 64 * ctx->sm_count;
  rt_launch(ctx, vec ? k->vector : k->single, grid, kRowThreads, sizeof(float) * q.cols, q);
  RT_LAUNCHED(ctx);
  return RT_OK;
}

}  // extern "C"
