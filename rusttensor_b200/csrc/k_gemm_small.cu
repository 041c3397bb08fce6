// Small and narrow products in exact fp32: C[M,N] = act(op(A) op(B) + bias) (+ C).
//
// What bounds them: with a few dozen output tiles a product of this size occupies a fraction of the chip for as long as one tile
// walks its reduction, and a second launch that adds split-K partial sums costs as much as the product.  So
//  * 32 x 64 tiles, and the reduction of a tile is split over the CTAs of a cluster (1, 2, 4 or 8), so that about one to two
//    CTAs land on every SM; their partial tiles meet in distributed shared memory and each CTA finishes a share of them:
//    bias, activation and accumulation included, one launch in all, sums in a fixed order;
//  * inside a CTA four groups of four warps take a quarter of every 64-deep K-block each (4 x 4 outputs a thread);
//  * operands arrive by cp.async, three K-blocks in flight, 16 bytes at a time where the rows allow it, else 4.
// fp32 FMAs rather than tensor cores: below a few hundred MFLOP the splitting of operands into TF32 parts and the tensor-memory
// set-up cost more than the arithmetic.
// The partial sums leave a thread as 128-bit slots, so that a slot, and not an element, is what a thread adds up and writes.
// Measured in a graph (M x K x N; with one group of threads and element-wise sums before): 64 x 64 x 64 3.5 us (4.5), of which the launch is
// 0.65 and the first operands 1.15; 512 x 64 x 65 4.4 (5.1); 30 x 250 x 800 5.1 (5.2); 64 x 784 x 128 6.2 (6.5); 90 x 1000 x 100 6.3 (6.6).
#include <cooperative_groups.h>

#include "finish.cuh"
#include "rt_internal.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kBM = 32, kBN = 64, kBK = 64, kStages = 3, kGroups = 4, kThreads = kGroups * 128;
constexpr int kPad = 4;

struct SmallGemm {
  const float *a, *b, *bias;
  float* c;
  int64_t lda, ldb, ldc;
  int m, n, k, k_per_split, act;
  bool a16, b16, accumulate;
};

__device__ __forceinline__ void async_copy(float* dst, const float* src, int bytes, bool wide) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// A ROWS x COLS piece of a row-major matrix (COLS contiguous) to shared memory with row stride COLS + kPad, zeros outside
// [row_end) x [col_end).
template <int ROWS, int COLS>
__device__ __forceinline__ void load_piece(float* s, const float* g, int64_t ld, int row0, int row_end, int col0, int col_end, bool wide) {
  if (wide) {
    constexpr int kChunks = ROWS * COLS / 4;
#pragma unroll
    for (int i = threadIdx.x; i < kChunks; i += kThreads) {
      const int r = i / (COLS / 4), c = i % (COLS / 4) * 4;
      int left = (col_end - (col0 + c)) * 4;
      left = row0 + r < row_end ? (left > 16 ? 16 : (left < 0 ? 0 : left)) : 0;
      async_copy(s + r * (COLS + kPad) + c, left ? g + (int64_t)(row0 + r) * ld + col0 + c : g, left, true);
    }
  } else {
#pragma unroll 8
    for (int i = threadIdx.x; i < ROWS * COLS; i += kThreads) {
      const int r = i / COLS, c = i % COLS;
      const bool in = row0 + r < row_end && col0 + c < col_end;
      async_copy(s + r * (COLS + kPad) + c, in ? g + (int64_t)(row0 + r) * ld + col0 + c : g, in ? 4 : 0, false);
    }
  }
}

template <bool TA, bool TB>
struct Shape {
  static constexpr int a_floats = TA ? kBK * (kBM + kPad) : kBM * (kBK + kPad);
  static constexpr int b_floats = TB ? kBN * (kBK + kPad) : kBK * (kBN + kPad);
  static constexpr size_t bytes = sizeof(float) * kStages * (a_floats + b_floats);
  static_assert(kGroups * kBM * kBN <= kStages * (a_floats + b_floats), "the partial tiles reuse the stages");
};

// Several left operands and results for one right operand: the row tiles of item i follow those of item i - 1.
constexpr int kListTerms = 256;
struct SmallList {
  const float* a[kListTerms];
  float* c[kListTerms];
  int row_tiles;
};
struct NoList {};

template <bool TA, bool TB, class List>
__global__ void __launch_bounds__(kThreads, 2) small_gemm_kernel(const SmallGemm args, const List list) {
  extern __shared__ __align__(16) float smem[];
  using S = Shape<TA, TB>;
  cg::cluster_group cluster = cg::this_cluster();
  const int splits = cluster.num_blocks(), rank = cluster.block_rank();
  RT_PDL_ENTRY();
  SmallGemm p = args;
  int row_tile = blockIdx.y;
  if constexpr (sizeof(List) > sizeof(NoList)) {
    const int item = row_tile / list.row_tiles;
    row_tile -= item * list.row_tiles;
    p.a = list.a[item];
    p.c = list.c[item];
  }
  const int m0 = row_tile * kBM, n0 = (int)(blockIdx.x / splits) * kBN;
  const int kbeg = rank * p.k_per_split, kend = min(p.k, kbeg + p.k_per_split);
  const int blocks = kend > kbeg ? (kend - kbeg + kBK - 1) / kBK : 0;
  const int group = threadIdx.x >> 7, warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const int tm = (lane >> 3) + 4 * (warp & 1), tn = (lane & 7) + 8 * (warp >> 1);  // 8 x 16 threads

  auto fetch = [&](int i) {
    if (i < blocks) {
      float* sa = smem + (i % kStages) * (S::a_floats + S::b_floats);
      float* sb = sa + S::a_floats;
      const int k0 = kbeg + i * kBK;
      if (TA) load_piece<kBK, kBM>(sa, p.a, p.lda, k0, kend, m0, p.m, p.a16);
      else load_piece<kBM, kBK>(sa, p.a, p.lda, m0, p.m, k0, kend, p.a16);
      if (TB) load_piece<kBN, kBK>(sb, p.b, p.ldb, n0, p.n, k0, kend, p.b16);
      else load_piece<kBK, kBN>(sb, p.b, p.ldb, k0, kend, n0, p.n, p.b16);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) fetch(i);
  for (int it = 0; it < blocks; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    fetch(it + kStages - 1);
    const float* sa = smem + (it % kStages) * (S::a_floats + S::b_floats);
    const float* sb = sa + S::a_floats;
#pragma unroll
    for (int q = 0; q < kBK / kGroups; q += 4) {
      const int k = group * (kBK / kGroups) + q;
      float av[4][4], bv[4][4];  // [row or column][k]
      if (TA) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const float4 t = *reinterpret_cast<const float4*>(sa + (k + kk) * (kBM + kPad) + 4 * tm);
          av[0][kk] = t.x; av[1][kk] = t.y; av[2][kk] = t.z; av[3][kk] = t.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 t = *reinterpret_cast<const float4*>(sa + (tm + 8 * i) * (kBK + kPad) + k);
          av[i][0] = t.x; av[i][1] = t.y; av[i][2] = t.z; av[i][3] = t.w;
        }
      }
      if (TB) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 t = *reinterpret_cast<const float4*>(sb + (tn + 16 * j) * (kBK + kPad) + k);
          bv[j][0] = t.x; bv[j][1] = t.y; bv[j][2] = t.z; bv[j][3] = t.w;
        }
      } else {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const float4 t = *reinterpret_cast<const float4*>(sb + (k + kk) * (kBN + kPad) + 4 * tn);
          bv[0][kk] = t.x; bv[1][kk] = t.y; bv[2][kk] = t.z; bv[3][kk] = t.w;
        }
      }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i][kk], bv[j][kk], acc[i][j]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // Every thread leaves its sums as four 128-bit slots; a slot is then added over the groups and the CTAs of the cluster by one thread
  // of one of them and written out.  Slot i * 128 + t belongs to thread t of a group: row i of its block (column i when B is stored
  // transposed, whose columns are 16 apart).
  float4* part = reinterpret_cast<float4*>(smem);
  constexpr int kSlots = 4 * 128;
  const int t128 = threadIdx.x & 127;
#pragma unroll
  for (int i = 0; i < 4; ++i) part[group * kSlots + i * 128 + t128] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  __syncthreads();
  static_assert(kSlots == kThreads, "a slot a thread");
  auto over_groups = [&](int slot) {
    float4 v = part[slot];
#pragma unroll
    for (int g = 1; g < kGroups; ++g) {
      const float4 u = part[g * kSlots + slot];
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    return v;
  };
  if (splits > 1) {
    part[threadIdx.x] = over_groups(threadIdx.x);
    cluster.sync();
  }
  const int share = kSlots / splits, slot = rank * share + threadIdx.x, i = slot >> 7, l = slot & 31, w = (slot >> 5) & 3;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if ((int)threadIdx.x < share) {
    if (splits == 1) {
      v = over_groups(slot);
    } else {
      float4 u[8];  // all remote reads are in flight before the first is added
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < splits) u[s] = cluster.map_shared_rank(part, s)[slot];
      v = u[0];
#pragma unroll
      for (int s = 1; s < 8; ++s)
        if (s < splits) {
          v.x += u[s].x; v.y += u[s].y; v.z += u[s].z; v.w += u[s].w;
        }
    }
  }
  // nobody leaves while its partial tile may still be read: the wait comes after the result is written
  if (splits > 1) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
  const bool plain = !p.bias && p.act == RT_ACT_NONE && !p.accumulate;
  if ((int)threadIdx.x < share) {
    const int sm = (l >> 3) + 4 * (w & 1), sn = (l & 7) + 8 * (w >> 1);
    const int m = m0 + (TA ? 4 * sm + i : sm + 8 * i), n = n0 + (TB ? sn : 4 * sn);
    if (m < p.m) {
      float* out = p.c + (int64_t)m * p.ldc + n;
      if (!TB) {
        const int left = p.n - n;
        if (left > 0) {
          if (!plain) v = rt_finish4(v, p.bias ? p.bias + n : nullptr, p.act, p.accumulate ? out : nullptr, left);
          if (left >= 4 && rt_aligned16(out)) {
            *reinterpret_cast<float4*>(out) = v;
          } else {
            out[0] = v.x;
            if (left > 1) out[1] = v.y;
            if (left > 2) out[2] = v.z;
            if (left > 3) out[3] = v.w;
          }
        }
      } else {
        const float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + 16 * j < p.n) {
            float r = o[j];
            if (!plain) r = rt_finish4(make_float4(r, 0.f, 0.f, 0.f), p.bias ? p.bias + n + 16 * j : nullptr, p.act, p.accumulate ? out + 16 * j : nullptr, 1).x;
            out[16 * j] = r;
          }
      }
    }
  }
  if (splits > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

template <bool TA, bool TB, class List = NoList>
rt_status launch_small(rt_ctx* ctx, const SmallGemm& p, int splits, const List& list = List{}, int items = 1) {
  auto kern = small_gemm_kernel<TA, TB, List>;
  using S = Shape<TA, TB>;
  static RtDeviceOnce once;
  RT_CUDA(ctx, once([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bytes); }));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.n + kBN - 1) / kBN * splits), (unsigned)((p.m + kBM - 1) / kBM * items), 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = S::bytes;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)splits;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  RT_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, p, list));
  RT_LAUNCHED(ctx);
  return RT_OK;
}

// As many splits as put a CTA on every SM, at least one K-block each.  (Two K-blocks in one CTA were slower than one in each of two,
// 64 x 65 x 512: 5.5 and 5.1 us.)
int choose_splits(rt_ctx* ctx, int64_t tiles, int64_t k) {
  int splits = 1;
  while (splits < 8 && tiles * splits <= (int64_t)ctx->sm_count && k > (int64_t)kBK * splits) splits *= 2;
  return splits;
}

}  // namespace

// Microseconds that a product takes here, fitted like rt_gemm_ts_estimate: a K-block costs 1.3 us where about one CTA comes to an SM and
// 2.8 where two do, a third more where its copies are of 4 bytes.
float rt_gemm_small_estimate(rt_ctx* ctx, int64_t m, int64_t n, int64_t k, bool wide) {
  const int64_t tiles = ((m + kBM - 1) / kBM) * ((n + kBN - 1) / kBN), blocks = (k + kBK - 1) / kBK;
  const int splits = choose_splits(ctx, tiles, k);
  const int64_t ctas = tiles * splits, waves = (ctas + 2 * ctx->sm_count - 1) / (2 * ctx->sm_count);
  const float block = ctas * 4 > (int64_t)ctx->sm_count * 3 ? 2.8f : 1.3f;
  return (splits > 1 ? 3.7f : 2.7f) + block * (wide || k <= kBK ? 1.f : 1.3f) * (float)(waves * ((blocks + splits - 1) / splits));
}

rt_status rt_gemm_small_internal(rt_ctx* ctx, int trans_a, int trans_b, int64_t m, int64_t n, int64_t k, const float* a, int64_t lda,
                                 const float* b, int64_t ldb, float* c, int64_t ldc, const float* bias, int act, int accumulate) {
  const int64_t tiles = ((m + kBM - 1) / kBM) * ((n + kBN - 1) / kBN);
  if (m >= (1 << 20) || n >= (1 << 20) || k >= (1 << 28) || (m + kBM - 1) / kBM > 65535) return RT_ERR_UNIMPLEMENTED;
  const int splits = choose_splits(ctx, tiles, k);
  int64_t per = (k + splits - 1) / splits;
  per = (per + kBK - 1) / kBK * kBK;
  SmallGemm p{a, b, bias, c, lda, ldb, ldc, (int)m, (int)n, (int)k, (int)per, act, rt_aligned16(a) && lda % 4 == 0, rt_aligned16(b) && ldb % 4 == 0,
              accumulate != 0};
  if (!trans_a && !trans_b) return launch_small<false, false>(ctx, p, splits);
  if (!trans_a && trans_b) return launch_small<false, true>(ctx, p, splits);
  if (trans_a && !trans_b) return launch_small<true, false>(ctx, p, splits);
  return launch_small<true, true>(ctx, p, splits);
}

rt_status rt_gemm_small_list_internal(rt_ctx* ctx, int count, const float* const* a, float* const* c, int64_t m, int64_t n, int64_t k,
                                      const float* b, const float* bias, int act) {
  const int64_t row_tiles = (m + kBM - 1) / kBM, tiles = row_tiles * ((n + kBN - 1) / kBN) * (count < kListTerms ? count : kListTerms);
  if (m >= (1 << 20) || n >= (1 << 20) || k >= (1 << 28) || row_tiles * kListTerms > 65535) return RT_ERR_UNIMPLEMENTED;
  const int splits = choose_splits(ctx, tiles, k);
  int64_t per = (k + splits - 1) / splits;
  per = (per + kBK - 1) / kBK * kBK;
  for (int q = 0; q < count; q += kListTerms) {
    const int items = count - q < kListTerms ? count - q : kListTerms;
    SmallList l{};
    l.row_tiles = (int)row_tiles;
    bool a16 = k % 4 == 0;
    for (int i = 0; i < items; ++i) {
      l.a[i] = a[q + i];
      l.c[i] = c[q + i];
      a16 = a16 && rt_aligned16(a[q + i]);
    }
    SmallGemm p{nullptr, b, bias, nullptr, k, n, n, (int)m, (int)n, (int)k, (int)per, act, a16, rt_aligned16(b) && n % 4 == 0, false};
    rt_status st = launch_small<false, false>(ctx, p, splits, l, items);
    if (st != RT_OK) return st;
  }
  return RT_OK;
}
