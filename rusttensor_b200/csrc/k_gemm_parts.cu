// Large products on the tensor cores with operands split into 16-bit parts beforehand.
//
// An fp32 operand is scaled by a power of two and split into two fp16 parts, hi = fp16(x)
// and lo = fp16((x - hi) * 2^11): 22 bits, each part rounded to nearest.  hi * hi goes to one fp32 accumulator, hi * lo and lo * hi to
// another that is scaled down at the end.  That is three MMAs of kind::f16 where 3xTF32 takes three of kind::tf32 at half the rate and twice
// the bytes, and it drops less: lo * lo is below 2^-24 of a product, 2^-20 with the truncated TF32 parts.
// The scale comes from a sample of the operand, whose largest magnitude becomes 2^9; the pass that splits looks at all of it.  lo is exact
// to 2^-36.  If an element reaches 2^15 after scaling, or a segment (128 columns of a row, 64 rows of a column) lies wholly below 2^-9, or more
// elements than one in 2^20 are not zero and below 2^-22, or there are infinities, NaN or scales beyond 2^100, a third pass, which otherwise ends
// at once, splits again into three bf16 parts (8 + 8 + 8 bits, exact, the exponents of fp32) and the same kernel runs six MMAs where it otherwise
// runs three.  Within these lines an element keeps its 22 bits or is off by less than 2^-36 after scaling, which is 2^-27 of its segment's largest
// and 2^-14 of itself.  Where the terms of a result all weigh the same, what the parts drop is 1.1e-7 of |A| |B| with magnitudes spread evenly over
// 2^31, 3.3e-7 with 3xTF32.  Over 2^33, which goes to three parts, it would be 8e-7 and 5e-7, over 2^40 6e-5 and 5e-7.
// The decision is made on the device; nothing waits for it on the host.
//
// A K-block in memory is four slots of 16 along the reduction: hi hi lo lo of 32 elements, or the three bf16 parts of 16 and the first once
// more, with zeros for infinities and NaN: the cross terms take that one, so that an infinity meets no zero which is none.  A row of it is
// 128 bytes (reduction contiguous) or the block is 64 rows (rows contiguous); TMA fetches it in boxes of 8 KB with the 128-byte swizzle and
// tcgen05.mma reads it as it lies, either way round, so that nothing is transposed.  A matrix that is an operand with its rows and with its columns as
// the reduction (the upstream gradient of a product) is looked at once and split both ways.
//
// Roles of a CTA (one per SM, walking over tiles of 128 x up to 256): a TMA warp up to four K-blocks ahead, an MMA warp, eight warps that
// empty the accumulator into registers and write the result.  The tensor core adds into its accumulator with truncation, an error that
// grows with the number of additions (one per 16 of the reduction here, six with 3xTF32); so hi * hi is emptied every `chunk` K-blocks,
// while the MMAs of the cross terms run.  The cross terms are 2^11 smaller and stay until the tile is done.
// Measured: 4096^3, both operands read from memory, 360 us with the power limit reached (320 of them here, 95 % of the rate that cuBLAS
// sustains with bf16), 3xTF32 with operands fetched by TMA 670 - 815.  Error against float64 at that size 6.5e-7 of the result, 3xTF32 1.04e-6;
// at 1000 2.7e-7 and 3.5e-7; with three bf16 parts 4.0e-7 in 650 us.  A pass over all operands for the largest magnitude instead of the sample
// made product and both gradients 1270 us instead of 1210.
// What bounds a tile otherwise is shared memory: per K-block 128 bytes written and six times 32 read for each row of A and B, 960 cycles for
// 128 x 256 against 768 of MMAs.
// Every wait is bounded; on expiry the kernel records a code in the status word, raises a flag that all other waits poll, lets its own
// copies land, frees tensor memory and returns.
#include "parts_common.cuh"

namespace tc {
namespace parts {

constexpr int kMaxSplits = 4;  // a matrix that is an operand both ways round is split twice

struct SplitSource {
  const float* p;
  uint16_t* out;
  int64_t ld, ldo;   // floats, halves
  int rows, cols, tiles_c;
  uint32_t tiles;
  int along_rows;    // the reduction runs down the rows
  int vec;
  int source;        // of the statistics
  int look;          // whether its magnitudes are looked at here (a source that is split twice: once)
};
struct SplitArgs {
  SplitSource s[kMaxSplits];
  int count, sources, sample_blocks;
  uint32_t most_faint[kMaxSources];
  const uint2* samples;       // [source][block] of sample_kernel
  uint32_t* verdicts;         // [source][block] of split_kernel<false>
  Decision* decision;
};
// A tile of 64 rows x 128 columns: a warp has eight rows, two at a time, a lane eight columns of one.
template <bool VEC, bool AGAIN>
__device__ __forceinline__ void split_tiles(const SplitSource& s, float scale, uint32_t faint, uint32_t (*cols)[16][kTileCols], Magnitudes& all) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, piece = lane & 15;
  constexpr int depth = AGAIN ? 16 : 32;  // elements of a K-block
  // the padding behind the reduction is written as zeros
  const int rows = s.along_rows ? (s.rows + depth - 1) / depth * depth : s.rows;
  const int width = s.along_rows ? (int)s.ldo : (s.cols + depth - 1) / depth * depth;
  const int64_t next = s.along_rows ? depth * s.ldo : depth;
  int turn = 0;
  for (uint32_t t = blockIdx.x; t < s.tiles; t += gridDim.x) {
    const int tr = (int)(t / (uint32_t)s.tiles_c), tc = (int)(t - (uint32_t)tr * (uint32_t)s.tiles_c);
    const int r0 = tr * kTileRows + warp * 8 + (lane >> 4), c = tc * kTileCols + piece * 8;
    float x[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + 2 * i;
      const float* p = s.p + (int64_t)r * s.ld + c;
      if (VEC) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 v = r < s.rows && c < s.cols ? __ldcs(reinterpret_cast<const float4*>(p)) : zero;
        const float4 w = r < s.rows && c + 4 < s.cols ? __ldcs(reinterpret_cast<const float4*>(p) + 1) : zero;
        x[i][0] = v.x; x[i][1] = v.y; x[i][2] = v.z; x[i][3] = v.w; x[i][4] = w.x; x[i][5] = w.y; x[i][6] = w.z; x[i][7] = w.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[i][j] = r < s.rows && c + j < s.cols ? __ldg(p + j) : 0.f;
      }
    }
    uint32_t col[8] = {};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + 2 * i;
      if (!AGAIN) {
        uint32_t row = 0, low = 0xffffffffu;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t m = __float_as_uint(x[i][j]) & 0x7fffffffu;
          row = max(row, m);
          low = lower(low, m);
          col[j] = max(col[j], m);
        }
        all.faint += low < faint;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) row = max(row, __shfl_xor_sync(0xffffffffu, row, o));
        all.most = max(all.most, row);
        if (row) all.least = min(all.least, row);
      }
      if (r < rows && c < width) {
        uint4 part[4];
        split8(x[i], AGAIN, scale, part);
        const unsigned along = s.along_rows ? r : c, block = along / depth, in_block = along % depth;
        uint16_t* o = s.along_rows ? s.out + ((int64_t)block * 64 + in_block) * s.ldo + c : s.out + (int64_t)r * s.ldo + block * 64 + in_block;
        *reinterpret_cast<uint4*>(o) = part[0];
        *reinterpret_cast<uint4*>(o + next) = part[1];
        if (AGAIN) {
          *reinterpret_cast<uint4*>(o + 2 * next) = part[2];
          *reinterpret_cast<uint4*>(o + 3 * next) = part[3];
        }
      }
    }
    if (AGAIN || !s.look) continue;
    turn ^= 1;  // two buffers, so that one barrier a tile is enough
    uint32_t* mine = &cols[turn][warp * 2 + (lane >> 4)][piece * 8];
    *reinterpret_cast<uint4*>(mine) = make_uint4(col[0], col[1], col[2], col[3]);
    *reinterpret_cast<uint4*>(mine + 4) = make_uint4(col[4], col[5], col[6], col[7]);
    __syncthreads();
    if (threadIdx.x < kTileCols) {
      uint32_t m = 0;
#pragma unroll
      for (int i = 0; i < 16; ++i) m = max(m, cols[turn][i][threadIdx.x]);
      if (m) all.least = min(all.least, m);
    }
  }
}
// Bound by memory: 4 bytes read and 4 written an element.  AGAIN: into three parts, if the first pass has found that two will not do; otherwise over
// in 4 us, of which most is the launch and the verdicts of 592 blocks.
template <bool AGAIN>
__global__ void __launch_bounds__(256, 4) split_kernel(const SplitArgs a) {
  RT_PDL_ENTRY();
  __shared__ uint32_t red[2 * kMaxSources][8];
  __shared__ uint32_t cols[AGAIN ? 1 : 2][16][kTileCols];
  Decision d{};
  if (AGAIN) {
    d = decide(a.verdicts, a.sources, gridDim.x, a.most_faint, red);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.decision->wide = d.wide;
      a.decision->special = d.special;
    }
    if (!d.wide) return;
  } else {
    uint2 v[kMaxSources];
    over_samples(a.samples, a.sources, a.sample_blocks, red, v);
#pragma unroll
    for (int q = 0; q < kMaxSources; ++q) {
      d.exponent[q] = exponent_for(v[q].x);
      if (blockIdx.x == 0 && threadIdx.x == 0) a.decision->exponent[q] = d.exponent[q];
    }
  }
  for (int q = 0; q < a.count; ++q) {
    const SplitSource& s = a.s[q];
    const int exponent = s.source == 0 ? d.exponent[0] : (s.source == 1 ? d.exponent[1] : d.exponent[2]);
    const float scale = AGAIN ? 1.f : ldexpf(1.f, exponent);
    const uint32_t faint = faint_below(exponent);
    Magnitudes all;
    if (s.vec) split_tiles<true, AGAIN>(s, scale, faint, cols, all);
    else split_tiles<false, AGAIN>(s, scale, faint, cols, all);
    if (AGAIN || !s.look) continue;
    all = over_block(all, red);
    if (threadIdx.x == 0) a.verdicts[s.source * gridDim.x + blockIdx.x] = verdict(all, exponent);
  }
}

// A matrix and its parts.  `along_rows`: the reduction of the products that it is an operand of runs down its rows.
struct Split {
  const float* p;
  int64_t ld;
  int rows, cols, along_rows, source;  // source: its number among those that the decision was made from
  RtScratch mem;
  int64_t ldo = 0;
  Split(rt_ctx* ctx, int src, const float* q, int64_t l, int64_t r, int64_t c, bool along)
      : p(q), ld(l), rows((int)r), cols((int)c), along_rows(along), source(src), mem(ctx) {}
  // room for the larger of the two forms: 64 values for every 16 of the reduction
  rt_status alloc() {
    const int64_t k = ((along_rows ? rows : cols) + 15) / 16 * 64;
    ldo = along_rows ? (int64_t)((cols + 7) / 8) * 8 : k;
    return mem.alloc(sizeof(uint16_t) * (size_t)((along_rows ? k : rows) * ldo));
  }
  bool map(CUtensorMap* m) {
    const int64_t k = ((along_rows ? rows : cols) + 15) / 16 * 64;
    return along_rows ? map_parts(m, mem.as<uint16_t>(), cols, k, ldo) : map_parts(m, mem.as<uint16_t>(), k, rows, ldo);
  }
};


// The passes that split matrices, the first `sources` of which are all different.  Preparing takes the memory and makes the tensor maps, so that
// what can be missing is missing before anything has been launched: a caller that takes another kernel then may be adding to what is there.
struct Splitting {
  SampleArgs sample{};
  SplitArgs split{};
  RtScratch work;
  explicit Splitting(rt_ctx* ctx) : work(ctx) {}
  rt_status prepare(rt_ctx* ctx, Split* const* s, int count, int sources) {
    const int sample_blocks = ctx->sm_count, blocks = 4 * ctx->sm_count;
    rt_status st = work.alloc((sizeof(uint2) * (size_t)sample_blocks + sizeof(uint32_t) * (size_t)blocks) * kMaxSources + sizeof(Decision));
    if (st != RT_OK) return st;
    uint2* samples = work.as<uint2>();
    sample.count = split.sources = sources;
    split.count = count;
    split.sample_blocks = sample_blocks;
    split.samples = samples;
    split.verdicts = reinterpret_cast<uint32_t*>(samples + (size_t)sample_blocks * kMaxSources);
    split.decision = reinterpret_cast<Decision*>(split.verdicts + (size_t)blocks * kMaxSources);
    for (int q = 0; q < count; ++q) {
      if ((st = s[q]->alloc()) != RT_OK) return st;
      const Sample m = sample_of(ctx, s[q]->p, s[q]->ld, s[q]->rows, s[q]->cols, false);
      if (q < sources) {
        sample.s[q] = m;
        split.most_faint[q] = most_faint((int64_t)s[q]->rows * s[q]->cols);
      }
      split.s[q] = {s[q]->p, s[q]->mem.as<uint16_t>(), s[q]->ld, s[q]->ldo, s[q]->rows, s[q]->cols, m.tiles_c, m.tiles, s[q]->along_rows, m.vec,
                    s[q]->source, q < sources};
    }
    return RT_OK;
  }
  rt_status run(rt_ctx* ctx) {
    rt_launch(ctx, sample_kernel, split.sample_blocks, 256, 0, sample, work.as<uint2>());
    RT_LAUNCHED(ctx);
    rt_launch(ctx, split_kernel<false>, 4 * ctx->sm_count, 256, 0, split);
    RT_LAUNCHED(ctx);
    rt_launch(ctx, split_kernel<true>, 4 * ctx->sm_count, 256, 0, split);
    RT_LAUNCHED(ctx);
    return RT_OK;
  }
};

// C = act(op(A) op(B) + bias) (+ C) of two split matrices.
struct Product {
  CUtensorMap map_a, map_b;
  Params p{};
  rt_status prepare(rt_ctx* ctx, Split& a, bool trans_a, Split& b, bool trans_b, const Decision* decision, float* c, int64_t ldc, const float* bias, int act,
                    int accumulate) {
    if (!a.map(&map_a) || !b.map(&map_b)) return RT_ERR_UNIMPLEMENTED;
    p.decision = decision;
    p.source_a = a.source;
    p.source_b = b.source;
    p.a_along_m = a.along_rows;
    p.b_along_n = b.along_rows;
    p.M = trans_a ? a.cols : a.rows;
    p.K = trans_a ? a.rows : a.cols;
    p.N = trans_b ? b.rows : b.cols;
    p.chunk = p.K < 1024 ? 6 : (p.K < 2048 ? 8 : 16);
    p.m_tiles = (p.M + BM - 1) / BM;
    choose_tiles(ctx, &p);
    p.c = c;
    p.ldc = ldc;
    p.bias = bias;
    p.act = act;
    p.accumulate = accumulate;
    return RT_OK;
  }
  rt_status run(rt_ctx* ctx) { return launch<kMatrices>(ctx, map_a, map_b, p); }
};
inline bool extents_fit(int64_t m, int64_t n, int64_t k) { return m < (1 << 24) && n < (1 << 24) && k < (1 << 24); }

}  // namespace parts
}  // namespace tc

// Microseconds that a product takes in this form: launches, 16 bytes an element of the operands (two reads, one write, one read), and the
// K-blocks' shared-memory traffic.  Measured: 1024 x 1024 x 1024 29 (estimate 29), 1559 x 277 x 2997 56 (56), 2902 x 2041 x 3921 174 (171).
float rt_gemm_parts_estimate(const rt_ctx* ctx, int64_t m, int64_t n, int64_t k) {
  using namespace tc::parts;
  if (!extents_fit(m, n, k)) return 1e30f;
  Params p{};
  p.N = (int)n;
  p.m_tiles = (int)((m + BM - 1) / BM);
  return 14.f + 3.2e-6f * (float)k * (float)(m + n) + 1.35e-3f * (float)((k + 31) / 32) * (float)choose_tiles(ctx, &p);
}

// C = act(op(A) op(B) + bias) (+ C).  RT_ERR_UNIMPLEMENTED: not a shape for this kernel, or no room for the parts.
rt_status rt_gemm_parts_internal(rt_ctx* ctx, int trans_a, int trans_b, int64_t m, int64_t n, int64_t k, const float* a, int64_t lda, const float* b,
                                 int64_t ldb, float* c, int64_t ldc, const float* bias, int act, int accumulate) {
  using namespace tc::parts;
  if (!extents_fit(m, n, k)) return RT_ERR_UNIMPLEMENTED;
  Split sa(ctx, 0, a, lda, trans_a ? k : m, trans_a ? m : k, trans_a), sb(ctx, 1, b, ldb, trans_b ? n : k, trans_b ? k : n, !trans_b);
  Split* both[2] = {&sa, &sb};
  Splitting splitting(ctx);
  Product product;
  rt_status st = splitting.prepare(ctx, both, 2, 2);
  if (st == RT_OK) st = product.prepare(ctx, sa, trans_a, sb, trans_b, splitting.split.decision, c, ldc, bias, act, accumulate);
  if (st != RT_OK) return st == RT_ERR_OOM ? RT_ERR_UNIMPLEMENTED : st;
  if ((st = splitting.run(ctx)) != RT_OK) return st;
  return product.run(ctx);
}
// da[m,k] = g[m,n] b[k,n]^T and db[k,n] (+)= a[m,k]^T g[m,n], the upstream gradient looked at once for both.
rt_status rt_matmul_backward_parts_internal(rt_ctx* ctx, const float* a, const float* b, const float* g, int64_t m, int64_t k, int64_t n, float* da,
                                            float* db, int accumulate_db) {
  using namespace tc::parts;
  if (!extents_fit(m, n, k)) return RT_ERR_UNIMPLEMENTED;
  Split sa(ctx, 0, a, k, m, k, true), sb(ctx, 1, b, n, k, n, false), g_rows(ctx, 2, g, n, m, n, false), g_cols(ctx, 2, g, n, m, n, true);
  Split* all[4] = {&sa, &sb, &g_rows, &g_cols};
  Splitting splitting(ctx);
  Product of_b, of_a;
  rt_status st = splitting.prepare(ctx, all, 4, 3);
  if (st == RT_OK) st = of_b.prepare(ctx, sa, true, g_cols, false, splitting.split.decision, db, n, nullptr, RT_ACT_NONE, accumulate_db);
  if (st == RT_OK) st = of_a.prepare(ctx, g_rows, false, sb, true, splitting.split.decision, da, k, nullptr, RT_ACT_NONE, 0);
  if (st != RT_OK) return st == RT_ERR_OOM ? RT_ERR_UNIMPLEMENTED : st;
  if ((st = splitting.run(ctx)) != RT_OK) return st;
  if ((st = of_b.run(ctx)) != RT_OK) return st;
  return of_a.run(ctx);
}
