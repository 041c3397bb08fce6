// Large products on the tensor cores with operands split into 16-bit parts beforehand.
//
// An fp32 operand is scaled by a power of two that brings its largest magnitude just below 2^15 and split into two fp16 parts, hi = fp16(x)
// and lo = fp16((x - hi) * 2^11): 22 bits, each part rounded to nearest.  hi * hi goes to one fp32 accumulator, hi * lo and lo * hi to
// another that is scaled down at the end.  That is three MMAs of kind::f16 where 3xTF32 takes three of kind::tf32 at half the rate and twice
// the bytes, and it drops less: lo * lo is below 2^-24 of a product, 2^-20 with the truncated TF32 parts.
// fp16 spans 2^40 below the largest element.  The pass that finds the largest magnitude also looks at every 128 columns of a row and every
// 64 rows of a column; if one of these segments lies wholly more than 2^24 below the largest (or there are infinities, NaN or magnitudes
// beyond 2^100), the operands are split into three bf16 parts instead (8 + 8 + 8 bits, exact, the exponents of fp32) and the same kernel
// runs six MMAs where it otherwise runs three.  Above that line an element keeps its 22 bits or is off by less than 2^-27 of its own segment.
// The decision is made on the device; nothing waits for it on the host.
//
// A K-block in memory is four slots of 16 along the reduction: hi hi lo lo of 32 elements, or the three bf16 parts of 16 and the first once
// more, with zeros for infinities and NaN: the cross terms take that one, so that an infinity meets no zero which is none.  A row of it is
// 128 bytes (reduction contiguous) or the block is 64 rows (rows contiguous); TMA fetches it in boxes of 8 KB with the 128-byte swizzle and
// tcgen05.mma reads it as it lies, either way round, so that nothing is transposed and a matrix that is an operand twice (the upstream
// gradient of a product) is split once.
//
// Roles of a CTA (one per SM, walking over tiles of 128 x up to 256): a TMA warp up to four K-blocks ahead, an MMA warp, eight warps that
// empty the accumulator into registers and write the result.  The tensor core adds into its accumulator with truncation, an error that
// grows with the number of additions (one per 16 of the reduction here, six with 3xTF32); so hi * hi is emptied every `chunk` K-blocks,
// while the MMAs of the cross terms run.  The cross terms are 2^11 smaller and stay until the tile is done.
// Measured: 4096^3, both operands read from memory, 368 us with the power limit reached (320 of them here, 95 % of the rate that cuBLAS
// sustains with bf16; 42 looking for magnitudes, 45 splitting), 3xTF32 with operands fetched by TMA 670 - 815.  Error against float64 at that
// size 6.5e-7 of the result, 3xTF32 1.04e-6; at 1000 2.7e-7 and 3.5e-7; with three bf16 parts 4.0e-7 in 650 us.
// What bounds a tile otherwise is shared memory: per K-block 128 bytes written and six times 32 read for each row of A and B, 960 cycles for
// 128 x 256 against 768 of MMAs.
// Every wait is bounded; on expiry the kernel records a code in the status word, raises a flag that all other waits poll, lets its own
// copies land, frees tensor memory and returns.
#include <cuda.h>
#include <cuda_fp16.h>

#include <climits>

#include "conv_geom.cuh"
#include "rt_internal.cuh"
#include "tc_common.cuh"

namespace tc {
namespace parts {

constexpr int BM = 128;
constexpr int kEpilogueWarps = 8, kTmaWarp = 8, kMmaWarp = 9, kThreads = 320;
constexpr uint32_t kBox = 64 * 128, kStage = 6 * kBox;  // 128 rows of A and up to 256 of B
constexpr int kStages = 4;
constexpr uint32_t kStageOffset = kStages * kStage;      // one 32 x 33 tile per accumulating warp
constexpr uint32_t kBarOffset = kStageOffset + kEpilogueWarps * 32 * 33 * 4;
constexpr int kBars = 2 * kStages + 3;
constexpr uint32_t kSmem = kBarOffset + kBars * 8 + 16 + 1024;  // + alignment of the base to 1024
static_assert(kSmem <= 232448, "shared memory");
constexpr uint32_t kCross = 256;  // tensor-memory column of the cross terms

constexpr int kMaxSources = 3, kMaxSplits = 4;  // a matrix that is an operand both ways round is split twice
constexpr int kStatTileRows = 64, kStatTileCols = 128;
constexpr int kNarrowestExponent = 24;  // a segment further below the largest magnitude than this makes the split one of three parts

struct Decision {
  int wide;                   // three bf16 parts
  int exponent[kMaxSources];  // an element is split after multiplication with 2^exponent
};

// ---- largest magnitudes -------------------------------------------------------------------------------------------------------
struct StatSource {
  const float* p;
  int64_t ld;
  int rows, cols, tiles_c, vec;
  uint32_t tiles;
};
struct StatArgs {
  StatSource s[kMaxSources];
  int count;
};
// Bound by memory: every element is read once, eight 128-bit loads a thread in flight, four blocks an SM.  Of each source a block leaves the largest magnitude
// and the smallest of its non-zero segments' largest, as the bits of floats (which order as they do; NaN above infinity).
__device__ __forceinline__ void load_tile(const StatSource& s, uint32_t t, int warp, int lane, uint32_t (&v)[8][4]) {
  const int tr = (int)(t / (uint32_t)s.tiles_c), tc = (int)(t - (uint32_t)tr * (uint32_t)s.tiles_c);
  const int r0 = tr * kStatTileRows + warp * 8, c0 = tc * kStatTileCols;
  const float* p = s.p + (int64_t)r0 * s.ld + c0;
#pragma unroll
  for (int i = 0; i < 8; ++i, p += s.ld) {
    const bool in = r0 + i < s.rows;
    if (s.vec) {
      const float4 f = in && c0 + 4 * lane < s.cols ? __ldg(reinterpret_cast<const float4*>(p) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[i][0] = __float_as_uint(f.x); v[i][1] = __float_as_uint(f.y); v[i][2] = __float_as_uint(f.z); v[i][3] = __float_as_uint(f.w);
    } else {  // a row's 128 elements as four coalesced loads: the lane has other columns of the tile
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] = in && c0 + 32 * j + lane < s.cols ? __float_as_uint(__ldg(p + 32 * j + lane)) : 0u;
    }
  }
}
__global__ void __launch_bounds__(256, 4) stat_kernel(const StatArgs a, uint2* __restrict__ out) {
  RT_PDL_ENTRY();
  __shared__ uint32_t cols[2][8][kStatTileCols];
  __shared__ uint32_t red[2][8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int turn = 0;
  for (int q = 0; q < a.count; ++q) {
    const StatSource& s = a.s[q];
    uint32_t most = 0, least = 0xffffffffu;
    for (uint32_t t = blockIdx.x; t < s.tiles; t += gridDim.x) {
      uint32_t v[8][4];
      load_tile(s, t, warp, lane, v);
      uint32_t col[4] = {0, 0, 0, 0};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint32_t row = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t m = v[i][j] & 0x7fffffffu;
          row = max(row, m);
          col[j] = max(col[j], m);
        }
        row = __reduce_max_sync(0xffffffffu, row);
        most = max(most, row);
        if (row) least = min(least, row);
      }
      turn ^= 1;  // two buffers, so that one barrier a tile is enough
#pragma unroll
      for (int j = 0; j < 4; ++j) cols[turn][warp][lane + 32 * j] = col[j];
      __syncthreads();
      if (threadIdx.x < kStatTileCols) {
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) m = max(m, cols[turn][i][threadIdx.x]);
        if (m) least = min(least, m);
      }
    }
    least = __reduce_min_sync(0xffffffffu, least);
    __syncthreads();
    if (lane == 0) {
      red[0][warp] = most;
      red[1][warp] = least;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int i = 1; i < 8; ++i) {
        most = max(most, red[0][i]);
        least = min(least, red[1][i]);
      }
      out[(int64_t)q * gridDim.x + blockIdx.x] = make_uint2(most, least);
    }
    __syncthreads();
  }
}
// What the blocks of stat_kernel left, as every block of a splitting kernel sees it.  `red`: 2 x 8 words; 256 threads.
__device__ __forceinline__ Decision decide(const uint2* stats, int blocks, int count, uint32_t (*red)[8]) {
  Decision d{};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int q = 0; q < count; ++q) {
    uint32_t most = 0, least = 0xffffffffu;
    for (int i = threadIdx.x; i < blocks; i += 256) {
      const uint2 v = __ldg(stats + (int64_t)q * blocks + i);
      most = max(most, v.x);
      least = min(least, v.y);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    least = __reduce_min_sync(0xffffffffu, least);
    __syncthreads();
    if (lane == 0) {
      red[0][warp] = most;
      red[1][warp] = least;
    }
    __syncthreads();
    most = red[0][lane & 7];
    least = red[1][lane & 7];
    most = __reduce_max_sync(0xffffffffu, most);
    least = __reduce_min_sync(0xffffffffu, least);
    if (most == 0) continue;  // all zero
    const int e = (int)(most >> 23) - 127;  // subnormal magnitudes: -127
    if (e > 100 || e < -100 || (int)(least >> 23) - 127 < e - kNarrowestExponent) d.wide = 1;
    d.exponent[q] = 14 - e;
  }
  if (d.wide)
    for (int q = 0; q < kMaxSources; ++q) d.exponent[q] = 0;
  return d;
}

// ---- splitting ----------------------------------------------------------------------------------------------------------------
// The parts of eight elements, two or four, as 16-byte pieces.
__device__ __forceinline__ void split8(const float (&x)[8], int wide, float scale, uint4 (&part)[4]) {
  uint32_t w[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (!wide) {
      const float a = x[2 * i] * scale, b = x[2 * i + 1] * scale;
      const __half2 hi = __floats2half2_rn(a, b);
      const float2 h = __half22float2(hi);
      const __half2 lo = __floats2half2_rn((a - h.x) * 2048.f, (b - h.y) * 2048.f);
      w[0][i] = *reinterpret_cast<const uint32_t*>(&hi);
      w[1][i] = *reinterpret_cast<const uint32_t*>(&lo);
      w[2][i] = w[3][i] = 0;
    } else {
      float a = x[2 * i], b = x[2 * i + 1];
      const bool fa = fabsf(a) <= 3.4028235e38f, fb = fabsf(b) <= 3.4028235e38f;
      const uint32_t special = (fa ? 0u : (a != a ? 0x7fc0u : __float_as_uint(a) >> 16)) | (fb ? 0u : (b != b ? 0x7fc00000u : __float_as_uint(b)));
      if (!fa) a = 0.f;
      if (!fb) b = 0.f;
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const uint32_t ta = __float_as_uint(a) & 0xffff0000u, tb = __float_as_uint(b) & 0xffff0000u;
        w[p][i] = ta >> 16 | tb;
        a -= __uint_as_float(ta);
        b -= __uint_as_float(tb);
      }
      w[3][i] = w[0][i];
      w[0][i] |= special;
    }
  }
#pragma unroll
  for (int p = 0; p < 4; ++p) part[p] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

struct SplitSource {
  const float* p;
  uint16_t* out;
  int64_t ld, ldo;   // floats, halves
  int rows, cols;
  int along_rows;    // the reduction runs down the rows
  int vec;
  int source;        // of the statistics
};
struct SplitArgs {
  SplitSource s[kMaxSplits];
  int count, stat_sources, stat_blocks;
  const uint2* stats;
  Decision* decision;
};
// VEC: every piece of eight lies within the columns and on a 16-byte boundary.
template <bool VEC>
__device__ __forceinline__ void split_source(const SplitSource& s, int wide, float scale) {
  const int depth = wide ? 16 : 32;  // elements of a K-block
  // the padding behind the reduction is written as zeros
  const int rows = s.along_rows ? (s.rows + depth - 1) / depth * depth : s.rows;
  const int pieces = s.along_rows ? (s.cols + 7) / 8 : (s.cols + depth - 1) / depth * depth / 8;
  const int64_t total = (int64_t)rows * pieces, step = (int64_t)gridDim.x * 256, first = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int step_r = (int)(step / pieces), step_c = (int)(step % pieces);
  int r = (int)(first / pieces), c8 = (int)(first % pieces);
  for (int64_t i = first; i < total; i += 2 * step) {
    float x[2][8];
    int rr[2], cc[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {  // both pieces are loaded before either is used
      rr[u] = r;
      cc[u] = c8 * 8;
      const float* p = s.p + (int64_t)r * s.ld + cc[u];
      if (VEC) {
        const bool in = r < s.rows && cc[u] < s.cols;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 v = in ? __ldcs(reinterpret_cast<const float4*>(p)) : zero, w = in ? __ldcs(reinterpret_cast<const float4*>(p) + 1) : zero;
        x[u][0] = v.x; x[u][1] = v.y; x[u][2] = v.z; x[u][3] = v.w; x[u][4] = w.x; x[u][5] = w.y; x[u][6] = w.z; x[u][7] = w.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[u][j] = r < s.rows && cc[u] + j < s.cols ? __ldg(p + j) : 0.f;
      }
      r += step_r;
      c8 += step_c;
      if (c8 >= pieces) {
        c8 -= pieces;
        ++r;
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (i + u * step >= total) break;
      uint4 part[4];
      split8(x[u], wide, scale, part);
      const unsigned along = s.along_rows ? rr[u] : cc[u], block = along / depth, in_block = along % depth;
      uint16_t* o = s.along_rows ? s.out + ((int64_t)block * 64 + in_block) * s.ldo + cc[u] : s.out + (int64_t)rr[u] * s.ldo + block * 64 + in_block;
      const int64_t next = s.along_rows ? depth * s.ldo : depth;
      *reinterpret_cast<uint4*>(o) = part[0];
      *reinterpret_cast<uint4*>(o + next) = part[1];
      if (wide) {
        *reinterpret_cast<uint4*>(o + 2 * next) = part[2];
        *reinterpret_cast<uint4*>(o + 3 * next) = part[3];
      }
    }
  }
}
// Bound by memory: 4 bytes read and 4 written an element.  The sources are taken in the opposite order to that in which stat_kernel read
// them, since the last of them is still in L2.
__global__ void __launch_bounds__(256) split_kernel(const SplitArgs a) {
  RT_PDL_ENTRY();
  __shared__ uint32_t red[2][8];
  const Decision d = decide(a.stats, a.stat_blocks, a.stat_sources, red);
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.decision = d;
  for (int q = a.count - 1; q >= 0; --q) {
    const SplitSource& s = a.s[q];
    const float scale = ldexpf(1.f, d.exponent[s.source]);
    if (s.vec && s.cols % 8 == 0) split_source<true>(s, d.wide, scale);
    else split_source<false>(s, d.wide, scale);
  }
}

// ---- the product --------------------------------------------------------------------------------------------------------------
struct Params {
  const Decision* decision;
  int source_a, source_b;
  int a_along_m, b_along_n;   // operand with its rows (of the product) contiguous instead of the reduction
  int M, N, K;
  int chunk;                  // K-blocks that the accumulator of hi * hi sums before it is emptied
  int m_tiles, width;         // columns of a tile: a multiple of 64, 256 at most
  int items, whole, part;     // the tiles from `whole` on are walked over in parts of `part` columns
  float* c;
  int64_t ldc;
  const float* bias;
  int act, accumulate;
};
__device__ __forceinline__ void item_of(const Params& p, int i, int& mt, int& n0, int& w) {
  int tile = i, sub = 0;
  w = p.width;
  if (i >= p.whole) {
    const int per = p.width / p.part, j = i - p.whole;
    tile = p.whole + j / per;
    sub = j % per;
    w = p.part;
  }
  mt = tile % p.m_tiles;
  n0 = tile / p.m_tiles * p.width + sub * p.part;
  const int left = (p.N - n0 + 63) & ~63;
  w = min(w, left);  // none or less: nothing to do
}

__device__ __forceinline__ void load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map),
               "r"(x), "r"(y), "r"(bar)
               : "memory");
}
// One MMA with both operands in shared memory; one elected lane of a converged warp issues.
__device__ __forceinline__ void mma(uint32_t d, uint32_t a, uint32_t a_hi, uint32_t b, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred pa, pe;\n\t"
      ".reg .b64 da, db;\n\t"
      "elect.sync _|pe, 0xffffffff;\n\t"
      "setp.ne.b32 pa, %6, 0;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, pa;\n\t}" ::"r"(d), "r"(a), "r"(a_hi), "r"(b), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Bounded wait that also ends when another role has given up.
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, int* status, int code, volatile int* abort) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (mbar_try(bar, parity)) return true;
    if ((i & 63) == 63 && *abort) return false;
  }
  *abort = 1;
  record_status(status, code);
  return false;
}
__device__ __forceinline__ float activated(float v, int act) {
  if (act == RT_ACT_RELU) return fmaxf(v, 0.f);
  if (act == RT_ACT_TANH) return tanhf(v);
  if (act == RT_ACT_SIGMOID) return 1.f / (1.f + expf(-v));
  return v;
}

__global__ void __launch_bounds__(kThreads, 1)
parts_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Params p, int* status) {
  RT_PDL_ENTRY();
  extern __shared__ char smem_raw[];
  __shared__ volatile int abort_flag;
  const uint32_t raw_base = smem_u32(smem_raw);
  const uint32_t base = (raw_base + 1023) & ~1023u;
  char* smem = smem_raw + (base - raw_base);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t bars = base + kBarOffset;
  auto full = [&](int i) { return bars + 8 * i; };
  auto empty = [&](int i) { return bars + 8 * (kStages + i); };
  const uint32_t acc_full = bars + 16 * kStages, acc_empty = acc_full + 8, cross_empty = acc_full + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kBarOffset + kBars * 8);

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full(i), 1);
      mbar_init(empty(i), 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, kEpilogueWarps);
    mbar_init(cross_empty, kEpilogueWarps);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) tmem_alloc(smem_u32(tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const int wide = __shfl_sync(0xffffffffu, p.decision->wide, 0);
  const int k_blocks = wide ? (p.K + 15) / 16 : (p.K + 31) / 32;
  bool ok = true;

  if (warp == kTmaWarp) {
    // ---------------- TMA ----------------
    if (lane == 0) {
      asm volatile("fence.proxy.async.global;" ::: "memory");  // the parts were written by ordinary stores
      int it = 0;
      for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
        int mt, n0, w;
        item_of(p, i, mt, n0, w);
        if (w <= 0) continue;
        const int boxes = w / 64;
        for (int kb = 0; kb < k_blocks && ok; ++kb, ++it) {
          const int s = it % kStages;
          if (it >= kStages) ok = wait(empty(s), (it / kStages - 1) & 1, status, 61, &abort_flag);
          if (!ok) break;
          const uint32_t dst = base + s * kStage;
          mbar_expect_tx(full(s), (2 + boxes) * kBox);
          for (int j = 0; j < 2; ++j) {
            const int m = mt * BM + j * 64;
            load_2d(dst + j * kBox, &map_a, p.a_along_m ? m : kb * 64, p.a_along_m ? kb * 64 : m, full(s));
          }
          for (int j = 0; j < boxes; ++j) {
            const int n = n0 + j * 64;
            load_2d(dst + (2 + j) * kBox, &map_b, p.b_along_n ? n : kb * 64, p.b_along_n ? kb * 64 : n, full(s));
          }
        }
      }
      // copies that nobody has waited for must have landed before the CTA may leave
      if (!ok)
        for (int i = it > kStages ? it - kStages : 0; i < it; ++i) mbar_wait(full(i % kStages), (i / kStages) & 1, status, 62);
    }
  } else if (warp == kMmaWarp) {
    // ---------------- MMAs ----------------
    // descriptors: 8-row (8-K) groups 1024 bytes apart, 128-byte swizzle; with the rows contiguous, groups of 64 rows a box apart
    constexpr uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
    const uint32_t lbo = (kBox >> 4) << 16;
    const uint32_t slot_a = p.a_along_m ? 2048 >> 4 : 32 >> 4, slot_b = p.b_along_n ? 2048 >> 4 : 32 >> 4;
    const uint32_t format = wide ? 1u : 0u;
    const uint32_t idesc0 = (1u << 4) | format << 7 | format << 10 | (uint32_t)p.a_along_m << 15 | (uint32_t)p.b_along_n << 16 |
                            (uint32_t)(BM >> 4) << 24;
    int it = 0, chunks = 0, t = 0;
    for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
      int mt, n0, w;
      item_of(p, i, mt, n0, w);
      if (w <= 0) continue;
      const uint32_t idesc = idesc0 | (uint32_t)(w >> 3) << 17;
      for (int kb = 0, in_chunk = 0; kb < k_blocks && ok; ++kb, ++it) {
        const int s = it % kStages;
        const bool first = in_chunk == 0, last = ++in_chunk == p.chunk || kb + 1 == k_blocks;
        if (last) in_chunk = 0;
        ok = wait(full(s), (it / kStages) & 1, status, 63, &abort_flag);
        if (ok && kb == 0 && t > 0) ok = wait(cross_empty, (t - 1) & 1, status, 64, &abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a = ((base + s * kStage) >> 4 & 0x3FFF) | lbo, b = ((base + s * kStage + 2 * kBox) >> 4 & 0x3FFF) | lbo;
        const uint32_t cross = tmem + kCross, more = kb > 0;
        // slots: hi 0 1, lo 2 3; or the parts 0 1 2 and 3 = the finite values of 0
        if (!wide) {
          mma(cross, a, desc_hi, b + 2 * slot_b, desc_hi, idesc, more);
          mma(cross, a + slot_a, desc_hi, b + 3 * slot_b, desc_hi, idesc, 1);
          mma(cross, a + 2 * slot_a, desc_hi, b, desc_hi, idesc, 1);
          mma(cross, a + 3 * slot_a, desc_hi, b + slot_b, desc_hi, idesc, 1);
        } else {
          mma(cross, a + slot_a, desc_hi, b + slot_b, desc_hi, idesc, more);
          mma(cross, a + 3 * slot_a, desc_hi, b + 2 * slot_b, desc_hi, idesc, 1);
          mma(cross, a + 2 * slot_a, desc_hi, b + 3 * slot_b, desc_hi, idesc, 1);
          mma(cross, a + 3 * slot_a, desc_hi, b + slot_b, desc_hi, idesc, 1);
          mma(cross, a + slot_a, desc_hi, b + 3 * slot_b, desc_hi, idesc, 1);
        }
        if (first && chunks > 0) {
          ok = __all_sync(0xffffffffu, wait(acc_empty, (chunks - 1) & 1, status, 65, &abort_flag));
          if (!ok) break;
          tc_fence_after();
        }
        mma(tmem, a, desc_hi, b, desc_hi, idesc, !first);
        if (!wide) mma(tmem, a + slot_a, desc_hi, b + slot_b, desc_hi, idesc, 1);
        umma_commit_elect(empty(s));
        if (last) {
          umma_commit_elect(acc_full);
          ++chunks;
        }
      }
      ++t;
    }
  } else {
    // ---------------- sums over the chunks, result ----------------
    float* stage = reinterpret_cast<float*>(smem + kStageOffset) + warp * 32 * 33;
    const int quad = warp & 3, group = warp >> 2;
    const int exponent = wide ? 0 : -(p.decision->exponent[p.source_a] + p.decision->exponent[p.source_b]);
    const float f1 = ldexpf(1.f, exponent / 2), f2 = ldexpf(1.f, exponent - exponent / 2), cross_scale = wide ? 1.f : 1.f / 2048.f;
    const int chunks = (k_blocks + p.chunk - 1) / p.chunk;  // of a tile
    uint32_t parity = 0;
    for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
      int mt, n0, w;
      item_of(p, i, mt, n0, w);
      if (w <= 0) continue;
      const int half = w / 2;  // columns of this group
      const uint32_t d = tmem + ((uint32_t)(quad * 32) << 16) + group * half;
      float sum[128];
#pragma unroll
      for (int j = 0; j < 128; ++j) sum[j] = 0.f;
      for (int ch = 0; ch < chunks && ok; ++ch) {
        ok = __all_sync(0xffffffffu, wait(acc_full, parity, status, 66, &abort_flag));
        if (!ok) break;
        parity ^= 1;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 128; c += 32)
          if (c < half) {
            float v[32];
            tmem_ld32(d + c, v);
#pragma unroll
            for (int j = 0; j < 32; ++j) sum[c + j] += v[j];
          }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty);
      }
      if (!ok) break;
#pragma unroll
      for (int c = 0; c < 128; c += 32)
        if (c < half) {
          float v[32];
          tmem_ld32(d + kCross + c, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) sum[c + j] = (sum[c + j] + v[j] * cross_scale) * f1 * f2;
        }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(cross_empty);
      const int m0 = mt * BM + quad * 32, n_first = n0 + group * half;
#pragma unroll
      for (int c = 0; c < 128; c += 32) {
        const int n = n_first + c + lane;
        if (c < half && n_first + c < p.N) {
#pragma unroll
          for (int j = 0; j < 32; ++j) stage[lane * 33 + j] = sum[c + j];
          __syncwarp();
          if (n < p.N) {
            const float bias = p.bias ? __ldg(p.bias + n) : 0.f;
            float* out = p.c + (int64_t)m0 * p.ldc + n;
            const int rows = min(32, p.M - m0);
#pragma unroll 4
            for (int r = 0; r < rows; ++r) {
              float u = stage[r * 33 + lane] + bias;
              if (p.act != RT_ACT_NONE) u = activated(u, p.act);
              if (p.accumulate) u += out[(int64_t)r * p.ldc];
              out[(int64_t)r * p.ldc] = u;
            }
          }
          __syncwarp();
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
    cudaGetLastError();
    return reinterpret_cast<EncodeTiledFn>(f);
  }();
  return fn;
}
// [rows][cols] 16-bit values, rows ld apart, boxes of 64 x 64, zeros outside.
inline bool map_parts(CUtensorMap* m, uint16_t* t, int64_t cols, int64_t rows, int64_t ld) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {64, 64}, one[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, t, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
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

// Splits matrices, the first `sources` of which are all different; decision: device memory of one Decision.
inline rt_status split_all(rt_ctx* ctx, Split* const* s, int count, int sources, RtScratch* work, Decision** decision) {
  const int stat_blocks = 4 * ctx->sm_count;
  const size_t stat_bytes = sizeof(uint2) * (size_t)stat_blocks * kMaxSources;
  rt_status st = work->alloc(stat_bytes + sizeof(Decision));
  if (st != RT_OK) return st;
  StatArgs a{};
  SplitArgs b{};
  a.count = b.stat_sources = sources;
  b.count = count;
  b.stat_blocks = stat_blocks;
  b.stats = work->as<uint2>();
  *decision = b.decision = reinterpret_cast<Decision*>(work->as<char>() + stat_bytes);
  for (int q = 0; q < count; ++q) {
    if ((st = s[q]->alloc()) != RT_OK) return st;
    const int vec = rt_aligned16(s[q]->p) && s[q]->ld % 4 == 0 && s[q]->cols % 4 == 0;
    const int tiles_c = (s[q]->cols + kStatTileCols - 1) / kStatTileCols;
    if (q < sources)
      a.s[q] = {s[q]->p, s[q]->ld, s[q]->rows, s[q]->cols, tiles_c, vec, (uint32_t)tiles_c * (uint32_t)((s[q]->rows + kStatTileRows - 1) / kStatTileRows)};
    b.s[q] = {s[q]->p, s[q]->mem.as<uint16_t>(), s[q]->ld, s[q]->ldo, s[q]->rows, s[q]->cols, s[q]->along_rows, vec, s[q]->source};
  }
  rt_launch(ctx, stat_kernel, stat_blocks, 256, 0, a, work->as<uint2>());
  RT_LAUNCHED(ctx);
  rt_launch(ctx, split_kernel, 8 * ctx->sm_count, 256, 0, b);
  RT_LAUNCHED(ctx);
  return RT_OK;
}

// Width of the tiles, and of the parts that those of the last wave are walked over in.  What a K-block costs is what crosses the shared
// memory of an SM: 128 bytes written and six times 32 read for each of the 128 rows and w columns.  Returns that, for the whole product
// and one K-block, in units of a row.
inline int choose_tiles(const rt_ctx* ctx, Params* p) {
  const int sms = ctx->sm_count;
  int best = INT_MAX;
  for (int w = 256; w >= 64; w -= 64) {
    const int tiles = p->m_tiles * ((p->N + w - 1) / w), whole = tiles / sms * sms, rest = tiles - whole;
    for (int part = w; part >= 64; part -= 64) {
      if (w % part) continue;
      const int parts = rest * (w / part), cost = tiles / sms * (BM + w) + (parts + sms - 1) / sms * (BM + part);
      if (cost >= best) continue;
      best = cost;
      p->width = w;
      p->part = part;
      p->whole = whole;
      p->items = whole + parts;
    }
  }
  return best;
}

// C = act(op(A) op(B) + bias) (+ C) of two split matrices.
inline rt_status product(rt_ctx* ctx, Split& a, bool trans_a, Split& b, bool trans_b, const Decision* decision, float* c, int64_t ldc, const float* bias,
                         int act, int accumulate) {
  Params p{};
  CUtensorMap ma, mb;
  if (!a.map(&ma) || !b.map(&mb)) return RT_ERR_UNIMPLEMENTED;
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
  static RtDeviceOnce once;
  RT_CUDA(ctx, once([&] { return cudaFuncSetAttribute(parts_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem); }));
  rt_launch(ctx, parts_gemm_kernel, p.items < ctx->sm_count ? p.items : ctx->sm_count, kThreads, kSmem, ma, mb, p, ctx->device_status);
  RT_LAUNCHED(ctx);
  return RT_OK;
}
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
  RtScratch work(ctx);
  Split sa(ctx, 0, a, lda, trans_a ? k : m, trans_a ? m : k, trans_a), sb(ctx, 1, b, ldb, trans_b ? n : k, trans_b ? k : n, !trans_b);
  Split* both[2] = {&sa, &sb};
  Decision* decision;
  rt_status st = split_all(ctx, both, 2, 2, &work, &decision);
  if (st == RT_ERR_OOM) return RT_ERR_UNIMPLEMENTED;
  if (st != RT_OK) return st;
  return product(ctx, sa, trans_a, sb, trans_b, decision, c, ldc, bias, act, accumulate);
}
// da[m,k] = g[m,n] b[k,n]^T and db[k,n] (+)= a[m,k]^T g[m,n], the upstream gradient looked at once for both.
rt_status rt_matmul_backward_parts_internal(rt_ctx* ctx, const float* a, const float* b, const float* g, int64_t m, int64_t k, int64_t n, float* da,
                                            float* db, int accumulate_db) {
  using namespace tc::parts;
  if (!extents_fit(m, n, k)) return RT_ERR_UNIMPLEMENTED;
  RtScratch work(ctx);
  Split sa(ctx, 0, a, k, m, k, true), sb(ctx, 1, b, n, k, n, false), g_rows(ctx, 2, g, n, m, n, false), g_cols(ctx, 2, g, n, m, n, true);
  Split* all[4] = {&sa, &sb, &g_rows, &g_cols};
  Decision* decision;
  rt_status st = split_all(ctx, all, 4, 3, &work, &decision);
  if (st == RT_ERR_OOM) return RT_ERR_UNIMPLEMENTED;
  if (st == RT_OK) st = product(ctx, sa, true, g_cols, false, decision, db, n, nullptr, RT_ACT_NONE, accumulate_db);
  if (st == RT_OK) st = product(ctx, g_rows, false, sb, true, decision, da, k, nullptr, RT_ACT_NONE, 0);
  return st;
}
