// What the products of operands in 16-bit parts share (k_gemm_parts.cu, k_conv_parts.cu): the scale and the decision between two fp16 and three
// bf16 parts, splitting, PTX wrappers, the product kernel.  k_gemm_parts.cu says how they work.
#pragma once
#include <cuda_fp16.h>

#include <climits>

#include "conv_geom.cuh"
#include "rt_internal.cuh"
#include "tc_common.cuh"
#include "tensor_map.cuh"

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

constexpr int kMaxSources = 3;
constexpr int kTileRows = 64, kTileCols = 128;
constexpr int kSampleExponent = 9;                         // where the sample's largest magnitude is scaled to
constexpr int kLargestExponent = 14, kSmallestExponent = -9;  // of any element, of a segment's largest
// Elements that are not zero and stay below 2^-22 after scaling are faint: they keep fewer than 14 bits, which shows where the other operand is large.
// Two parts will do while there are next to none.  Of 2^24 numbers from a normal distribution 0.03 are, of the gate gradients of a recurrent network
// 4; of magnitudes spread evenly over 2^31 none, over 2^33 one in 20.
constexpr int kFaintExponent = -22;
// An image's pixel is multiplied as a whole, all channels: its largest element stays above this, where two parts keep 20 bits at least.
constexpr int kFaintPixelExponent = -16;
inline uint32_t most_faint(int64_t elements) { return 4 + (uint32_t)(elements >> 20); }

struct Decision {
  int wide;                   // three bf16 parts
  int special;                // convolutions: there are infinities or NaN
  int exponent[kMaxSources];  // an element is split after multiplication with 2^exponent
};

// ---- magnitudes: the largest, and the smallest of the non-zero segments' largest, as the bits of floats (which order as they do; NaN
// above infinity), and in how many pieces (of eight or sixteen elements) there is a faint one ------------------------------------------
struct Magnitudes {
  uint32_t most = 0, least = 0xffffffffu, faint = 0;
};
// What a block makes of its own, in a word: whether two parts are out of the question, whether there are infinities or NaN, the faint pieces.
constexpr uint32_t kOutOfRange = 1u << 31, kSpecial = 1u << 30, kFaintOfBlock = 1u << 20;
struct Sample {
  const float* p;
  int64_t ld;
  int rows, cols, tiles_c, vec;
  uint32_t tiles, step;  // one of `step` tiles is looked at
};
struct SampleArgs {
  Sample s[kMaxSources];
  int count;
};
inline Sample sample_of(const rt_ctx* ctx, const float* p, int64_t ld, int64_t rows, int64_t cols, bool all) {
  const int64_t tiles_c = (cols + kTileCols - 1) / kTileCols, tiles = tiles_c * ((rows + kTileRows - 1) / kTileRows);
  return {p, ld, (int)rows, (int)cols, (int)tiles_c, rt_aligned16(p) && ld % 4 == 0 && cols % 4 == 0, (uint32_t)tiles,
          all ? 1u : (uint32_t)((tiles + ctx->sm_count - 1) / ctx->sm_count)};
}
// The block's, in all its threads.  red: 3 x 8 words; 256 threads.
__device__ __forceinline__ Magnitudes over_block(Magnitudes m, uint32_t (*red)[8]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  m.most = __reduce_max_sync(0xffffffffu, m.most);
  m.least = __reduce_min_sync(0xffffffffu, m.least);
  m.faint = __reduce_add_sync(0xffffffffu, m.faint);
  __syncthreads();
  if (lane == 0) {
    red[0][warp] = m.most;
    red[1][warp] = m.least;
    red[2][warp] = m.faint;
  }
  __syncthreads();
  m.most = __reduce_max_sync(0xffffffffu, red[0][lane & 7]);
  m.least = __reduce_min_sync(0xffffffffu, red[1][lane & 7]);
  m.faint = __reduce_add_sync(0xffffffffu, lane < 8 ? red[2][lane] : 0u);
  return m;
}
// Most and least over all blocks' samples, [source][block].  red: 6 x 8 words.
__device__ __forceinline__ void over_samples(const uint2* samples, int sources, int blocks, uint32_t (*red)[8], uint2 (&v)[kMaxSources]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < kMaxSources; ++q) v[q] = make_uint2(0u, 0xffffffffu);
  for (int i = threadIdx.x; i < blocks; i += 256)
#pragma unroll
    for (int q = 0; q < kMaxSources; ++q)
      if (q < sources) {
        const uint2 w = __ldg(samples + q * blocks + i);
        v[q] = make_uint2(max(v[q].x, w.x), min(v[q].y, w.y));
      }
#pragma unroll
  for (int q = 0; q < kMaxSources; ++q) {
    const uint32_t most = __reduce_max_sync(0xffffffffu, v[q].x), least = __reduce_min_sync(0xffffffffu, v[q].y);
    if (lane == 0) {
      red[2 * q][warp] = most;
      red[2 * q + 1][warp] = least;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kMaxSources; ++q)
    v[q] = make_uint2(__reduce_max_sync(0xffffffffu, red[2 * q][lane & 7]), __reduce_min_sync(0xffffffffu, red[2 * q + 1][lane & 7]));
  __syncthreads();
}
// The exponent that a sample asks for; more than 100 either way is refused by verdict().
__device__ __forceinline__ int exponent_for(uint32_t most) { return most == 0 || most >= 0x7f800000u ? 0 : kSampleExponent + 127 - (int)(most >> 23); }
// An element of magnitude m (its bits) is faint if m - 1 is below this: zero is not.
__device__ __forceinline__ uint32_t faint_below(int exponent, int power = kFaintExponent) { return max(__float_as_uint(ldexpf(1.f, power - exponent)), 1u) - 1u; }
// The least of m - 1 over a piece, an element more.
__device__ __forceinline__ uint32_t lower(uint32_t least, uint32_t m) { return __viaddmin_u32(m, 0xffffffffu, least); }
__device__ __forceinline__ uint32_t verdict(const Magnitudes& v, int exponent) {
  uint32_t w = min(v.faint, kFaintOfBlock);
  if (v.most >= 0x7f800000u) w |= kSpecial | kOutOfRange;
  else if (v.most && (exponent > 100 || exponent < -100 || (int)(v.most >> 23) - 127 + exponent > kLargestExponent ||
                      (int)(v.least >> 23) - 127 + exponent < kSmallestExponent))
    w |= kOutOfRange;
  return w;
}
// All blocks' verdicts, [source][block].  red: 4 x 8 words.
__device__ __forceinline__ Decision decide(const uint32_t* verdicts, int sources, int blocks, const uint32_t (&most_faint)[kMaxSources], uint32_t (*red)[8]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t flags = 0, faint[kMaxSources] = {};
#pragma unroll 4
  for (int i = threadIdx.x; i < blocks; i += 256)
#pragma unroll
    for (int q = 0; q < kMaxSources; ++q)
      if (q < sources) {
        const uint32_t w = __ldg(verdicts + q * blocks + i);
        flags |= w;
        faint[q] += w & (kSpecial - 1);
      }
  flags = __reduce_or_sync(0xffffffffu, flags);
#pragma unroll
  for (int q = 0; q < kMaxSources; ++q) faint[q] = __reduce_add_sync(0xffffffffu, faint[q]);
  if (lane == 0) {
    red[kMaxSources][warp] = flags;
#pragma unroll
    for (int q = 0; q < kMaxSources; ++q) red[q][warp] = faint[q];
  }
  __syncthreads();
  flags = __reduce_or_sync(0xffffffffu, red[kMaxSources][lane & 7]);
  Decision d{};
  d.wide = (flags & kOutOfRange) != 0;
  d.special = (flags & kSpecial) != 0;
#pragma unroll
  for (int q = 0; q < kMaxSources; ++q)
    if (q < sources && __reduce_add_sync(0xffffffffu, lane < 8 ? red[q][lane] : 0u) > most_faint[q]) d.wide = 1;
  return d;
}
// A warp has eight rows of a tile of 64 x 128, eight 128-bit loads in flight.
static __global__ void __launch_bounds__(256) sample_kernel(const SampleArgs a, uint2* __restrict__ out) {
  RT_PDL_ENTRY();
  __shared__ uint32_t cols[2][8][kTileCols];
  __shared__ uint32_t red[3][8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int turn = 0;
  for (int q = 0; q < a.count; ++q) {
    const Sample& s = a.s[q];
    Magnitudes all;
    for (uint32_t k = blockIdx.x; k * s.step < s.tiles; k += gridDim.x) {
      // not always the same place of `step` tiles: rows of them may repeat
      const uint32_t t = min(k * s.step + (s.step > 1 ? (k * 40503u >> 8) % s.step : 0), s.tiles - 1);
      const int tr = (int)(t / (uint32_t)s.tiles_c), tc = (int)(t - (uint32_t)tr * (uint32_t)s.tiles_c);
      const int r0 = tr * kTileRows + warp * 8, c0 = tc * kTileCols;
      const float* p = s.p + (int64_t)r0 * s.ld + c0;
      uint32_t v[8][4];
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
        all.most = max(all.most, row);
        if (row) all.least = min(all.least, row);
      }
      turn ^= 1;  // two buffers, so that one barrier a tile is enough
#pragma unroll
      for (int j = 0; j < 4; ++j) cols[turn][warp][lane + 32 * j] = col[j];
      __syncthreads();
      if (threadIdx.x < kTileCols) {
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) m = max(m, cols[turn][i][threadIdx.x]);
        if (m) all.least = min(all.least, m);
      }
    }
    all = over_block(all, red);
    if (threadIdx.x == 0) out[q * gridDim.x + blockIdx.x] = make_uint2(all.most, all.least);
    __syncthreads();
  }
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

// ---- the product --------------------------------------------------------------------------------------------------------------
struct Params {
  const Decision* decision;
  int source_a, source_b;
  int a_along_m, b_along_n;   // operand with its rows (of the product) contiguous instead of the reduction
  int M, N, K;
  int chunk;                  // K-blocks that the accumulator of hi * hi sums before it is emptied
  int m_tiles, width;         // columns of a tile: a multiple of 64, 256 at most
  int items, whole, part;     // the tiles from `whole` on are walked over in parts of `part` columns
  // A = the pixels of a channels-last image at one kernel tap: a tile is a box of bw x bh x bn of them
  int C, taps, kw;
  int bw, bh, bn, tiles_w, tiles_h;
  int rows_w, rows_h, rows_n;              // extent of the row side
  int sx, sy, px, py;                      // source coordinate = row coordinate * s - p + tap
  int out_h, out_w;                        // output pixel = row coordinate, channels as planes
  int pairs;                               // of 2 x 2 outputs (columns channel * 4 + 2 * ry + rx) two may be written at a time
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

__device__ __forceinline__ void load_4d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, int w, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
               : "memory");
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

// The first pixel of a box of which there are tiles_w x tiles_h to an image.
__device__ __forceinline__ void box_origin(int box, int tiles_w, int tiles_h, int bw, int bh, int bn, int& x, int& y, int& n) {
  const int r = box / tiles_w;
  x = box % tiles_w * bw;
  y = r % tiles_h * bh;
  n = r / tiles_h * bn;
}

// A: matrices, the pixels of an image, or those with 2 x 2 outputs each.
enum { kMatrices, kPixels, kPhases };
template <int KIND>
__global__ void __launch_bounds__(kThreads, 1)
parts_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Params p, int* status) {
  constexpr bool PIXELS = KIND != kMatrices;
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
  const int c_blocks = PIXELS ? (wide ? (p.C + 15) / 16 : (p.C + 31) / 32) : 0;
  const int k_blocks = PIXELS ? p.taps * c_blocks : (wide ? (p.K + 15) / 16 : (p.K + 31) / 32);
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
        int x0 = 0, y0 = 0, i0 = 0, cb = 0, kx = 0, ky = 0;
        if (PIXELS) {
          box_origin(mt, p.tiles_w, p.tiles_h, p.bw, p.bh, p.bn, x0, y0, i0);
          x0 = x0 * p.sx - p.px;
          y0 = y0 * p.sy - p.py;
        }
        for (int kb = 0; kb < k_blocks && ok; ++kb, ++it) {
          const int s = it % kStages;
          if (it >= kStages) ok = wait(empty(s), (it / kStages - 1) & 1, status, 61, &abort_flag);
          if (!ok) break;
          const uint32_t dst = base + s * kStage;
          mbar_expect_tx(full(s), (2 + boxes) * kBox);
          if (PIXELS) {
            load_4d(dst, &map_a, cb * 64, x0 + kx, y0 + ky, i0, full(s));
            if (++cb == c_blocks) {
              cb = 0;
              if (++kx == p.kw) {
                kx = 0;
                ++ky;
              }
            }
          }
          if constexpr (!PIXELS) for (int j = 0; j < 2; ++j) {
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
      if constexpr (PIXELS) {  // a thread has a pixel: runs of at least eight along a row, a plane apart from channel to channel
        constexpr int shift = KIND == kPhases ? 2 : 0;
        if (p.bias) {
#pragma unroll
          for (int c = 0; c < 128; c += 32)
            if (c < half) {
              const float bias = n_first + c + lane < p.N ? __ldg(p.bias + ((n_first + c + lane) >> shift)) : 0.f;
#pragma unroll
              for (int j = 0; j < 32; ++j) sum[c + j] += __shfl_sync(0xffffffffu, bias, j);
            }
        }
        const int q = quad * 32 + lane, z = q / p.bw;
        int x, y, im;
        box_origin(mt, p.tiles_w, p.tiles_h, p.bw, p.bh, p.bn, x, y, im);
        x += q % p.bw;
        y += z % p.bh;
        im += z / p.bh;
        if (x < p.rows_w && y < p.rows_h && im < p.rows_n) {
          const int64_t plane = (int64_t)p.out_h * p.out_w;
          float* out = p.c + ((int64_t)im * (p.N >> shift) + (n_first >> shift)) * plane + (int64_t)(y << (shift >> 1)) * p.out_w + (x << (shift >> 1));
          if constexpr (KIND == kPhases) {
            const bool right = 2 * x + 1 < p.out_w, below = 2 * y + 1 < p.out_h;
#pragma unroll
            for (int j = 0; j < 128; j += 4) {
              if (j >= half || n_first + j >= p.N) break;
              if (p.pairs) {
                *reinterpret_cast<float2*>(out) = make_float2(sum[j], sum[j + 1]);
                if (below) *reinterpret_cast<float2*>(out + p.out_w) = make_float2(sum[j + 2], sum[j + 3]);
              } else {
                out[0] = sum[j];
                if (right) out[1] = sum[j + 1];
                if (below) out[p.out_w] = sum[j + 2];
                if (right && below) out[p.out_w + 1] = sum[j + 3];
              }
              out += plane;
            }
          } else {
#pragma unroll
            for (int c = 0; c < 128; c += 32) {
              if (c >= half) break;
              if (n_first + c + 32 <= p.N) {
#pragma unroll
                for (int j = 0; j < 32; ++j, out += plane) *out = sum[c + j];
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j, out += plane)
                  if (n_first + c + j < p.N) *out = sum[c + j];
              }
            }
          }
        }
      } else {
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
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
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

template <int KIND>
rt_status launch(rt_ctx* ctx, const CUtensorMap& ma, const CUtensorMap& mb, const Params& p) {
  static RtDeviceOnce once;
  RT_CUDA(ctx, once([&] { return cudaFuncSetAttribute(parts_gemm_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem); }));
  rt_launch(ctx, parts_gemm_kernel<KIND>, p.items < ctx->sm_count ? p.items : ctx->sm_count, kThreads, kSmem, ma, mb, p, ctx->device_status);
  RT_LAUNCHED(ctx);
  return RT_OK;
}


}  // namespace parts
}  // namespace tc
