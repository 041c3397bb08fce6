// Large convolutions on the tensor cores with operands split into 16-bit parts (k_gemm_parts.cu).
//
// Images are split into channels-last parts: a pixel is a row of K-blocks of its channels, padded with zeros.  As the A operand of a
// forward-like product 128 pixels at one kernel tap are one TMA box (zeros outside the image, element strides for strided convolutions: no
// im2col buffer).  The gather of a stride of two (transposed convolution, input gradient) computes the 2 x 2 outputs that belong to an input
// pixel as four columns: each needs its own taps, the others' have weights of zero there.  That is 9 taps for 4 with a 4 x 4 kernel, but 256
// columns instead of 64, which cost half as much each, and whole sectors are written: 75 us for each of four launches before (with 23 of a
// 25 us tile spent on writing every other float).
// For a weight gradient the reduction runs over the pixels: 64 of them, one K-block of channels wide, are the same boxes read the other way
// round, in which the parts of a channel lie along the rows and columns of the product.  All pairs of parts are multiplied, lo * lo among
// them; the pass that adds the splits of the reduction picks the pairs.
#include "parts_common.cuh"

namespace tc {
namespace parts {

constexpr int kSplitPixels = 128;
struct ImageSplit {
  const float* p;
  uint16_t* out;
  float* sums;          // of a channel's pixels in a tile: [tile][C]; or null
  int C, HW, pitch;     // pitch: 16-bit values of a pixel
  int tiles;            // in all
  FastDiv d_tiles;      // of an image
};
// Rows n of the weights, K-block tap * c_blocks + channel block: element (n, c, ky, kx) at n * sn + c * sc + ky * sky + kx * skx + off.  With
// phases n is channel * 4 + 2 * ry + rx, and tap u of a phase is its own a = u + shift, 0 <= a < count, which is ky = first + 2 * (count - 1 - a).
struct TapSplit {
  const float* w;
  uint16_t* out;
  int64_t sn, sc, sky, skx, off, pitch;
  int N, C, kh, kw, phases;
  int shift_y[2], count_y[2], first_y[2], shift_x[2], count_x[2], first_x[2];
};
constexpr int kMaxImages = 2;
struct ConvSplitArgs {
  ImageSplit image[kMaxImages];
  TapSplit taps;        // w null: none
  int images, sample_blocks;
  uint32_t most_faint[kMaxSources];
  const uint2* samples;       // [source][block]; the weights, the last source, are looked at as a whole
  uint32_t* verdicts;         // [source][block] of conv_split_kernel<false>
  Decision* decision;
};
// Bound by memory: 4 bytes read and 4 written an element.  A block turns 32 channels x 128 pixels at a time through shared memory; what is
// looked at is 128 pixels of a channel, and all channels of a pixel.  AGAIN: into three parts, if the first pass has found that two will not do.
template <bool AGAIN>
__global__ void __launch_bounds__(256, 4) conv_split_kernel(const ConvSplitArgs a) {
  RT_PDL_ENTRY();
  __shared__ uint32_t red[2 * kMaxSources][8];
  __shared__ float tile[32][kSplitPixels + 1];
  constexpr int depth = AGAIN ? 16 : 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, weights = a.taps.w ? 1 : 0;
  Decision d{};
  Magnitudes of_weights;
  if (AGAIN) {
    d = decide(a.verdicts, a.images + weights, gridDim.x, a.most_faint, red);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.decision->wide = d.wide;
      a.decision->special = d.special;
    }
    if (!d.wide) return;
  } else {
    uint2 v[kMaxSources];
    over_samples(a.samples, a.images + weights, a.sample_blocks, red, v);
#pragma unroll
    for (int q = 0; q < kMaxSources; ++q) {
      d.exponent[q] = exponent_for(v[q].x);
      if (blockIdx.x == 0 && threadIdx.x == 0) a.decision->exponent[q] = d.exponent[q];
      if (q == a.images) {
        of_weights.most = v[q].x;
        of_weights.least = v[q].y;
      }
    }
  }
  for (int q = 0; q < a.images; ++q) {
    const ImageSplit& s = a.image[q];
    const int exponent = q == 0 ? d.exponent[0] : d.exponent[1];
    const float scale = AGAIN ? 1.f : ldexpf(1.f, exponent);
    const uint32_t faint = faint_below(exponent), faint_pixel = faint_below(exponent, kFaintPixelExponent);
    Magnitudes all;
    for (int i0 = blockIdx.x; i0 < s.tiles; i0 += gridDim.x) {
      uint32_t im, t;
      s.d_tiles.divmod((uint32_t)i0, im, t);
      const int p0 = (int)t * kSplitPixels, left = s.HW - p0;
      uint32_t pixel[2] = {};  // largest of this thread's channels of its two pixels
      for (int c0 = 0; c0 < s.C; c0 += 32) {
        const float* src = s.p + ((int64_t)im * s.C + c0) * s.HW + p0;
        float v[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // a warp has four channels
          const int c = warp * 4 + i;
#pragma unroll
          for (int j = 0; j < 4; ++j) v[i][j] = c0 + c < s.C && lane + 32 * j < left ? __ldcs(src + (int64_t)c * s.HW + lane + 32 * j) : 0.f;
        }
        __syncthreads();  // the tile before has been read
        uint32_t low = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = warp * 4 + i;
          uint32_t row = 0;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            tile[c][lane + 32 * j] = v[i][j];
            const uint32_t m = __float_as_uint(v[i][j]) & 0x7fffffffu;
            row = max(row, m);
            low = lower(low, m);
          }
          if (AGAIN) continue;
          row = __reduce_max_sync(0xffffffffu, row);
          all.most = max(all.most, row);
          if (row) all.least = min(all.least, row);
          if (s.sums) {
            float sum = (v[i][0] + v[i][1]) + (v[i][2] + v[i][3]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane == 0 && c0 + c < s.C) s.sums[(int64_t)i0 * s.C + c0 + c] = sum;
          }
        }
        all.faint += low < faint;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; ++i) {  // eight channels of a pixel
          const int item = i * 256 + threadIdx.x, px = item >> 2, c = (item & 3) * 8;
          float x[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            x[j] = tile[c + j][px];
            if (!AGAIN) pixel[i] = max(pixel[i], __float_as_uint(x[j]) & 0x7fffffffu);
          }
          // the K-blocks that hold channels are written to their end
          if (px < left && c0 + c < (s.C + depth - 1) / depth * depth) {
            uint4 part[4];
            split8(x, AGAIN, scale, part);
            uint16_t* o = s.out + ((int64_t)im * s.HW + p0 + px) * s.pitch + (c0 + c) / depth * 64 + (c0 + c) % depth;
            *reinterpret_cast<uint4*>(o) = part[0];
            *reinterpret_cast<uint4*>(o + depth) = part[1];
            if (AGAIN) {
              *reinterpret_cast<uint4*>(o + 2 * depth) = part[2];
              *reinterpret_cast<uint4*>(o + 3 * depth) = part[3];
            }
          }
        }
      }
      if (AGAIN) continue;
#pragma unroll
      for (int i = 0; i < 2; ++i) {  // four lanes have a pixel
        uint32_t m = pixel[i];
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
        if (m - 1 < faint_pixel) all.least = min(all.least, m);  // which is below what a segment's may be
      }
    }
    if (!AGAIN) {
      all = over_block(all, red);
      if (threadIdx.x == 0) a.verdicts[q * gridDim.x + blockIdx.x] = verdict(all, exponent);
    }
  }
  if (!weights) return;
  const TapSplit& s = a.taps;
  const int exponent = a.images == 0 ? d.exponent[0] : (a.images == 1 ? d.exponent[1] : d.exponent[2]);
  const float scale = AGAIN ? 1.f : ldexpf(1.f, exponent);
  const int eighths = (s.C + depth - 1) / depth * depth / 8, taps = s.kh * s.kw;
  const int64_t total = (int64_t)s.N * taps * eighths;
  const uint32_t faint = faint_below(exponent);
  // from the last block on, which has had the least to do
  for (int64_t i = (int64_t)(gridDim.x - 1 - blockIdx.x) * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
    const int c = (int)(i % eighths) * 8, tap = (int)(i / eighths % taps), n = (int)(i / eighths / taps);
    int ky = tap / s.kw, kx = tap % s.kw, row = n;
    bool there = true;
    if (s.phases) {
      const int ry = n >> 1 & 1, rx = n & 1, u = ky + s.shift_y[ry], v = kx + s.shift_x[rx];
      there = u >= 0 && u < s.count_y[ry] && v >= 0 && v < s.count_x[rx];
      ky = s.first_y[ry] + 2 * (s.count_y[ry] - 1 - u);
      kx = s.first_x[rx] + 2 * (s.count_x[rx] - 1 - v);
      row = n >> 2;
    }
    const float* w = s.w + row * s.sn + ky * s.sky + kx * s.skx + s.off;
    float x[8];
    uint32_t low = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      x[j] = there && c + j < s.C ? __ldg(w + (c + j) * s.sc) : 0.f;
      low = lower(low, __float_as_uint(x[j]) & 0x7fffffffu);
    }
    of_weights.faint += low < faint;
    uint4 part[4];
    split8(x, AGAIN, scale, part);
    uint16_t* o = s.out + n * s.pitch + ((int64_t)tap * (eighths * 8 / depth) + c / depth) * 64 + c % depth;
    *reinterpret_cast<uint4*>(o) = part[0];
    *reinterpret_cast<uint4*>(o + depth) = part[1];
    if (AGAIN) {
      *reinterpret_cast<uint4*>(o + 2 * depth) = part[2];
      *reinterpret_cast<uint4*>(o + 3 * depth) = part[3];
    }
  }
  if (!AGAIN) {
    of_weights = over_block(of_weights, red);
    if (threadIdx.x == 0) a.verdicts[a.images * gridDim.x + blockIdx.x] = verdict(of_weights, exponent);
  }
}

// ---- weight gradient ----------------------------------------------------------------------------------------------------------
struct GradParams {
  const Decision* decision;
  int Cy, Cx, taps, kw;
  int boxes, splits;                       // boxes of 64 pixels, spread over the splits
  int bw, bh, bn, tiles_w, tiles_h;
  int sx, sy, px, py;
  int chunk;                               // K-blocks between two emptyings of the accumulator
  float* partial;                          // [split][tile][column][row]
};
struct GradTiles {
  int c_rows, c_cols, m_tiles, n_tiles;    // K-blocks of the channels on either side; tiles of two and four of them
};
__host__ __device__ inline GradTiles grad_tiles(int Cy, int Cx, int taps, int wide) {
  GradTiles t;
  const int depth = wide ? 16 : 32;
  t.c_rows = (Cy + depth - 1) / depth;
  t.c_cols = (Cx + depth - 1) / depth;
  t.m_tiles = (t.c_rows + 1) / 2;
  t.n_tiles = (t.c_cols * taps + 3) / 4;
  return t;
}
constexpr uint32_t kGradBars = kStages * kStage;
constexpr uint32_t kGradSmem = kGradBars + (2 * kStages + 4) * 8 + 16 + 1024;

// An item is a tile of 128 rows (two K-blocks of Cy's parts) x up to 256 columns (four of a tap's Cx's) of one split of the pixels.  Bound by
// what crosses an SM's shared memory: 48 KB written and as much read for 512 cycles of MMAs.
__global__ void __launch_bounds__(kThreads, 1)
parts_grad_kernel(const __grid_constant__ CUtensorMap map_y, const __grid_constant__ CUtensorMap map_x, const GradParams p, int* status) {
  RT_PDL_ENTRY();
  extern __shared__ char smem_raw[];
  __shared__ volatile int abort_flag;
  const uint32_t raw_base = smem_u32(smem_raw);
  const uint32_t base = (raw_base + 1023) & ~1023u;
  char* smem = smem_raw + (base - raw_base);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t bars = base + kGradBars;
  auto full = [&](int i) { return bars + 8 * i; };
  auto empty = [&](int i) { return bars + 8 * (kStages + i); };
  auto acc_full = [&](int i) { return bars + 8 * (2 * kStages + i); };
  auto acc_empty = [&](int i) { return bars + 8 * (2 * kStages + 2 + i); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kGradBars + (2 * kStages + 4) * 8);
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full(i), 1);
      mbar_init(empty(i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(acc_full(i), 1);
      mbar_init(acc_empty(i), kEpilogueWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) tmem_alloc(smem_u32(tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const int wide = __shfl_sync(0xffffffffu, p.decision->wide, 0);
  const GradTiles g = grad_tiles(p.Cy, p.Cx, p.taps, wide);
  const int tiles = g.m_tiles * g.n_tiles, items = tiles * p.splits;
  auto range = [&](int split, int& begin, int& end) {
    begin = (int)((int64_t)p.boxes * split / p.splits);
    end = (int)((int64_t)p.boxes * (split + 1) / p.splits);
  };
  auto columns = [&](int nt) { return min(4, g.c_cols * p.taps - nt * 4); };  // boxes of B
  bool ok = true;

  if (warp == kTmaWarp) {
    if (lane == 0) {
      asm volatile("fence.proxy.async.global;" ::: "memory");  // the parts were written by ordinary stores
      int it = 0;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        const int tile = item % tiles, mt = tile % g.m_tiles, nt = tile / g.m_tiles, nb = columns(nt);
        int begin, end;
        range(item / tiles, begin, end);
        // where the columns' boxes lie beside the rows', and the boxes' positions counted up: one thread does all this, and a K-block's
        // MMAs take 512 cycles
        int dc[4], dx[4], dy[4], x, y, im;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int block = nt * 4 + j, tap = block / g.c_cols;
          dc[j] = block % g.c_cols * 64;
          dx[j] = tap % p.kw - p.px;
          dy[j] = tap / p.kw - p.py;
        }
        box_origin(begin, p.tiles_w, p.tiles_h, p.bw, p.bh, p.bn, x, y, im);
        const int end_x = p.tiles_w * p.bw, end_y = p.tiles_h * p.bh;
        for (int kb = begin; kb < end && ok; ++kb, ++it) {
          const int s = it % kStages;
          if (it >= kStages) ok = wait(empty(s), (it / kStages - 1) & 1, status, 71, &abort_flag);
          if (!ok) break;
          const uint32_t dst = base + s * kStage;
          mbar_expect_tx(full(s), (2 + nb) * kBox);
          for (int j = 0; j < 2; ++j) load_4d(dst + j * kBox, &map_y, (mt * 2 + j) * 64, x, y, im, full(s));  // zeros behind the last block
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < nb) load_4d(dst + (2 + j) * kBox, &map_x, dc[j], x * p.sx + dx[j], y * p.sy + dy[j], im, full(s));
          if ((x += p.bw) == end_x) {
            x = 0;
            if ((y += p.bh) == end_y) {
              y = 0;
              im += p.bn;
            }
          }
        }
      }
      if (!ok)
        for (int i = it > kStages ? it - kStages : 0; i < it; ++i) mbar_wait(full(i % kStages), (i / kStages) & 1, status, 72);
    }
  } else if (warp == kMmaWarp) {
    constexpr uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
    const uint32_t lbo = (kBox >> 4) << 16, format = wide ? 1u : 0u;
    const uint32_t idesc0 = (1u << 4) | format << 7 | format << 10 | 1u << 15 | 1u << 16 | (uint32_t)(BM >> 4) << 24;
    int it = 0, chunks = 0;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      const uint32_t idesc = idesc0 | (uint32_t)(columns(item % tiles / g.m_tiles) * 64 >> 3) << 17;
      int begin, end;
      range(item / tiles, begin, end);
      for (int kb = begin, in_chunk = 0; kb < end && ok; ++kb, ++it) {
        const int s = it % kStages, acc = chunks & 1;
        const bool first = in_chunk == 0, last = ++in_chunk == p.chunk || kb + 1 == end;
        if (last) in_chunk = 0;
        ok = wait(full(s), (it / kStages) & 1, status, 73, &abort_flag);
        if (ok && first && chunks >= 2) ok = wait(acc_empty(acc), (chunks / 2 - 1) & 1, status, 74, &abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a = ((base + s * kStage) >> 4 & 0x3FFF) | lbo, b = ((base + s * kStage + 2 * kBox) >> 4 & 0x3FFF) | lbo;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          mma(tmem + acc * 256, a + j * (2048 >> 4), desc_hi, b + j * (2048 >> 4), desc_hi, idesc, j > 0 || !first);
        umma_commit_elect(empty(s));
        if (last) {
          umma_commit_elect(acc_full(acc));
          ++chunks;
        }
      }
    }
  } else {
    const int quad = warp & 3, group = warp >> 2;
    int done = 0;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      const int half = columns(item % tiles / g.m_tiles) * 32;
      int begin, end;
      range(item / tiles, begin, end);
      float sum[128];
#pragma unroll
      for (int j = 0; j < 128; ++j) sum[j] = 0.f;
      for (int kb = begin; kb < end && ok; kb += p.chunk, ++done) {
        const int acc = done & 1;
        ok = __all_sync(0xffffffffu, wait(acc_full(acc), (done / 2) & 1, status, 75, &abort_flag));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem + acc * 256 + ((uint32_t)(quad * 32) << 16) + group * half;
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
        if (lane == 0) mbar_arrive(acc_empty(acc));
      }
      if (!ok) break;
      float* out = p.partial + ((int64_t)item * 256 + group * half) * BM + quad * 32 + lane;
#pragma unroll
      for (int j = 0; j < 128; ++j)
        if (j < half) out[(int64_t)j * BM] = sum[j];
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// dw[cy][cx][tap] = sum over the splits and the pairs of parts; db[c] = sum over the tiles of the upstream gradient's image.
// A warp has a column's 32 rows of a channel block at a time: coalesced reads.  Fixed order.
// Where a box overhangs the image y there are zeros, which x is multiplied with all the same: an infinity among it makes NaN.  With infinities or
// NaN in the images an element that came out NaN is therefore computed once more from the images themselves.
struct GradFinish {
  const Decision* decision;
  const float* partial;
  float* dw;
  int Cy, Cx, taps, splits, source_y, source_x;
  const float* sums;
  float* db;
  int sum_tiles, sum_C;
  const float *x, *y;
  int Nb, Hx, Wx, Hy, Wy, kw, sx, sy, px, py;
};
__device__ __noinline__ float grad_from_images(const GradFinish& p, int cy, int cx, int tap) {
  const int lane = threadIdx.x & 31, ky = tap / p.kw, kx = tap % p.kw, pixels = p.Nb * p.Hy * p.Wy;
  double sum = 0;
  for (int i = lane; i < pixels; i += 32) {
    const int xo = i % p.Wy, yo = i / p.Wy % p.Hy, n = i / p.Wy / p.Hy, v = yo * p.sy - p.py + ky, u = xo * p.sx - p.px + kx;
    const bool in = v >= 0 && v < p.Hx && u >= 0 && u < p.Wx;
    sum += (double)__ldg(p.y + (((int64_t)n * p.Cy + cy) * p.Hy + yo) * p.Wy + xo) * (in ? __ldg(p.x + (((int64_t)n * p.Cx + cx) * p.Hx + v) * p.Wx + u) : 0.f);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return (float)sum;
}
__global__ void __launch_bounds__(256) parts_grad_finish_kernel(const __grid_constant__ GradFinish p) {
  RT_PDL_ENTRY();
  const int wide = p.decision->wide, special = p.decision->special, depth = wide ? 16 : 32;
  const GradTiles g = grad_tiles(p.Cy, p.Cx, p.taps, wide);
  const int tiles = g.m_tiles * g.n_tiles, lane = threadIdx.x & 31;
  const int exponent = wide ? 0 : -(p.decision->exponent[p.source_y] + p.decision->exponent[p.source_x]);
  const float f1 = ldexpf(1.f, exponent / 2), f2 = ldexpf(1.f, exponent - exponent / 2);
  const int64_t cy_padded = (int64_t)g.c_rows * depth;
  const int64_t total = cy_padded * p.Cx * p.taps;
  for (int64_t first = (int64_t)blockIdx.x * 256 + (threadIdx.x & ~31u); first < total; first += (int64_t)gridDim.x * 256) {
    const int64_t i = first + lane;
    const int cy = (int)(i % cy_padded), rest = (int)(i / cy_padded), cx = rest % p.Cx, tap = rest / p.Cx;
    float v = 0.f;
    if (i < total && cy < p.Cy) {
      const int rb = cy / depth, column_block = tap * g.c_cols + cx / depth;
      const int tile = rb / 2 + column_block / 4 * g.m_tiles;
      const int row = rb % 2 * 64 + cy % depth, col = column_block % 4 * 64 + cx % depth;
      const float* q = p.partial + ((int64_t)tile * 256 + col) * BM + row;
      auto at = [&](const float* t, int part_y, int part_x) { return __ldcs(t + (int64_t)part_x * depth * BM + part_y * depth); };
      float main = 0.f, cross = 0.f;
#pragma unroll 4
      for (int s = 0; s < p.splits; ++s) {
        const float* t = q + (int64_t)s * tiles * 256 * BM;
        main += at(t, 0, 0);
        if (wide) cross += (at(t, 3, 1) + at(t, 1, 3)) + (at(t, 1, 1) + (at(t, 3, 2) + at(t, 2, 3)));
        else cross += (at(t, 0, 1) + at(t, 1, 0)) + at(t, 1, 1) * (1.f / 2048.f);
      }
      v = (main + cross * (wide ? 1.f : 1.f / 2048.f)) * f1 * f2;
    }
    if (special)
      for (unsigned bad = __ballot_sync(0xffffffffu, v != v); bad; bad &= bad - 1) {
        const int of = __ffs((int)bad) - 1;
        const float again = grad_from_images(p, __shfl_sync(0xffffffffu, cy, of), __shfl_sync(0xffffffffu, cx, of), __shfl_sync(0xffffffffu, tap, of));
        if (lane == of) v = again;
      }
    if (i < total && cy < p.Cy) p.dw[((int64_t)cy * p.Cx + cx) * p.taps + tap] = v;
  }
  if (!p.db) return;
  __shared__ float red[8];
  const int warp = threadIdx.x >> 5;
  for (int c = blockIdx.x; c < p.sum_C; c += gridDim.x) {
    float v = 0.f;
#pragma unroll 4
    for (int t = threadIdx.x; t < p.sum_tiles; t += 256) v += __ldg(p.sums + (int64_t)t * p.sum_C + c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w) v += red[w];
      p.db[c] = v;
    }
    __syncthreads();
  }
}

// The columns of the phases have weights of zero at the taps that are not theirs, which an infinity or NaN makes NaN of: with such in the images or
// weights an output that came out NaN is computed once more from its own taps.  Otherwise over at once.
struct Repair {
  const Decision* decision;
  const float *y, *w, *bias;
  float* out;
  int64_t total;
  int Cm, Cy, Hy, Wy, Hx, Wx, kh, kw, sh, sw, ph, pw;
};
__global__ void __launch_bounds__(256) repair_gather_kernel(const Repair p) {
  RT_PDL_ENTRY();
  if (!p.decision->special) return;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < p.total; i += (int64_t)gridDim.x * 256) {
    if (p.out[i] == p.out[i]) continue;
    const int u = (int)(i % p.Wx), v = (int)(i / p.Wx % p.Hx), c = (int)(i / p.Wx / p.Hx % p.Cm);
    const float* y = p.y + i / p.Wx / p.Hx / p.Cm * p.Cy * p.Hy * p.Wy;
    double sum = p.bias ? __ldg(p.bias + c) : 0.f;
    for (int ky = 0; ky < p.kh; ++ky) {
      const int yo = (v + p.ph - ky) / p.sh;
      if (v + p.ph < ky || (v + p.ph - ky) % p.sh || yo >= p.Hy) continue;
      for (int kx = 0; kx < p.kw; ++kx) {
        const int xo = (u + p.pw - kx) / p.sw;
        if (u + p.pw < kx || (u + p.pw - kx) % p.sw || xo >= p.Wy) continue;
        for (int k = 0; k < p.Cy; ++k)
          sum += (double)__ldg(y + ((int64_t)k * p.Hy + yo) * p.Wy + xo) * __ldg(p.w + (((int64_t)k * p.Cm + c) * p.kh + ky) * p.kw + kx);
      }
    }
    p.out[i] = (float)sum;
  }
}

// ---- host ---------------------------------------------------------------------------------------------------------------------
// An image [Nb][C][H][W] and its parts.
struct Image {
  const float* p;
  int Nb, C, H, W, source;
  bool sums;
  RtScratch mem, sum_mem;
  Image(rt_ctx* ctx, int src, const float* q, int n, int c, int h, int w, bool want_sums = false)
      : p(q), Nb(n), C(c), H(h), W(w), source(src), sums(want_sums), mem(ctx), sum_mem(ctx) {}
  int pitch() const { return (C + 15) / 16 * 64; }
  int tiles() const { return (H * W + kSplitPixels - 1) / kSplitPixels; }
  rt_status alloc() {
    rt_status st = mem.alloc(sizeof(uint16_t) * (size_t)Nb * H * W * pitch());
    if (st == RT_OK && sums) st = sum_mem.alloc(sizeof(float) * (size_t)Nb * tiles() * C);
    return st;
  }
  // Boxes of bw x bh x bn pixels, sx and sy apart, one K-block deep.
  bool map(CUtensorMap* m, int bw, int bh, int bn, int sx, int sy) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t row = (cuuint64_t)pitch() * 2;
    const cuuint64_t dims[4] = {(cuuint64_t)pitch(), (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)Nb};
    const cuuint64_t strides[3] = {row, W * row, (cuuint64_t)H * W * row};
    const cuuint32_t box[4] = {64, (cuuint32_t)((bw - 1) * sx + 1), (cuuint32_t)((bh - 1) * sy + 1), (cuuint32_t)bn};
    const cuuint32_t step[4] = {1, (cuuint32_t)sx, (cuuint32_t)sy, 1};
    if (box[1] > 256 || box[2] > 256) return false;
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 4, mem.ptr, dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
};
struct Taps {
  TapSplit t{};
  const float* all = nullptr;  // the whole weight tensor
  int64_t all_rows = 0, all_cols = 0;
  RtScratch mem;
  explicit Taps(rt_ctx* ctx) : mem(ctx) {}
  rt_status alloc() {
    t.pitch = (int64_t)t.kh * t.kw * ((t.C + 15) / 16) * 64;
    rt_status st = mem.alloc(sizeof(uint16_t) * (size_t)(t.N * t.pitch));
    t.out = mem.as<uint16_t>();
    return st;
  }
};
// The box of `pixels` (a power of two) that wastes least at the edges; runs of fewer than eight along a row make scattered accesses.
inline void choose_box(int pixels, int w, int h, int n, int* bw, int* bh, int* bn) {
  double best = -1;
  for (int a = 1; a <= pixels; a *= 2)
    for (int b = 1; a * b <= pixels; b *= 2) {
      const int c = pixels / (a * b);
      auto used = [](int extent, int box) { return (double)extent / ((extent + box - 1) / box * box); };
      const double score = used(w, a) * used(h, b) * used(n, c) * (a >= 8 ? 1.0 : (a == 4 ? 0.9 : (a == 2 ? 0.7 : 0.5)));
      if (score > best + 1e-9) {
        best = score;
        *bw = a;
        *bh = b;
        *bn = c;
      }
    }
}
// Parts of images and weights (taps null: none).
inline rt_status split_conv(rt_ctx* ctx, Image* const* images, int n_images, Taps* taps, RtScratch* work, Decision** decision) {
  const int sample_blocks = ctx->sm_count, blocks = 4 * ctx->sm_count;
  rt_status st = work->alloc((sizeof(uint2) * (size_t)sample_blocks + sizeof(uint32_t) * (size_t)blocks) * kMaxSources + sizeof(Decision));
  if (st != RT_OK) return st;
  SampleArgs a{};
  ConvSplitArgs b{};
  uint2* samples = work->as<uint2>();
  a.count = n_images + (taps ? 1 : 0);
  b.sample_blocks = sample_blocks;
  b.samples = samples;
  b.verdicts = reinterpret_cast<uint32_t*>(samples + (size_t)sample_blocks * kMaxSources);
  *decision = b.decision = reinterpret_cast<Decision*>(b.verdicts + (size_t)blocks * kMaxSources);
  b.images = n_images;
  for (int q = 0; q < n_images; ++q) {
    Image& im = *images[q];
    if ((st = im.alloc()) != RT_OK) return st;
    const int64_t hw = (int64_t)im.H * im.W;
    a.s[q] = sample_of(ctx, im.p, hw, (int64_t)im.Nb * im.C, hw, false);
    b.most_faint[q] = most_faint((int64_t)im.Nb * im.C * hw);
    ImageSplit& s = b.image[q];
    s.p = im.p;
    s.out = im.mem.as<uint16_t>();
    s.sums = im.sums ? im.sum_mem.as<float>() : nullptr;
    s.C = im.C;
    s.HW = im.H * im.W;
    s.pitch = im.pitch();
    s.tiles = im.Nb * im.tiles();
    s.d_tiles.init((uint32_t)im.tiles());
  }
  if (taps) {
    if ((st = taps->alloc()) != RT_OK) return st;
    b.taps = taps->t;
    a.s[n_images] = sample_of(ctx, taps->all, taps->all_cols, taps->all_rows, taps->all_cols, true);
    b.most_faint[n_images] = most_faint(taps->all_rows * taps->all_cols);
  }
  rt_launch(ctx, sample_kernel, sample_blocks, 256, 0, a, samples);
  RT_LAUNCHED(ctx);
  rt_launch(ctx, conv_split_kernel<false>, blocks, 256, 0, b);
  RT_LAUNCHED(ctx);
  rt_launch(ctx, conv_split_kernel<true>, blocks, 256, 0, b);
  RT_LAUNCHED(ctx);
  return RT_OK;
}
// out(n, co, y, x) (+ bias) = sum over taps and channels of src(n, c, y * sy - py + ky, x * sx - px + kx) * w(co, c, ky, kx); with phases y and x
// are those of 2 x 2 outputs.
inline rt_status pixel_product(rt_ctx* ctx, Image& src, Taps& w, int source_w, const Decision* decision, int rows_h, int rows_w, int sy, int sx, int py, int px,
                               const float* bias, float* out, int out_h, int out_w) {
  Params p{};
  choose_box(BM, rows_w, rows_h, src.Nb, &p.bw, &p.bh, &p.bn);
  CUtensorMap ma, mb;
  if (!src.map(&ma, p.bw, p.bh, p.bn, sx, sy) || !map_parts(&mb, w.t.out, w.t.pitch, w.t.N, w.t.pitch)) return RT_ERR_UNIMPLEMENTED;
  p.decision = decision;
  p.source_a = src.source;
  p.source_b = source_w;
  p.N = w.t.N;
  p.C = src.C;
  p.taps = w.t.kh * w.t.kw;
  p.kw = w.t.kw;
  p.K = src.C * p.taps;
  p.chunk = p.K < 512 ? 6 : (p.K < 1024 ? 8 : 16);
  p.tiles_w = (rows_w + p.bw - 1) / p.bw;
  p.tiles_h = (rows_h + p.bh - 1) / p.bh;
  p.rows_w = rows_w; p.rows_h = rows_h; p.rows_n = src.Nb;
  p.m_tiles = p.tiles_w * p.tiles_h * ((src.Nb + p.bn - 1) / p.bn);
  choose_tiles(ctx, &p);
  p.sx = sx; p.sy = sy; p.px = px; p.py = py;
  p.out_h = out_h; p.out_w = out_w;
  p.pairs = out_w % 2 == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
  p.c = out;
  p.bias = bias;
  return w.t.phases ? launch<kPhases>(ctx, ma, mb, p) : launch<kPixels>(ctx, ma, mb, p);
}
// Which convolutions: so many multiply-adds, boxes that TMA steps over, indices of 32 bits.  Tiles of 64 columns pay later (64 x 64 x 28 x 28 to
// 64, 1.85 G: 47 us, as 3xTF32 44), the strided gather, whose phases are one launch instead of four, much earlier (40 x 128 x 14 x 14 to 64, 1.03
// G: 149 us as four).
inline int64_t least_work(int N, bool phases) { return int64_t(1) << (phases ? 28 : (N > 64 ? 30 : 31)); }
inline bool conv_worth_it(int64_t work, int64_t least, int C, int N, int sy, int sx, int64_t image_rows, int64_t hw) {
  return work >= least && C >= 16 && N >= 16 && sy <= 8 && sx <= 8 && hw < (1 << 24) && image_rows < (1 << 24) &&
         image_rows * ((hw + kSplitPixels - 1) / kSplitPixels) < (int64_t(1) << 30);
}
// The weights w[Cy,Cx,kh,kw] as a convolution has them.
inline Taps* forward_taps(Taps* t, const float* w, const ConvGeom& g) {
  const int64_t taps = (int64_t)g.kh * g.kw;
  t->t = {w, nullptr, g.Cx * taps, taps, g.kw, 1, 0, 0, g.Cy, g.Cx, g.kh, g.kw, 0};
  t->all = w;
  t->all_rows = g.Cy;
  t->all_cols = g.Cx * taps;
  return t;
}
// The two phases of one dimension: output 2 * y + r meets the taps k = first + 2 * a; in terms of y they are a unit-stride convolution with
// `count` taps turned round, of which the first is `pad` before y.
inline void phases_of(int k, int pad, int* shift, int* count, int* first, int* taps, int* lead) {
  int p[2];
  for (int r = 0; r < 2; ++r) {
    first[r] = (r + pad) % 2;
    count[r] = (k - first[r] + 1) / 2;
    p[r] = count[r] - 1 - (r + pad - first[r]) / 2;
  }
  *lead = p[0] > p[1] ? p[0] : p[1];
  int after = INT_MIN;
  for (int r = 0; r < 2; ++r) {
    shift[r] = p[r] - *lead;
    if (count[r] - p[r] > after) after = count[r] - p[r];
  }
  *taps = *lead + after;
}
// What a gather of y[Nb,Cy,Hy,Wy] with w[Cy,Cm,kh,kw] needs: the weights turned round, and where the first tap lies.
struct Gather {
  Taps taps;
  int rows_h, rows_w, py, px;
  explicit Gather(rt_ctx* ctx) : taps(ctx) {}
  bool set(const float* w, const ConvGeom& g, int cm) {
    const int64_t all = (int64_t)g.kh * g.kw;
    taps.all = w;
    taps.all_rows = g.Cy;
    taps.all_cols = cm * all;
    if (g.sh == 1 && g.sw == 1) {
      taps.t = {w, nullptr, all, cm * all, -(int64_t)g.kw, -1, all - 1, 0, cm, g.Cy, g.kh, g.kw, 0};
      rows_h = g.Hx;
      rows_w = g.Wx;
      py = g.kh - 1 - g.ph;
      px = g.kw - 1 - g.pw;
      return true;
    }
    if (g.sh != 2 || g.sw != 2 || g.kh < 2 || g.kw < 2) return false;  // every output has a tap
    taps.t = {w, nullptr, all, cm * all, g.kw, 1, 0, 0, 4 * cm, g.Cy, 0, 0, 1};
    TapSplit& t = taps.t;
    phases_of(g.kh, g.ph, t.shift_y, t.count_y, t.first_y, &t.kh, &py);
    phases_of(g.kw, g.pw, t.shift_x, t.count_x, t.first_x, &t.kw, &px);
    rows_h = (g.Hx + 1) / 2;
    rows_w = (g.Wx + 1) / 2;
    return true;
  }
  rt_status run(rt_ctx* ctx, Image& y, int source_w, const Decision* decision, const ConvGeom& g, int cm, const float* bias, float* out) {
    rt_status st = pixel_product(ctx, y, taps, source_w, decision, rows_h, rows_w, 1, 1, py, px, bias, out, g.Hx, g.Wx);
    if (st != RT_OK || !taps.t.phases) return st;
    const Repair r{decision, y.p, taps.all, bias, out, (int64_t)g.Nb * cm * g.Hx * g.Wx, cm, g.Cy, g.Hy, g.Wy, g.Hx, g.Wx, g.kh, g.kw, g.sh, g.sw, g.ph, g.pw};
    rt_launch(ctx, repair_gather_kernel, 4 * ctx->sm_count, 256, 0, r);
    RT_LAUNCHED(ctx);
    return RT_OK;
  }
};
inline bool gather_worth_it(const ConvGeom& g, int cm) {
  return conv_worth_it((int64_t)g.Nb * g.Hy * g.Wy * g.Cy * cm * g.kh * g.kw, least_work(cm, g.sh == 2 && g.sw == 2), g.Cy, cm, 1, 1, (int64_t)g.Nb * g.Cy, (int64_t)g.Hy * g.Wy) &&
         (int64_t)g.Nb * g.Hx * g.Wx < (1ll << 31);
}
inline bool grad_worth_it(const ConvGeom& g) {
  return conv_worth_it((int64_t)g.Nb * g.Hy * g.Wy * g.Cy * g.Cx * g.kh * g.kw, 0, g.Cx, g.Cy, g.sh, g.sw, (int64_t)g.Nb * g.Cx, (int64_t)g.Hx * g.Wx) &&
         (int64_t)g.Nb * g.Cy < (1 << 24) && (int64_t)g.Nb * g.Hy * g.Wy < (1ll << 31) && (int64_t)g.Cx * g.Cy * g.kh * g.kw < (1ll << 28);
}
// dw[Cy,Cx,kh,kw] from the parts of both images, and db (or null): the channel sums of one of them.
inline rt_status weight_grad(rt_ctx* ctx, Image& x, Image& y, const Decision* decision, const ConvGeom& g, float* dw, float* db, const Image& of) {
  GradParams p{};
  p.decision = decision;
  p.Cy = g.Cy; p.Cx = g.Cx; p.taps = g.kh * g.kw; p.kw = g.kw;
  choose_box(64, g.Wy, g.Hy, g.Nb, &p.bw, &p.bh, &p.bn);
  p.tiles_w = (g.Wy + p.bw - 1) / p.bw;
  p.tiles_h = (g.Hy + p.bh - 1) / p.bh;
  p.boxes = p.tiles_w * p.tiles_h * ((g.Nb + p.bn - 1) / p.bn);
  p.sx = g.sw; p.sy = g.sh; p.px = g.pw; p.py = g.ph;
  p.chunk = 8;  // 32 additions with truncation
  CUtensorMap my, mx;
  if (!y.map(&my, p.bw, p.bh, p.bn, 1, 1) || !x.map(&mx, p.bw, p.bh, p.bn, g.sw, g.sh)) return RT_ERR_UNIMPLEMENTED;
  const GradTiles t = grad_tiles(p.Cy, p.Cx, p.taps, 0), w = grad_tiles(p.Cy, p.Cx, p.taps, 1);
  const int tiles = t.m_tiles * t.n_tiles;
  // as many splits as give every SM an item; of at least eight K-blocks
  p.splits = tiles >= ctx->sm_count ? 1 : ctx->sm_count / tiles;
  if (p.splits > (p.boxes + 7) / 8) p.splits = (p.boxes + 7) / 8;
  RtScratch partial(ctx);
  rt_status st = partial.alloc(sizeof(float) * (size_t)p.splits * w.m_tiles * w.n_tiles * 256 * BM);
  if (st != RT_OK) return st;
  p.partial = partial.as<float>();
  static RtDeviceOnce once;
  RT_CUDA(ctx, once([&] { return cudaFuncSetAttribute(parts_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGradSmem); }));
  rt_launch(ctx, parts_grad_kernel, ctx->sm_count, kThreads, kGradSmem, my, mx, p, ctx->device_status);
  RT_LAUNCHED(ctx);
  GradFinish f{decision, p.partial, dw, p.Cy, p.Cx, p.taps, p.splits, y.source, x.source, static_cast<const float*>(of.sum_mem.ptr), db, of.Nb * of.tiles(),
               of.C, x.p, y.p, g.Nb, g.Hx, g.Wx, g.Hy, g.Wy, g.kw, g.sw, g.sh, g.pw, g.ph};
  rt_launch(ctx, parts_grad_finish_kernel, rt_grid_for(ctx, (int64_t)t.c_rows * 32 * p.Cx * p.taps, 256), 256, 0, f);
  RT_LAUNCHED(ctx);
  return RT_OK;
}
inline rt_status or_another_kernel(rt_status st) { return st == RT_ERR_OOM ? RT_ERR_UNIMPLEMENTED : st; }

}  // namespace parts
}  // namespace tc

// RT_ERR_UNIMPLEMENTED: not a convolution for these kernels, or no room for the parts.
// y[Nb,Cy,Hy,Wy] = conv(x, w[Cy,Cx,kh,kw]) (+ bias).
rt_status rt_conv_forward_parts_internal(rt_ctx* ctx, const float* x, const float* w, const float* bias, const ConvGeom& g, float* y) {
  using namespace tc::parts;
  const int64_t pixels = (int64_t)g.Nb * g.Hy * g.Wy;
  if (!conv_worth_it(pixels * g.Cy * g.Cx * g.kh * g.kw, least_work(g.Cy, false), g.Cx, g.Cy, g.sh, g.sw, (int64_t)g.Nb * g.Cx, (int64_t)g.Hx * g.Wx) ||
      pixels >= (1ll << 31))
    return RT_ERR_UNIMPLEMENTED;
  Image src(ctx, 0, x, g.Nb, g.Cx, g.Hx, g.Wx);
  Image* images[1] = {&src};
  Taps t(ctx);
  RtScratch work(ctx);
  Decision* decision;
  rt_status st = split_conv(ctx, images, 1, forward_taps(&t, w, g), &work, &decision);
  if (st == RT_OK) st = pixel_product(ctx, src, t, 1, decision, g.Hy, g.Wy, g.sh, g.sw, g.ph, g.pw, bias, y, g.Hy, g.Wy);
  return or_another_kernel(st);
}
// out[Nb,Cm,Hx,Wx] (+ bias) = gather of y[Nb,Cy,Hy,Wy] with w[Cy,Cm,kh,kw]: input gradient of a convolution, forward of a transposed one.
rt_status rt_conv_gather_parts_internal(rt_ctx* ctx, const float* y, const float* w, const float* bias, const ConvGeom& g, int cm, float* out) {
  using namespace tc::parts;
  Gather gather(ctx);
  if (!gather_worth_it(g, cm) || !gather.set(w, g, cm)) return RT_ERR_UNIMPLEMENTED;
  Image src(ctx, 0, y, g.Nb, g.Cy, g.Hy, g.Wy);
  Image* images[1] = {&src};
  RtScratch work(ctx);
  Decision* decision;
  rt_status st = split_conv(ctx, images, 1, &gather.taps, &work, &decision);
  if (st == RT_OK) st = gather.run(ctx, src, 1, decision, g, cm, bias, out);
  return or_another_kernel(st);
}
// dw[Cy,Cx,kh,kw] = sum over images and pixels of y * (x at the tap); db[Cy] = sum of y.
rt_status rt_conv_weight_grad_parts_internal(rt_ctx* ctx, const float* x, const float* y, const ConvGeom& g, float* dw, float* db) {
  using namespace tc::parts;
  if (!grad_worth_it(g)) return RT_ERR_UNIMPLEMENTED;
  Image ix(ctx, 0, x, g.Nb, g.Cx, g.Hx, g.Wx), iy(ctx, 1, y, g.Nb, g.Cy, g.Hy, g.Wy, db != nullptr);
  Image* images[2] = {&ix, &iy};
  RtScratch work(ctx);
  Decision* decision;
  rt_status st = split_conv(ctx, images, 2, nullptr, &work, &decision);
  if (st == RT_OK) st = weight_grad(ctx, ix, iy, decision, g, dw, db, iy);
  return or_another_kernel(st);
}
// dx[Nb,Cx,Hx,Wx], dw[Cy,Cx,kh,kw] and db[Cy] (or null) of a convolution from its upstream gradient y, which is split once for all.
rt_status rt_conv_backward_parts_internal(rt_ctx* ctx, const float* x, const float* w, const float* y, const ConvGeom& g, float* dx, float* dw, float* db) {
  using namespace tc::parts;
  Gather gather(ctx);
  if (!grad_worth_it(g) || !gather_worth_it(g, g.Cx) || !gather.set(w, g, g.Cx)) return RT_ERR_UNIMPLEMENTED;
  Image ix(ctx, 0, x, g.Nb, g.Cx, g.Hx, g.Wx), iy(ctx, 1, y, g.Nb, g.Cy, g.Hy, g.Wy, db != nullptr);
  Image* images[2] = {&ix, &iy};
  RtScratch work(ctx);
  Decision* decision;
  rt_status st = split_conv(ctx, images, 2, &gather.taps, &work, &decision);
  if (st == RT_OK) st = weight_grad(ctx, ix, iy, decision, g, dw, db, iy);
  if (st == RT_OK) st = gather.run(ctx, iy, 2, decision, g, g.Cx, nullptr, dx);
  return or_another_kernel(st);
}
// The same of a transposed convolution: y is its input, x (the wide side) the upstream gradient, whose channel sums db is.
rt_status rt_conv_transpose_backward_parts_internal(rt_ctx* ctx, const float* x, const float* w, const float* y, const ConvGeom& g, float* dy, float* dw,
                                                    float* db) {
  using namespace tc::parts;
  if (!grad_worth_it(g)) return RT_ERR_UNIMPLEMENTED;
  Image ix(ctx, 0, x, g.Nb, g.Cx, g.Hx, g.Wx, db != nullptr), iy(ctx, 1, y, g.Nb, g.Cy, g.Hy, g.Wy);
  Image* images[2] = {&ix, &iy};
  Taps t(ctx);
  RtScratch work(ctx);
  Decision* decision;
  rt_status st = split_conv(ctx, images, 2, forward_taps(&t, w, g), &work, &decision);
  if (st == RT_OK) st = weight_grad(ctx, ix, iy, decision, g, dw, db, ix);
  if (st == RT_OK) st = pixel_product(ctx, ix, t, 2, decision, g.Hy, g.Wy, g.sh, g.sw, g.ph, g.pw, nullptr, dy, g.Hy, g.Wy);
  return or_another_kernel(st);
}
