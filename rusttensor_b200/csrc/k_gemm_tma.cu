// Products of more than one wave of small tiles and convolutions on the tensor cores (tcgen05 3xTF32), operands fetched by TMA; the largest of
// either go to k_gemm_parts.cu and k_conv_parts.cu.
//
// What bounds a 3xTF32 product is the 128 B/cycle shared-memory path, not the tensor pipe: an fp32 operand element is 4 bytes as
// TMA brings it, and every copy, split and operand read of an MMA crosses that path.  This kernel therefore
//  * feeds the raw fp32 tile to the MMA as the hi operand - the tensor core ignores the low 13 mantissa bits of a TF32 operand,
//    which is the truncation hi = a & 0xffffe000 - so that only lo = a - hi has to be made;
//  * keeps the A operand (hi and lo) in tensor memory, from which an MMA reads at no cost to shared memory.
// The tensor core adds every partial product into its fp32 accumulator with truncation: on one accumulator over the whole reduction
// the error grows to 2.9e-5 of the result at 4096.  An accumulator is therefore emptied after every K-block of 32, or every
// few, and these are summed in registers with rounding (error 3.5e-7 - 1e-6 whatever the length); accumulators are used in turn, so
// that the MMAs do not wait for it.
// Roles of a CTA (one per SM, walking over tiles): one TMA warp several K-blocks ahead; six converter warps (A raw -> tensor
// memory hi / lo; B raw -> B lo at the same swizzled address, so the swizzle needs no decoding), four of them at work where B comes
// already split; one MMA warp; eight accumulating warps, which also write the result.
// Measured: 1024^3 31 us.  Without the conversions (in a copy made for timing) the MMAs and copies of a large product take two thirds of its
// time: shared memory is what is full.
// A operand: a matrix with the reduction contiguous, one with the rows contiguous, or the pixels of a channels-last image at one
// kernel tap (4-D boxes, zeros outside the image, element strides for strided convolutions: no im2col buffer).  B operand: a
// matrix with the reduction contiguous.  Whatever is not in such a form or not 16-byte aligned is brought into it by one pass of
// pack_kernel beforehand.
// Every wait is bounded; on expiry the kernel records a code in the status word, raises a flag that all other waits poll, lets its
// own copies land, frees tensor memory and returns.
#include "conv_geom.cuh"
#include "rt_internal.cuh"
#include "tc_common.cuh"
#include "tensor_map.cuh"

namespace tc {
namespace tma {

constexpr int BM = 128, BK = 32;
constexpr int kEpilogueWarps = 8, kConverterWarps = 6;
constexpr int kThreads = (kEpilogueWarps + kConverterWarps + 2) * 32;  // 512: 128 registers a thread, which 128 sums just fit
constexpr int kTmaWarp = kEpilogueWarps + kConverterWarps, kMmaWarp = kTmaWarp + 1;
constexpr uint32_t kARaw = BM * BK * 4;  // 16 KB

// SPLIT: B comes as two matrices, hi and lo (the packed weights of a convolution, used by every tile).
template <int BN, bool SPLIT>
struct Config {
  static_assert(BN <= 128, "columns of one MMA and of one accumulator");
  // The two groups of accumulating warps: each takes half the columns; or they take turns, a tile each, so that one writes a
  // result while the other sums the next tile (convolutions: short reductions, scattered stores).
  static constexpr bool turns = SPLIT;
  static constexpr int NC = turns ? BN : BN / 2;
  static constexpr int ACC = 2;                   // accumulators, used in turn
  static constexpr int L = 4;                     // converted A (tensor memory) and B lo
  static constexpr uint32_t b_raw = BN * BK * 4;
  static constexpr uint32_t raw = kARaw + (SPLIT ? 2 : 1) * b_raw;
  static constexpr int R = BN == 64 && SPLIT ? 6 : 4;  // raw tiles in flight
  static constexpr uint32_t lo_offset = R * raw;
  static constexpr uint32_t stage_offset = lo_offset + (SPLIT ? 0 : L * b_raw);  // result: one 32 x 17 tile per accumulating warp
  static constexpr uint32_t bar_offset = stage_offset + kEpilogueWarps * 32 * 17 * 4;
  static constexpr int n_bars = 2 * R + 2 * L + 3 * ACC;
  static constexpr uint32_t total = bar_offset + n_bars * 8 + 16 + 1024;  // + alignment of the base to 1024
  static constexpr uint32_t a_cols = 2 * BK;                              // tensor-memory columns of a converted A block
  static constexpr int converters = SPLIT ? 4 : kConverterWarps;
  static_assert(ACC * BN + L * a_cols <= 512, "tensor memory");
  static_assert(total <= 232448, "shared memory");
};

enum { kRowsMajorK = 0, kRowsMajorM = 1, kPixels = 2 };

struct Params {
  int a_mode;
  int tiles, m_tiles, k_blocks, chunk;     // chunk: K-blocks that one accumulator sums before it is emptied
  // matrices
  int M, N;
  float* c;
  int64_t ldc;
  const float* bias;
  int act, accumulate;
  // pixels: a tile is a box of bw x bh x bn pixels of the row side
  int bw, bh, bn, tiles_w, tiles_h;        // tiles along the width, the height
  int rows_w, rows_h, rows_n;              // extent of the row side
  int c_blocks, kw;                        // blocks of 32 channels, kernel width: k-block = (ky * kw + kx) * c_blocks + channel block
  int sx, sy, px, py;                      // source coordinate = row coordinate * s - p + tap
  int out_h, out_w, osx, osy, ox, oy;      // output pixel = row coordinate * os + o, channels as planes
};

__device__ __forceinline__ void load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map),
               "r"(x), "r"(y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void load_4d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, int w, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void store_tmem16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
      "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
// lo * hi, hi * lo and hi * hi of one K-step into one accumulator, A in tensor memory; one elected lane of a converged warp issues.
__device__ __forceinline__ void mma_step(uint32_t d, uint32_t a_hi, uint32_t a_lo, uint32_t b_hi, uint32_t b_lo, uint32_t b_desc_hi, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred pa, pt, pe;\n\t"
      ".reg .b64 dbh, dbl;\n\t"
      "elect.sync _|pe, 0xffffffff;\n\t"
      "setp.ne.b32 pa, %7, 0;\n\t"
      "setp.eq.b32 pt, 0, 0;\n\t"
      "mov.b64 dbh, {%3, %5};\n\t"
      "mov.b64 dbl, {%4, %5};\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::tf32 [%0], [%2], dbh, %6, pa;\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], dbl, %6, pt;\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], dbh, %6, pt;\n\t}" ::"r"(d), "r"(a_hi), "r"(a_lo), "r"(b_hi), "r"(b_lo),
      "r"(b_desc_hi), "r"(idesc), "r"(accumulate)
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
// a - (a truncated to TF32), with half a unit of the last place that the tensor core keeps added: it truncates what it is given, which
// would make every lo too small.
__device__ __forceinline__ uint32_t low_part(float a) {
  return __float_as_uint(a - __uint_as_float(__float_as_uint(a) & 0xFFFFE000u)) + 0x1000u;
}
__device__ __forceinline__ float activated(float v, int act) {
  if (act == RT_ACT_RELU) return fmaxf(v, 0.f);
  if (act == RT_ACT_TANH) return tanhf(v);
  if (act == RT_ACT_SIGMOID) return 1.f / (1.f + expf(-v));
  return v;
}

template <int BN, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
tma_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Params p, int* status) {
  extern __shared__ char smem_raw[];
  using C = Config<BN, SPLIT>;
  __shared__ volatile int abort_flag;
  const uint32_t raw_base = smem_u32(smem_raw);
  const uint32_t base = (raw_base + 1023) & ~1023u;
  char* smem = smem_raw + (base - raw_base);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t bars = base + C::bar_offset;
  auto raw_full = [&](int i) { return bars + 8 * i; };
  auto raw_empty = [&](int i) { return bars + 8 * (C::R + i); };
  auto conv_full = [&](int i) { return bars + 8 * (2 * C::R + i); };
  auto conv_empty = [&](int i) { return bars + 8 * (2 * C::R + C::L + i); };
  // one "full" barrier per accumulator and group of accumulating warps: a group sees only the uses that are its own, so that the phases
  // of its barriers follow them
  auto acc_full = [&](int group, int i) { return bars + 8 * (2 * C::R + 2 * C::L + group * C::ACC + i); };
  auto acc_empty = [&](int i) { return bars + 8 * (2 * C::R + 2 * C::L + 2 * C::ACC + i); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::bar_offset + C::n_bars * 8);

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < C::R; ++i) {
      mbar_init(raw_full(i), 1);
      mbar_init(raw_empty(i), 1);
    }
    for (int i = 0; i < C::L; ++i) {
      mbar_init(conv_full(i), C::converters);
      mbar_init(conv_empty(i), 1);
    }
    for (int i = 0; i < C::ACC; ++i) {
      mbar_init(acc_full(0, i), 1);
      mbar_init(acc_full(1, i), 1);
      mbar_init(acc_empty(i), C::turns ? kEpilogueWarps / 2 : kEpilogueWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) tmem_alloc(smem_u32(tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t tmem_a = tmem + C::ACC * BN;
  bool ok = true;

  if (warp == kTmaWarp) {
    // ---------------- TMA: raw tiles ----------------
    if (lane == 0) {
      int it = 0;
      for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
        const int mt = tile % p.m_tiles, nt = tile / p.m_tiles;
        int x0 = 0, y0 = 0, n0 = 0;
        if (p.a_mode == kPixels) {
          const int tw = mt % p.tiles_w, r = mt / p.tiles_w;
          x0 = tw * p.bw * p.sx - p.px;
          y0 = r % p.tiles_h * p.bh * p.sy - p.py;
          n0 = r / p.tiles_h * p.bn;
        }
        int cb = 0, kx = 0, ky = 0;
        for (int kb = 0; kb < p.k_blocks && ok; ++kb, ++it) {
          const int s = it % C::R;
          if (it >= C::R) ok = wait(raw_empty(s), (it / C::R - 1) & 1, status, 41, &abort_flag);
          if (!ok) break;
          const uint32_t dst = base + s * C::raw;
          mbar_expect_tx(raw_full(s), C::raw);
          if (p.a_mode == kRowsMajorK) load_2d(dst, &map_a, kb * BK, mt * BM, raw_full(s));
          else if (p.a_mode == kRowsMajorM) load_2d(dst, &map_a, mt * BM, kb * BK, raw_full(s));
          else load_4d(dst, &map_a, cb * BK, x0 + kx, y0 + ky, n0, raw_full(s));
          load_2d(dst + kARaw, &map_b, kb * BK, nt * BN, raw_full(s));
          if (SPLIT) load_2d(dst + kARaw + C::b_raw, &map_b, kb * BK, p.N + nt * BN, raw_full(s));
          if (++cb == p.c_blocks) {
            cb = 0;
            if (++kx == p.kw) {
              kx = 0;
              ++ky;
            }
          }
        }
      }
      // copies that nobody has waited for must have landed before the CTA may leave
      if (!ok)
        for (int i = it > C::R ? it - C::R : 0; i < it; ++i) mbar_wait(raw_full(i % C::R), (i / C::R) & 1, status, 42);
    }
  } else if (warp == kMmaWarp) {
    // ---------------- MMAs ----------------
    constexpr uint32_t idesc = make_idesc(BN);
    constexpr uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);  // 8-row groups of 1024 bytes, 128-byte swizzle
    int it = 0, chunks = 0, t = 0;  // chunks that are complete
    for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x, ++t) {
      for (int kb = 0, in_chunk = 0; kb < p.k_blocks && ok; ++kb, ++it) {
        const int s = it % C::R, l = it % C::L;
        const bool first = in_chunk == 0, last = ++in_chunk == p.chunk || kb + 1 == p.k_blocks;
        if (last) in_chunk = 0;
        ok = __all_sync(0xffffffffu, wait(raw_full(s), (it / C::R) & 1, status, 44, &abort_flag) &&
                                         wait(conv_full(l), (it / C::L) & 1, status, 45, &abort_flag));
        if (!ok) break;
        tc_fence_after();
        const uint32_t b_hi = ((base + s * C::raw + kARaw) >> 4 & 0x3FFF) | (1u << 16);
        const uint32_t b_lo = ((SPLIT ? base + s * C::raw + kARaw + C::b_raw : base + C::lo_offset + l * C::b_raw) >> 4 & 0x3FFF) | (1u << 16);
        const uint32_t a_hi = tmem_a + l * C::a_cols, a_lo = a_hi + BK;
        const int acc = chunks % C::ACC, use = chunks / C::ACC;
        if (first && use > 0) {
          ok = __all_sync(0xffffffffu, wait(acc_empty(acc), (use - 1) & 1, status, 43, &abort_flag));
          tc_fence_after();
        }
        if (ok) {
#pragma unroll
          for (int j = 0; j < BK / 8; ++j)
            mma_step(tmem + acc * BN, a_hi + 8 * j, a_lo + 8 * j, b_hi + 2 * j, b_lo + 2 * j, desc_hi, idesc, first && j == 0 ? 0u : 1u);
          if (last) umma_commit_elect(acc_full(C::turns ? t & 1 : 0, acc));
        }
        if (ok) {
          umma_commit_elect(raw_empty(s));
          umma_commit_elect(conv_empty(l));
        }
        if (last) ++chunks;
      }
    }
  } else if (warp >= kEpilogueWarps && warp < kEpilogueWarps + C::converters) {
    // ---------------- converters ----------------
    // Four of the six convert A (a row a thread; tensor-memory lanes 32 * (warp % 4) ..) and a smaller share of B than the other two.
    const int cw = warp - kEpilogueWarps, row = cw * 32 + lane;
    constexpr int chunks = BN * 8, share_a = chunks * 9 / 64 / 32 * 32, share_b = (chunks - 4 * share_a) / 2;  // 16-byte pieces of B
    const int b_begin = (cw < 4 ? cw * share_a : 4 * share_a + (cw - 4) * share_b) + lane, b_end = b_begin - lane + (cw < 4 ? share_a : share_b);
    int it = 0;
    for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
      for (int kb = 0; kb < p.k_blocks && ok; ++kb, ++it) {
        const int s = it % C::R, l = it % C::L;
        ok = wait(raw_full(s), (it / C::R) & 1, status, 46, &abort_flag);
        if (ok && it >= C::L) ok = wait(conv_empty(l), (it / C::L - 1) & 1, status, 47, &abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const char* a = smem + s * C::raw;
        if (cw < 4) {
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t hi[16], lo[16];
            if (p.a_mode == kRowsMajorM) {
              const float* q = reinterpret_cast<const float*>(a) + half * 16 * BM + row;
#pragma unroll
              for (int i = 0; i < 16; ++i) hi[i] = __float_as_uint(q[i * BM]);
            } else {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float4 v = *reinterpret_cast<const float4*>(a + row * 128 + ((half * 4 + i) ^ (row & 7)) * 16);
                hi[4 * i] = __float_as_uint(v.x); hi[4 * i + 1] = __float_as_uint(v.y);
                hi[4 * i + 2] = __float_as_uint(v.z); hi[4 * i + 3] = __float_as_uint(v.w);
              }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float v = __uint_as_float(hi[i]);
              lo[i] = low_part(v);
            }
            const uint32_t ta = tmem_a + ((uint32_t)(cw * 32) << 16) + l * C::a_cols + half * 16;
            store_tmem16(ta, hi);
            store_tmem16(ta + BK, lo);
          }
        }
        const float4* b = reinterpret_cast<const float4*>(a + kARaw);
        float4* bl = reinterpret_cast<float4*>(smem + C::lo_offset + l * C::b_raw);
#pragma unroll 5
        for (int j = b_begin; !SPLIT && j < b_end; j += 32) {
          const float4 v = b[j];
          bl[j] = make_float4(__uint_as_float(low_part(v.x)), __uint_as_float(low_part(v.y)), __uint_as_float(low_part(v.z)),
                              __uint_as_float(low_part(v.w)));
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(conv_full(l));
      }
    }
  } else if (warp < kEpilogueWarps) {
    // ---------------- sums over the K-blocks, result ----------------
    float* stage = reinterpret_cast<float*>(smem + C::stage_offset) + warp * 32 * 17;
    const int quad = warp & 3, group = warp >> 2, full = C::turns ? group : 0;
    const int col0 = C::turns ? 0 : group * C::NC;  // of this warp's columns in the tile
    const int chunks = (p.k_blocks + p.chunk - 1) / p.chunk;  // of a tile
    int t = 0;
    uint32_t phases = 0;  // bit i: parity of this group's next use of accumulator i
    for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x, ++t) {
      if (C::turns && (t & 1) != group) continue;
      float sum[C::NC];
#pragma unroll
      for (int j = 0; j < C::NC; ++j) sum[j] = 0.f;
      for (int i = 0; i < chunks && ok; ++i) {
        const int acc = (t * chunks + i) % C::ACC;
        ok = __all_sync(0xffffffffu, wait(acc_full(full, acc), (phases >> acc) & 1, status, 48, &abort_flag));
        if (!ok) break;
        phases ^= 1u << acc;
        tc_fence_after();
        const uint32_t d = tmem + acc * BN + col0 + ((uint32_t)(quad * 32) << 16);
#pragma unroll
        for (int c = 0; c < C::NC; c += 16) {
          uint32_t v[16];
          tmem_ld16_nowait(d + c, v);
          tmem_wait_ld();
          if (c + 16 == C::NC) {  // all read
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(acc));
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) sum[c + j] += __uint_as_float(v[j]);
        }
      }
      if (!ok) break;
      const int mt = tile % p.m_tiles, n0 = tile / p.m_tiles * BN + col0, n_left = p.N - n0;
      if (SPLIT) {
        const int tw = mt % p.tiles_w, r = mt / p.tiles_w, row = quad * 32 + lane;
        const int w = row % p.bw, q = row / p.bw;
        const int x = tw * p.bw + w, y = r % p.tiles_h * p.bh + q % p.bh, n = r / p.tiles_h * p.bn + q / p.bh;
        if (x < p.rows_w && y < p.rows_h && n < p.rows_n) {
          const int64_t plane = (int64_t)p.out_h * p.out_w;
          float* out = p.c + ((int64_t)n * p.N + n0) * plane + (int64_t)(y * p.osy + p.oy) * p.out_w + x * p.osx + p.ox;
#pragma unroll
          for (int j = 0; j < C::NC; ++j) {
            if (j < n_left) *out = p.bias ? sum[j] + __ldg(p.bias + n0 + j) : sum[j];
            out += plane;
          }
        }
      } else {
        const int m0 = mt * BM + quad * 32, cc = lane & 15;
#pragma unroll
        for (int c = 0; c < C::NC; c += 16) {
          if (c < n_left) {
#pragma unroll
            for (int j = 0; j < 16; ++j) stage[lane * 17 + j] = sum[c + j];
            __syncwarp();
            if (c + cc < n_left) {
              const float bias = p.bias ? __ldg(p.bias + n0 + c + cc) : 0.f;
              float* out = p.c + (int64_t)m0 * p.ldc + n0 + c + cc;
#pragma unroll 2
              for (int i = lane >> 4; i < 32; i += 2)
                if (m0 + i < p.M) {
                  float u = stage[i * 17 + cc] + bias;
                  if (p.act != RT_ACT_NONE) u = activated(u, p.act);
                  if (p.accumulate) u += out[(int64_t)i * p.ldc];
                  out[(int64_t)i * p.ldc] = u;
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

// ---- operands brought into a form that TMA can fetch ------------------------------------------------------------------------
// dst[b][c][r] = src[b][r][c] (TRANSPOSE) or dst[b][r][c] = src[b][r][c], rows of dst `ldd` floats apart.
template <bool TRANSPOSE>
__global__ void __launch_bounds__(256) pack_kernel(const float* __restrict__ src, float* __restrict__ dst, int rows, int cols, int64_t lds, int64_t ldd,
                                                   int64_t batch_src, int64_t batch_dst) {
  __shared__ float tile[32][33];
  const float* s = src + (int64_t)blockIdx.z * batch_src;
  float* d = dst + (int64_t)blockIdx.z * batch_dst;
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    const int r = r0 + ty + j, c = c0 + tx;
    const float v = r < rows && c < cols ? __ldg(s + (int64_t)r * lds + c) : 0.f;
    if (TRANSPOSE) tile[ty + j][tx] = v;
    else if (r < rows && c < cols) d[(int64_t)r * ldd + c] = v;
  }
  if (!TRANSPOSE) return;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    const int c = c0 + ty + j, r = r0 + tx;
    if (r < rows && c < cols) d[(int64_t)c * ldd + r] = tile[tx][ty + j];
  }
}
// The transpose with 128-bit accesses on both sides: a block turns 32 rows x 128 columns, four independent loads a thread.  16-byte aligned
// pointers and rows on both sides; bound by memory bandwidth (103 MB turned: see the figures at channels_last).
__global__ void __launch_bounds__(256) transpose4_kernel(const float* __restrict__ src, float* __restrict__ dst, int rows, int cols, int64_t lds, int64_t ldd,
                                                         int64_t batch_src, int64_t batch_dst) {
  RT_PDL_ENTRY();
  __shared__ float tile[32][129];
  const float* s = src + (int64_t)blockIdx.z * batch_src;
  float* d = dst + (int64_t)blockIdx.z * batch_dst;
  const int c0 = blockIdx.x * 128, r0 = blockIdx.y * 32;
  float4 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + (threadIdx.x >> 5) + 8 * i, c = c0 + (threadIdx.x & 31) * 4;
    v[i] = r < rows && c < cols ? __ldcs(reinterpret_cast<const float4*>(s + (int64_t)r * lds + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float* t = &tile[(threadIdx.x >> 5) + 8 * i][(threadIdx.x & 31) * 4];
    t[0] = v[i].x; t[1] = v[i].y; t[2] = v[i].z; t[3] = v[i].w;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = (threadIdx.x >> 3) + 32 * i, r = (threadIdx.x & 7) * 4;
    if (c0 + c < cols && r0 + r < rows)
      *reinterpret_cast<float4*>(d + (int64_t)(c0 + c) * ldd + r0 + r) = make_float4(tile[r][c], tile[r + 1][c], tile[r + 2][c], tile[r + 3][c]);
  }
}
// B operand of a convolution, hi rows and then lo rows: row n, column ((ky * kw + kx) * c_blocks + channel block) * 32 + channel; zeros
// behind the last channel.
__global__ void __launch_bounds__(256) pack_taps_kernel(const float* __restrict__ w, float* __restrict__ dst, int N, int C, int c_blocks, int kw, int taps,
                                                        int64_t sn, int64_t sc, int64_t sky, int64_t skx, int64_t off0) {
  RT_PDL_ENTRY();
  const int64_t cols = (int64_t)taps * c_blocks * BK;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N * cols; i += (int64_t)gridDim.x * blockDim.x) {
    const int n = (int)(i / cols), k = (int)(i % cols), tap = k / (c_blocks * BK), c = k % (c_blocks * BK);
    const float v = c < C ? __ldg(w + n * sn + c * sc + tap / kw * sky + tap % kw * skx + off0) : 0.f;
    dst[i] = v;
    dst[N * cols + i] = __uint_as_float(low_part(v));
  }
}

// [rows][cols] floats, rows ld floats apart, boxes of box_cols x box_rows, zeros outside.
inline bool map_matrix(CUtensorMap* m, const float* t, int64_t cols, int64_t rows, int64_t ld, int box_cols, int box_rows, bool swizzle) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 4};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, one[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(t), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
             swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, bool SPLIT = false>
rt_status launch(rt_ctx* ctx, const CUtensorMap& a, const CUtensorMap& b, const Params& p) {
  using C = Config<BN, SPLIT>;
  auto kern = tma_gemm_kernel<BN, SPLIT>;
  static RtDeviceOnce once;
  RT_CUDA(ctx, once([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::total); }));
  kern<<<p.tiles < ctx->sm_count ? p.tiles : ctx->sm_count, kThreads, C::total, ctx->stream>>>(a, b, p, ctx->device_status);
  RT_LAUNCHED(ctx);
  return RT_OK;
}
// K-blocks per accumulator.  Errors of 3.5e-7, 5.8e-7 and 1.0e-6 of the result for 1, 2 and 4 blocks, at any length; emptying an
// accumulator costs 3 - 7 % of the time.  The lines lie where the error stays below that of the kernel for smaller products
// (4.5e-7 + 8e-10 k) at the same length.
inline int chunk_of(int64_t k) { return k < 1024 ? 1 : (k < 2048 ? 2 : 4); }
inline int64_t up4(int64_t v) { return (v + 3) & ~int64_t(3); }
inline rt_status pack(rt_ctx* ctx, const float* src, float* dst, int64_t rows, int64_t cols, int64_t lds, int64_t ldd, bool transpose, int64_t batch,
                      int64_t batch_src, int64_t batch_dst) {
  const dim3 grid((unsigned)((cols + 31) / 32), (unsigned)((rows + 31) / 32), (unsigned)batch);
  if (transpose && rt_aligned16(src) && rt_aligned16(dst) && ((rows | cols | lds | ldd | batch_src | batch_dst) & 3) == 0)
    rt_launch(ctx, transpose4_kernel, dim3((unsigned)((cols + 127) / 128), grid.y, grid.z), 256, 0, src, dst, (int)rows, (int)cols, lds, ldd, batch_src,
                                                                                                    batch_dst);
  else if (transpose) pack_kernel<true><<<grid, 256, 0, ctx->stream>>>(src, dst, (int)rows, (int)cols, lds, ldd, batch_src, batch_dst);
  else pack_kernel<false><<<grid, 256, 0, ctx->stream>>>(src, dst, (int)rows, (int)cols, lds, ldd, batch_src, batch_dst);
  RT_LAUNCHED(ctx);
  return RT_OK;
}

}  // namespace tma
}  // namespace tc

// C = act(op(A) op(B) + bias) (+ C).  RT_ERR_UNIMPLEMENTED: not a shape for this kernel.
rt_status rt_gemm_tma_internal(rt_ctx* ctx, int trans_a, int trans_b, int64_t m, int64_t n, int64_t k, const float* a, int64_t lda, const float* b,
                               int64_t ldb, float* c, int64_t ldc, const float* bias, int act, int accumulate) {
  using namespace tc::tma;
  if (m >= (1 << 24) || n >= (1 << 24) || k >= (1 << 24)) return RT_ERR_UNIMPLEMENTED;
  const int64_t mt = (m + BM - 1) / BM, nt = (n + 127) / 128;
  if ((m + 31) / 32 > 65535 || (k + 31) / 32 > 65535 || (n + 31) / 32 > 65535) return RT_ERR_UNIMPLEMENTED;
  auto direct = [](const float* p, int64_t ld) { return rt_aligned16(p) && ld % 4 == 0; };
  RtScratch wa(ctx), wb(ctx);
  Params p{};
  p.a_mode = kRowsMajorK;
  CUtensorMap ma, mb;
  bool mapped = true;
  rt_status st = RT_OK;
  // A with the rows contiguous is read from shared memory a word at a time; from sixteen tile columns on, turning it once is cheaper
  // (4096^3: 0.70 against 0.76 ms)
  if (trans_a && direct(a, lda) && n < 2048) {
    p.a_mode = kRowsMajorM;
    mapped = map_matrix(&ma, a, m, k, lda, BM, BK, false);
  } else {
    const float* q = a;
    int64_t ld = lda;
    if (trans_a || !direct(a, lda)) {
      ld = up4(k);
      if ((st = wa.alloc(sizeof(float) * (size_t)(m * ld))) != RT_OK) return st;
      q = wa.as<float>();
      st = trans_a ? pack(ctx, a, wa.as<float>(), k, m, lda, ld, true, 1, 0, 0) : pack(ctx, a, wa.as<float>(), m, k, lda, ld, false, 1, 0, 0);
      if (st != RT_OK) return st;
    }
    mapped = map_matrix(&ma, q, k, m, ld, BK, BM, true);
  }
  const float* q = b;
  int64_t ld = ldb;
  if (!trans_b || !direct(b, ldb)) {
    ld = up4(k);
    if ((st = wb.alloc(sizeof(float) * (size_t)(n * ld))) != RT_OK) return st;
    q = wb.as<float>();
    st = trans_b ? pack(ctx, b, wb.as<float>(), n, k, ldb, ld, false, 1, 0, 0) : pack(ctx, b, wb.as<float>(), k, n, ldb, ld, true, 1, 0, 0);
    if (st != RT_OK) return st;
  }
  mapped = mapped && map_matrix(&mb, q, k, n, ld, BK, 128, true);
  if (!mapped) return RT_ERR_UNIMPLEMENTED;
  p.M = (int)m;
  p.N = (int)n;
  p.c = c;
  p.ldc = ldc;
  p.bias = bias;
  p.act = act;
  p.accumulate = accumulate;
  p.m_tiles = (int)mt;
  p.tiles = (int)(mt * nt);
  p.k_blocks = (int)((k + BK - 1) / BK);
  p.c_blocks = p.k_blocks;
  p.chunk = chunk_of(k);
  p.kw = 1;
  return launch<128>(ctx, ma, mb, p);
}

namespace tc {
namespace tma {

// A convolution-shaped product over the pixels (n, y, x) of the row side: out(n, co, y * osy + oy, x * osx + ox) (+ bias) =
// sum over taps and channels of src(n, c, y * sy - py + ky, x * sx - px + kx) * w(co, c, ky, kx), zeros outside the source.
struct PixelProduct {
  int Nb, C, H, W;                      // source
  int rows_h, rows_w;                   // row side
  int N, kh, kw, sy, sx, py, px;
  const float* w;                       // element (co, c, ky, kx) at co * sn + c * sc + ky * sky + kx * skx + off0
  int64_t sn, sc, sky, skx, off0;
  const float* bias;
  float* out;
  int out_h, out_w, osy, osx, oy, ox;
};

// The box of 128 pixels (powers of two) that wastes least at the edges; short runs along a row make scattered stores.
inline void choose_box(int w, int h, int n, int* bw, int* bh, int* bn) {
  double best = -1;
  for (int a = 1; a <= 128; a *= 2)
    for (int b = 1; a * b <= 128; b *= 2) {
      const int c = 128 / (a * b);
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

// src in channels-last form: [Nb][H * W][up4(C)].
inline rt_status channels_last(rt_ctx* ctx, const float* src, int Nb, int C, int64_t hw, RtScratch* ws) {
  const int64_t cp = up4(C);
  rt_status st = ws->alloc(sizeof(float) * (size_t)Nb * hw * cp);
  if (st != RT_OK) return st;
  for (int n = 0; n < Nb && st == RT_OK; n += 32768)
    st = pack(ctx, src + (int64_t)n * C * hw, ws->as<float>() + (int64_t)n * hw * cp, C, hw, hw, cp, true, Nb - n < 32768 ? Nb - n : 32768, C * hw, hw * cp);
  return st;
}

inline rt_status pixel_product(rt_ctx* ctx, const PixelProduct& q, const float* nhwc) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return RT_ERR_UNIMPLEMENTED;
  Params p{};
  p.a_mode = kPixels;
  choose_box(q.rows_w, q.rows_h, q.Nb, &p.bw, &p.bh, &p.bn);
  const int64_t cp = up4(q.C);
  CUtensorMap ma, mb;
  const cuuint64_t dims[4] = {(cuuint64_t)q.C, (cuuint64_t)q.W, (cuuint64_t)q.H, (cuuint64_t)q.Nb};
  const cuuint64_t strides[3] = {(cuuint64_t)cp * 4, (cuuint64_t)q.W * cp * 4, (cuuint64_t)q.H * q.W * cp * 4};
  const cuuint32_t box[4] = {BK, (cuuint32_t)((p.bw - 1) * q.sx + 1), (cuuint32_t)((p.bh - 1) * q.sy + 1), (cuuint32_t)p.bn};
  const cuuint32_t step[4] = {1, (cuuint32_t)q.sx, (cuuint32_t)q.sy, 1};
  if (box[1] > 256 || box[2] > 256) return RT_ERR_UNIMPLEMENTED;
  if (enc(&ma, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(nhwc), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return RT_ERR_UNIMPLEMENTED;
  const int bn_cols = q.N <= 64 ? 64 : 128;
  p.c_blocks = (q.C + BK - 1) / BK;
  p.kw = q.kw;
  p.k_blocks = p.c_blocks * q.kh * q.kw;
  const int64_t cols = (int64_t)p.k_blocks * BK;
  RtScratch wb(ctx);
  rt_status st = wb.alloc(sizeof(float) * (size_t)(2 * q.N * cols));
  if (st != RT_OK) return st;
  rt_launch(ctx, pack_taps_kernel, rt_grid_for(ctx, q.N * cols, 256), 256, 0, q.w, wb.as<float>(), q.N, q.C, p.c_blocks, q.kw, q.kh * q.kw, q.sn, q.sc, q.sky,
                                                                               q.skx, q.off0);
  RT_LAUNCHED(ctx);
  if (!map_matrix(&mb, wb.as<float>(), cols, 2 * q.N, cols, BK, bn_cols, true)) return RT_ERR_UNIMPLEMENTED;
  p.tiles_w = (q.rows_w + p.bw - 1) / p.bw;
  p.tiles_h = (q.rows_h + p.bh - 1) / p.bh;
  p.rows_w = q.rows_w;
  p.rows_h = q.rows_h;
  p.rows_n = q.Nb;
  p.m_tiles = p.tiles_w * p.tiles_h * ((q.Nb + p.bn - 1) / p.bn);
  p.tiles = p.m_tiles * ((q.N + bn_cols - 1) / bn_cols);
  p.N = q.N;
  p.c = q.out;
  p.bias = q.bias;
  const int64_t k = (int64_t)q.C * q.kh * q.kw;
  p.chunk = k < 512 ? 2 : (k < 1024 ? 3 : 4);  // the gather kernel's errors: 6e-7 at 300, 9e-7 at 576, 1.5e-6 at 1152
  p.sx = q.sx; p.sy = q.sy; p.px = q.px; p.py = q.py;
  p.out_h = q.out_h; p.out_w = q.out_w; p.osx = q.osx; p.osy = q.osy; p.ox = q.ox; p.oy = q.oy;
  return bn_cols == 64 ? launch<64, true>(ctx, ma, mb, p) : launch<128, true>(ctx, ma, mb, p);
}

// Which convolutions: a whole wave of tiles, enough channels to fill most of a block of 32, strides that TMA steps over.
inline bool worth_it(rt_ctx* ctx, int64_t pixels, int C, int N, int sy, int sx, int H, int W) {
  return pixels >= 128ll * ctx->sm_count && pixels < (1ll << 31) && C >= 16 && N >= 16 && sy <= 8 && sx <= 8 && (int64_t)H * W < (1ll << 31);
}

}  // namespace tma
}  // namespace tc

// y[Nb,Cy,Hy,Wy] = conv(x, w[Cy,Cx,kh,kw]) (+ bias).
rt_status rt_conv_forward_tma_internal(rt_ctx* ctx, const float* x, const float* w, const float* bias, const ConvGeom& g, float* y) {
  using namespace tc::tma;
  if (!worth_it(ctx, (int64_t)g.Nb * g.Hy * g.Wy, g.Cx, g.Cy, g.sh, g.sw, g.Hx, g.Wx)) return RT_ERR_UNIMPLEMENTED;
  RtScratch ws(ctx);
  rt_status st = channels_last(ctx, x, g.Nb, g.Cx, (int64_t)g.Hx * g.Wx, &ws);
  if (st != RT_OK) return st;
  const int64_t taps = (int64_t)g.kh * g.kw;
  PixelProduct q{g.Nb, g.Cx, g.Hx, g.Wx, g.Hy, g.Wy, g.Cy, g.kh, g.kw, g.sh, g.sw, g.ph, g.pw, w, g.Cx * taps, taps, g.kw, 1, 0, bias, y,
                 g.Hy, g.Wy, 1, 1, 0, 0};
  return pixel_product(ctx, q, ws.as<float>());
}

// out[Nb,Cm,Hx,Wx] (+ bias) = gather of y[Nb,Cy,Hy,Wy] with w[Cy,Cm,kh,kw]: input gradient of a convolution, forward of a transposed one.
// The outputs of one stride phase (iy % sh, ix % sw) only meet the taps ky = ky0 + sh * a, kx = kx0 + sw * b; with those the phase is a
// unit-stride convolution of y with the kernel turned round that writes every sh-th / sw-th output.
rt_status rt_conv_gather_tma_internal(rt_ctx* ctx, const float* y, const float* w, const float* bias, const ConvGeom& g, int cm, float* out) {
  using namespace tc::tma;
  if (!worth_it(ctx, (int64_t)g.Nb * g.Hx * g.Wx / (g.sh * g.sw), g.Cy, cm, 1, 1, g.Hy, g.Wy)) return RT_ERR_UNIMPLEMENTED;
  for (int ry = 0; ry < g.sh; ++ry)  // every phase needs a tap (otherwise its outputs are the bias alone)
    if ((ry + g.ph) % g.sh >= g.kh) return RT_ERR_UNIMPLEMENTED;
  for (int rx = 0; rx < g.sw; ++rx)
    if ((rx + g.pw) % g.sw >= g.kw) return RT_ERR_UNIMPLEMENTED;
  RtScratch ws(ctx);
  rt_status st = channels_last(ctx, y, g.Nb, g.Cy, (int64_t)g.Hy * g.Wy, &ws);
  const int64_t taps = (int64_t)g.kh * g.kw;
  for (int ry = 0; ry < g.sh && st == RT_OK; ++ry)
    for (int rx = 0; rx < g.sw && st == RT_OK; ++rx) {
      const int rows_h = (g.Hx - ry + g.sh - 1) / g.sh, rows_w = (g.Wx - rx + g.sw - 1) / g.sw;
      if (rows_h <= 0 || rows_w <= 0) continue;
      const int ky0 = (ry + g.ph) % g.sh, kx0 = (rx + g.pw) % g.sw;
      const int nay = (g.kh - ky0 + g.sh - 1) / g.sh, nax = (g.kw - kx0 + g.sw - 1) / g.sw;
      const int py = (nay - 1) - (ry + g.ph - ky0) / g.sh, px = (nax - 1) - (rx + g.pw - kx0) / g.sw;
      PixelProduct q{g.Nb, g.Cy, g.Hy, g.Wy, rows_h, rows_w, cm, nay, nax, 1, 1, py, px, w, taps, cm * taps, -(int64_t)g.sh * g.kw, -(int64_t)g.sw,
                     (int64_t)(ky0 + g.sh * (nay - 1)) * g.kw + kx0 + g.sw * (nax - 1), bias, out, g.Hx, g.Wx, g.sh, g.sw, ry, rx};
      st = pixel_product(ctx, q, ws.as<float>());
    }
  return st;
}
