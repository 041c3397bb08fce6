// A whole LSTM sequence in one kernel, and its gradient in another.
//
// Timestep by timestep the recurrence is a product of [batch, H] x [H, 4H] and a few element operations, each a kernel that is over before
// it has started: 8 + 4 us of a timestep at batch 64, H 512, of which the arithmetic is two.  Here the kernel stays: every block keeps its
// slice of the recurrent weights in shared memory for the whole sequence, and what the blocks tell one another per timestep is written to
// and polled in memory, value and timestep number side by side in 8 bytes, so that seeing the number is having the value: no barrier.
//
// A block has 16 rows of the batch and U hidden units (all four gates of them).  Rows are independent of one another, so only the blocks
// of the same rows exchange anything.  Forward a block publishes h of its units and gathers everybody's: the 16 warps split the reduction
// and add up in shared memory.  Backward a block has the gate gradients of its own units and multiplies them with its slice (its columns
// of the weights) into a partial gradient of ALL units, which it sends to the blocks that own them: 32 KB in and out either way, where
// gathering the gate gradients would take 128.  All sums are fp32 in a fixed order.
// The blocks wait for one another, so they are launched cooperatively (all resident or an error).  Every wait is bounded; a block whose wait
// expires records a code in the status word and goes on without waiting.
//
// Bound by latency.  Measured at batch 30, H 200: 2.3 us a timestep forward, 4.2 backward; as kernels of their own the product, the cell and
// the concatenation took 9.7 forward, 12.3 backward.  Sizes whose blocks do not fit beside one another, or whose slice of the weights does not
// fit into a block, run timestep by timestep.
#include "rt_internal.cuh"
#include "tc_common.cuh"

namespace {

constexpr int kRows = 16, kWarps = 16, kThreads = kWarps * 32;
constexpr int kPitch = 20;  // words between the 16 rows' values of one reduction index and the next: 16-byte aligned, few bank conflicts
constexpr uint32_t kPolls = 1u << 21;

struct SeqArgs {
  int steps, batch, hidden, groups;  // groups of U units
  const float* w;                    // [hidden][4 * hidden], rows ldw apart
  int64_t ldw;
  const float* c0;
  uint4* mail;                       // zeroed before the launch
  int* gave_up;                      // zeroed before the launch
  int* status;
  // forward: the part of the gates' inputs that does not depend on h; activated gates, cell, its hyperbolic tangent and the output,
  // each [steps * batch][hidden]
  const float *pre, *h0;
  float *ig, *fg, *gg, *og, *c, *tc, *h;
  // backward
  const float* dh;
  float *dgates, *dh0, *dc0;
};

__device__ __forceinline__ uint4 peek(const uint4* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void post(uint2* p, float v, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(__float_as_uint(v)), "r"(tag) : "memory");
}
__device__ __forceinline__ void post2(uint4* p, float v, float w, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %3, %2, %3};" ::"l"(p), "r"(__float_as_uint(v)), "r"(__float_as_uint(w)), "r"(tag) : "memory");
}
__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + expf(-x)); }

// Waits until N pieces of mail carry `tag`.  False: the wait ran out, here or in another block.  (Polling one piece until it is there and
// only then the others is a round trip more: 693 -> 714 us for 128 timesteps at batch 64, H 512.)
template <int N>
__device__ __forceinline__ bool receive(const uint4* const (&from)[N], const bool (&want)[N], uint32_t tag, uint4 (&v)[N], const SeqArgs& a) {
  for (uint32_t i = 0; i < kPolls; ++i) {
    bool there = true;
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (want[j]) v[j] = peek(from[j]);
#pragma unroll
    for (int j = 0; j < N; ++j) there = there && (!want[j] || (v[j].y == tag && v[j].w == tag));
    if (__all_sync(0xffffffffu, there)) return true;
    if ((i & 1023) == 1023 && *(volatile int*)a.gave_up) return false;
  }
  *(volatile int*)a.gave_up = 1;
  tc::record_status(a.status, 81);
  return false;
}

template <int U>
__global__ void __launch_bounds__(kThreads, 1) lstm_sequence_kernel(const SeqArgs a) {
  extern __shared__ float4 smem4[];
  constexpr int kRegion = kRows * U;  // 16-byte pieces of a warp's region: its sums, before that 2 U reduction indices of h
  static_assert(2 * U * kPitch * 4 <= kRegion * 16, "region");
  constexpr int UL = U / 8, P = 32 / U, NL = U / 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rg = lane >> 3, cg = lane & 7;
  const int H = a.hidden, group = blockIdx.x % a.groups, row0 = blockIdx.x / a.groups * kRows;
  const int first_block = blockIdx.x - group, padded = a.groups * U;
  float4* const regions = smem4 + padded * U;
  float* const stage = reinterpret_cast<float*>(regions + warp * kRegion);
  for (int i = threadIdx.x; i < padded * U; i += kThreads) {  // [reduction index][unit]: the four gates
    const int k = i / U, unit = group * U + i % U;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < H && unit < H) {
      const float* q = a.w + (int64_t)k * a.ldw + unit;
      v = make_float4(__ldg(q), __ldg(q + H), __ldg(q + 2 * H), __ldg(q + 3 * H));
    }
    smem4[i] = v;
  }
  // for the cell: warp = row, lane = unit; the lanes beyond U help adding up
  const int row = row0 + warp, u = lane % U, part = lane / U, unit = group * U + u;
  const bool active = row < a.batch && unit < H;
  const int64_t cell = (int64_t)row * H + unit, per_step = (int64_t)a.batch * H;
  float c = active && a.c0 ? __ldg(a.c0 + cell) : 0.f;
  const int q_begin = warp * a.groups / kWarps, q_end = (warp + 1) * a.groups / kWarps;
  bool ok = true;
  __syncthreads();
  for (int t = 0; t < a.steps; ++t) {
    float pre[4] = {0.f, 0.f, 0.f, 0.f};
    if (active && part == 0) {
      const float* q = a.pre + ((int64_t)t * a.batch + row) * 4 * H + unit;
#pragma unroll
      for (int g = 0; g < 4; ++g) pre[g] = __ldg(q + (int64_t)g * H);
    }
    float acc[UL][4][4] = {};
    if (t > 0 || a.h0) {
      for (int q = q_begin; q < q_end; q += 2) {
        uint4 v[2 * NL] = {};
        int at[2 * NL];
        const uint4* from[2 * NL];
        bool want[2 * NL];
#pragma unroll
        for (int j = 0; j < 2 * NL; ++j) {
          const int piece = j % NL * 32 + lane, r = piece / (U / 2), pair = piece % (U / 2);
          want[j] = q + j / NL < q_end;
          at[j] = (j / NL * U + 2 * pair) * kPitch + r;
          from[j] = a.mail + (((int64_t)((t - 1) & 1) * gridDim.x + first_block + q + j / NL) * kRows + r) * (U / 2) + pair;
          if (t == 0 && want[j] && row0 + r < a.batch) {
            const int k = (q + j / NL) * U + 2 * pair;
            const float* h = a.h0 + (int64_t)(row0 + r) * H + k;
            v[j].x = k < H ? __float_as_uint(__ldg(h)) : 0u;
            v[j].z = k + 1 < H ? __float_as_uint(__ldg(h + 1)) : 0u;
          }
        }
        if (t > 0 && ok) ok = receive(from, want, (uint32_t)t, v, a);
#pragma unroll
        for (int j = 0; j < 2 * NL; ++j) {
          stage[at[j]] = __uint_as_float(v[j].x);
          stage[at[j] + kPitch] = __uint_as_float(v[j].z);
        }
        __syncwarp();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (q + half >= q_end) break;
          const float4* w = smem4 + (q + half) * U * U + cg;
          const float* h = stage + half * U * kPitch + 4 * rg;
#pragma unroll 8
          for (int k = 0; k < U; ++k) {
            const float4 x = *reinterpret_cast<const float4*>(h + k * kPitch);
            const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int j = 0; j < UL; ++j) {
              const float4 y = w[k * U + 8 * j];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                acc[j][i][0] = fmaf(xs[i], y.x, acc[j][i][0]);
                acc[j][i][1] = fmaf(xs[i], y.y, acc[j][i][1]);
                acc[j][i][2] = fmaf(xs[i], y.z, acc[j][i][2]);
                acc[j][i][3] = fmaf(xs[i], y.w, acc[j][i][3]);
              }
            }
          }
        }
        __syncwarp();
      }
    }
#pragma unroll
    for (int j = 0; j < UL; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        regions[warp * kRegion + (4 * rg + i) * U + cg + 8 * j] = make_float4(acc[j][i][0], acc[j][i][1], acc[j][i][2], acc[j][i][3]);
    __syncthreads();
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < kWarps / P; ++i) {
      const float4 v = regions[(part * (kWarps / P) + i) * kRegion + warp * U + u];
      s[0] += v.x; s[1] += v.y; s[2] += v.z; s[3] += v.w;
    }
    __syncthreads();  // the regions may be written again
#pragma unroll
    for (int g = 0; g < 4; ++g) {
#pragma unroll
      for (int d = U; d < 32; d *= 2) s[g] += __shfl_xor_sync(0xffffffffu, s[g], d);
      s[g] += pre[g];
    }
    const float ig = sigmoid(s[0]), fg = sigmoid(s[1]), gg = tanhf(s[2]), og = sigmoid(s[3]);
    c = fg * c + ig * gg;
    const float tc = tanhf(c), h = og * tc;
    if (part == 0) {
      // the padding's h is never used: it meets weights of zero, and must therefore be finite
      if (t + 1 < a.steps)
        post(reinterpret_cast<uint2*>(a.mail) + (((int64_t)(t & 1) * gridDim.x + blockIdx.x) * kRows + warp) * U + u, active ? h : 0.f, (uint32_t)t + 1);
      if (active) {
        const int64_t e = t * per_step + cell;
        a.ig[e] = ig; a.fg[e] = fg; a.gg[e] = gg; a.og[e] = og; a.c[e] = c; a.tc[e] = tc; a.h[e] = h;
      }
    }
  }
}

template <int U>
__global__ void __launch_bounds__(kThreads, 1) lstm_sequence_backward_kernel(const SeqArgs a) {
  extern __shared__ float4 smem4[];
  constexpr int pairs = U / 2, at_once = 32 / pairs, N = 4;  // pieces of 16 bytes in a row's mail, sources that the lanes read at once
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rg = lane >> 3, cg = lane & 7;
  const int H = a.hidden, S = a.groups, group = blockIdx.x % S, rows = blockIdx.x / S, row0 = rows * kRows;
  const int pitch_w = (S * U + 31) / 32 * 32;
  float* const ws = reinterpret_cast<float*>(smem4);           // [gate * U + unit][unit of the gradient]
  float* const dgs = ws + 4 * U * pitch_w;                       // two turns of [gate * U + unit][row]
  for (int i = threadIdx.x; i < 4 * U * pitch_w; i += kThreads) {
    const int u = i % U, gate = i / U % 4, j = i / (4 * U), unit = group * U + u;
    ws[(gate * U + u) * pitch_w + j] = j < H && unit < H ? __ldg(a.w + (int64_t)j * a.ldw + (int64_t)gate * H + unit) : 0.f;
  }
  const int row = row0 + warp, u = lane % U, unit = group * U + u;
  const bool active = row < a.batch && unit < H;
  const int64_t cell = (int64_t)row * H + unit, per_step = (int64_t)a.batch * H;
  const int bands = (int)gridDim.x / S;
  // mail to block `dest` from block `src` of these rows
  auto box = [&](int turn, int dest, int src) { return a.mail + (((int64_t)(turn * bands + rows) * S + dest) * S + src) * kRows * pairs; };
  float dc = 0.f;
  bool ok = true;
  for (int step = 0; step <= a.steps; ++step) {
    const int t = a.steps - 1 - step;
    if (t < 0 && !a.dh0) break;
    float ig = 0.f, fg = 0.f, gg = 0.f, og = 0.f, tc = 0.f, before = 0.f, dh = 0.f;
    if (active && t >= 0) {
      const int64_t e = t * per_step + cell;
      ig = __ldg(a.ig + e); fg = __ldg(a.fg + e); gg = __ldg(a.gg + e); og = __ldg(a.og + e); tc = __ldg(a.tc + e); dh = __ldg(a.dh + e);
      before = t > 0 ? __ldg(a.c + e - per_step) : (a.c0 ? __ldg(a.c0 + cell) : 0.f);
    }
    if (step > 0) {
      float x = 0.f, y = 0.f;
      for (int s0 = 0; s0 < S; s0 += N * at_once) {
        uint4 v[N] = {};
        const uint4* from[N];
        bool want[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const int src = s0 + j * at_once + lane / pairs;
          want[j] = src < S;
          from[j] = box((step - 1) & 1, group, src) + warp * pairs + lane % pairs;
        }
        if (ok) ok = receive(from, want, (uint32_t)step, v, a);
#pragma unroll
        for (int j = 0; j < N; ++j)
          if (want[j]) {
            x += __uint_as_float(v[j].x);
            y += __uint_as_float(v[j].z);
          }
      }
#pragma unroll
      for (int d = pairs; d < 32; d *= 2) {
        x += __shfl_xor_sync(0xffffffffu, x, d);
        y += __shfl_xor_sync(0xffffffffu, y, d);
      }
      x = __shfl_sync(0xffffffffu, x, u / 2);
      y = __shfl_sync(0xffffffffu, y, u / 2);
      dh += u & 1 ? y : x;
    }
    if (t < 0) {
      if (active && lane < U) a.dh0[cell] = dh;
      break;
    }
    float* const turn = dgs + (step & 1) * 4 * U * kPitch;
    dc += dh * og * (1.f - tc * tc);
    const float d[4] = {dc * gg * ig * (1.f - ig), dc * before * fg * (1.f - fg), dc * ig * (1.f - gg * gg), dh * tc * og * (1.f - og)};
    dc *= fg;
    if (lane < U) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        turn[(g * U + u) * kPitch + warp] = active ? d[g] : 0.f;
        if (active) a.dgates[((int64_t)t * a.batch + row) * 4 * H + (int64_t)g * H + unit] = d[g];
      }
    }
    if (t == 0 && !a.dh0) break;
    __syncthreads();
    for (int j0 = warp * 32; j0 < pitch_w; j0 += kWarps * 32) {
      float acc[4][4] = {};
      const float *w = ws + j0 + 4 * cg, *x = turn + 4 * rg;
#pragma unroll 8
      for (int k = 0; k < 4 * U; ++k) {
        const float4 p = *reinterpret_cast<const float4*>(x + k * kPitch), q = *reinterpret_cast<const float4*>(w + k * pitch_w);
        const float xs[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[i][0] = fmaf(xs[i], q.x, acc[i][0]);
          acc[i][1] = fmaf(xs[i], q.y, acc[i][1]);
          acc[i][2] = fmaf(xs[i], q.z, acc[i][2]);
          acc[i][3] = fmaf(xs[i], q.w, acc[i][3]);
        }
      }
      const int j = j0 + 4 * cg, dest = j / U;
      if (dest < S) {
        uint4* to = box(step & 1, dest, group) + 4 * rg * pairs + j % U / 2;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          post2(to + i * pairs, acc[i][0], acc[i][1], (uint32_t)step + 1);
          post2(to + i * pairs + 1, acc[i][2], acc[i][3], (uint32_t)step + 1);
        }
      }
    }
  }
  if (a.dc0 && active && lane < U) a.dc0[cell] = dc;
}

// ---- a timestep at a time, for sizes that do not fit ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) lstm_step_kernel(const float* __restrict__ pre, const float* __restrict__ z, const float* __restrict__ before,
                                                        const SeqArgs a, int t) {
  RT_PDL_ENTRY();
  const int64_t n = (int64_t)a.batch * a.hidden, H = a.hidden;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < n; e += (int64_t)gridDim.x * 256) {
    const int64_t q = e / H * 4 * H + e % H;
    float s[4];
    for (int g = 0; g < 4; ++g) s[g] = __ldg(pre + q + g * H) + (z ? __ldg(z + q + g * H) : 0.f);
    const float ig = sigmoid(s[0]), fg = sigmoid(s[1]), gg = tanhf(s[2]), og = sigmoid(s[3]);
    const float c = fg * (before ? __ldg(before + e) : 0.f) + ig * gg, tc = tanhf(c);
    const int64_t o = t * n + e;
    a.ig[o] = ig; a.fg[o] = fg; a.gg[o] = gg; a.og[o] = og; a.c[o] = c; a.tc[o] = tc; a.h[o] = og * tc;
  }
}
__global__ void __launch_bounds__(256) lstm_step_backward_kernel(const SeqArgs a, int t, const float* __restrict__ from_next, const float* dc_next,
                                                                 float* dc) {
  RT_PDL_ENTRY();
  const int64_t n = (int64_t)a.batch * a.hidden, H = a.hidden;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < n; e += (int64_t)gridDim.x * 256) {
    const int64_t o = t * n + e;
    const float ig = a.ig[o], fg = a.fg[o], gg = a.gg[o], og = a.og[o], tc = a.tc[o], before = t > 0 ? a.c[o - n] : (a.c0 ? a.c0[e] : 0.f);
    const float dh = __ldg(a.dh + o) + (from_next ? from_next[e] : 0.f), d = (dc_next ? dc_next[e] : 0.f) + dh * og * (1.f - tc * tc);
    float* q = a.dgates + t * 4 * n + e / H * 4 * H + e % H;
    q[0] = d * gg * ig * (1.f - ig);
    q[H] = d * before * fg * (1.f - fg);
    q[2 * H] = d * ig * (1.f - gg * gg);
    q[3 * H] = dh * tc * og * (1.f - og);
    dc[e] = d * fg;
  }
}

// Units a block: as few as give every block an SM of its own and its slice of the weights room.  0: they do not fit.
struct Fit {
  int units = 0, groups = 0, blocks = 0;
  size_t smem = 0;
};
Fit fit(const rt_ctx* ctx, int64_t batch, int64_t hidden, bool backward) {
  if (batch > 1 << 20 || hidden > 1 << 20) return {};
  for (int u = 8; u <= 16; u += 8) {
    Fit f;
    f.units = u;
    f.groups = (int)((hidden + u - 1) / u);
    const int64_t blocks = (batch + kRows - 1) / kRows * f.groups;
    const size_t pitch_w = ((size_t)f.groups * u + 31) / 32 * 32;
    f.smem = backward ? sizeof(float) * 4 * u * (pitch_w + 2 * kPitch)
                      : 16 * ((size_t)f.groups * u * u + kWarps * kRows * u);
    f.blocks = (int)blocks;
    if (blocks <= ctx->sm_count && f.smem <= 232448) return f;
  }
  return {};
}
rt_status launch_together(rt_ctx* ctx, void (*kern)(SeqArgs), RtDeviceOnce& once, const Fit& f, const SeqArgs& a) {
  RT_CUDA(ctx, once([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448); }));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = f.blocks;
  cfg.blockDim = kThreads;
  cfg.dynamicSmemBytes = f.smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  RT_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, a));
  RT_LAUNCHED(ctx);
  return RT_OK;
}
// `mail`: 8 bytes a value and a word for giving up, cleared.
rt_status clear_mail(rt_ctx* ctx, RtScratch* mem, size_t values, SeqArgs* a) {
  const size_t bytes = 8 * values + 16;
  rt_status st = mem->alloc(bytes);
  if (st != RT_OK) return st;
  RT_CUDA(ctx, cudaMemsetAsync(mem->ptr, 0, bytes, ctx->stream));
  a->mail = mem->as<uint4>();
  a->gave_up = reinterpret_cast<int*>(mem->as<char>() + 8 * values);
  return RT_OK;
}
rt_status check_sizes(rt_ctx* ctx, const char* name, int64_t steps, int64_t batch, int64_t hidden, int64_t ldw) {
  if (steps <= 0 || batch <= 0 || hidden <= 0 || steps >= (1 << 30)) RT_FAIL(ctx, RT_ERR_INVALID_INDEX, "%s: extents must be positive", name);
  if (ldw < 4 * hidden) RT_FAIL(ctx, RT_ERR_SHAPE_MISMATCH, "%s: leading dimension smaller than the row length", name);
  return RT_OK;
}
void set_saved(SeqArgs* a, const float* saved, int64_t plane) {
  float** p[6] = {&a->ig, &a->fg, &a->gg, &a->og, &a->c, &a->tc};
  for (int i = 0; i < 6; ++i) *p[i] = const_cast<float*>(saved) + i * plane;
}

}  // namespace

extern "C" {

rt_status rt_lstm_sequence(rt_ctx* ctx, const float* pre, const float* w, int64_t ldw, const float* h0, const float* c0, int64_t steps, int64_t batch,
                           int64_t hidden, float* saved, float* h) {
  RT_CHECK_CTX(ctx);
  rt_status st = check_sizes(ctx, "rt_lstm_sequence", steps, batch, hidden, ldw);
  if (st != RT_OK) return st;
  RT_CHECK_PTR(ctx, pre);
  RT_CHECK_PTR(ctx, w);
  RT_CHECK_PTR(ctx, saved);
  RT_CHECK_PTR(ctx, h);
  const int64_t n = batch * hidden;
  SeqArgs a{};
  a.steps = (int)steps;
  a.batch = (int)batch;
  a.hidden = (int)hidden;
  a.w = w;
  a.ldw = ldw;
  a.pre = pre;
  a.h0 = h0;
  a.c0 = c0;
  a.h = h;
  a.status = ctx->device_status;
  set_saved(&a, saved, steps * n);
  ctx->fused_compiled += 2 * steps;
  const Fit f = fit(ctx, batch, hidden, false);
  if (f.units) {
    a.groups = f.groups;
    RtScratch mail(ctx);
    if ((st = clear_mail(ctx, &mail, (size_t)2 * f.blocks * kRows * f.units, &a)) != RT_OK) return st;
    static RtDeviceOnce once8, once16;
    return f.units == 8 ? launch_together(ctx, lstm_sequence_kernel<8>, once8, f, a) : launch_together(ctx, lstm_sequence_kernel<16>, once16, f, a);
  }
  RtScratch z(ctx);
  if ((st = z.alloc(sizeof(float) * (size_t)(4 * n))) != RT_OK) return st;
  for (int64_t t = 0; t < steps; ++t) {
    const float* hp = t > 0 ? h + (t - 1) * n : h0;
    if (hp && (st = rt_gemm(ctx, 0, 0, batch, 4 * hidden, hidden, hp, hidden, w, ldw, z.as<float>(), 4 * hidden, 0)) != RT_OK) return st;
    rt_launch(ctx, lstm_step_kernel, rt_grid_for(ctx, n, 256), 256, 0, pre + t * 4 * n, hp ? z.as<float>() : nullptr,
              t > 0 ? a.c + (t - 1) * n : c0, a, (int)t);
    RT_LAUNCHED(ctx);
  }
  return RT_OK;
}

rt_status rt_lstm_sequence_backward(rt_ctx* ctx, const float* saved, const float* w, int64_t ldw, const float* c0, const float* dh, int64_t steps,
                                    int64_t batch, int64_t hidden, float* dgates, float* dh0, float* dc0) {
  RT_CHECK_CTX(ctx);
  rt_status st = check_sizes(ctx, "rt_lstm_sequence_backward", steps, batch, hidden, ldw);
  if (st != RT_OK) return st;
  RT_CHECK_PTR(ctx, saved);
  RT_CHECK_PTR(ctx, w);
  RT_CHECK_PTR(ctx, dh);
  RT_CHECK_PTR(ctx, dgates);
  const int64_t n = batch * hidden;
  SeqArgs a{};
  a.steps = (int)steps;
  a.batch = (int)batch;
  a.hidden = (int)hidden;
  a.w = w;
  a.ldw = ldw;
  a.c0 = c0;
  a.dh = dh;
  a.dgates = dgates;
  a.dh0 = dh0;
  a.dc0 = dc0;
  a.status = ctx->device_status;
  set_saved(&a, saved, steps * n);
  ctx->fused_compiled += 2 * steps;
  const Fit f = fit(ctx, batch, hidden, true);
  if (f.units) {
    a.groups = f.groups;
    RtScratch mail(ctx);
    if ((st = clear_mail(ctx, &mail, (size_t)2 * f.blocks * f.groups * kRows * f.units, &a)) != RT_OK) return st;
    static RtDeviceOnce once8, once16;
    return f.units == 8 ? launch_together(ctx, lstm_sequence_backward_kernel<8>, once8, f, a)
                        : launch_together(ctx, lstm_sequence_backward_kernel<16>, once16, f, a);
  }
  RtScratch rec(ctx), dc(ctx);
  if ((st = rec.alloc(sizeof(float) * (size_t)n)) != RT_OK || (st = dc.alloc(sizeof(float) * (size_t)n)) != RT_OK) return st;
  for (int64_t t = steps - 1; t >= 0; --t) {
    const bool last = t == steps - 1;
    rt_launch(ctx, lstm_step_backward_kernel, rt_grid_for(ctx, n, 256), 256, 0, a, (int)t, last ? nullptr : rec.as<float>(), last ? nullptr : dc.as<float>(),
              t == 0 && dc0 ? dc0 : dc.as<float>());
    RT_LAUNCHED(ctx);
    if (t == 0 && !dh0) break;
    st = rt_gemm(ctx, 0, 1, batch, hidden, 4 * hidden, dgates + t * 4 * n, 4 * hidden, w, ldw, t == 0 ? dh0 : rec.as<float>(), hidden, 0);
    if (st != RT_OK) return st;
  }
  return RT_OK;
}

}  // extern "C"
