// A whole LSTM sequence in one kernel, and its gradient in another.
//
// Timestep by timestep the recurrence is a product of [batch, H] x [H, 4H] and a few element operations, each a kernel that is over before
// it has started: 8 + 4 us of a timestep at batch 64, H 512, of which the arithmetic is two.  Here the kernel stays: every block keeps its
// slice of the recurrent weights in shared memory for the whole sequence, and what the blocks tell one another per timestep is written to
// and polled in memory, the value and what tells its timestep in one element of 4 or 8 bytes, so that seeing the one is having the other: no
// barrier.  (A vector access is one access per element, in no order: value and number must not be two of them.)
//
// A block has 16 rows of the batch and U hidden units (all four gates of them).  Rows are independent of one another, so only the blocks
// of the same rows exchange anything.  Forward a block publishes h of its units and gathers everybody's (4 bytes a value): the 16 warps
// split the reduction and add up in shared memory.  Backward a block has the gate gradients of its own units and multiplies them with its
// slice (its columns of the weights) into a partial gradient of ALL units, which it sends to the blocks that own them (8 bytes a value):
// 64 KB in and out at H 512, where gathering the gate gradients would take twice that.  All sums are fp32 in a fixed order.
// Operands lie as pairs of reduction indices, even and odd sums apart, for two multiply-adds an instruction: that halves what the warps
// issue, though not the time of the multiply-adds themselves (36 cycles for 16 of these, 32 for 32 single ones).  A lane's results
// backward are 16 units apart, so that eight lanes write 128 bytes together.
// The blocks wait for one another, so they are launched cooperatively (all resident or an error).  Every wait is bounded; a block whose wait
// expires records a code in the status word and goes on without waiting.
//
// Bound by latency; at H 512 forward two of the 5.3 us are multiply-adds.  Measured, a timestep: batch 30, H 200: 2.3 us forward, 3.0
// backward (2.4 and 3.9 before the pairs and the shorter mail); batch 64, H 512: 5.3 and 6.6 (5.4 and 7.9).  As kernels of their own the
// product, the cell and the concatenation took 9.7 forward, 12.3 backward at the first size.  Sizes whose blocks do not fit beside one
// another, or whose slice of the weights does not fit into a block, run timestep by timestep.
#include "packed_fma.cuh"
#include "rt_internal.cuh"
#include "tc_common.cuh"

namespace {

constexpr int kRows = 16, kWarps = 16, kThreads = kWarps * 32;
constexpr int kPitch = 36;  // words between the 16 rows' values of two reduction indices and those of the next two: 16-byte aligned, few bank conflicts

struct SeqArgs {
  int steps, batch, hidden, groups;  // groups of U units
  const float* w;                    // [hidden][4 * hidden], rows ldw apart
  int64_t ldw;
  const float* c0;
  uint4* mail;                       // zeroed before the launch
  int* gave_up;                      // zeroed before the launch
  int* status;
  uint32_t polls;
  // forward: the part of the gates' inputs that does not depend on h; activated gates, cell, its hyperbolic tangent and the output,
  // each [steps * batch][hidden]
  const float *pre, *h0;
  float *ig, *fg, *gg, *og, *c, *tc, *h;
  // backward
  const float* dh;
  float *dgates, *dh0, *dc0;
};

// Forward mail: four values, each with its turn.
__device__ __forceinline__ uint4 peek(const uint4* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
// Backward mail: two elements of {value, number of the timestep}.  (848 us for 128 timesteps at batch 64, H 512; as four elements of 32 bits, which
// would say nothing about their order, 840.)
__device__ __forceinline__ uint4 peek2(const uint4* p) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .b64 a, b;\n\t"
      "ld.relaxed.gpu.global.v2.b64 {a, b}, [%4];\n\t"
      "mov.b64 {%0, %1}, a;\n\t"
      "mov.b64 {%2, %3}, b;\n\t}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p)
      : "memory");
  return v;
}
__device__ __forceinline__ void post2(uint4* p, float v, float w, uint32_t tag) {
  asm volatile(
      "{\n\t.reg .b64 a, b;\n\t"
      "mov.b64 a, {%1, %3};\n\t"
      "mov.b64 b, {%2, %3};\n\t"
      "st.relaxed.gpu.global.v2.b64 [%0], {a, b};\n\t}" ::"l"(p),
      "r"(__float_as_uint(v)), "r"(__float_as_uint(w)), "r"(tag)
      : "memory");
}
// Two multiply-adds in one instruction: what the accumulators hold apart are the sums over the even and over the odd reduction indices.
struct Pair {
  unsigned long long v = 0;
  __device__ __forceinline__ float sum() const {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a + b;
  }
};
__device__ __forceinline__ ulonglong2 pairs_at(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + expf(-x)); }

// Forward a value carries the number of its timestep in one bit: h lies within [-1, 1], whose floats leave bit 30 zero, and a place is
// written every second timestep, so that the bit need only tell a message from the one before it.  NaN goes as a number that h cannot be.
// (With the number beside the value, twice the bytes to poll: 5.5 us a timestep at batch 64, H 512.)
constexpr uint32_t kTurnBit = 1u << 30, kNanCode = 0x3fffffffu;
__device__ __forceinline__ uint32_t turn_bit(int t) { return (t >> 1) & 1 ? 0u : kTurnBit; }  // memory starts as zeros
__device__ __forceinline__ void post_output(uint32_t* p, float h, uint32_t bit) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"((h == h ? __float_as_uint(h) : kNanCode) | bit) : "memory");
}
__device__ __forceinline__ uint32_t output_of(uint32_t v) {
  v &= ~kTurnBit;
  return v == kNanCode ? 0x7fc00000u : v;
}

// Waits until the wanted ones of N pieces of mail, STRIDE apart, have arrived.  False: the wait ran out, here or in another block.  (Polling
// one piece until it is there and only then the others is a round trip more: 693 -> 714 us for 128 timesteps at batch 64, H 512.)
template <int STRIDE, int N, class Peek, class Arrived>
__device__ __forceinline__ bool receive(const uint4* from, bool (&want)[N], uint4 (&v)[N], const SeqArgs& a, const Peek& look, const Arrived& arrived) {
  for (uint32_t i = 0; i < a.polls; ++i) {
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (want[j]) v[j] = look(from + j * STRIDE);
    bool there = true;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      want[j] = want[j] && !arrived(v[j]);
      there = there && !want[j];
    }
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
  static_assert(U * kPitch * 4 <= kRegion * 16, "region");
  constexpr int UL = U / 8, P = 32 / U, NL = U / 8, quads = U / 4;  // quads: 16-byte pieces of a row's mail
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rg = lane >> 3, cg = lane & 7;
  const int H = a.hidden, group = blockIdx.x % a.groups, row0 = blockIdx.x / a.groups * kRows;
  const int first_block = blockIdx.x - group, padded = a.groups * U;
  float4* const regions = smem4 + padded * U;
  float* const stage = reinterpret_cast<float*>(regions + warp * kRegion);
  for (int i = threadIdx.x; i < padded * U; i += kThreads) {  // [pair of reduction indices][pair of gates][unit]: gate, index within the pairs
    const int pair = i / (2 * U), gate = i / U % 2 * 2, unit = group * U + i % U;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (2 * pair < H && unit < H) {
      const float* q = a.w + (int64_t)(2 * pair) * a.ldw + (int64_t)gate * H + unit;
      v.x = __ldg(q);
      v.z = __ldg(q + H);
      if (2 * pair + 1 < H) {
        v.y = __ldg(q + a.ldw);
        v.w = __ldg(q + a.ldw + H);
      }
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
    Pair acc[UL][4][4];
    if (t > 0 || a.h0) {
      for (int q = q_begin; q < q_end; q += 2) {
        // piece j of the lane: rows of U / 4 pieces, sources of 16 rows, all one after the other
        uint4 v[2 * NL] = {};
        bool want[2 * NL];
        const int quad = lane % quads, r0 = lane / quads;
#pragma unroll
        for (int j = 0; j < 2 * NL; ++j) want[j] = j < NL || q + 1 < q_end;
        if (t > 0) {
          const uint32_t bit = turn_bit(t - 1);
          const uint4* from = a.mail + ((int64_t)((t - 1) & 1) * gridDim.x + first_block + q) * kRows * quads + lane;
          if (ok)
            ok = receive<32>(from, want, v, a, peek, [bit](const uint4& m) { return (((m.x ^ bit) | (m.y ^ bit) | (m.z ^ bit) | (m.w ^ bit)) & kTurnBit) == 0; });
#pragma unroll
          for (int j = 0; j < 2 * NL; ++j) v[j] = make_uint4(output_of(v[j].x), output_of(v[j].y), output_of(v[j].z), output_of(v[j].w));
        } else {
#pragma unroll
          for (int j = 0; j < 2 * NL; ++j) {
            const int r = j % NL * (128 / U) + r0, k = (q + j / NL) * U + 4 * quad;
            const float* h = a.h0 + (int64_t)(row0 + r) * H + k;
            if (want[j] && row0 + r < a.batch) {
              v[j].x = k < H ? __float_as_uint(__ldg(h)) : 0u;
              v[j].y = k + 1 < H ? __float_as_uint(__ldg(h + 1)) : 0u;
              v[j].z = k + 2 < H ? __float_as_uint(__ldg(h + 2)) : 0u;
              v[j].w = k + 3 < H ? __float_as_uint(__ldg(h + 3)) : 0u;
            }
          }
        }
        float* const to = stage + 2 * quad * kPitch + 2 * r0;
#pragma unroll
        for (int j = 0; j < 2 * NL; ++j) {
          float* const o = to + j / NL * (U / 2) * kPitch + j % NL * (256 / U);
          *reinterpret_cast<uint2*>(o) = make_uint2(v[j].x, v[j].y);
          *reinterpret_cast<uint2*>(o + kPitch) = make_uint2(v[j].z, v[j].w);
        }
        __syncwarp();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (q + half >= q_end) break;
          const float* w = reinterpret_cast<const float*>(smem4 + (q + half) * U * U + cg);
          const float* h = stage + half * (U / 2) * kPitch + 8 * rg;
#pragma unroll 4
          for (int k = 0; k < U / 2; ++k) {
            const ulonglong2 x01 = pairs_at(h + k * kPitch), x23 = pairs_at(h + k * kPitch + 4);
            const unsigned long long xs[4] = {x01.x, x01.y, x23.x, x23.y};
#pragma unroll
            for (int j = 0; j < UL; ++j) {
              const ulonglong2 y01 = pairs_at(w + (k * 2 * U + 8 * j) * 4), y23 = pairs_at(w + (k * 2 * U + U + 8 * j) * 4);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                fma2(acc[j][i][0].v, xs[i], y01.x);
                fma2(acc[j][i][1].v, xs[i], y01.y);
                fma2(acc[j][i][2].v, xs[i], y23.x);
                fma2(acc[j][i][3].v, xs[i], y23.y);
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
        regions[warp * kRegion + (4 * rg + i) * U + cg + 8 * j] = make_float4(acc[j][i][0].sum(), acc[j][i][1].sum(), acc[j][i][2].sum(), acc[j][i][3].sum());
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
        post_output(reinterpret_cast<uint32_t*>(a.mail) + (((int64_t)(t & 1) * gridDim.x + blockIdx.x) * kRows + warp) * U + u, active ? h : 0.f, turn_bit(t));
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
  float* const ws = reinterpret_cast<float*>(smem4);           // [pair of gate * U + unit][unit of the gradient][index within the pair]
  float* const dgs = ws + 4 * U * pitch_w;                       // two turns of [pair of gate * U + unit][row][index within the pair]
  for (int i = threadIdx.x; i < 4 * U * pitch_w; i += kThreads) {
    const int u = i % U, gate = i / U % 4, j = i / (4 * U), unit = group * U + u;
    ws[((gate * U + u) / 2 * pitch_w + j) * 2 + u % 2] = j < H && unit < H ? __ldg(a.w + (int64_t)j * a.ldw + (int64_t)gate * H + unit) : 0.f;
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
        bool want[N];
#pragma unroll
        for (int j = 0; j < N; ++j) want[j] = s0 + j * at_once + lane / pairs < S;
        const uint4* from = box((step - 1) & 1, group, s0 + lane / pairs) + warp * pairs + lane % pairs;
        const uint32_t tag = (uint32_t)step;
        if (ok) ok = receive<at_once * kRows * pairs>(from, want, v, a, peek2, [tag](const uint4& m) { return m.y == tag && m.w == tag; });
#pragma unroll
        for (int j = 0; j < N; ++j) {  // zeros where there is no source
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
    float* const turn = dgs + (step & 1) * 2 * U * kPitch;
    dc += dh * og * (1.f - tc * tc);
    const float d[4] = {dc * gg * ig * (1.f - ig), dc * before * fg * (1.f - fg), dc * ig * (1.f - gg * gg), dh * tc * og * (1.f - og)};
    dc *= fg;
    if (lane < U) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        turn[(g * U + u) / 2 * kPitch + 2 * warp + u % 2] = active ? d[g] : 0.f;
        if (active) a.dgates[((int64_t)t * a.batch + row) * 4 * H + (int64_t)g * H + unit] = d[g];
      }
    }
    if (t == 0 && !a.dh0) break;
    __syncthreads();
    for (int j0 = warp * 32; j0 < pitch_w; j0 += kWarps * 32) {
      // a lane has four rows and the units j0 + 2 cg, j0 + 16 + 2 cg and those after them
      Pair acc[4][4];
      const float *w = ws + (j0 + 2 * cg) * 2, *x = turn + 8 * rg;
#pragma unroll 4
      for (int k = 0; k < 2 * U; ++k) {
        const ulonglong2 p01 = pairs_at(x + k * kPitch), p23 = pairs_at(x + k * kPitch + 4);
        const ulonglong2 q01 = pairs_at(w + k * 2 * pitch_w), q23 = pairs_at(w + k * 2 * pitch_w + 32);
        const unsigned long long xs[4] = {p01.x, p01.y, p23.x, p23.y};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          fma2(acc[i][0].v, xs[i], q01.x);
          fma2(acc[i][1].v, xs[i], q01.y);
          fma2(acc[i][2].v, xs[i], q23.x);
          fma2(acc[i][3].v, xs[i], q23.y);
        }
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int j = j0 + 16 * half + 2 * cg, dest = j / U;
        if (dest < S) {
          uint4* to = box(step & 1, dest, group) + 4 * rg * pairs + j % U / 2;
#pragma unroll
          for (int i = 0; i < 4; ++i) post2(to + i * pairs, acc[i][2 * half].sum(), acc[i][2 * half + 1].sum(), (uint32_t)step + 1);
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
    f.smem = backward ? sizeof(float) * 4 * u * (pitch_w + kPitch)
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
// `mail` and a word for giving up, cleared.
rt_status clear_mail(rt_ctx* ctx, RtScratch* mem, size_t mail, SeqArgs* a) {
  const size_t bytes = mail + 16;
  rt_status st = mem->alloc(bytes);
  if (st != RT_OK) return st;
  RT_CUDA(ctx, cudaMemsetAsync(mem->ptr, 0, bytes, ctx->stream));
  a->mail = mem->as<uint4>();
  a->gave_up = reinterpret_cast<int*>(mem->as<char>() + mail);
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

rt_status rt_lstm_sequence_polls(rt_ctx* ctx, int64_t polls) {
  RT_CHECK_CTX(ctx);
  if (polls > UINT32_MAX) RT_FAIL(ctx, RT_ERR_INVALID_INDEX, "rt_lstm_sequence_polls: 2^32 and more");
  ctx->sequence_polls = polls < 0 ? rt_ctx().sequence_polls : (uint32_t)polls;
  return RT_OK;
}

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
  a.polls = ctx->sequence_polls;
  set_saved(&a, saved, steps * n);
  const Fit f = fit(ctx, batch, hidden, false);
  if (f.units) {
    a.groups = f.groups;
    RtScratch mail(ctx);
    if ((st = clear_mail(ctx, &mail, (size_t)2 * f.blocks * kRows * f.units * 4, &a)) != RT_OK) return st;
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
  a.polls = ctx->sequence_polls;
  set_saved(&a, saved, steps * n);
  const Fit f = fit(ctx, batch, hidden, true);
  if (f.units) {
    a.groups = f.groups;
    RtScratch mail(ctx);
    if ((st = clear_mail(ctx, &mail, (size_t)2 * f.blocks * f.groups * kRows * f.units * 8, &a)) != RT_OK) return st;
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
