// Elementwise programs as straight-line kernels.
//
// The interpreter pays 0.16 us per instruction on a small tensor (decoding is a chain of dependent branches) and as much again as
// the arithmetic on a large one.  The chains that the networks of host/models.hpp and plain layers (bias, activation, their
// gradients, a mean squared error, the LSTM cell) consist of are therefore listed in fused_programs_*.inc and compiled: the same
// instruction words as template arguments, registers and operand numbers become constants, immediates and shapes stay run-time.
// An unlisted program is interpreted, with the same results: a program is found by its instructions, so a user's expression with one
// op more or in another form is not (rt_fused_launch_counts tells).  Those of the LSTM written op by op serve steps that are not captured (in a
// capture its timesteps are one sequence, k_lstm_seq.cu); there the first and last timesteps are interpreted.
//
// Measured, kernel time inside a graph: the gate gradient of the LSTM cell (30 instructions, 12 operands, 4 windows) on [64, 2048]
// 12.5 us interpreted, 4.2 us compiled; an elementwise gradient with four transcendentals on [4096, 4096] 300 us interpreted, 77 us
// compiled (its 268 MB take 41 us at the copy bandwidth: bound by instruction issue, as everything here that has more than two or three
// transcendentals an element is).  Issue slots that a warp takes for one: exp 9, tanh 19, sin 27, cos 29, both by sincosf 34, 1/x 14, x/y 15.
#pragma once
#define RT_FUSED_EXPAND_MATH
#include "fused_common.cuh"

namespace {

using namespace fused;

// Four elements of the iteration space: consecutive ones (VEC) or ones THREADS apart.
template <bool VEC>
struct Quad {
  static constexpr int G = VEC ? 1 : 4;
  uint32_t at[G];
  int c0[G], c1[G];  // coordinates; c1 runs fastest
  bool live[G];
};

template <bool VEC>
__device__ __forceinline__ bool inside(const FusedParams& p, int region, const Quad<VEC>& e, int g) {
  const rt_fused_region& r = p.region[region];
  if (p.nd == 1) return e.c1[g] >= r.lo[0] && e.c1[g] < r.hi[0];
  return e.c0[g] >= r.lo[0] && e.c0[g] < r.hi[0] && e.c1[g] >= r.lo[1] && e.c1[g] < r.hi[1];
}

template <int K, bool VEC>
__device__ __forceinline__ void load_operand(const FusedParams& p, const Quad<VEC>& e, float (&v)[4]) {
  const rt_fused_operand& o = p.operand[K];
  const int s1 = o.stride[p.nd == 1 ? 0 : 1], s0 = p.nd == 1 ? 0 : o.stride[0];
#pragma unroll
  for (int g = 0; g < Quad<VEC>::G; ++g) {
    const bool ok = e.live[g] && (o.region == RT_FUSED_NONE || inside<VEC>(p, o.region, e, g));
    const float* q = o.ptr + (int64_t)(e.c0[g] * s0 + e.c1[g] * s1);
    if (VEC) {
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
      if (ok) {
        if (p.mode[K] == kVector) {
          t = __ldg(reinterpret_cast<const float4*>(q));
        } else if (s1 == 0) {
          const float s = __ldg(q);
          t = make_float4(s, s, s, s);
        } else {
          t = make_float4(__ldg(q), __ldg(q + s1), __ldg(q + 2 * s1), __ldg(q + 3 * s1));
        }
      }
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
      v[g] = ok ? __ldg(q) : 0.f;
    }
  }
}

template <int OP>
__device__ __forceinline__ float apply_one(float x, float y, float imm) {
#define RT_CASE(code, expr) \
  if constexpr (OP == code) return (expr);
  RT_FUSED_OPS(RT_CASE)
#undef RT_CASE
  return x;
}

// What becomes of an output: it is written.
struct Store {
  template <int OUT, bool VEC>
  __device__ __forceinline__ void put(const FusedParams& p, const Quad<VEC>& e, const float (&acc)[4]) {
#pragma unroll
    for (int g = 0; g < Quad<VEC>::G; ++g)
      if (e.live[g]) {
        if constexpr (VEC) *reinterpret_cast<float4*>(p.out[OUT] + e.at[g]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        else p.out[OUT][e.at[g]] = acc[g];
      }
  }
};

// A sine and a cosine of one register's value, the earlier (first) and the later instruction: sincosf reduces the argument once for both (the
// program with column sums over [4096, 4096] that has them: 98 us apart, 88 us together, without a spill).
struct Pair {
  int first = -1, later = -1;
};
template <class P>
__host__ __device__ constexpr Pair find_pair() {
  auto op = [](int i) { return P::code[i] & 0xff; };
  for (int i = 1; i < P::n; ++i)
    for (int j = i + 2; j < P::n && op(i - 1) == RT_F_REG; ++j) {
      const uint32_t reg = (P::code[i - 1] >> 8) & 0xff;
      bool same = ((op(i) == RT_F_SIN && op(j) == RT_F_COS) || (op(i) == RT_F_COS && op(j) == RT_F_SIN)) && op(j - 1) == RT_F_REG &&
                  ((P::code[j - 1] >> 8) & 0xff) == reg;
      for (int k = i; k < j && same; ++k) same = ((P::code[k] >> 16) & 0xff) != reg;
      if (same) return {i, j};
    }
  return {};
}

template <class P, int PC, bool VEC, class Sink>
__device__ __forceinline__ void execute(const FusedParams& p, const Quad<VEC>& e, float (&r)[RT_FUSED_REGS][4], float (&other)[4], float (&acc)[4], Sink& sink) {
  if constexpr (PC < P::n) {
    constexpr uint32_t word = P::code[PC];
    constexpr int op = word & 0xff, src = (word >> 8) & 0xff, dst = (word >> 16) & 0xff, region = word >> 24;
    constexpr Pair pair = find_pair<P>();
    if constexpr (op == RT_F_LOAD) {
      load_operand<src, VEC>(p, e, acc);
    } else if constexpr (op == RT_F_OUT) {
      sink.template put<src, VEC>(p, e, acc);
    } else if constexpr (PC == pair.later) {
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] = other[i];
    } else if constexpr (PC == pair.first) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float x = acc[i];
        if constexpr (op == RT_F_SIN) sincosf(x, &acc[i], &other[i]);
        else sincosf(x, &other[i], &acc[i]);
      }
    } else {
      const float imm = __uint_as_float(p.code[PC].y);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float y;
        if constexpr (src == RT_FUSED_IMM) y = imm;
        else y = r[src][i];
        if constexpr (op == RT_F_SELECT) acc[i] = inside<VEC>(p, region, e, VEC ? 0 : i) ? acc[i] : y;
        else acc[i] = apply_one<op>(acc[i], y, imm);
      }
    }
    if constexpr (dst != RT_FUSED_NONE) {
#pragma unroll
      for (int i = 0; i < 4; ++i) r[dst][i] = acc[i];
    }
    execute<P, PC + 1, VEC>(p, e, r, other, acc, sink);
  }
}
// The program for four elements.
template <class P, bool VEC, class Sink>
__device__ __forceinline__ void run(const FusedParams& p, const Quad<VEC>& e, Sink& sink) {
  float r[RT_FUSED_REGS][4], other[4], acc[4];
  if constexpr (P::preload > 0) load_operand<0, VEC>(p, e, r[0]);
  if constexpr (P::preload > 1) load_operand<1, VEC>(p, e, r[1]);
  if constexpr (P::preload > 2) load_operand<2, VEC>(p, e, r[2]);
  if constexpr (P::preload > 3) load_operand<3, VEC>(p, e, r[3]);
  if constexpr (P::preload > 4) load_operand<4, VEC>(p, e, r[4]);
  execute<P, 0, VEC>(p, e, r, other, acc, sink);
}

constexpr int kKnownThreads = 128;
template <class P, bool VEC>
__global__ void __launch_bounds__(kKnownThreads) known_kernel(const __grid_constant__ FusedParams p) {
  RT_PDL_ENTRY();
  for (uint32_t tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
    Quad<VEC> e;
#pragma unroll
    for (int g = 0; g < Quad<VEC>::G; ++g) {
      e.at[g] = VEC ? (tile * kKnownThreads + threadIdx.x) * 4 : (tile * 4 + g) * kKnownThreads + threadIdx.x;
      e.live[g] = e.at[g] < p.numel;
      uint32_t q = 0, m = e.live[g] ? e.at[g] : 0;
      if (p.nd == 2) p.dim[1].divmod(m, q, m);
      e.c0[g] = (int)q;
      e.c1[g] = (int)m;
    }
    Store sink;
    run<P, VEC>(p, e, sink);
  }
}

template <class P>
rt_status launch_program(rt_ctx* ctx, FusedParams& p, bool vec, int64_t numel) {
  const int64_t tiles = (numel + kKnownThreads * 4 - 1) / (kKnownThreads * 4), cap = (int64_t)ctx->sm_count * 32;
  p.tiles = (uint32_t)tiles;
  const unsigned grid = (unsigned)(tiles < cap ? tiles : cap);
  if (vec) rt_launch(ctx, known_kernel<P, true>, grid, kKnownThreads, 0, p);
  else rt_launch(ctx, known_kernel<P, false>, grid, kKnownThreads, 0, p);
  RT_LAUNCHED(ctx);
  return RT_OK;
}

template <int PRELOAD, uint32_t... WORDS>
struct Program {
  static constexpr int n = sizeof...(WORDS), preload = PRELOAD;
  static constexpr uint32_t code[sizeof...(WORDS)] = {WORDS...};
  static constexpr KnownProgram entry{code, n, preload, &launch_program<Program>};
};

// I(op, source register / operand / output, register written or X, region); X: none, C: the immediate
constexpr uint32_t X = RT_FUSED_NONE, C = RT_FUSED_IMM;
#define I(op, src, dst, region) (uint32_t(op) | uint32_t(src) << 8 | uint32_t(dst) << 16 | uint32_t(region) << 24)

}  // namespace
