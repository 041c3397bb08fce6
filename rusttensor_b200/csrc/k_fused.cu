// rt_fused_elementwise: a whole chain of elementwise ops in one launch.
//
// The ops of a model arrive one by one; launched one by one each of them costs a kernel (1.3 - 2 us inside a graph whatever its
// size) and a pass over memory for its operands and its result.  Here the host hands over the chain as a short program and the
// kernel runs it.  Programs that are listed in fused_programs_*.inc are kernels of their own (fused_known.cuh); all others are
// interpreted by the kernel below: the instruction words are copied to shared memory, one switch decodes an instruction, which works
// on V elements of the thread.
//
// What bounds it: instruction decoding, a chain of dependent branches of about 300 cycles per instruction.  Measured, time in a
// graph: 2.3 us + 0.16 us per instruction for [64, 2048]; on [4096, 4096] 5.6 us per instruction (a separate kernel per op takes 25 us
// there).  The register file is shared memory (naming a register is then an address, not a branch: with a file of registers behind
// switches an instruction cost 0.28 us).  Operands 0..4 are loaded before the first instruction so that their latencies overlap.
#include <cmath>
#include <cstring>
#include <unordered_map>

#include "fused_common.cuh"

namespace {

using namespace fused;

// Elements of one thread: V of them in G groups; a group is 4 consecutive elements (VEC) or a single one.
template <int V, bool VEC>
struct Elements {
  static constexpr int G = VEC ? V / 4 : V;
  uint32_t at[G];                        // linear index of the group's first element
  uint32_t c[RT_FUSED_MAX_DIMS][G];      // its coordinates
  bool live[G];
};

template <int V, bool VEC>
__device__ __forceinline__ bool in_box(const FusedParams& p, int region, const Elements<V, VEC>& e, int g, int j) {
  const rt_fused_region& r = p.region[region];
  bool in = true;
#pragma unroll
  for (int d = 0; d < RT_FUSED_MAX_DIMS; ++d) {
    if (d < p.nd) {
      const int c = (int)e.c[d][g] + (d == p.nd - 1 ? j : 0);
      in = in && c >= r.lo[d] && c < r.hi[d];
    }
  }
  return in;
}

template <int V, bool VEC>
__device__ __forceinline__ void load_operand(const FusedParams& p, int k, const Elements<V, VEC>& e, float (&v)[V]) {
  const rt_fused_operand& o = p.operand[k];
  const int mode = p.mode[k], region = o.region;
  if (mode == kSame && region == RT_FUSED_NONE) {
    const float s = __ldg(o.ptr);
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = s;
    return;
  }
#pragma unroll
  for (int g = 0; g < Elements<V, VEC>::G; ++g) {
    int64_t off = 0;
    int inner = 0;
#pragma unroll
    for (int d = 0; d < RT_FUSED_MAX_DIMS; ++d)
      if (d < p.nd) {
        off += (int64_t)(int)e.c[d][g] * o.stride[d];
        if (VEC && d == p.nd - 1) inner = o.stride[d];
      }
    const float* q = o.ptr + off;
    if (VEC) {
      if (mode == kScalar || region != RT_FUSED_NONE) {
        // a vector that lies inside the box as a whole is still one load
        const bool first = e.live[g] && (region == RT_FUSED_NONE || in_box<V, VEC>(p, region, e, g, 0));
        if (mode == kVector && first && in_box<V, VEC>(p, region, e, g, 3)) {
          const float4 t = __ldg(reinterpret_cast<const float4*>(q));
          v[4 * g] = t.x; v[4 * g + 1] = t.y; v[4 * g + 2] = t.z; v[4 * g + 3] = t.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const bool ok = e.live[g] && (region == RT_FUSED_NONE || in_box<V, VEC>(p, region, e, g, j));
            v[4 * g + j] = ok ? __ldg(q + j * inner) : 0.f;
          }
        }
      } else if (mode == kVector) {
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e.live[g]) t = __ldg(reinterpret_cast<const float4*>(q));
        v[4 * g] = t.x; v[4 * g + 1] = t.y; v[4 * g + 2] = t.z; v[4 * g + 3] = t.w;
      } else {
        const float s = e.live[g] ? __ldg(q) : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) v[4 * g + j] = s;
      }
    } else {
      const bool ok = e.live[g] && (region == RT_FUSED_NONE || in_box<V, VEC>(p, region, e, g, 0));
      v[g] = ok ? __ldg(q) : 0.f;
    }
  }
}

// acc = op(acc, b), one switch for everything.
template <int V>
__device__ __forceinline__ void apply(int op, float imm, const float (&b)[V], float (&acc)[V]) {
  switch (op) {
#define RT_CASE(code, expr)                           \
  case code:                                          \
    _Pragma("unroll") for (int i = 0; i < V; ++i) {   \
      const float x = acc[i], y = b[i];               \
      acc[i] = (expr);                                \
    }                                                 \
    break;
    RT_FUSED_OPS(RT_CASE)
#undef RT_CASE
    default: break;
  }
}

// The register file is shared memory, so that naming a register is an address and not a branch: [register][quad][thread] of
// float4, each thread's own slots, conflict free.
template <int V, int THREADS>
struct Registers {
  static constexpr int kStride = V / 4 * THREADS;  // float4s of one register
  float4* base;
  __device__ __forceinline__ void read(int k, float (&v)[V]) const {
#pragma unroll
    for (int i = 0; i < V / 4; ++i) {
      const float4 t = base[k * kStride + i * THREADS];
      v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
    }
  }
  __device__ __forceinline__ void write(int k, const float (&v)[V]) const {
#pragma unroll
    for (int i = 0; i < V / 4; ++i) base[k * kStride + i * THREADS] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  }
};

template <int V, bool VEC, int THREADS, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS) fused_kernel(const __grid_constant__ FusedParams p) {
  using E = Elements<V, VEC>;
  extern __shared__ float4 file[];
  __shared__ uint2 code[RT_FUSED_MAX_CODE + 1];
  RT_PDL_ENTRY();
  for (int i = threadIdx.x; i < p.n_code; i += THREADS) code[i] = p.code[i];
  __syncthreads();
  const Registers<V, THREADS> r{file + threadIdx.x};
  for (uint32_t tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
    E e;
#pragma unroll
    for (int g = 0; g < E::G; ++g) {
      const uint32_t unit = (tile * E::G + g) * THREADS + threadIdx.x;
      e.at[g] = VEC ? unit * 4 : unit;
      e.live[g] = e.at[g] < p.numel;
      uint32_t rest = e.live[g] ? e.at[g] : 0;
#pragma unroll
      for (int d = RT_FUSED_MAX_DIMS - 1; d >= 0; --d) {
        e.c[d][g] = 0;
        if (d == 0) e.c[0][g] = rest;
        else if (d < p.nd) {
          uint32_t q, m;
          p.dim[d].divmod(rest, q, m);
          e.c[d][g] = m;
          rest = q;
        }
      }
    }
    float acc[V];
    {
      float first[RT_FUSED_PRELOAD][V];
#pragma unroll
      for (int k = 0; k < RT_FUSED_PRELOAD; ++k)
        if (k < p.n_preload) load_operand<V, VEC>(p, k, e, first[k]);
#pragma unroll
      for (int k = 0; k < RT_FUSED_PRELOAD; ++k)
        if (k < p.n_preload) r.write(k, first[k]);
    }
    uint2 word = code[0];
    for (int pc = 0; pc < p.n_code; ++pc) {
      const uint2 next = code[pc + 1];  // the entry behind the last one is never executed
      const int op = word.x & 0xff, src = (word.x >> 8) & 0xff, dst = (word.x >> 16) & 0xff, region = word.x >> 24;
      const float imm = __uint_as_float(word.y);
      if (op >= kPlain) {
        float b[V];
        const bool is_imm = src == RT_FUSED_IMM;
        r.read(is_imm ? 0 : src, b);
#pragma unroll
        for (int i = 0; i < V; ++i) b[i] = is_imm ? imm : b[i];
        apply<V>(op, imm, b, acc);
      } else if (op == RT_F_LOAD) {
        load_operand<V, VEC>(p, src, e, acc);
      } else if (op == RT_F_OUT) {
        float* o = p.out[src];
#pragma unroll
        for (int g = 0; g < E::G; ++g)
          if (e.live[g]) {
            if (VEC) *reinterpret_cast<float4*>(o + e.at[g]) = make_float4(acc[VEC ? 4 * g : g], acc[VEC ? 4 * g + 1 : g], acc[VEC ? 4 * g + 2 : g], acc[VEC ? 4 * g + 3 : g]);
            else o[e.at[g]] = acc[g];
          }
      } else {  // RT_F_SELECT
        float b[V];
        const bool is_imm = src == RT_FUSED_IMM;
        r.read(is_imm ? 0 : src, b);
#pragma unroll
        for (int i = 0; i < V; ++i)
          acc[i] = in_box<V, VEC>(p, region, e, VEC ? i / 4 : i, VEC ? i % 4 : 0) ? acc[i] : (is_imm ? imm : b[i]);
      }
      if (dst != RT_FUSED_NONE) r.write(dst, acc);
      word = next;
    }
  }
}

template <int V, bool VEC, int THREADS, int BLOCKS>
rt_status launch_fused(rt_ctx* ctx, FusedParams& p, int64_t numel) {
  const int64_t per_block = (int64_t)V * THREADS, tiles = (numel + per_block - 1) / per_block;
  p.tiles = (uint32_t)tiles;
  const int64_t cap = (int64_t)ctx->sm_count * BLOCKS * 4;
  const size_t smem = (size_t)RT_FUSED_REGS * V * THREADS * sizeof(float);
  auto kern = fused_kernel<V, VEC, THREADS, BLOCKS>;
  static RtDeviceOnce once;
  RT_CUDA(ctx, once([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }));
  rt_launch(ctx, kern, (unsigned)(tiles < cap ? tiles : cap), THREADS, smem, p);
  RT_LAUNCHED(ctx);
  return RT_OK;
}

// The program compiled ahead of time that has these instructions, or null.
const KnownProgram* find_known(const FusedParams& p) {
  auto hash = [](const uint32_t* w, int n, int step) {
    uint64_t h = 1469598103934665603ull;
    for (int i = 0; i < n; ++i) h = (h ^ w[i * step]) * 1099511628211ull;
    return h;
  };
  static const std::unordered_multimap<uint64_t, const KnownProgram*> table = [&] {
    std::unordered_multimap<uint64_t, const KnownProgram*> t;
    int n;
    for (auto list : {known_programs, known_recurrent_programs}) {
      const KnownProgram* k = list(&n);
      for (int i = 0; i < n; ++i) t.emplace(hash(k[i].code, k[i].n_code, 1), &k[i]);
    }
    return t;
  }();
  auto range = table.equal_range(hash(&p.code[0].x, p.n_code, 2));
  for (auto it = range.first; it != range.second; ++it) {
    const KnownProgram* k = it->second;
    bool same = k->n_code == p.n_code && k->n_preload == p.n_preload;
    for (int i = 0; i < p.n_code && same; ++i) same = k->code[i] == p.code[i].x;
    if (same) return k;
  }
  return nullptr;
}
// Whether every box begins and ends between groups of four elements.
bool regions_in_quads(const FusedParams& p) {
  for (int k = 0; k < p.n_regions; ++k)
    if (p.region[k].lo[p.nd - 1] % 4 != 0 || p.region[k].hi[p.nd - 1] % 4 != 0) return false;
  return true;
}

}  // namespace

// The instruction as the kernel decodes it: reversed operands become ops of their own.
uint2 fused::encode(const rt_fused_instr& in) {
  int op = in.op;
  if (in.swap && op != RT_F_SELECT) switch (op) {
      case RT_F_SUB: op = kReverseSub; break;
      case RT_F_DIV: op = kReverseDiv; break;
      case RT_F_POWF: op = kReversePow; break;
      case RT_F_GT: op = RT_F_LT; break;
      case RT_F_GE: op = RT_F_LE; break;
      case RT_F_LT: op = RT_F_GT; break;
      case RT_F_LE: op = RT_F_GE; break;
      default: break;
    }
  const bool unary = op >= RT_F_RELU && op <= RT_F_ELU_SLOPE;
  const uint32_t src = unary ? 0u : in.src, region = in.op == RT_F_SELECT ? in.swap : 0u;
  uint2 w;
  w.x = (uint32_t)op | src << 8 | (uint32_t)in.dst << 16 | region << 24;
  static_assert(sizeof(in.imm) == 4, "");
  memcpy(&w.y, &in.imm, 4);
  return w;
}

rt_status fused::prepare(rt_ctx* ctx, const rt_fused_program* f, FusedParams* out, bool* in_vectors, int64_t* count) {
  RT_CHECK_CTX(ctx);
  RT_CHECK_PTR(ctx, f);
  if (f->nd < 1 || f->nd > RT_FUSED_MAX_DIMS || f->n_operands < 0 || f->n_operands > RT_FUSED_MAX_OPERANDS || f->n_regions < 0 ||
      f->n_regions > RT_FUSED_MAX_REGIONS || f->n_outputs < 1 || f->n_outputs > RT_FUSED_MAX_OUTPUTS || f->n_code < 1 ||
      f->n_code > RT_FUSED_MAX_CODE || f->n_preload < 0 || f->n_preload > RT_FUSED_PRELOAD || f->n_preload > f->n_operands)
    RT_FAIL(ctx, RT_ERR_INVALID_OPERATION, "rt_fused_elementwise: a count of the program is out of range");
  int64_t numel = 1;
  for (int d = 0; d < f->nd; ++d) {
    if (f->shape[d] < 0) RT_FAIL(ctx, RT_ERR_INVALID_OPERATION, "rt_fused_elementwise: negative extent");
    numel *= f->shape[d];
    if (numel >= (1ll << 31)) RT_FAIL(ctx, RT_ERR_UNIMPLEMENTED, "rt_fused_elementwise: 2^31 or more elements");
  }
  for (int i = 0; i < f->n_code; ++i) {
    const rt_fused_instr& in = f->code[i];
    const bool unary = in.op >= RT_F_RELU && in.op <= RT_F_ELU_SLOPE;
    const int most = in.op == RT_F_LOAD ? f->n_operands : (in.op == RT_F_OUT ? f->n_outputs : RT_FUSED_REGS);
    if (in.op >= RT_F_COUNT || (!unary && in.src >= most && !(in.op != RT_F_LOAD && in.op != RT_F_OUT && in.src == RT_FUSED_IMM)) ||
        (in.dst != RT_FUSED_NONE && in.dst >= RT_FUSED_REGS) || (in.op == RT_F_SELECT && in.swap >= f->n_regions))
      RT_FAIL(ctx, RT_ERR_INVALID_OPERATION, "rt_fused_elementwise: instruction %d is malformed", i);
  }
  for (int k = 0; k < f->n_operands; ++k) {
    RT_CHECK_PTR(ctx, f->operand[k].ptr);
    if (f->operand[k].region != RT_FUSED_NONE && (f->operand[k].region < 0 || f->operand[k].region >= f->n_regions))
      RT_FAIL(ctx, RT_ERR_INVALID_OPERATION, "rt_fused_elementwise: operand %d names region %d", k, f->operand[k].region);
  }
  *count = numel;
  if (numel == 0) return RT_OK;
  FusedParams& p = *out;
  p.nd = f->nd;
  p.n_preload = f->n_preload;
  p.n_code = f->n_code;
  p.n_regions = f->n_regions;
  p.numel = (uint32_t)numel;
  bool vec = f->shape[f->nd - 1] % 4 == 0;  // a group of four elements then never straddles the end of a row
  for (int k = 0; k < f->n_outputs; ++k) {
    RT_CHECK_PTR(ctx, f->out[k]);
    p.out[k] = f->out[k];
    vec = vec && rt_aligned16(f->out[k]);
  }
  for (int d = 0; d < f->nd; ++d) p.dim[d].init((uint32_t)(f->shape[d] ? f->shape[d] : 1));
  for (int k = 0; k < f->n_operands; ++k) {
    const rt_fused_operand& o = f->operand[k];
    p.operand[k] = o;
    bool same = true, quads = rt_aligned16(o.ptr) && o.stride[f->nd - 1] == 1;
    for (int d = 0; d < f->nd; ++d) {
      same = same && o.stride[d] == 0;
      if (d < f->nd - 1) quads = quads && o.stride[d] % 4 == 0;
    }
    p.mode[k] = same ? kSame : (quads ? kVector : (o.stride[f->nd - 1] == 0 ? kBroadcast : kScalar));
  }
  for (int k = 0; k < f->n_regions; ++k) p.region[k] = f->region[k];
  for (int i = 0; i < f->n_code; ++i) p.code[i] = encode(f->code[i]);
  *in_vectors = vec && regions_in_quads(p);
  return RT_OK;
}

extern "C" rt_status rt_fused_elementwise(rt_ctx* ctx, const rt_fused_program* f) {
  FusedParams p;
  bool vec;
  int64_t numel;
  rt_status st = prepare(ctx, f, &p, &vec, &numel);
  if (st != RT_OK || numel == 0) return st;
  if (p.nd <= 2)
    if (const KnownProgram* k = find_known(p)) {
      ctx->fused_compiled++;
      return k->launch(ctx, p, vec, numel);
    }
  ctx->fused_interpreted++;
  // Eight elements per thread halve the decoding per element, four give twice the warps: the line lies where eight still fill
  // every SM with its 512 threads.
  const bool wide = numel >= (int64_t)ctx->sm_count * 512 * 8;
  if (wide) return vec ? launch_fused<8, true, 256, 2>(ctx, p, numel) : launch_fused<8, false, 256, 2>(ctx, p, numel);
  return vec ? launch_fused<4, true, 128, 8>(ctx, p, numel) : launch_fused<4, false, 128, 8>(ctx, p, numel);
}
