// Shared by the two kernels behind rt_fused_elementwise: the interpreter (k_fused.cu) and the programs compiled ahead of time
// (k_fused_known.cu).
#pragma once
#include "conv_geom.cuh"
#include "rt_internal.cuh"

namespace fused {

struct FusedParams {
  int nd, n_preload, n_code, n_regions;
  uint32_t numel, tiles;
  FastDiv dim[RT_FUSED_MAX_DIMS];
  uint8_t mode[RT_FUSED_MAX_OPERANDS];  // how a group of four consecutive elements is read (kernels with VEC)
  rt_fused_operand operand[RT_FUSED_MAX_OPERANDS];
  rt_fused_region region[RT_FUSED_MAX_REGIONS];
  float* out[RT_FUSED_MAX_OUTPUTS];
  uint2 code[RT_FUSED_MAX_CODE];  // x: op | src << 8 | dst << 16 | region << 24, y: the immediate
};
// one value for the whole iteration space; four consecutive floats as one 128-bit load; one value for the group; four loads
enum { kSame = 0, kVector = 1, kBroadcast = 2, kScalar = 3 };
// ops from kPlain on work on registers alone; reversed operands are ops of their own
enum { kPlain = RT_F_REG, kReverseSub = RT_F_COUNT, kReverseDiv, kReversePow };

// The functions behind sin, cos, tan and powf are long: the interpreter calls them instead of expanding them once per element.
#ifdef RT_FUSED_EXPAND_MATH
#define RT_FUSED_MATH __forceinline__
#else
#define RT_FUSED_MATH __noinline__
#endif
static __device__ RT_FUSED_MATH float call_sin(float x) { return sinf(x); }
static __device__ RT_FUSED_MATH float call_cos(float x) { return cosf(x); }
static __device__ RT_FUSED_MATH float call_tan(float x) { return tanf(x); }
static __device__ RT_FUSED_MATH float call_pow(float x, float y) { return powf(x, y); }

// Every op in one place: OP(code, expression in the accumulator x, the operand y and the immediate imm).
#define RT_FUSED_OPS(OP)                                   \
  OP(RT_F_REG, y)                                          \
  OP(RT_F_ADD, x + y)                                      \
  OP(RT_F_MUL, x * y)                                      \
  OP(RT_F_SUB, x - y)                                      \
  OP(kReverseSub, y - x)                                   \
  OP(RT_F_DIV, x / y)                                      \
  OP(kReverseDiv, y / x)                                   \
  OP(RT_F_POWF, call_pow(x, y))                            \
  OP(kReversePow, call_pow(y, x))                          \
  OP(RT_F_MAX, fmaxf(x, y))                                \
  OP(RT_F_MIN, fminf(x, y))                                \
  OP(RT_F_EQ, fabsf(x - y) < 1e-9f ? 1.f : 0.f)            \
  OP(RT_F_NE, fabsf(x - y) >= 1e-9f ? 1.f : 0.f)           \
  OP(RT_F_GT, x > y ? 1.f : 0.f)                           \
  OP(RT_F_GE, x >= y ? 1.f : 0.f)                          \
  OP(RT_F_LT, x < y ? 1.f : 0.f)                           \
  OP(RT_F_LE, x <= y ? 1.f : 0.f)                          \
  OP(RT_F_RELU, fmaxf(x, 0.f))                             \
  OP(RT_F_STEP, x > 0.f ? 1.f : 0.f)                       \
  OP(RT_F_EXP, expf(x))                                    \
  OP(RT_F_LN, logf(x))                                     \
  OP(RT_F_SIN, call_sin(x))                                \
  OP(RT_F_COS, call_cos(x))                                \
  OP(RT_F_TAN, call_tan(x))                                \
  OP(RT_F_TANH, tanhf(x))                                  \
  OP(RT_F_SIGMOID, 1.f / (1.f + expf(-x)))                 \
  OP(RT_F_SOFTPLUS, logf(1.f + expf(x)))                   \
  OP(RT_F_SQRT, sqrtf(x))                                  \
  OP(RT_F_ABS, fabsf(x))                                   \
  OP(RT_F_SIGN, x > 0.f ? 1.f : (x < 0.f ? -1.f : 0.f))    \
  OP(RT_F_NEG, -x)                                         \
  OP(RT_F_RECIP, 1.f / x)                                  \
  OP(RT_F_ONE_MINUS_SQUARE, 1.f - x * x)                   \
  OP(RT_F_LOGISTIC_SLOPE, x * (1.f - x))                   \
  OP(RT_F_HALF_RSQRT, 0.5f / sqrtf(x))                     \
  OP(RT_F_RECIP_SQUARE, 1.f / (x * x))                     \
  OP(RT_F_SQUARE, x * x)                                   \
  OP(RT_F_ELU, x < 0.f ? imm * (expf(x) - 1.f) : x)        \
  OP(RT_F_ELU_SLOPE, x < 0.f ? imm * expf(x) : 1.f)

// Programs compiled ahead of time register themselves here.
struct KnownProgram {
  const uint32_t* code;  // the words of the instructions, without immediates
  int n_code, n_preload;
  rt_status (*launch)(rt_ctx* ctx, FusedParams& p, bool vec, int64_t numel);
};
// Checks a program and brings it into the kernels' form; vec: groups of four consecutive elements may be read and written as vectors.
rt_status prepare(rt_ctx* ctx, const rt_fused_program* f, FusedParams* p, bool* vec, int64_t* numel);  // k_fused.cu
uint2 encode(const rt_fused_instr& in);                  // k_fused.cu
const KnownProgram* known_programs(int* n);            // k_fused_known.cu
const KnownProgram* known_recurrent_programs(int* n);  // k_fused_lstm.cu

}  // namespace fused
