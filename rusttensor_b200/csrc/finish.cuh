// What a product's epilogue does to its sums.
#pragma once
#include "rt_internal.cuh"

// act(v + bias) + old for four neighbouring results of a product, `left` of which exist.  Not inlined: with four copies of tanh and the
// logistic function in its tail, a kernel that uses neither spent 2 us more (128 x 64 tile, 32 values a thread).
static __device__ __noinline__ float4 rt_finish4(float4 v, const float* bias, int act, const float* old, int left) {
  float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < left) {
      if (bias) o[j] += __ldg(bias + j);
      if (act == RT_ACT_RELU) o[j] = fmaxf(o[j], 0.f);
      else if (act == RT_ACT_TANH) o[j] = tanhf(o[j]);
      else if (act == RT_ACT_SIGMOID) o[j] = 1.f / (1.f + expf(-o[j]));
      if (old) o[j] += old[j];
    }
  return make_float4(o[0], o[1], o[2], o[3]);
}
