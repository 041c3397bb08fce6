// Checks of the CUDA backend's host logic (host/b200_backend.hpp, host/lazy.hpp) without a GPU: the few C-ABI entry points that they
// reach are stubs over host memory, which count blocks and fail on demand.  Usage: engine_checks NAME; test_engine_host.py runs them.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include "../../rusttensor_b200/csrc/host/b200_backend.hpp"

using namespace rt;
using B = B200Backend;

namespace {
std::map<void*, size_t> live;  // blocks that are allocated
int failures;                  // of the checks
int mallocs_left = -1;         // rt_malloc fails once they are used up; < 0: never
int mallocs;
bool kernels_fail = false;
int masked_pool_gradients;     // launches of the pooling gradient that masks by the relu in front
int forward_sequences, backward_sequences;
int row_gradients, programs;   // launches of the gradient of a logsumexp by its own kernel, of elementwise programs
int logsumexps;                // launches of a logsumexp, by its own kernel or within a program
int asked_of_programs;         // programs built for a kernel with a reduction
bool reductions_known = false; // kernels for programs with a reduction
bool recording = false;
int unrecorded;                // kernels while nothing is recorded
rt_status kernel() {
  unrecorded += !recording;
  return kernels_fail ? RT_ERR_CUDA : RT_OK;
}

void expect(bool ok, const char* what, int line) {
  if (ok) return;
  std::printf("line %d: %s\n", line, what);
  ++failures;
}
#define EXPECT(x) expect((x), #x, __LINE__)

B::Storage make(const Shape& s, float first, float step = 1.f) {
  B::Storage x = B::alloc(s);
  for (size_t i = 0; i < x.numel(); ++i) x.buf->ptr[i] = first + step * (float)i;
  return x;
}
bool holds(const B::Storage& x, float first, float step = 1.f) {
  const float* p = x.ptr();
  for (size_t i = 0; i < x.numel(); ++i)
    if (p[i] != first + step * (float)i) return false;
  return true;
}
void scribble(float* p, size_t n) {
  for (size_t i = 0; i < n; ++i) p[i] = -77.f;
}
}  // namespace

// ---- the stubs ------------------------------------------------------------------------------------------------------------
extern "C" {
const char* rt_last_error(rt_ctx*) { return "stub"; }
rt_status rt_malloc(rt_ctx*, size_t bytes, void** out) {
  if (mallocs_left == 0) return RT_ERR_OOM;
  if (mallocs_left > 0) --mallocs_left;
  ++mallocs;
  *out = std::calloc(1, bytes);
  live[*out] = bytes;
  return RT_OK;
}
rt_status rt_free(rt_ctx*, void* p) {
  if (!p) return RT_OK;
  if (!live.erase(p)) {
    std::printf("a block is freed twice, or is none\n");
    ++failures;
    return RT_OK;
  }
  std::free(p);
  return RT_OK;
}
rt_status rt_memcpy_d2d(rt_ctx*, void* d, const void* s, size_t n) {
  std::memmove(d, s, n);
  return RT_OK;
}
rt_status rt_unary(rt_ctx*, int op, const float* x, float* y, int64_t n, float, float) {
  if (kernel() != RT_OK) return RT_ERR_CUDA;
  for (int64_t i = 0; i < n; ++i) y[i] = op == RT_SQUARE ? x[i] * x[i] : (op == RT_TANH ? std::tanh(x[i]) : (op == RT_SIGMOID ? 1.f / (1.f + std::exp(-x[i])) : x[i]));
  return RT_OK;
}
rt_status rt_binary(rt_ctx*, int op, const float* a, const int64_t* as, int na, const float* b, const int64_t*, int, float* out) {
  int64_t n = 1;
  for (int d = 0; d < na; ++d) n *= as[d];
  for (int64_t i = 0; i < n && (op == RT_ADD || op == RT_MUL); ++i) out[i] = op == RT_ADD ? a[i] + b[i] : a[i] * b[i];  // of one shape
  return kernel();
}
rt_status rt_relu_max_pool2d(rt_ctx*, const float*, int64_t, int64_t, int64_t, int64_t, int, int, int, int, int, int, float*, float*) {
  return RT_OK;
}
rt_status rt_max_pool2d_backward(rt_ctx*, const float*, const float*, int64_t, int64_t, int64_t, int64_t, int, int, int, int, int, int, float*) {
  return RT_OK;
}
rt_status rt_relu_max_pool2x2_backward_from_output(rt_ctx*, const float*, const float*, const float*, int64_t, int64_t, int64_t, int64_t, float*) {
  ++masked_pool_gradients;
  return RT_OK;
}
rt_status rt_column_sums_list(rt_ctx*, int count, const float* const* xs, const int64_t* rows, const int64_t* cols, float* const* outs) {
  if (kernel() != RT_OK) return RT_ERR_CUDA;
  for (int k = 0; k < count; ++k)
    for (int64_t i = 0; i < rows[k] * cols[k]; ++i) outs[k][i % cols[k]] = (i < cols[k] ? 0.f : outs[k][i % cols[k]]) + xs[k][i];
  return RT_OK;
}
rt_status rt_sum_rows_accumulate_list(rt_ctx*, int count, const float* const* xs, int64_t rows, int64_t cols, float* out) {
  if (kernel() != RT_OK) return RT_ERR_CUDA;
  for (int k = 0; k < count; ++k)
    for (int64_t i = 0; i < rows * cols; ++i) out[i % cols] += xs[k][i];
  return RT_OK;
}
rt_status rt_gemm_bias_act_list(rt_ctx* ctx, int count, const float* const* as, float* const* outs, int64_t m, int64_t n, int64_t k, const float* b,
                                const float* bias, int act) {
  for (int i = 0; i < count; ++i) rt_gemm_bias_act(ctx, m, n, k, as[i], k, b, n, bias, act, outs[i], n);
  return kernel();
}
uint64_t possible_ops = ~uint64_t(0);  // of kernels with a reduction; all ones: any
rt_status rt_fused_reduction_possible(rt_ctx*, int, uint64_t ops) { return possible_ops == ~uint64_t(0) || ops == possible_ops ? RT_OK : RT_ERR_UNIMPLEMENTED; }
rt_status rt_fused_reduction_known(rt_ctx*, const rt_fused_program*, int) { return ++asked_of_programs, reductions_known ? RT_OK : RT_ERR_UNIMPLEMENTED; }
rt_status rt_fused_column_sums(rt_ctx*, const rt_fused_program*, int, float*) { return kernel(); }
rt_status rt_fused_logsumexp(rt_ctx*, const rt_fused_program*, float*) { return ++logsumexps, kernel(); }
rt_status rt_reduce_backward(rt_ctx*, int, const float* x, const float*, int64_t outer, int64_t len, int64_t, float* dx) {
  ++row_gradients;
  for (int64_t i = 0; i < outer * len; ++i) dx[i] = x[i];  // to tell which values it has read
  return kernel();
}
rt_status rt_fused_elementwise(rt_ctx*, const rt_fused_program* p) {  // the ops that the checks use; others pass the accumulator on
  if (kernel() != RT_OK) return RT_ERR_CUDA;
  ++programs;
  int64_t n = 1;
  for (int d = 0; d < p->nd; ++d) n *= p->shape[d];
  for (int64_t e = 0; e < n; ++e) {
    int64_t c[RT_FUSED_MAX_DIMS], rest = e;
    for (int d = p->nd; d-- > 0; rest /= p->shape[d]) c[d] = rest % p->shape[d];
    auto inside = [&](int r) {
      bool in = true;
      for (int d = 0; d < p->nd && r != RT_FUSED_NONE; ++d) in = in && c[d] >= p->region[r].lo[d] && c[d] < p->region[r].hi[d];
      return in;
    };
    auto load = [&](int k) {
      const float* q = p->operand[k].ptr;
      for (int d = 0; d < p->nd; ++d) q += c[d] * p->operand[k].stride[d];
      return inside(p->operand[k].region) ? *q : 0.f;
    };
    float reg[RT_FUSED_REGS] = {}, acc = 0.f;
    for (int k = 0; k < p->n_preload; ++k) reg[k] = load(k);
    for (int i = 0; i < p->n_code; ++i) {
      const rt_fused_instr& in = p->code[i];
      const float other = in.src == RT_FUSED_IMM ? in.imm : (in.src < RT_FUSED_REGS ? reg[in.src] : 0.f);
      const float x = in.swap ? other : acc, y = in.swap ? acc : other;
      switch (in.op) {
        case RT_F_LOAD: acc = load(in.src); break;
        case RT_F_REG: acc = other; break;
        case RT_F_OUT: p->out[in.src][e] = acc; break;
        case RT_F_SELECT: acc = inside(in.swap) ? acc : other; break;
        case RT_F_ADD: acc = x + y; break;
        case RT_F_SUB: acc = x - y; break;
        case RT_F_MUL: acc = x * y; break;
        case RT_F_SQUARE: acc = acc * acc; break;
        case RT_F_TANH: acc = std::tanh(acc); break;
        case RT_F_EXP: acc = std::exp(acc); break;
        case RT_F_SIGMOID: acc = 1.f / (1.f + std::exp(-acc)); break;
        default: break;
      }
      if (in.dst != RT_FUSED_NONE) reg[in.dst] = acc;
    }
  }
  return RT_OK;
}
// products and the recurrence, as far as the forward pass goes
rt_status rt_gemm_bias_act(rt_ctx*, int64_t m, int64_t n, int64_t k, const float* a, int64_t lda, const float* b, int64_t ldb, const float* bias, int, float* c,
                           int64_t ldc) {
  for (int64_t i = 0; i < m; ++i)
    for (int64_t j = 0; j < n; ++j) {
      float sum = bias ? bias[j] : 0.f;
      for (int64_t l = 0; l < k; ++l) sum += a[i * lda + l] * b[l * ldb + j];
      c[i * ldc + j] = sum;
    }
  return kernel();
}
rt_status rt_gemm(rt_ctx* ctx, int ta, int tb, int64_t m, int64_t n, int64_t k, const float* a, int64_t lda, const float* b, int64_t ldb, float* c, int64_t ldc,
                  int acc) {
  return ta || tb || acc ? kernel() : rt_gemm_bias_act(ctx, m, n, k, a, lda, b, ldb, nullptr, 0, c, ldc);
}
rt_status rt_lstm_sequence(rt_ctx*, const float* pre, const float* w, int64_t ldw, const float* h0, const float* c0, int64_t steps, int64_t batch, int64_t hidden,
                           float* saved, float* h) {
  ++forward_sequences;
  const int64_t n = batch * hidden, plane = steps * n;
  for (int64_t t = 0; t < steps; ++t)
    for (int64_t e = 0; e < n; ++e) {
      const int64_t row = e / hidden, u = e % hidden, o = t * n + e;
      float z[4];
      for (int g = 0; g < 4; ++g) {
        z[g] = pre[(t * batch + row) * 4 * hidden + g * hidden + u];
        const float* before = t ? h + (t - 1) * n + row * hidden : (h0 ? h0 + row * hidden : nullptr);
        for (int64_t l = 0; before && l < hidden; ++l) z[g] += before[l] * w[l * ldw + g * hidden + u];
        z[g] = g == 2 ? std::tanh(z[g]) : 1.f / (1.f + std::exp(-z[g]));
      }
      const float c = z[1] * (t ? saved[4 * plane + o - n] : (c0 ? c0[e] : 0.f)) + z[0] * z[2];
      const float kept[6] = {z[0], z[1], z[2], z[3], c, std::tanh(c)};
      for (int k = 0; k < 6; ++k) saved[k * plane + o] = kept[k];
      h[o] = z[3] * kept[5];
    }
  return kernel();
}
// their results stay zero
rt_status rt_graph_begin(rt_ctx*) { return recording = true, RT_OK; }
rt_status rt_graph_end(rt_ctx*, rt_graph**) { return recording = false, RT_OK; }
rt_status rt_fill(rt_ctx*, float*, float, int64_t) { return kernel(); }
rt_status rt_softmax_nll_list(rt_ctx*, int, const float* const*, const float* const*, int64_t, int64_t, float, float, int, const float* const*, float*) {
  return kernel();
}
rt_status rt_softmax_nll_with_grad(rt_ctx*, const float*, const float*, int64_t, int64_t, float, float, const float*, float, float*, float*) { return kernel(); }
rt_status rt_softmax_nll_scaled_backward(rt_ctx*, const float*, const float*, int64_t, int64_t, float, float*) { return kernel(); }
rt_status rt_matmul_backward(rt_ctx*, const float*, const float*, const float*, int64_t, int64_t, int64_t, float*, float*) { return kernel(); }
rt_status rt_gemm_sum_products(rt_ctx*, int, const float* const*, const float* const*, int64_t, int64_t, int64_t, float*) { return kernel(); }
rt_status rt_reduce(rt_ctx*, int op, const float*, int64_t, int64_t, int64_t, float*) { return logsumexps += op == RT_RED_LOGSUMEXP, kernel(); }
rt_status rt_unbroadcast(rt_ctx*, const float*, const int64_t*, int, const int64_t*, int, float*) { return kernel(); }
rt_status rt_broadcast_to(rt_ctx*, const float*, const int64_t*, int, const int64_t*, int, float*) { return kernel(); }
rt_status rt_slice_assign(rt_ctx*, float*, const int64_t*, int, const int64_t*, const float*, const int64_t*) { return kernel(); }
rt_status rt_lstm_sequence_backward(rt_ctx*, const float*, const float*, int64_t, const float*, const float*, int64_t, int64_t, int64_t, float*, float*,
                                    float*) {
  ++backward_sequences;
  return kernel();
}
}

// ---- the checks -----------------------------------------------------------------------------------------------------------
namespace {

// A slice of whole rows and its base do not see each other's writes through a device pointer.
void rows_do_not_alias() {
  const Shape s{6, 4};
  for (int first : {0, 2}) {
    B::Storage x = make(s, 1.f), y = B::slice(x, {{2, 4}, {0, 4}}), z = B::unary(RT_SQUARE, y);
    EXPECT(holds(y, 9.f));
    scribble(B::escape(first == 0 ? x : y), first == 0 ? 24 : 8);
    EXPECT(first == 0 ? holds(y, 9.f) : holds(x, 1.f));
    for (int i = 0; i < 8; ++i) EXPECT(z.ptr()[i] == (9.f + i) * (9.f + i));  // asked for before the write
  }
  {  // a slice of a slice, of one row
    B::Storage x = make(s, 1.f), y = B::slice(x, {{1, 5}, {0, 4}}), w = B::slice(y, {{3, 4}, {1, 3}});
    EXPECT(holds(w, 18.f));
    scribble(B::escape(y), 16);
    scribble(B::escape(x), 24);
    EXPECT(holds(w, 18.f));
  }
  {  // the base's memory goes with the base
    B::Storage x = make(s, 1.f), y = B::slice(x, {{2, 4}, {0, 4}});
    y.ptr();
    x = B::Storage{};
    EXPECT(live.size() == 1 && live.begin()->second == 8 * sizeof(float));
  }
  EXPECT(live.empty());
}
// A tensor broadcast to its own shape is a tensor of its own.
void broadcast_does_not_alias() {
  B::Storage x = make({2, 3}, 1.f), y = B::broadcast_to(x, {2, 3});
  scribble(B::escape(y), 6);
  EXPECT(holds(x, 1.f));
}
// Inside a capture rows are not copied; what a step leaves behind has a block of its own.
void rows_in_a_capture() {
  B::Storage x = make({6, 4}, 1.f);
  lazy::capturing() = true;
  B::Storage y = B::slice(x, {{2, 4}, {0, 4}});
  EXPECT(y.ptr() == x.ptr() + 8);
  B::Storage w = B::slice(y, {{1, 2}, {0, 4}});
  EXPECT(w.ptr() == x.ptr() + 12);
  B::own(y);
  lazy::capturing() = false;
  scribble(B::escape(x), 24);
  EXPECT(holds(y, 9.f));
  EXPECT(B::escape(w) != x.ptr() + 12);
}
// The gradient of a pooling is masked by the relu in front of it, not by one whose buffer happens to lie where that one's was.
void pooling_knows_its_relu() {
  const Shape s{1, 1, 4, 4};
  for (bool same : {true, false}) {
    masked_pool_gradients = 0;
    B::Storage gradient, mask, other = make(s, 3.f);
    const DeviceBuffer* old;
    {
      B::Storage x = B::unary(RT_RELU, make(s, -5.f));
      old = x.buf.get();
      auto pooled = B::max_pool2d(x, {2, 2}, {2, 2}, {0, 0});
      OpType t(OpType::MaxPool2D);
      t.kernel_size = t.stride = {2, 2};
      t.padding = {0, 0};
      Op<B> op(t, {Tensor<B>(x, true), Tensor<B>(pooled.second, false)}, nullptr);
      op.cached_outputs = pooled.first;
      gradient = B::max_pool2d_backward(op, make(pooled.first.shape, 1.f));
      if (same) mask = B::lz_unary(RT_F_STEP, x);
    }
    std::vector<B::Storage> tried;
    for (int i = 0; i < 1000 && !same && !mask.buf; ++i) {
      tried.push_back(B::unary(RT_RELU, other));
      if (tried.back().buf.get() == old) mask = B::lz_unary(RT_F_STEP, tried.back());
    }
    if (!mask.buf) continue;  // the address was not used again
    B::lz_mul(gradient, mask).ptr();
    EXPECT(masked_pool_gradients == (same ? 1 : 0));
  }
}
// A launch or an allocation that fails leaves nothing behind: no block is lost, and asking again gives the values.
template <class F>
void fails_and_recovers(size_t most_blocks, F ask) {
  const size_t before = live.size();
  for (size_t k = 0; k <= most_blocks; ++k) {
    mallocs_left = k < most_blocks ? (int)k : -1;
    kernels_fail = k == most_blocks;
    bool threw = false;
    try {
      ask();
    } catch (const Error&) {
      threw = true;
    }
    EXPECT(threw);
    EXPECT(live.size() == before);
  }
  mallocs_left = -1;
  kernels_fail = false;
  ask();
}
void errors_lose_nothing() {
  {  // the bias gradients of several layers
    std::vector<B::Storage> g;
    for (int i = 0; i < 3; ++i) g.push_back(B::unbroadcast(make({2, 4}, (float)i), {4}));
    fails_and_recovers(3, [&] { B::evaluate_column_sums({&g[0], &g[1], &g[2], &g[1]}); });
    for (int i = 0; i < 3; ++i) EXPECT(holds(g[i], 2 * i + 4.f, 2.f));
  }
  for (bool shared : {false, true}) {  // terms added to a gradient, in its own block or in a new one
    B::Storage x = make({2, 4}, 1.f), acc = make({4}, 10.f), other;
    if (shared) other = acc;
    B::append_terms(acc, lazy::Tag::SumRows, {B::input(x)}, {2, 4}, B::run_sum_rows);
    fails_and_recovers(shared ? 1 : 0, [&] { acc.ptr(); });
    EXPECT(holds(acc, 16.f, 3.f));
    if (shared) EXPECT(holds(other, 10.f));
  }
  {  // at once, because the term's address has been handed out
    B::Storage x = make({2, 4}, 1.f), acc = make({4}, 10.f);
    B::escape(x);
    kernels_fail = true;
    try {
      B::append_terms(acc, lazy::Tag::SumRows, {B::input(x)}, {2, 4}, B::run_sum_rows);
      EXPECT(false);
    } catch (const Error&) {
    }
    kernels_fail = false;
    EXPECT(acc.buf && holds(acc, 16.f, 3.f));
  }
  {  // another contribution to a gradient, likewise
    B::Storage g = make({4}, 1.f);
    Tensor<B> p(make({4}, 0.f), true);
    p.set_grad(make({4}, 10.f));
    B::escape(g);
    kernels_fail = true;
    try {
      p.add_grad(g);
      EXPECT(false);
    } catch (const Error&) {
    }
    kernels_fail = false;
    EXPECT(p.grad()->buf && holds(*p.grad(), 10.f));
  }
  {  // products of one layer in a list
    const B::Storage w = make({4, 3}, 0.f);
    std::vector<B::Storage> y;
    for (int i = 0; i < 4; ++i) y.push_back(B::matmul(make({2, 4}, 0.f), w));
    fails_and_recovers(4, [&] { y[0].ptr(); });
  }
  EXPECT(live.empty());
}
// What has been handed out may be written at any time: a gradient does not count on a forward result whose address is known outside,
// and a term that joins others is added on the spot.
bool reads(const DeviceBuffer* b, const DeviceBuffer* of) {
  if (b == of) return true;
  if (b->node)
    for (auto& i : b->node->in)
      if (reads(i.buf.get(), of)) return true;
  return false;
}
void written_from_outside() {
  for (int op : {RT_RELU, RT_EXP, RT_TANH, RT_SIGMOID})
    for (bool known : {false, true}) {
      B::Storage x = make({2, 3}, 1.f), y = B::unary(op, x);
      Op<B> o(OpType(OpType::Relu), {Tensor<B>(x, true)}, nullptr);
      o.cached_outputs = y;
      y.buf->drop_node();  // as if it had been computed
      y.buf->ptr = lazy::Block(B::ctx(), 6).release();
      if (known) B::escape(y);
      B::Storage d = B::unary_bwd(op, o, make({2, 3}, 1.f));
      EXPECT(reads(d.buf.get(), y.buf.get()) == !known);
      EXPECT(reads(d.buf.get(), x.buf.get()) == known);
    }
  for (int known : {0, 1, 2}) {  // the gradient of an LSTM cell's output takes the gate and tanh(c) that the forward pass has kept
    const B::Storage gates = make({2, 12}, 0.f, 0.1f), c = make({2, 3}, 0.f, 0.1f), h = B::lstm_cell_h(gates, c);
    Op<B> o(OpType(OpType::FusedLstmCellH), {Tensor<B>(gates, true), Tensor<B>(c, true)}, nullptr);
    o.cached_outputs = h;
    const auto gate = h.buf->saved[0], th = h.buf->saved[1];
    if (known) B::escape(known == 1 ? gates : c);
    const auto d = B::lstm_cell_h_backward(o, make({2, 3}, 1.f));
    EXPECT(reads(d.second.buf.get(), gate.get()) == (known != 1));
    EXPECT(reads(d.second.buf.get(), th.get()) == (known == 0));
  }
  B::Storage a = make({2, 4}, 1.f), b = make({2, 4}, 1.f), acc = make({4}, 10.f);
  float* p = B::escape(b);
  B::append_terms(acc, lazy::Tag::SumRows, {B::input(a)}, {2, 4}, B::run_sum_rows);
  EXPECT(acc.buf->node != nullptr);
  B::append_terms(acc, lazy::Tag::SumRows, {B::input(b)}, {2, 4}, B::run_sum_rows);
  scribble(p, 8);
  EXPECT(holds(acc, 22.f, 5.f));
}

// A matrix that is both operands of a product is listed twice among its readers; the product is computed once.
void a_product_of_a_matrix_with_itself() {
  {
    const B::Storage x = make({3, 3}, 1.f), y = make({3, 3}, 2.f);
    std::vector<B::Storage> p{B::matmul(y, x), B::matmul(x, x), B::matmul(x, x)};
    p[0].ptr();
    for (auto& q : p) EXPECT(!q.buf->node);
    EXPECT(live.size() == 5);
  }
  EXPECT(live.empty());
}

// An LSTM written op by op, in a capture: one sequence forward; backward one, unless somebody could miss a gradient of what lies between.
void cells_become_a_sequence() {
  using Tn = Tensor<B>;
  const size_t T = 5, Bn = 3, V = 4, H = 2;
  enum { kPlain, kHeld, kCellUsed, kOtherGates, kStateUsedTwice, kInputsOutOfOrder, kGivenState, kCases };
  for (int way = 0; way < kCases; ++way) {
    forward_sequences = backward_sequences = 0;
    {
      const Tn x(make({(T + 1) * Bn, V}, 0.f, .01f), false), w(make({V + H, 4 * H}, 0.f, .01f), true), b(make({4 * H}, 0.f, .01f), true);
      const Tn given(make({Bn, H}, 0.f), false);
      std::vector<Tn> held;
      Tn total;
      B::begin_capture();
      {
        Tn h = way == kGivenState ? given : Tn::zeros({Bn, H}, false), c = Tn::zeros({Bn, H}, false), sum;
        for (size_t t = 0; t < T; ++t) {
          const size_t r = (way == kInputsOutOfOrder && t == 2 ? t + 2 : t) * Bn;
          const Tn xh = ops::concat<B>({ops::slice(x, {{r, r + Bn}, {0, V}}), h}, 1);
          const Tn z = ops::add(ops::matmul(xh, w), b.broadcast_to({Bn, 4 * H}));
          auto gate = [&](size_t k) { return ops::slice(z, {{0, Bn}, {k * H, (k + 1) * H}}); };
          const Tn f = ops::sigmoid(gate(way == kOtherGates ? 0 : 1)), i = ops::sigmoid(gate(way == kOtherGates ? 1 : 0));
          c = ops::add(ops::mul(f, c), ops::mul(i, ops::tanh(gate(2))));
          h = ops::mul(ops::sigmoid(gate(3)), ops::tanh(c));
          if (way == kHeld && t == 2) held.push_back(c);
          Tn out = ops::sum(way == kStateUsedTwice ? ops::mul(h, h) : h, std::nullopt);
          if (way == kCellUsed && t == 2) out = ops::add(out, ops::sum(c, std::nullopt));
          sum = t ? ops::add(sum, out) : out;
        }
        total = sum;
      }
      total.backward();
      EXPECT(w.grad().has_value() && b.grad().has_value());
      for (auto& g : {*w.grad(), *b.grad()}) g.ptr();
      if (way == kHeld) EXPECT(held[0].grad().has_value());
      total.detach_graph();
      rt_graph* graph = nullptr;
      B::end_capture(&graph);
    }
    const bool cells = way != kOtherGates && way != kGivenState;  // out of order: the first two timesteps
    EXPECT(forward_sequences == (cells ? 1 : 0));
    EXPECT(backward_sequences == (way == kPlain || way == kStateUsedTwice ? 1 : 0));
    EXPECT(live.empty());
  }
}

// In a capture every state has the values of the recurrence, whatever is asked for first: the last state, a state, a gate, a cell state, a timestep's
// inputs, what a product takes.
void recurrences_have_their_values() {
  using Tn = Tensor<B>;
  const size_t T = 7, Bn = 3, V = 4, H = 2;
  std::vector<float> xs(T * Bn * V), ws((V + H) * 4 * H), bs(4 * H), want_h, want_c;
  for (size_t i = 0; i < xs.size(); ++i) xs[i] = std::sin(1.f + (float)i);
  for (size_t i = 0; i < ws.size(); ++i) ws[i] = .7f * std::cos(2.f + (float)i);
  for (size_t i = 0; i < bs.size(); ++i) bs[i] = .3f * std::sin(3.f * (float)i);
  for (size_t t = 0; t < T; ++t)
    for (size_t r = 0; r < Bn; ++r)
      for (size_t u = 0; u < H; ++u) {
        float z[4];
        for (size_t g = 0; g < 4; ++g) {
          z[g] = bs[g * H + u];
          for (size_t v = 0; v < V; ++v) z[g] += xs[(t * Bn + r) * V + v] * ws[v * 4 * H + g * H + u];
          for (size_t l = 0; l < H && t; ++l) z[g] += want_h[((t - 1) * Bn + r) * H + l] * ws[(V + l) * 4 * H + g * H + u];
          z[g] = g == 2 ? std::tanh(z[g]) : 1.f / (1.f + std::exp(-z[g]));
        }
        const float c = z[1] * (t ? want_c[((t - 1) * Bn + r) * H + u] : 0.f) + z[0] * z[2];
        want_c.push_back(c);
        want_h.push_back(z[3] * std::tanh(c));
      }
  auto filled = [](const Shape& shape, const std::vector<float>& v) {
    B::Storage x = B::alloc(shape);
    std::copy(v.begin(), v.end(), x.buf->ptr);
    return x;
  };
  enum { kLast, kState, kGate, kCellState, kInputs, kFirstInputs, kOperand, kSum, kWays };
  for (int way = 0; way < kWays; ++way)
    for (size_t at : {size_t(0), size_t(3), T - 1}) {
      {
        const Tn x(filled({T * Bn, V}, xs), false), w(filled({V + H, 4 * H}, ws), true), b(filled({4 * H}, bs), true);
        std::vector<Tn> hs, cs;
        B::begin_capture();
        {
          Tn h = Tn::zeros({Bn, H}, false), c = Tn::zeros({Bn, H}, false), asked;
          for (size_t t = 0; t < T; ++t) {
            const Tn xt = ops::slice(x, {{t * Bn, (t + 1) * Bn}, {0, V}}), xh = ops::concat<B>({xt, h}, 1);
            const Tn z = ops::add(ops::matmul(xh, w), b.broadcast_to({Bn, 4 * H}));
            auto gate = [&](size_t k) { return ops::slice(z, {{0, Bn}, {k * H, (k + 1) * H}}); };
            const Tn i = ops::sigmoid(gate(0)), f = ops::sigmoid(gate(1));
            c = ops::add(ops::mul(f, c), ops::mul(i, ops::tanh(gate(2))));
            h = ops::mul(ops::sigmoid(gate(3)), ops::tanh(c));
            hs.push_back(h);
            cs.push_back(c);
            if (t == at) asked = way == kState ? h : way == kGate ? f : way == kCellState ? c : way == kOperand ? xh : way == kSum ? ops::add(h, c) : xt;
            if (t == 0 && way == kFirstInputs) xt.data().ptr();  // while the recurrence is being written
          }
          if (way != kLast && way != kFirstInputs) asked.data().ptr();
          hs.back().data().ptr();
        }
        rt_graph* graph = nullptr;
        for (size_t t = 0; t < T; ++t)
          for (size_t e = 0; e < Bn * H; ++e) {
            EXPECT(std::abs(hs[t].data().ptr()[e] - want_h[t * Bn * H + e]) < 1e-5f);
            EXPECT(std::abs(cs[t].data().ptr()[e] - want_c[t * Bn * H + e]) < 1e-5f);
          }
        B::end_capture(&graph);
      }
      EXPECT(live.empty() && DeviceBuffer::waiting() == 0);
    }
}

// What a captured step computes as rows of one matrix (the states of a sequence, the output layer's results, the gradients of the losses) and
// somebody keeps stays where every replay writes it when its address is asked for; a slice of it goes elsewhere.
void kept_results_stay_where_they_are_written() {
  using Tn = Tensor<B>;
  const size_t T = 4, Bn = 2, V = 3, H = 2;
  for (bool states : {true, false}) {  // with states kept the backward pass goes timestep by timestep
    const Tn x(make({T * Bn, V}, 0.f, .01f), false), y(make({T * Bn, V}, 0.f, .01f), false), w(make({V + H, 4 * H}, 0.f, .01f), true);
    const Tn b(make({4 * H}, 0.f, .01f), true), wo(make({H, V}, 0.f, .1f), true), bo(make({V}, 0.f, .1f), true);
    std::vector<Tn> kept;
    std::vector<B::Storage> slices;
    B::begin_capture();
    Tn sum;
    {
      Tn h = Tn::zeros({Bn, H}, false), c = Tn::zeros({Bn, H}, false);
      for (size_t t = 0; t < T; ++t) {
        const Tn xh = ops::concat<B>({ops::slice(x, {{t * Bn, (t + 1) * Bn}, {0, V}}), h}, 1);
        const Tn z = ops::add(ops::matmul(xh, w), b.broadcast_to({Bn, 4 * H}));
        auto gate = [&](size_t k) { return ops::slice(z, {{0, Bn}, {k * H, (k + 1) * H}}); };
        const Tn i = ops::sigmoid(gate(0)), f = ops::sigmoid(gate(1));
        c = ops::add(ops::mul(f, c), ops::mul(i, ops::tanh(gate(2))));
        h = ops::mul(ops::sigmoid(gate(3)), ops::tanh(c));
        const Tn logits = ops::add(ops::matmul(h, wo), bo.broadcast_to({Bn, V}));
        const Tn l = ops::softmax_cross_entropy(logits, ops::slice(y, {{t * Bn, (t + 1) * Bn}, {0, V}}), 1, Reduction::Mean);
        sum = t ? ops::add(sum, l) : l;
        if (t == 1) kept = states ? std::vector<Tn>{logits, h, c, i} : std::vector<Tn>{logits};
      }
    }
    sum.backward();
    for (auto& g : {sum.data(), *w.grad(), *b.grad(), *wo.grad(), *bo.grad()}) B::own(g);
    slices = {B::slice(kept[0].data(), {{1, 2}, {0, V}}), B::slice(kept[0].data(), {{1, 2}, {0, V}})};
    sum.detach_graph();
    std::vector<B::Storage> all;
    for (auto& k : kept) all.push_back(k.data());
    if (!states) all.push_back(*kept[0].grad());
    std::vector<float*> where;
    for (auto& s : all) where.push_back(s.ptr());
    for (auto& s : all) EXPECT(s.buf->owner != nullptr);
    for (auto& s : slices) EXPECT(s.ptr() == where[0] + V);
    rt_graph* graph = nullptr;
    B::end_capture(&graph);
    for (size_t k = 0; k < all.size(); ++k) {
      EXPECT(B::escape(all[k]) == where[k]);
      scribble(where[k], all[k].numel());
      EXPECT(all[k].ptr() == where[k]);
    }
    EXPECT(B::escape(slices[0]) != where[0] + V);
    B::Storage logits = kept[0].data();
    all.clear();
    kept.clear();
    B::make_unique(logits);  // the other slice still reads the rows
    EXPECT(logits.ptr() != where[0] && slices[1].ptr() == where[0] + V);
    slices.clear();
    float* const own = logits.ptr();
    B::make_unique(logits);
    EXPECT(logits.ptr() == own);
  }
  EXPECT(live.empty());
}

// However long a recurrence in a capture is, evaluating it and letting go of it takes a bounded stack, whatever is asked for first.
void long_recurrences() {
  using Tn = Tensor<B>;
  const size_t T = 20000, Bn = 1, V = 1, H = 1;
  enum { kGateFirst, kInputFirst, kLastGateAlone, kCellState, kOfTheLastState, kNothing, kWays };
  for (int way = 0; way < kWays; ++way) {
    forward_sequences = 0;
    {
      const Tn x(make({T * Bn, V}, 0.f, .01f), false), w(make({V + H, 4 * H}, 0.f, .01f), true), b(make({4 * H}, 0.f, .01f), true);
      B::begin_capture();
      {
        Tn h = Tn::zeros({Bn, H}, false), c = Tn::zeros({Bn, H}, false), asked;
        for (size_t t = 0; t < T; ++t) {
          const Tn xt = ops::slice(x, {{t * Bn, (t + 1) * Bn}, {0, V}}), xh = ops::concat<B>({xt, h}, 1);
          const Tn z = ops::add(ops::matmul(xh, w), b.broadcast_to({Bn, 4 * H}));
          auto gate = [&](size_t k) { return ops::slice(z, {{0, Bn}, {k * H, (k + 1) * H}}); };
          const Tn i = ops::sigmoid(gate(0)), f = ops::sigmoid(gate(1));
          c = ops::add(ops::mul(f, c), ops::mul(i, ops::tanh(gate(2))));
          h = ops::mul(ops::sigmoid(gate(3)), ops::tanh(c));
          if (way == kGateFirst && t == 3) asked = f;
          if (way == kInputFirst && t == 3) asked = xt;
          if (way == kLastGateAlone && t + 1 == T) asked = i;
          if (way == kCellState && t + 1 == T) asked = c;
          if (way == kOfTheLastState && t + 1 == T) asked = ops::square(ops::exp(h));
          if (way == kLastGateAlone) {  // no tape: nothing but the next timestep holds a state
            h.detach_graph();
            c.detach_graph();
          }
        }
        if (way == kLastGateAlone) h = c = Tn();
        if (asked.inner) asked.data().ptr();
        if (way == kGateFirst || way == kInputFirst) h.data().ptr();
      }
      rt_graph* graph = nullptr;
      B::end_capture(&graph);
    }
    EXPECT(forward_sequences == (way == kNothing ? 0 : 1));  // of the timesteps that are one still
    EXPECT(live.empty() && !DeviceBuffer::head());
  }
}

// A capture that goes on in another graph in the middle of the backward pass (an exchange of the gradients that are ready runs between the two):
// everything is in one of the graphs.
void a_capture_in_two_parts() {
  using Tn = Tensor<B>;
  const size_t T = 4, Bn = 2, V = 3, H = 2;
  {
    const Tn x(make({T * Bn, V}, 0.f, .01f), false), w(make({V + H, 4 * H}, 0.f, .01f), true), b(make({4 * H}, 0.f, .01f), true);
    const Tn wo(make({H, V}, 0.f, .1f), true), bo(make({V}, 0.f, .1f), true);
    rt_graph *first = nullptr, *second = nullptr;
    int ready = 0;
    B::begin_capture();
    unrecorded = 0;
    {
      Tn h = Tn::zeros({Bn, H}, false), c = Tn::zeros({Bn, H}, false), sum;
      for (size_t t = 0; t < T; ++t) {
        const Tn z = ops::add(ops::matmul(ops::concat<B>({ops::slice(x, {{t * Bn, (t + 1) * Bn}, {0, V}}), h}, 1), w), b.broadcast_to({Bn, 4 * H}));
        auto gate = [&](size_t k) { return ops::slice(z, {{0, Bn}, {k * H, (k + 1) * H}}); };
        c = ops::add(ops::mul(ops::sigmoid(gate(1)), c), ops::mul(ops::sigmoid(gate(0)), ops::tanh(gate(2))));
        h = ops::mul(ops::sigmoid(gate(3)), ops::tanh(c));
        const Tn l = ops::sum(ops::square(ops::add(ops::matmul(h, wo), bo.broadcast_to({Bn, V}))), std::nullopt);
        sum = t ? ops::add(sum, l) : l;
      }
      Tn::leaf_ready_hook() = [&](const Tn& leaf) {
        if (ready++ > 0) return;
        B::own(*leaf.grad());
        B::split_capture(&first);
      };
      sum.backward();
      Tn::leaf_ready_hook() = nullptr;
      for (auto& g : {sum.data(), *w.grad(), *b.grad(), *wo.grad(), *bo.grad()}) B::own(g);
      sum.detach_graph();
    }
    B::end_capture(&second);
    EXPECT(ready == 4 && unrecorded == 0);
  }
  EXPECT(live.empty());
}

// A program that no kernel with a reduction has been compiled for takes no memory before it is refused.
void refused_programs_take_no_memory() {
  {
    const B::Storage x = make({4, 8}, 0.f), b = make({8}, 0.f);
    const B::Storage y = B::add(B::tanh(B::mul(x, b)), x);
    mallocs = 0;
    const B::Storage lse = B::logsumexp(y, 1);
    EXPECT(!y.buf->node && mallocs == 2);
    const B::Storage u = B::mul(x, b), v = B::exp(u), sums = B::unbroadcast(B::mul(B::tanh(u), x), {8});
    mallocs = 0;
    v.ptr();
    EXPECT(!v.buf->node && mallocs <= 2);  // v, and u beside it, which somebody holds
    sums.ptr();
  }
  {  // nor is one built whose ops are not those of any
    const B::Storage x = make({4, 8}, 0.f), b = make({8}, 0.f);
    for (bool other : {false, true}) {
      possible_ops = uint64_t(1) << RT_F_TANH | uint64_t(1) << RT_F_ADD | uint64_t(1) << RT_F_MUL;
      asked_of_programs = 0;
      B::logsumexp(B::add(B::tanh(B::mul(x, b)), other ? B::exp(x) : x), 1).ptr();
      EXPECT(asked_of_programs == (other ? 0 : 1));
      possible_ops = ~uint64_t(0);
    }
  }
  EXPECT(live.empty());
}

// A logsumexp is computed whatever else waits for what its rows are made of: the rows may be evaluated by looking at that.
void logsumexps_are_computed() {
  for (bool known : {false, true})
    for (bool whole : {false, true}) {
      reductions_known = known;
      const B::Storage x = make({4, 8}, 0.f), b = make({8}, 0.f);
      const B::Storage h = B::tanh(x), y = B::add(h, B::broadcast_to(b, {4, 8}));
      const B::Storage s = B::reduce(RT_RED_SUM, y, whole ? std::optional<size_t>() : std::optional<size_t>(0));
      const B::Storage sums = B::unbroadcast(B::mul(h, B::broadcast_to(s, {4, 8})), {8});
      EXPECT(sums.buf->node != nullptr);
      logsumexps = 0;
      const B::Storage lse = B::logsumexp(y, 1);
      EXPECT(logsumexps == 1 && !y.buf->node);
      sums.ptr();
      reductions_known = false;
    }
  EXPECT(live.empty());
}

// The gradient of a logsumexp is part of a program that carries a reduction, where there is one; elsewhere it has a kernel of its own, which the
// program around it reads.
void gradients_of_rows() {
  for (bool known : {false, true}) {
    B::Storage x = make({4, 8}, 0.f), b = make({8}, 0.f);
    const B::Storage y = B::tanh(B::add(x, b)), lse = B::logsumexp(y, 1);
    Op<B> o(OpType::with_axis(OpType::LogSumExp, 1), {Tensor<B>(y, true)}, nullptr);
    o.cached_outputs = lse;
    reductions_known = known;
    row_gradients = programs = 0;
    const B::Storage d = B::logsumexp_backward(o, make({4}, 1.f)), dx = B::lz_mul(d, B::lz_unary(RT_F_ONE_MINUS_SQUARE, y));
    const B::Storage db = B::unbroadcast(B::lz_mul(dx, x), {8});
    EXPECT(d.buf->node && row_gradients == 0);
    dx.ptr();
    EXPECT(row_gradients == (known ? 0 : 1) && programs == (known ? 0 : 1));
    db.ptr();
    reductions_known = false;
  }
  {  // what it reads changes in place: it is computed before
    B::Storage x = make({4, 8}, 3.f);
    const B::Storage lse = B::logsumexp(x, 1);
    Op<B> o(OpType::with_axis(OpType::LogSumExp, 1), {Tensor<B>(x, true)}, nullptr);
    o.cached_outputs = lse;
    const B::Storage d = B::logsumexp_backward(o, make({4}, 1.f));
    EXPECT(d.buf->node != nullptr);
    scribble(B::escape(x), 32);
    EXPECT(!d.buf->node && holds(d, 3.f));
  }
  EXPECT(live.empty() && DeviceBuffer::row_gradients() == 0);
}

const struct {
  const char* name;
  void (*run)();
} kChecks[] = {{"cells_become_a_sequence", cells_become_a_sequence}, {"long_recurrences", long_recurrences}, {"recurrences_have_their_values", recurrences_have_their_values}, {"gradients_of_rows", gradients_of_rows}, {"logsumexps_are_computed", logsumexps_are_computed}, {"refused_programs_take_no_memory", refused_programs_take_no_memory}, {"a_capture_in_two_parts", a_capture_in_two_parts},
               {"kept_results_stay_where_they_are_written", kept_results_stay_where_they_are_written},
               {"rows_do_not_alias", rows_do_not_alias}, {"rows_in_a_capture", rows_in_a_capture},
               {"broadcast_does_not_alias", broadcast_does_not_alias},
               {"pooling_knows_its_relu", pooling_knows_its_relu},
               {"errors_lose_nothing", errors_lose_nothing},
               {"written_from_outside", written_from_outside},
               {"a_product_of_a_matrix_with_itself", a_product_of_a_matrix_with_itself}};

}  // namespace

int main(int argc, char** argv) {
  B::ctx_slot() = reinterpret_cast<rt_ctx*>(&failures);  // never looked into
  for (auto& c : kChecks)
    if (argc == 2 && std::strcmp(argv[1], c.name) == 0) {
      c.run();
      return failures ? 1 : 0;
    }
  std::printf("unknown check\n");
  return 2;
}
