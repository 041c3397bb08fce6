// `B200Backend`: the Backend implementation that forwards every trait method of the
// reference (src/backend/mod.rs:14-656) to one C-ABI entry point of librt_b200.so
// (include/rt_b200.h).  This is the C++ twin of the Rust shim a maintainer would write
// as `impl Backend for B200Backend`; it owns no math, only shape bookkeeping (integer,
// host side) and device-buffer lifetime.
//
// Storage is a reference-counted device buffer plus a shape.  Buffers are immutable once
// produced by an op, so copying a Storage is O(1) yet indistinguishable from the deep
// copy the reference's `Clone` performs; the in-place mutators (optimizer steps,
// update_from_host) first make the buffer unique.
#pragma once
#include <algorithm>
#include <memory>
#include <cmath>
#include <cstring>
#include <optional>
#include <random>
#include <tuple>
#include <unordered_map>
#include <vector>

#include "../../../include/rt_b200.h"
#include "autograd.hpp"
#include "lazy.hpp"

namespace rt {

struct DeviceStorage {
  std::shared_ptr<DeviceBuffer> buf;
  Shape shape;
  float* ptr() const { return buf ? buf->data() : nullptr; }  // evaluates a deferred expression
  size_t numel() const { return shape_numel(shape); }
};

struct B200Backend {
  using Storage = DeviceStorage;
  using OpB = Op<B200Backend>;

  static rt_ctx*& ctx_slot() {
    static rt_ctx* c = nullptr;
    return c;
  }
  static rt_ctx* ctx() {
    if (!ctx_slot()) throw Error(ErrorKind::CudaError, "B200Backend: no context (call rth_init first)");
    return ctx_slot();
  }
  static void check(rt_status st) {
    if (st != RT_OK) throw Error((ErrorKind)st, rt_last_error(ctx_slot()));
  }
  static std::vector<int64_t> dims(const Shape& s) { return std::vector<int64_t>(s.begin(), s.end()); }

  static Storage alloc(const Shape& s) {
    size_t n = shape_numel(s);
    void* p = nullptr;
    check(rt_malloc(ctx(), sizeof(float) * std::max<size_t>(n, 1), &p));
    return Storage{std::make_shared<DeviceBuffer>(ctx(), (float*)p, n), s};
  }
  // Before a buffer is changed in place: deferred expressions that read it are evaluated, and a buffer that somebody else
  // holds too is replaced by a copy.
  static void make_unique(Storage& s) {
    if (!s.buf) return;
    s.buf->data();
    bool costly = false;  // a product or convolution that nobody has asked for yet: keep its operand instead of computing it
    if (!s.buf->escaped)
      for (auto* r : s.buf->readers) costly = costly || r->node->kind == lazy::Kind::Opaque;
    if (!costly) s.buf->flush_readers();
    if (s.buf.use_count() > 1 || s.buf->shares_rows()) {
      Storage c = alloc(s.shape);
      check(rt_memcpy_d2d(ctx(), c.ptr(), s.ptr(), sizeof(float) * s.numel()));
      s.buf = std::move(c.buf);
    }
    s.buf->id = DeviceBuffer::next_id();
  }

  // ---- deferred elementwise ops (lazy.hpp) --------------------------------------------------------------------------
  static bool deferrable(const Shape& s) {
    const size_t n = shape_numel(s);
    return lazy::deferring() && n > 0 && n < ((size_t)1 << 31) && s.size() <= (size_t)lazy::kMaxRawDims;
  }
  static Storage defer(lazy::Node n, const Shape& shape) {
    bool now;
    Storage s = pend(std::move(n), shape, &now);
    if (now) s.buf->data();
    return s;
  }
  // The same, but left to the caller to evaluate when it has to be done `now`.
  static Storage pend(lazy::Node n, const Shape& shape, bool* at_once) {
    n.shape = shape;
    bool now = false;
    for (auto& i : n.in) {
      if (i.buf->node) {
        n.depth = std::max(n.depth, i.buf->node->depth + 1);
        n.weight += i.buf->node->weight;
      }
      now = now || (i.buf->escaped && !lazy::capturing());
    }
    const bool scalar_sum = n.kind == lazy::Kind::Binary && n.op == RT_F_ADD && shape_numel(shape) == 1;
    now = now || n.depth >= (scalar_sum ? lazy::kMaxChain : lazy::kMaxDepth);
    n.weight = std::min(n.weight, 1 << 20);
    if (n.tag == lazy::Tag::Matmul) n.depth = 1;  // of a sequence, which is evaluated from its first timestep on
    *at_once = now;
    return Storage{std::make_shared<DeviceBuffer>(ctx(), std::make_unique<lazy::Node>(std::move(n)), shape_numel(shape)), shape};
  }
  static lazy::Input input(const Storage& x) { return lazy::Input{x.buf, x.shape}; }
  static bool is_const(const Storage& x) { return x.buf && x.buf->node && x.buf->node->kind == lazy::Kind::Const; }
  static Storage lz_unary(uint8_t op, const Storage& x, float imm = 0.f) {
    lazy::Node n{lazy::Kind::Unary};
    n.op = op;
    n.imm = imm;
    n.weight = lazy::op_weight(op);
    n.in.push_back(input(x));
    Storage y = defer(std::move(n), x.shape);
    y.buf->made_from = x.buf->id;
    return y;
  }
  static Storage lz_imm(uint8_t op, const Storage& x, float imm, bool swap = false) {
    if (is_const(x)) {  // both operands known: the same IEEE operation here (a loss gradient starts as a chain of these)
      const float c = x.buf->node->imm;
      if (op == RT_F_MUL) return filled(x.shape, c * imm);
      if (op == RT_F_DIV && !swap) return filled(x.shape, c / imm);
    }
    lazy::Node n{lazy::Kind::BinaryImm};
    n.op = op;
    n.imm = imm;
    n.swap = swap;
    n.weight = lazy::op_weight(op);
    n.in.push_back(input(x));
    return defer(std::move(n), x.shape);
  }
  static Storage lz_binary(uint8_t op, const Storage& a, const Storage& b, const Shape& shape) {
    if (is_const(a) && is_const(b) && op == RT_F_MUL) return filled(shape, a.buf->node->imm * b.buf->node->imm);
    lazy::Node n{lazy::Kind::Binary};
    n.op = op;
    n.weight = lazy::op_weight(op);
    n.in.push_back(input(a));
    n.in.push_back(input(b));
    return defer(std::move(n), shape);
  }
  static Storage lz_mul(const Storage& a, const Storage& b) { return lz_binary(RT_F_MUL, a, b, a.shape); }
  static Storage lz_box(lazy::Kind kind, const Storage& x, const Shape& shape, Shape starts) {
    if (kind == lazy::Kind::Broadcast && is_const(x)) return filled(shape, x.buf->node->imm);
    lazy::Node n{kind};
    n.starts = std::move(starts);
    n.in.push_back(input(x));
    return defer(std::move(n), shape);
  }
  // A result with a kernel of its own.  `run` gets the node and the block to fill.
  template <class F>
  static Storage lz_opaque(lazy::Tag tag, std::vector<int64_t> geo, std::vector<lazy::Input> in, const Shape& shape, F run) {
    lazy::Node n{lazy::Kind::Opaque};
    n.tag = tag;
    n.geo = std::move(geo);
    n.in = std::move(in);
    n.weight = 1 << 10;
    n.run = [run](lazy::Node& nd, DeviceBuffer* b) {
      lazy::Block out(b->ctx, b->numel);
      check(run(nd, out.ptr));
      b->ptr = out.release();
    };
    return defer(std::move(n), shape);
  }
  // Rows that point into another tensor's block (a slice taken inside a capture) get a block of their own.  Results that were computed as
  // rows of one matrix have theirs to themselves already, and replays of the capture go on writing there.
  static void own(const Storage& s) {
    if (!s.buf) return;
    const float* p = s.buf->data();
    if (!s.buf->shares_rows()) return;
    lazy::Block block(ctx(), s.buf->numel);
    check(rt_memcpy_d2d(ctx(), block.ptr, p, sizeof(float) * s.buf->numel));
    s.buf->ptr = block.release();
    s.buf->owner.reset();
  }
  // The address of a tensor's values for use outside the engine: whoever has it may write there at any time.
  static float* escape(const Storage& s) {
    if (!s.buf) return nullptr;
    own(s);
    s.buf->flush_readers();
    s.buf->escaped = true;
    return s.buf->ptr;
  }
  static void begin_capture() {
    lazy::flush_all();  // what was asked for before the capture must not become part of the graph
    check(rt_graph_begin(ctx()));
    lazy::capturing() = true;
  }
  static void end_capture(rt_graph** out) {
    lazy::capturing() = false;
    check(rt_graph_end(ctx(), out));
  }
  // Goes on in another graph.  What is still deferred belongs to the first: between the two it would be computed once, and no replay would
  // compute it again.
  static void split_capture(rt_graph** first) {
    lazy::flush_all();
    end_capture(first);
    begin_capture();
  }

  // ---- factories / access (mod.rs:44-88, 248-252) --------------------------------------
  static Storage filled(const Shape& s, float v) {
    if (deferrable(s)) {
      lazy::Node n{lazy::Kind::Const};
      n.imm = v;
      return defer(std::move(n), s);
    }
    Storage r = alloc(s);
    check(rt_fill(ctx(), r.ptr(), v, (int64_t)r.numel()));
    return r;
  }
  static Storage zeros(const Shape& s) { return filled(s, 0.f); }
  static Storage ones(const Shape& s) { return filled(s, 1.f); }
  static Storage from_vec(std::vector<float> v, const Shape& s) {
    if (v.size() != shape_numel(s)) throw Error::shape_mismatch(s, Shape{v.size()});
    if (v.size() == 1) return filled(s, v[0]);  // a constant: no host copy, safe inside graph capture
    Storage r = alloc(s);
    check(rt_memcpy_h2d(ctx(), r.ptr(), v.data(), sizeof(float) * v.size()));
    return r;
  }
  // ---- random factories (mod.rs:57-69; src/backend/cpu.rs:133-194; src/init.rs:7-52) ------------------------
  // The generator state is (seed, counter offset); manual_seed restarts the stream.  Without a seed the first use
  // takes one from the operating system, like rand's thread-local generator.
  struct RngState { uint64_t seed = 0, offset = 0; bool seeded = false; };
  static RngState& rng() {
    static RngState s;
    return s;
  }
  static void manual_seed(uint64_t seed) { rng() = RngState{seed, 0, true}; }
  static RngState& rng_ready() {
    RngState& s = rng();
    if (!s.seeded) {
      std::random_device rd;
      s = RngState{((uint64_t)rd() << 32) ^ rd(), 0, true};
    }
    return s;
  }
  static Storage random_uniform(const Shape& shape, float low, float high) {
    if (shape_numel(shape) == 0) return zeros(shape);
    RngState& s = rng_ready();
    Storage r = alloc(shape);
    check(rt_random_uniform(ctx(), r.ptr(), (int64_t)r.numel(), low, high, s.seed, s.offset));
    s.offset += (r.numel() + 3) / 4;
    return r;
  }
  static Storage random_normal(const Shape& shape, float mean, float std_dev) {
    if (shape_numel(shape) == 0) return zeros(shape);
    RngState& s = rng_ready();
    Storage r = alloc(shape);
    check(rt_random_normal(ctx(), r.ptr(), (int64_t)r.numel(), mean, std_dev, s.seed, s.offset));
    s.offset += (r.numel() + 3) / 4;
    return r;
  }
  static Storage bernoulli(const Shape& shape, float p) {
    if (shape_numel(shape) == 0) return zeros(shape);
    RngState& s = rng_ready();
    Storage r = alloc(shape);
    check(rt_bernoulli(ctx(), r.ptr(), (int64_t)r.numel(), p, s.seed, s.offset));
    s.offset += (r.numel() + 3) / 4;
    return r;
  }
  static Storage kaiming_uniform(size_t fan_in, const Shape& shape) {  // src/init.rs:7-52
    if (shape.empty()) throw Error::invalid_op("Cannot initialize tensor with empty shape");
    if (shape_numel(shape) == 0) return zeros(shape);
    if (fan_in == 0) throw Error::invalid_op("Fan-in cannot be zero for Kaiming initialization");
    const float bound = std::sqrt(6.0f / (float)fan_in);
    return random_uniform(shape, -bound, bound);
  }
  // Rows idx[i] of x viewed as [rows, row_len] -> [idx.size(), row_len] (the gather of data::get_random_batch on the
  // device: only the indices travel).  Indices are checked on the host.
  static Storage gather_rows(const Storage& x, size_t rows, size_t row_len, const std::vector<size_t>& idx) {
    std::vector<int32_t> h(idx.size());
    for (size_t i = 0; i < idx.size(); ++i) {
      if (idx[i] >= rows) throw Error(ErrorKind::InvalidIndex, "gather_rows: index out of range");
      h[i] = (int32_t)idx[i];
    }
    Storage out = alloc(Shape{idx.size(), row_len});
    if (idx.empty() || row_len == 0) return out;
    const float* src = x.ptr();
    void* d = nullptr;
    check(rt_malloc(ctx(), sizeof(int32_t) * h.size(), &d));
    rt_status st = rt_memcpy_h2d(ctx(), d, h.data(), sizeof(int32_t) * h.size());
    if (st == RT_OK) st = rt_gather_rows(ctx(), src, (int64_t)rows, (int64_t)row_len, static_cast<const int32_t*>(d), (int64_t)h.size(), out.ptr());
    rt_free(ctx(), d);
    check(st);
    return out;
  }
  static const Shape& shape(const Storage& s) { return s.shape; }
  static size_t size(const Storage& s) { return s.numel(); }
  static std::vector<float> copy_to_host(const Storage& s) {
    std::vector<float> v(s.numel());
    check(rt_memcpy_d2h(ctx(), v.data(), s.ptr(), sizeof(float) * v.size()));
    return v;
  }
  static void update_from_host(Storage& s, const std::vector<float>& d) {
    if (s.numel() != d.size()) throw Error::shape_mismatch(s.shape, Shape{d.size()});
    make_unique(s);
    check(rt_memcpy_h2d(ctx(), s.ptr(), d.data(), sizeof(float) * d.size()));
  }
  static void set_data(Storage& s, Storage d) { s = std::move(d); }
  static Storage reshaped(Storage s, const Shape& shape) {
    set_shape(s, shape);
    return s;
  }
  static void set_shape(Storage& s, const Shape& shape) {
    if (shape_numel(shape) != s.numel()) throw Error::shape_mismatch(shape, s.shape);
    s.shape = shape;
  }
  // Gradient slot of an input that never receives a gradient (the index tensor of
  // max_pool2d): the reference allocates zeros that are dropped unread.
  static Storage unused_grad(const Shape& s) { return Storage{nullptr, s}; }

  // ---- elementwise -----------------------------------------------------------------------
  static Storage unary(int op, const Storage& x, float p0 = 0.f, float p1 = 0.f) {
    if (deferrable(x.shape)) {
      switch (op) {
        case RT_RELU: return lz_unary(RT_F_RELU, x);
        case RT_ELU: return lz_unary(RT_F_ELU, x, p0);
        case RT_EXP: return lz_unary(RT_F_EXP, x);
        case RT_LN: return lz_unary(RT_F_LN, x);
        case RT_SIN: return lz_unary(RT_F_SIN, x);
        case RT_COS: return lz_unary(RT_F_COS, x);
        case RT_TAN: return lz_unary(RT_F_TAN, x);
        case RT_TANH: return lz_unary(RT_F_TANH, x);
        case RT_SIGMOID: return lz_unary(RT_F_SIGMOID, x);
        case RT_SOFTPLUS: return lz_unary(RT_F_SOFTPLUS, x);
        case RT_SQUARE: return lz_unary(RT_F_SQUARE, x);
        case RT_SQRT: return lz_unary(RT_F_SQRT, x);
        case RT_ABS: return lz_unary(RT_F_ABS, x);
        case RT_CLIP: return lz_imm(RT_F_MIN, lz_imm(RT_F_MAX, x, p0), p1);
        case RT_MUL_SCALAR: return lz_imm(RT_F_MUL, x, p0);
        case RT_DIV_SCALAR: return lz_imm(RT_F_DIV, x, p0);
        default: break;
      }
    }
    Storage y = alloc(x.shape);
    check(rt_unary(ctx(), op, x.ptr(), y.ptr(), (int64_t)x.numel(), p0, p1));
    return y;
  }
  static Storage unary_bwd(int op, const OpB& o, const Storage& g, float p0 = 0.f, float p1 = 0.f) {
    if (o.inputs.empty()) throw Error::invalid_op("backward requires 1 input");
    const Storage& x = o.inputs[0].data();
    if (x.shape != g.shape) throw Error::shape_mismatch(x.shape, g.shape);
    if (deferrable(x.shape)) {  // g * f'(x), each f' in the form of the stand-alone kernel
      // where f' follows from f(x), which the forward pass has (unless x or the result may have been changed since)
      if (o.cached_outputs && o.cached_outputs->buf && o.cached_outputs->buf->made_from == x.buf->id &&
          ((!x.buf->escaped && !o.cached_outputs->buf->escaped) || lazy::capturing())) {
        const Storage& y = *o.cached_outputs;
        switch (op) {
          case RT_RELU: return lz_mul(g, lz_unary(RT_F_STEP, y));
          case RT_EXP: return lz_mul(g, y);
          case RT_TANH: return lz_mul(g, lz_unary(RT_F_ONE_MINUS_SQUARE, y));
          case RT_SIGMOID: return lz_mul(g, lz_unary(RT_F_LOGISTIC_SLOPE, y));
          default: break;
        }
      }
      switch (op) {
        case RT_RELU: return lz_mul(g, lz_unary(RT_F_STEP, x));
        case RT_ELU: return lz_mul(g, lz_unary(RT_F_ELU_SLOPE, x, p0));
        case RT_EXP: return lz_mul(g, lz_unary(RT_F_EXP, x));
        case RT_LN: return lz_mul(g, lz_unary(RT_F_RECIP, x));
        case RT_SIN: return lz_mul(lz_unary(RT_F_COS, x), g);
        case RT_COS: return lz_mul(lz_unary(RT_F_NEG, lz_unary(RT_F_SIN, x)), g);
        case RT_TAN: return lz_mul(g, lz_unary(RT_F_RECIP_SQUARE, lz_unary(RT_F_COS, x)));
        case RT_TANH: return lz_mul(g, lz_unary(RT_F_ONE_MINUS_SQUARE, lz_unary(RT_F_TANH, x)));
        case RT_SIGMOID: return lz_mul(g, lz_unary(RT_F_LOGISTIC_SLOPE, lz_unary(RT_F_SIGMOID, x)));
        case RT_SOFTPLUS: return lz_mul(g, lz_unary(RT_F_SIGMOID, x));
        case RT_SQUARE: return lz_mul(g, lz_imm(RT_F_MUL, x, 2.f));
        case RT_SQRT: return lz_mul(g, lz_unary(RT_F_HALF_RSQRT, x));
        case RT_ABS: return lz_mul(g, lz_unary(RT_F_SIGN, x));
        case RT_CLIP: return lz_mul(g, lz_mul(lz_imm(RT_F_GE, x, p0), lz_imm(RT_F_LE, x, p1)));
        default: break;
      }
    }
    Storage dx = alloc(x.shape);
    check(rt_unary_backward(ctx(), op, x.ptr(), g.ptr(), dx.ptr(), (int64_t)x.numel(), p0, p1));
    return dx;
  }
  // Broadcast shape.  For add/mul/powf/maximum/minimum/comparisons the reference takes the larger
  // extent when one side is 1 and then asks ndarray to stretch each operand, which fails when an
  // extent 0 meets an extent 1 (src/ops/cpu_ops.rs:319-352; src/util.rs:2-26); sub/div use ndarray's
  // operator broadcasting, where 1 stretches to 0 (src/backend/cpu.rs:1259-1269).
  static Shape bshape(const Shape& a, const Shape& b, const char* op, bool ndarray_operator = false) {
    size_t nd = std::max(a.size(), b.size());
    Shape out(nd);
    for (size_t i = 0; i < nd; ++i) {
      size_t ad = i < nd - a.size() ? 1 : a[i - (nd - a.size())];
      size_t bd = i < nd - b.size() ? 1 : b[i - (nd - b.size())];
      if (ad == bd) out[i] = ad;
      else if (ad == 1 || bd == 1) {
        out[i] = ndarray_operator ? (ad == 1 ? bd : ad) : std::max(ad, bd);
        if ((out[i] != ad && ad != 1) || (out[i] != bd && bd != 1)) throw Error::incompatible(op, a, b);
      } else throw Error::incompatible(op, a, b);
    }
    return out;
  }
  static bool is_operator_op(int op) { return op == RT_SUB || op == RT_DIV; }
  static Storage binary(int op, const Storage& a, const Storage& b, const char* name) {
    const Shape os = bshape(a.shape, b.shape, name, is_operator_op(op));
    if (deferrable(os)) return lz_binary((uint8_t)(RT_F_ADD + (op - RT_ADD)), a, b, os);
    Storage out = alloc(os);
    auto as = dims(a.shape), bs = dims(b.shape);
    check(rt_binary(ctx(), op, a.ptr(), as.data(), (int)as.size(), b.ptr(), bs.data(), (int)bs.size(), out.ptr()));
    return out;
  }
  // d/da (or d/db) of a binary op times g, over g's shape, in the form of the stand-alone kernels
  static Storage binary_term(int op, const Storage& a, const Storage& b, const Storage& g, bool second) {
    const Shape& s = g.shape;
    switch (op) {
      case RT_ADD: return g;
      case RT_SUB: return second ? lz_unary(RT_F_NEG, g) : g;
      case RT_MUL: return lz_binary(RT_F_MUL, g, second ? a : b, s);
      case RT_DIV:
        if (!second) return lz_binary(RT_F_MUL, g, lz_unary(RT_F_RECIP, b), s);
        return lz_mul(g, lz_unary(RT_F_NEG, lz_binary(RT_F_DIV, a, lz_binary(RT_F_MUL, b, b, b.shape), s)));
      case RT_POWF:
        if (!second) return lz_mul(g, lz_binary(RT_F_MUL, b, lz_binary(RT_F_POWF, a, lz_imm(RT_F_SUB, b, 1.f), s), s));
        return lz_mul(g, lz_binary(RT_F_MUL, lz_binary(RT_F_POWF, a, b, s), lz_unary(RT_F_LN, a), s));
      case RT_MAXIMUM: return lz_mul(g, second ? lz_binary(RT_F_GT, b, a, s) : lz_binary(RT_F_GE, a, b, s));
      case RT_MINIMUM: return lz_mul(g, second ? lz_binary(RT_F_LT, b, a, s) : lz_binary(RT_F_LE, a, b, s));
      default: return filled(s, 0.f);  // comparisons
    }
  }
  static Storage reduced(const Storage& term, const Shape& target) { return unbroadcast(term, target); }
  static std::pair<Storage, Storage> binary_bwd(int op, const OpB& o, const Storage& g, const char* name) {
    if (o.inputs.size() != 2) throw Error::invalid_op(std::string(name) + " requires 2 inputs");
    const Storage& a = o.inputs[0].data();
    const Storage& b = o.inputs[1].data();
    Shape os = bshape(a.shape, b.shape, name, is_operator_op(op));
    if (g.numel() != shape_numel(os)) throw Error::incompatible(name, os, g.shape);
    bool need_a = o.inputs[0].requires_grad(), need_b = o.inputs[1].requires_grad();
    if (deferrable(os)) {
      // each term over the full shape; the side that was stretched is then summed down to its own shape
      Storage gf = g;
      set_shape(gf, os);
      Storage da = need_a ? reduced(binary_term(op, a, b, gf, false), a.shape) : Storage{nullptr, a.shape};
      Storage db = need_b ? reduced(binary_term(op, a, b, gf, true), b.shape) : Storage{nullptr, b.shape};
      return {std::move(da), std::move(db)};
    }
    Storage da = need_a ? alloc(a.shape) : Storage{nullptr, a.shape};
    Storage db = need_b ? alloc(b.shape) : Storage{nullptr, b.shape};
    auto as = dims(a.shape), bs = dims(b.shape);
    check(rt_binary_backward(ctx(), op, a.ptr(), as.data(), (int)as.size(), b.ptr(), bs.data(), (int)bs.size(), g.ptr(),
                             da.ptr(), db.ptr()));
    return {std::move(da), std::move(db)};
  }
  static Storage mul(const Storage& a, const Storage& b) { return binary(RT_MUL, a, b, "mul"); }
  static Storage add(const Storage& a, const Storage& b) { return binary(RT_ADD, a, b, "add"); }
  static Storage sub(const Storage& a, const Storage& b) { return binary(RT_SUB, a, b, "sub"); }
  static Storage div(const Storage& a, const Storage& b) { return binary(RT_DIV, a, b, "div"); }
  static Storage powf(const Storage& a, const Storage& b) { return binary(RT_POWF, a, b, "powf"); }
  static Storage maximum(const Storage& a, const Storage& b) { return binary(RT_MAXIMUM, a, b, "maximum"); }
  static Storage minimum(const Storage& a, const Storage& b) { return binary(RT_MINIMUM, a, b, "minimum"); }
  static Storage equal(const Storage& a, const Storage& b) { return binary(RT_EQUAL, a, b, "equal"); }
  static Storage not_equal(const Storage& a, const Storage& b) { return binary(RT_NOT_EQUAL, a, b, "not_equal"); }
  static Storage greater(const Storage& a, const Storage& b) { return binary(RT_GREATER, a, b, "greater"); }
  static Storage greater_equal(const Storage& a, const Storage& b) { return binary(RT_GREATER_EQUAL, a, b, "greater_equal"); }
  static Storage less(const Storage& a, const Storage& b) { return binary(RT_LESS, a, b, "less"); }
  static Storage less_equal(const Storage& a, const Storage& b) { return binary(RT_LESS_EQUAL, a, b, "less_equal"); }
  // true when `small` (rank <= rank of `full`, no empty axis) broadcasts onto `full` by stretching 1s only
  static bool stretches_onto(const Shape& small, const Shape& full) {
    if (small.size() > full.size()) return false;
    const size_t off = full.size() - small.size();
    for (size_t i = 0; i < small.size(); ++i)
      if (small[i] != full[i + off] && small[i] != 1) return false;
    return true;
  }
  static std::pair<Storage, Storage> mul_backward(const OpB& o, const Storage& g) { return binary_bwd(RT_MUL, o, g, "mul"); }
  static std::pair<Storage, Storage> add_backward(const OpB& o, const Storage& g) {
    // same-shape add: both gradients are the upstream gradient itself (no copy)
    if (o.inputs.size() == 2 && o.inputs[0].data().shape == g.shape && o.inputs[1].data().shape == g.shape) return {g, g};
    // full-shape a + broadcast b (a bias): da is the upstream gradient itself, db its sum over the stretched axes
    if (o.inputs.size() == 2 && o.inputs[0].data().shape == g.shape && g.numel() > 0 && stretches_onto(o.inputs[1].data().shape, g.shape)) {
      const Shape& bs = o.inputs[1].data().shape;
      const auto& bias = o.inputs[1];
      if (bias.requires_grad() && bias.grad() && deferrable(g.shape) && g.shape.size() == 2 && bs.size() == 1 && bs[0] == g.shape[1] &&
          bias.grad()->shape == bs) {
        // the bias already holds a gradient (it is used at every timestep): this one's column sums join a list that is added in one go
        append_terms(bias.grad_mut(), lazy::Tag::SumRows, {input(g)}, {(int64_t)g.shape[0], (int64_t)g.shape[1]}, run_sum_rows);
        return {g, unused_grad(bs)};
      }
      return {g, bias.requires_grad() ? unbroadcast(g, bs) : unused_grad(bs)};
    }
    return binary_bwd(RT_ADD, o, g, "add");
  }
  static std::pair<Storage, Storage> sub_backward(const OpB& o, const Storage& g) { return binary_bwd(RT_SUB, o, g, "sub"); }
  static std::pair<Storage, Storage> div_backward(const OpB& o, const Storage& g) { return binary_bwd(RT_DIV, o, g, "div"); }
  static std::pair<Storage, Storage> powf_backward(const OpB& o, const Storage& g) { return binary_bwd(RT_POWF, o, g, "powf"); }
  static std::pair<Storage, Storage> maximum_backward(const OpB& o, const Storage& g) { return binary_bwd(RT_MAXIMUM, o, g, "maximum"); }
  static std::pair<Storage, Storage> minimum_backward(const OpB& o, const Storage& g) { return binary_bwd(RT_MINIMUM, o, g, "minimum"); }

  static Storage div_scalar(const Storage& x, float s) {
    if (s == 0.0f) throw Error::invalid_op("Division by zero scalar");
    return unary(RT_DIV_SCALAR, x, s);
  }
  static Storage mul_scalar(const Storage& x, float s) { return unary(RT_MUL_SCALAR, x, s); }
  static Storage exp(const Storage& x) { return unary(RT_EXP, x); }
  static Storage ln(const Storage& x) { return unary(RT_LN, x); }
  static Storage abs(const Storage& x) { return unary(RT_ABS, x); }
  static Storage tanh(const Storage& x) { return unary(RT_TANH, x); }
  static Storage sin(const Storage& x) { return unary(RT_SIN, x); }
  static Storage cos(const Storage& x) { return unary(RT_COS, x); }
  static Storage tan(const Storage& x) { return unary(RT_TAN, x); }
  static Storage relu(const Storage& x) { return unary(RT_RELU, x); }
  static Storage sigmoid(const Storage& x) { return unary(RT_SIGMOID, x); }
  static Storage softplus(const Storage& x) { return unary(RT_SOFTPLUS, x); }
  static Storage square(const Storage& x) { return unary(RT_SQUARE, x); }
  static Storage elu(const Storage& x, float alpha) { return unary(RT_ELU, x, alpha); }
  static Storage clip(const Storage& x, float lo, float hi) { return unary(RT_CLIP, x, lo, hi); }
  static Storage sqrt(const Storage& x) {
    // The reference rejects any negative input (src/backend/cpu.rs:1717-1723); the check
    // is a device min-reduction read back to the host.
    if (x.numel() > 0) {
      Storage m = min(x, std::nullopt);
      if (copy_to_host(m).at(0) < 0.0f) throw Error::invalid_op("sqrt: input contains negative values");
    }
    return unary(RT_SQRT, x);
  }
  static Storage relu_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_RELU, o, g); }
  static Storage elu_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_ELU, o, g, o.op_type.scalar); }
  static Storage exp_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_EXP, o, g); }
  static Storage ln_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_LN, o, g); }
  static Storage abs_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_ABS, o, g); }
  static Storage sigmoid_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_SIGMOID, o, g); }
  static Storage tanh_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_TANH, o, g); }
  static Storage sqrt_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_SQRT, o, g); }
  static Storage softplus_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_SOFTPLUS, o, g); }
  static Storage square_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_SQUARE, o, g); }
  static Storage sin_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_SIN, o, g); }
  static Storage cos_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_COS, o, g); }
  static Storage tan_backward(const OpB& o, const Storage& g) { return unary_bwd(RT_TAN, o, g); }
  static Storage clip_backward(const OpB& o, const Storage& g) {
    return unary_bwd(RT_CLIP, o, g, o.op_type.min_val, o.op_type.max_val);
  }

  // ---- layout -----------------------------------------------------------------------------
  static Storage transpose(const Storage& x) {
    if (x.shape.size() <= 1) return x;
    if (x.shape.size() != 2) throw Error::unimplemented("transpose of more than 2 dimensions");
    Storage y = alloc(Shape{x.shape[1], x.shape[0]});
    check(rt_transpose2d(ctx(), x.ptr(), (int64_t)x.shape[0], (int64_t)x.shape[1], y.ptr()));
    return y;
  }
  static Storage broadcast_to(const Storage& x, const Shape& shape) {
    if (shape.size() < x.shape.size()) throw Error::incompatible("broadcast", x.shape, shape);
    size_t off = shape.size() - x.shape.size();
    for (size_t i = 0; i < x.shape.size(); ++i)
      if (x.shape[i] != shape[i + off] && x.shape[i] != 1) throw Error::incompatible("broadcast", x.shape, shape);
    if (deferrable(shape)) return lz_box(lazy::Kind::Broadcast, x, shape, {});  // also to its own shape: a tensor of its own
    Storage y = alloc(shape);
    auto xs = dims(x.shape), os = dims(shape);
    check(rt_broadcast_to(ctx(), x.ptr(), xs.data(), (int)xs.size(), os.data(), (int)os.size(), y.ptr()));
    return y;
  }
  static Storage unbroadcast(const Storage& g, const Shape& target) {
    if (g.shape == target) return g;
    // The reduction works on the right-aligned target; a target that is rank-compatible
    // only after reshaping (same element count) is reshaped, as the reference does last.
    Shape t = target;
    auto gs = dims(g.shape), ts = dims(t);
    if (ts.size() > gs.size()) {
      if (shape_numel(t) == g.numel()) {
        Storage r = g;
        r.shape = t;
        return r;
      }
      throw Error::incompatible("unbroadcast (final shape/size)", g.shape, target);
    }
    if (deferrable(g.shape) && deferrable(t) && gs.size() == 2 && shape_numel(t) == g.shape[1] && !t.empty() && t.back() == g.shape[1])
      // the column sums of a matrix (the gradient of a bias): deferred, because a bias that is used again takes more of them
      return lz_opaque(lazy::Tag::SumRows, {-1}, {input(g)}, t, [](lazy::Node& n, float* o) {
        const int64_t gd[2] = {(int64_t)n.in[0].shape[0], (int64_t)n.in[0].shape[1]}, td[1] = {gd[1]};
        return rt_unbroadcast(ctx(), n.in[0].buf->data(), gd, 2, td, 1, o);
      });
    Storage out = alloc(t);
    check(rt_unbroadcast(ctx(), g.ptr(), gs.data(), (int)gs.size(), ts.data(), (int)ts.size(), out.ptr()));
    return out;
  }
  // Those of `grads` that are unevaluated column sums of matrices of up to 2048 rows (more are better split over blocks), in one launch.
  static void evaluate_column_sums(const std::vector<const Storage*>& grads) {
    std::vector<std::shared_ptr<DeviceBuffer>> sums;
    for (auto* g : grads) {
      const lazy::Node* n = g->buf ? g->buf->node.get() : nullptr;
      if (n && n->tag == lazy::Tag::SumRows && n->geo[0] < 0 && n->in[0].shape[0] <= 2048 && n->in[0].shape[1] == g->buf->numel &&
          std::find(sums.begin(), sums.end(), g->buf) == sums.end())
        sums.push_back(g->buf);
    }
    if (sums.size() < 2) return;
    for (auto& b : sums)
      if (b->node) {
        const std::shared_ptr<DeviceBuffer> x = b->node->in[0].buf;
        x->data();
      }
    sums.erase(std::remove_if(sums.begin(), sums.end(), [](auto& b) { return !b->node; }), sums.end());  // evaluated on the way
    std::vector<const float*> xs;
    std::vector<int64_t> rows, cols;
    std::vector<float*> outs;
    std::vector<lazy::Block> blocks;
    for (auto& b : sums) {
      const lazy::Input& x = b->node->in[0];
      xs.push_back(x.buf->data());
      rows.push_back((int64_t)x.shape[0]);
      cols.push_back((int64_t)x.shape[1]);
      blocks.emplace_back(b->ctx, b->numel);
      outs.push_back(blocks.back().ptr);
    }
    check(rt_column_sums_list(ctx(), (int)sums.size(), xs.data(), rows.data(), cols.data(), outs.data()));
    for (size_t i = 0; i < sums.size(); ++i) blocks[i].to(sums[i].get());
  }
  static Storage slice(const Storage& x, const std::vector<Range>& ranges) {
    if (ranges.size() != x.shape.size()) throw Error::invalid_op("Slice ranges do not match input dimensionality");
    Shape os(ranges.size());
    std::vector<int64_t> starts(ranges.size());
    for (size_t i = 0; i < ranges.size(); ++i) {
      os[i] = ranges[i].end - ranges[i].start;
      starts[i] = (int64_t)ranges[i].start;
    }
    if (deferrable(os) && deferrable(x.shape)) return lz_box(lazy::Kind::Slice, x, os, Shape(starts.begin(), starts.end()));
    Storage y = alloc(os);
    auto xs = dims(x.shape), od = dims(os);
    check(rt_slice(ctx(), x.ptr(), xs.data(), (int)xs.size(), starts.data(), od.data(), y.ptr()));
    return y;
  }
  static Storage slice_backward(const OpB& o, const Storage& g) {
    if (o.op_type.kind != OpType::Slice) throw Error::internal("Incorrect OpType for slice_backward");
    const Shape& is = o.op_type.input_shape;
    std::vector<int64_t> starts;
    Shape gs;
    for (auto& r : o.op_type.ranges) {
      starts.push_back((int64_t)r.start);
      gs.push_back(r.end - r.start);
    }
    if (shape_numel(gs) != g.numel()) throw Error::incompatible("slice_backward", gs, g.shape);
    if (deferrable(is) && deferrable(gs)) {
      Storage gb = g;
      set_shape(gb, gs);
      return lz_box(lazy::Kind::Pad, gb, is, Shape(starts.begin(), starts.end()));
    }
    Storage dx = zeros(is);
    auto id = dims(is), gd = dims(gs);
    check(rt_slice_assign(ctx(), dx.ptr(), id.data(), (int)id.size(), starts.data(), g.ptr(), gd.data()));
    return dx;
  }
  static Storage concat(const std::vector<const Storage*>& xs, size_t axis) {
    if (xs.empty()) throw Error::invalid_op("Cannot concat empty list of storages");
    Shape os = xs[0]->shape;
    if (axis >= os.size()) throw Error(ErrorKind::ShapeError, "concatenate: axis out of bounds");
    size_t total = 0;
    for (auto* x : xs) {
      if (x->shape.size() != os.size()) throw Error(ErrorKind::ShapeError, "concatenate: incompatible shapes");
      for (size_t d = 0; d < os.size(); ++d)
        if (d != axis && x->shape[d] != os[d]) throw Error(ErrorKind::ShapeError, "concatenate: incompatible shapes");
      total += x->shape[axis];
    }
    os[axis] = total;
    bool defers = deferrable(os) && xs.size() <= 4;  // each piece costs a region of the program
    for (auto* x : xs) defers = defers && x->numel() > 0;
    if (defers) {
      lazy::Node n{lazy::Kind::Concat};
      n.starts = Shape{axis};
      for (auto* x : xs) n.in.push_back(input(*x));
      return defer(std::move(n), os);
    }
    Storage y = alloc(os);
    int64_t outer = 1;
    for (size_t d = 0; d < axis; ++d) outer *= (int64_t)os[d];
    std::vector<const float*> srcs;
    std::vector<int64_t> lens;
    for (auto* x : xs) {
      srcs.push_back(x->numel() ? x->ptr() : nullptr);
      lens.push_back(outer ? (int64_t)x->numel() / outer : 0);
    }
    check(rt_concat_list(ctx(), (int)xs.size(), srcs.data(), lens.data(), outer, y.ptr()));
    return y;
  }
  // concat({x[r0:r1, :], h}, axis 1) for 2-D x and h without materialising the row slice: rows r0..r1 of a row-major matrix are
  // one contiguous block, which goes straight into the left columns of the result.
  static Storage concat_rows_with(const Storage& x, size_t r0, size_t r1, const Storage& h) {
    if (x.shape.size() != 2 || h.shape.size() != 2 || r0 > r1 || r1 > x.shape[0] || h.shape[0] != r1 - r0)
      throw Error(ErrorKind::ShapeError, "concat_rows_with: incompatible shapes");
    Shape os{r1 - r0, x.shape[1] + h.shape[1]};
    if (deferrable(os) && r1 > r0 && x.shape[1] > 0 && h.shape[1] > 0) {
      const Storage rows = slice(x, {{r0, r1}, {0, x.shape[1]}});
      return concat({&rows, &h}, 1);
    }
    Storage y = alloc(os);
    auto od = dims(os);
    std::vector<int64_t> starts{0, 0};
    Shape xs{r1 - r0, x.shape[1]};
    auto xd = dims(xs), hd = dims(h.shape);
    if (shape_numel(xs) > 0) check(rt_slice_assign(ctx(), y.ptr(), od.data(), 2, starts.data(), x.ptr() + r0 * x.shape[1], xd.data()));
    starts[1] = (int64_t)x.shape[1];
    if (h.numel() > 0) check(rt_slice_assign(ctx(), y.ptr(), od.data(), 2, starts.data(), h.ptr(), hd.data()));
    return y;
  }
  static std::vector<Storage> concat_backward(const OpB& o, const Storage& g) {
    if (o.op_type.kind != OpType::Concat) throw Error::internal("Incorrect OpType for concat_backward");
    size_t axis = *o.op_type.axis;
    std::vector<Storage> grads;
    size_t off = 0;
    for (size_t i = 0; i < o.op_type.input_shapes.size(); ++i) {
      const Shape& s = o.op_type.input_shapes[i];
      if (i < o.inputs.size() && !o.inputs[i].requires_grad()) {
        grads.push_back(Storage{nullptr, s});  // never accumulated
      } else {
        std::vector<Range> r;
        for (size_t d = 0; d < g.shape.size(); ++d) r.push_back(d == axis ? Range{off, off + s[axis]} : Range{0, g.shape[d]});
        grads.push_back(slice(g, r));
      }
      off += s[axis];
    }
    return grads;
  }
  static Storage expand_dims(const Storage& x, size_t axis) {
    if (axis > x.shape.size()) throw Error::invalid_index(axis);
    Storage y = x;
    y.shape.insert(y.shape.begin() + axis, 1);
    return y;
  }
  static Storage expand_dims_backward(const OpB& o, const Storage& g) {
    size_t axis = *o.op_type.axis;
    Shape orig = o.inputs[0].shape();
    Storage out = g;
    if (axis < g.shape.size() && g.shape[axis] == 1) {
      set_shape(out, orig);
    } else if (axis < g.shape.size()) {
      out = sum_along_axis(g, axis);
      set_shape(out, orig);
    } else {
      throw Error::internal("expand_dims_backward: axis out of bounds for grad_output");
    }
    return out;
  }
  static Storage squeeze(const Storage& x, std::optional<size_t> axis) {
    Shape ns;
    if (axis) {
      if (*axis >= x.shape.size()) throw Error::invalid_index(*axis);
      if (x.shape[*axis] != 1) throw Error::invalid_op("Cannot squeeze axis (not size 1)");
      ns = x.shape;
      ns.erase(ns.begin() + *axis);
    } else {
      for (size_t d : x.shape)
        if (d != 1) ns.push_back(d);
    }
    Storage y = x;
    set_shape(y, ns);
    return y;
  }
  static Storage squeeze_backward(const OpB& o, const Storage& g) {
    Storage y = g;
    set_shape(y, o.op_type.input_shape);
    return y;
  }

  // ---- reductions ---------------------------------------------------------------------------
  struct Axis3 {
    int64_t outer, len, inner;
    Shape out_shape;
  };
  static Axis3 split(const Shape& s, std::optional<size_t> axis) {
    Axis3 a{1, 1, 1, {}};
    if (!axis) {
      a.len = (int64_t)shape_numel(s);
      return a;
    }
    if (*axis >= s.size()) throw Error::invalid_index(*axis);
    for (size_t d = 0; d < *axis; ++d) a.outer *= (int64_t)s[d];
    a.len = (int64_t)s[*axis];
    for (size_t d = *axis + 1; d < s.size(); ++d) a.inner *= (int64_t)s[d];
    a.out_shape = s;
    a.out_shape.erase(a.out_shape.begin() + *axis);
    return a;
  }
  static Storage reduce(int kind, const Storage& x, std::optional<size_t> axis) {
    Axis3 a = split(x.shape, axis);
    if ((kind == RT_RED_SUM || kind == RT_RED_MEAN) && deferrable(x.shape))
      return lz_opaque(lazy::Tag::Reduce, {kind, axis ? (int64_t)*axis : -1}, {input(x)}, a.out_shape, [a, kind](lazy::Node& n, float* out) {
        return rt_reduce(ctx(), kind, n.in[0].buf->data(), a.outer, a.len, a.inner, out);
      });
    Storage out = alloc(a.out_shape);
    const bool fused = kind == RT_RED_LOGSUMEXP && a.inner == 1 && !x.shape.empty() && a.len == (int64_t)x.shape.back() && x.buf && x.buf->node &&
                       x.buf->node->shape == x.shape && lazy::evaluate_with_logsumexp(x.buf.get(), out.buf->ptr);
    if (!fused) check(rt_reduce(ctx(), kind, x.ptr(), a.outer, a.len, a.inner, out.ptr()));
    if (x.buf) out.buf->made_from = x.buf->id;
    return out;
  }
  static Storage sum_along_axis(const Storage& x, size_t axis) { return reduce(RT_RED_SUM, x, axis); }
  static Storage max_along_axis(const Storage& x, size_t axis) { return reduce(RT_RED_MAX, x, axis); }
  static float sum_all(const Storage& x) {
    float v = 0.f;
    check(rt_sum_all_host(ctx(), x.ptr(), (int64_t)x.numel(), &v));
    return v;
  }
  static Storage sum_all_scalar(const Storage& x) { return reduce(RT_RED_SUM, x, std::nullopt); }
  static Storage mean(const Storage& x, std::optional<size_t> axis) {
    if (axis) {
      if (*axis >= x.shape.size()) throw Error::invalid_index(*axis);
      if (x.shape[*axis] == 0) throw Error::invalid_op("Mean failed along axis");
    } else if (x.numel() == 0) {
      throw Error(ErrorKind::EmptyTensor, "empty tensor");
    }
    return reduce(RT_RED_MEAN, x, axis);
  }
  static Storage reduce_or_empty(int kind, const Storage& x, std::optional<size_t> axis) {
    if (x.numel() == 0) return zeros(x.shape);
    return reduce(kind, x, axis);
  }
  static Storage max(const Storage& x, std::optional<size_t> axis) { return reduce_or_empty(RT_RED_MAX, x, axis); }
  static Storage min(const Storage& x, std::optional<size_t> axis) { return reduce_or_empty(RT_RED_MIN, x, axis); }
  static Storage prod(const Storage& x, std::optional<size_t> axis) { return reduce_or_empty(RT_RED_PROD, x, axis); }
  static Storage logsumexp(const Storage& x, std::optional<size_t> axis) { return reduce_or_empty(RT_RED_LOGSUMEXP, x, axis); }
  static Storage argmax(const Storage& x, size_t axis) { return reduce_or_empty(RT_RED_ARGMAX, x, axis); }
  static Storage argmin(const Storage& x, size_t axis) { return reduce_or_empty(RT_RED_ARGMIN, x, axis); }
  static Storage log_softmax(const Storage& x, size_t axis) {
    Axis3 a = split(x.shape, axis);
    if (deferrable(x.shape))
      return lz_opaque(lazy::Tag::LogSoftmax, {(int64_t)axis}, {input(x)}, x.shape, [a](lazy::Node& n, float* out) {
        return rt_log_softmax(ctx(), n.in[0].buf->data(), a.outer, a.len, a.inner, out);
      });
    Storage y = alloc(x.shape);
    check(rt_log_softmax(ctx(), x.ptr(), a.outer, a.len, a.inner, y.ptr()));
    return y;
  }
  static Storage reduce_bwd(int kind, const OpB& o, const Storage& g, const char* name) {
    if (o.inputs.size() != 1) throw Error::invalid_op(std::string(name) + " backward expects 1 input");
    const Storage& x = o.inputs[0].data();
    Axis3 a = split(x.shape, o.op_type.axis);
    if ((int64_t)g.numel() != a.outer * a.inner) throw Error::incompatible(name, x.shape, g.shape);
    Storage dx = alloc(x.shape);
    check(rt_reduce_backward(ctx(), kind, x.ptr(), g.ptr(), a.outer, a.len, a.inner, dx.ptr()));
    return dx;
  }
  static Storage sum_backward(const OpB& o, const Storage& g) {
    if (!o.op_type.axis && !g.shape.empty()) throw Error::shape_mismatch(Shape{}, g.shape);  // cpu.rs:1480-1485
    return spread(RT_RED_SUM, o, g, "sum");
  }
  static Storage mean_backward(const OpB& o, const Storage& g) { return spread(RT_RED_MEAN, o, g, "mean"); }
  // Gradient of a sum or mean: the upstream gradient repeated along the reduced axis (divided by its length for a mean).
  static Storage spread(int kind, const OpB& o, const Storage& g, const char* name) {
    if (o.inputs.size() != 1) throw Error::invalid_op(std::string(name) + " backward expects 1 input");
    const Storage& x = o.inputs[0].data();
    Axis3 a = split(x.shape, o.op_type.axis);
    if ((int64_t)g.numel() != a.outer * a.inner) throw Error::incompatible(name, x.shape, g.shape);
    if (!deferrable(x.shape)) return reduce_bwd(kind, o, g, name);
    Storage gs = g;
    Shape one = o.op_type.axis ? x.shape : Shape{};
    if (o.op_type.axis) one[*o.op_type.axis] = 1;
    gs = reshaped(gs, one);
    Storage scaled = kind == RT_RED_MEAN ? lz_imm(RT_F_DIV, gs, (float)a.len) : gs;
    return one == x.shape ? scaled : lz_box(lazy::Kind::Broadcast, scaled, x.shape, {});
  }
  static Storage max_backward(const OpB& o, const Storage& g) { return reduce_bwd(RT_RED_MAX, o, g, "max"); }
  static Storage min_backward(const OpB& o, const Storage& g) { return reduce_bwd(RT_RED_MIN, o, g, "min"); }
  static Storage prod_backward(const OpB& o, const Storage& g) { return reduce_bwd(RT_RED_PROD, o, g, "prod"); }
  static Storage logsumexp_backward(const OpB& o, const Storage& g) {
    // g exp(x - logsumexp(x)): elementwise, with the forward result, unless it or x may have been changed since (Tag::RowGrad)
    if (o.inputs.size() == 1 && o.cached_outputs && o.cached_outputs->buf) {
      const Storage &x = o.inputs[0].data(), &lse = *o.cached_outputs;
      const Axis3 a = split(x.shape, o.op_type.axis);
      if (x.buf && a.inner == 1 && !x.shape.empty() && a.len == (int64_t)x.shape.back() && deferrable(x.shape) && lse.buf->made_from == x.buf->id &&
          (int64_t)g.numel() == a.outer && lse.numel() == g.numel() && ((!x.buf->escaped && !lse.buf->escaped) || lazy::capturing())) {
        Shape rows = x.shape;
        rows.back() = 1;
        lazy::Node n{lazy::Kind::Binary};
        n.op = RT_F_MUL;
        n.tag = lazy::Tag::RowGrad;
        n.weight = lazy::op_weight(RT_F_MUL);
        n.in = {input(reshaped(g, rows)), input(lz_unary(RT_F_EXP, lz_binary(RT_F_SUB, x, reshaped(lse, rows), x.shape))), input(x)};
        n.run = [a](lazy::Node& nd, DeviceBuffer* b) {
          const float *px = nd.in[2].buf->data(), *pg = nd.in[0].buf->data();
          lazy::Block out(b->ctx, b->numel);
          check(rt_reduce_backward(ctx(), RT_RED_LOGSUMEXP, px, pg, a.outer, a.len, a.inner, out.ptr));
          b->ptr = out.release();
        };
        return defer(std::move(n), x.shape);
      }
    }
    return reduce_bwd(RT_RED_LOGSUMEXP, o, g, "logsumexp");
  }
  static Storage log_softmax_backward(const OpB& o, const Storage& g) {
    if (o.inputs.empty()) throw Error::invalid_op("LogSoftmax requires 1 input");
    const Storage& x = o.inputs[0].data();
    Axis3 a = split(x.shape, o.op_type.axis);
    if (g.shape != x.shape) throw Error::shape_mismatch(x.shape, g.shape);
    // upstream = constant * targets (a classification loss): without the product in memory
    float c;
    if (g.buf && g.buf->node && a.inner == 1 && a.len <= 4096)
      if (const lazy::Input* t = lazy::times_constant(g.buf->node.get(), &c)) {
        const float* tp = t->buf->data();
        if (g.buf->node) {
          const float* xp = x.ptr();
          Storage dx;
          lazy::Loss l;
          DeviceBuffer* loss = lazy::loss_over(x.buf.get(), t->buf.get(), &l);
          if (loss && l.rows == (int64_t)a.outer && l.classes == (int64_t)a.len) {  // the loss itself comes out of the same pass
            auto keep = loss->shared_from_this();
            lazy::Block out(loss->ctx, loss->numel);
            dx = alloc(x.shape);
            check(rt_softmax_nll_with_grad(ctx(), xp, tp, a.outer, a.len, l.scale, l.divisor, nullptr, c, out.ptr, dx.ptr()));
            out.to(loss);
            return dx;
          }
          if (lazy::capturing() && deferrable(x.shape)) {  // may join those of the other timesteps
            int64_t bits = 0;
            std::memcpy(&bits, &c, sizeof(float));
            return lz_opaque(lazy::Tag::NllGrad, {a.outer, a.len, bits}, {input(x), *t}, x.shape, [c](lazy::Node& n, float* out) {
              return rt_softmax_nll_scaled_backward(ctx(), n.in[0].buf->data(), n.in[1].buf->data(), n.geo[0], n.geo[1], c, out);
            });
          }
          dx = alloc(x.shape);
          check(rt_softmax_nll_scaled_backward(ctx(), x.ptr(), tp, a.outer, a.len, c, dx.ptr()));
          return dx;
        }
      }
    Storage dx = alloc(x.shape);
    check(rt_log_softmax_backward(ctx(), x.ptr(), g.ptr(), a.outer, a.len, a.inner, dx.ptr()));
    return dx;
  }

  // ---- contractions / pooling -------------------------------------------------------------------
  static Storage matmul(const Storage& a, const Storage& b) {
    if (a.shape.size() != 2) throw Error(ErrorKind::ShapeError, "Input 'a' is not 2D");
    if (b.shape.size() != 2) throw Error(ErrorKind::ShapeError, "Input 'b' is not 2D");
    if (a.shape[1] != b.shape[0]) throw Error::incompatible("matmul", a.shape, b.shape);
    int64_t m = (int64_t)a.shape[0], k = (int64_t)a.shape[1], n = (int64_t)b.shape[1];
    if (k > 0 && deferrable(Shape{a.shape[0], b.shape[1]})) {
      // the operands are evaluated now (expressions do not grow through products); the product itself may still join a bias, an
      // activation, or its siblings.  In a capture the timesteps of an LSTM wait for the last one, and so does what takes their states.
      b.ptr();
      std::vector<int64_t> geo;
      lazy::Cell cell;
      if (const int64_t t = a.buf->node ? lazy::timestep_of(input(a), input(b)) : 0) geo.push_back(t);
      else if (!(lazy::capturing() && a.buf->node && a.shape == a.buf->node->shape && lazy::match_cell(a.buf.get(), &cell))) a.ptr();
      return lz_opaque(lazy::Tag::Matmul, std::move(geo), {input(a), input(b)}, Shape{a.shape[0], b.shape[1]}, [m, n, k](lazy::Node& nd, float* out) {
        return rt_gemm(ctx(), 0, 0, m, n, k, nd.in[0].buf->data(), k, nd.in[1].buf->data(), n, out, n, 0);
      });
    }
    Storage c = alloc(Shape{a.shape[0], b.shape[1]});
    check(rt_gemm(ctx(), 0, 0, m, n, k, a.ptr(), k, b.ptr(), n, c.ptr(), n, 0));
    return c;
  }
  // In a capture: a state of a sequence that was computed as one, whose gradient comes from all its timesteps at once.
  static bool of_a_sequence(const Storage& a) { return lazy::capturing() && a.buf && a.buf->sequence; }
  static Storage state_gradient(const Storage& g, const Storage& b, const Shape& shape) {
    return lz_opaque(lazy::Tag::MatmulNT, {}, {input(g), input(b)}, shape, [](lazy::Node& n, float* out) {
      const int64_t m = (int64_t)n.in[0].shape[0], cols = (int64_t)n.in[0].shape[1], k = (int64_t)n.in[1].shape[0];
      return rt_gemm(ctx(), 0, 1, m, k, cols, n.in[0].buf->data(), cols, n.in[1].buf->data(), cols, out, k, 0);
    });
  }
  static std::pair<Storage, Storage> matmul_backward(const OpB& o, const Storage& g) {
    if (o.inputs.size() != 2) throw Error::invalid_op("Matmul requires 2 inputs");
    const Storage& a = o.inputs[0].data();
    const Storage& b = o.inputs[1].data();
    int64_t m = (int64_t)a.shape[0], k = (int64_t)a.shape[1], n = (int64_t)b.shape[1];
    if (g.shape != Shape{a.shape[0], b.shape[1]}) throw Error::incompatible("matmul", g.shape, b.shape);
    bool need_a = o.inputs[0].requires_grad(), need_b = o.inputs[1].requires_grad();
    if (of_a_sequence(a) && deferrable(b.shape)) {  // the other timesteps' products follow: both wait for them
      Storage db{nullptr, b.shape};
      if (need_b) {
        db = filled(b.shape, 0.f);
        append_terms(db, lazy::Tag::SumProducts, {input(a), input(g)}, {m, k, n}, run_sum_products);
      }
      return {need_a ? state_gradient(g, b, a.shape) : Storage{nullptr, a.shape}, std::move(db)};
    }
    Storage da = need_a ? alloc(a.shape) : Storage{nullptr, a.shape};
    Storage db = need_b ? alloc(b.shape) : Storage{nullptr, b.shape};
    check(rt_matmul_backward(ctx(), a.ptr(), b.ptr(), g.ptr(), m, k, n, da.ptr(), db.ptr()));
    return {std::move(da), std::move(db)};
  }
  static std::pair<Storage, Storage> matmul_closure_backward(const OpB& o, const Storage& g) { return matmul_backward(o, g); }
  // matmul backward when the second operand already holds a gradient: returns dA and adds A^T g to `acc` in place (the
  // product kernel accumulates into its output; one launch instead of a product and an addition)
  static Storage matmul_backward_accumulate(const OpB& o, const Storage& g, Storage& acc) {
    const Storage& a = o.inputs[0].data();
    const Storage& b = o.inputs[1].data();
    int64_t m = (int64_t)a.shape[0], k = (int64_t)a.shape[1], n = (int64_t)b.shape[1];
    if (g.shape != Shape{a.shape[0], b.shape[1]}) throw Error::incompatible("matmul", g.shape, b.shape);
    if (acc.shape != b.shape) throw Error::shape_mismatch(b.shape, acc.shape);
    if (of_a_sequence(a) && deferrable(b.shape)) {
      append_terms(acc, lazy::Tag::SumProducts, {input(a), input(g)}, {m, k, n}, run_sum_products);
      return o.inputs[0].requires_grad() ? state_gradient(g, b, a.shape) : Storage{nullptr, a.shape};
    }
    Storage da = o.inputs[0].requires_grad() ? alloc(a.shape) : Storage{nullptr, a.shape};
    if (deferrable(a.shape) && deferrable(g.shape) && deferrable(b.shape)) {
      // the weight's gradient is a sum over all its uses: the products are collected and computed as one with a longer reduction
      append_terms(acc, lazy::Tag::SumProducts, {input(a), input(g)}, {m, k, n}, run_sum_products);
      if (da.buf) check(rt_gemm(ctx(), 0, 1, m, k, n, g.ptr(), n, b.ptr(), n, da.ptr(), k, 0));
      return da;
    }
    make_unique(acc);  // nobody else may see the sum appear in a buffer they share
    check(rt_matmul_backward_accumulate(ctx(), a.ptr(), b.ptr(), g.ptr(), m, k, n, da.ptr(), acc.ptr()));
    return da;
  }
  static bool is_accumulated(const Storage& s) { return !s.buf; }
  static bool accumulates_well(const Storage& b) { return b.shape.size() == 2 && (deferrable(b.shape) || b.shape[1] % 4 == 0); }

  // acc += a term that is computed later, together with the others of its kind.  Node: in[0] is what was there before.
  static constexpr size_t kMaxTerms = 512;  // operands: twice what one launch of rt_gemm_sum_products takes
  static void append_terms(Storage& acc, lazy::Tag tag, std::vector<lazy::Input> term, std::vector<int64_t> geo,
                           void (*run)(lazy::Node&, DeviceBuffer*)) {
    DeviceBuffer* b = acc.buf.get();
    if (b->node && b->node->tag == tag && b->node->geo == geo && acc.buf.use_count() == 1 && b->readers.empty() &&
        b->node->in.size() + term.size() <= 1 + kMaxTerms) {
      bool now = false;
      for (auto& t : term) {
        now = now || (t.buf->escaped && !lazy::capturing());
        t.buf->readers.push_back(b);
        b->node->in.push_back(std::move(t));
      }
      if (now) b->data();
      return;
    }
    acc.buf->data();
    lazy::Node n{lazy::Kind::Opaque};
    n.tag = tag;
    n.geo = std::move(geo);
    n.weight = 1 << 10;
    n.in.push_back(input(acc));
    for (auto& t : term) n.in.push_back(std::move(t));
    n.run = run;
    const Shape s = acc.shape;
    bool now;
    acc = Storage{};  // the node now holds the old values, alone unless somebody else does too
    acc = pend(std::move(n), s, &now);
    if (now) acc.buf->data();
  }
  // Adds to the old values: in their own block when nobody else needs it.  After an error the old values still have their block.
  template <class F>
  static void add_to(lazy::Node& n, DeviceBuffer* b, F add) {
    DeviceBuffer* base = n.in[0].buf.get();
    float* old = base->data();
    if (n.in[0].buf.use_count() == 1 && !base->escaped && !base->owner) {
      check(add(old));
      base->ptr = nullptr;
      b->ptr = old;
      return;
    }
    lazy::Block out(b->ctx, b->numel);
    check(rt_memcpy_d2d(ctx(), out.ptr, old, sizeof(float) * b->numel));
    check(add(out.ptr));
    b->ptr = out.release();
  }
  static void run_sum_products(lazy::Node& n, DeviceBuffer* b) {
    std::vector<const float*> as, gs;
    for (size_t i = 1; i < n.in.size(); i += 2) {
      as.push_back(n.in[i].buf->data());
      gs.push_back(n.in[i + 1].buf->data());
    }
    add_to(n, b, [&](float* out) { return rt_gemm_sum_products(ctx(), (int)as.size(), as.data(), gs.data(), n.geo[0], n.geo[1], n.geo[2], out); });
  }
  // existing += g for a gradient that receives another contribution (Tensor::add_grad).  After an error it is what it was.
  static void accumulate(Storage& existing, const Storage& g) {
    const lazy::Node* n = g.buf ? g.buf->node.get() : nullptr;
    if (n && n->tag == lazy::Tag::SumRows && n->geo[0] < 0 && g.buf->readers.empty() && g.shape.size() == 1 && existing.buf && existing.shape == g.shape) {
      const lazy::Input x = n->in[0];
      const lazy::Node* e = existing.buf->node.get();
      const std::vector<int64_t> geo{(int64_t)x.shape[0], (int64_t)x.shape[1]};
      if (lazy::capturing() && e && e->tag == lazy::Tag::SumRows && e->geo[0] < 0 && existing.buf.use_count() == 1 && existing.buf->readers.empty()) {
        const lazy::Input first = e->in[0];  // the first of a sequence's waits with the others
        existing = filled(existing.shape, 0.f);
        append_terms(existing, lazy::Tag::SumRows, {first}, {(int64_t)first.shape[0], (int64_t)first.shape[1]}, run_sum_rows);
      }
      append_terms(existing, lazy::Tag::SumRows, {x}, geo, run_sum_rows);
      return;
    }
    existing = add(existing, g);
  }
  static void run_sum_rows(lazy::Node& n, DeviceBuffer* b) {
    std::vector<const float*> xs;
    for (size_t i = 1; i < n.in.size(); ++i) xs.push_back(n.in[i].buf->data());
    add_to(n, b, [&](float* out) { return rt_sum_rows_accumulate_list(ctx(), (int)xs.size(), xs.data(), n.geo[0], n.geo[1], out); });
  }
  static void conv_shapes(const Storage& x, const Storage& w, const char* name) {
    if (x.shape.size() != 4 || w.shape.size() != 4) throw Error::invalid_op(std::string(name) + " expects 4D input and weights");
  }
  static Storage conv2d(const Storage& x, const Storage& w, const Storage* bias, Pair s, Pair p) {
    conv_shapes(x, w, "conv2d");
    if (x.shape[1] != w.shape[1]) throw Error::invalid_op("conv2d: input channels != weight channels");
    if (bias && bias->numel() != w.shape[0]) throw Error::invalid_op("conv2d: bias shape mismatch");
    size_t ho = (x.shape[2] + 2 * p.first - w.shape[2]) / s.first + 1, wo = (x.shape[3] + 2 * p.second - w.shape[3]) / s.second + 1;
    const Shape ys{x.shape[0], w.shape[0], ho, wo};
    if (deferrable(ys) && deferrable(x.shape) && deferrable(w.shape)) {
      x.ptr();
      w.ptr();
      std::vector<lazy::Input> in{input(x), input(w)};
      if (bias) in.push_back(input(*bias));
      const std::vector<int64_t> q{(int64_t)x.shape[0], (int64_t)x.shape[1], (int64_t)x.shape[2], (int64_t)x.shape[3], (int64_t)w.shape[0],
                                   (int64_t)w.shape[2], (int64_t)w.shape[3], (int64_t)s.first, (int64_t)s.second, (int64_t)p.first, (int64_t)p.second};
      return lz_opaque(lazy::Tag::Conv, q, std::move(in), ys, [](lazy::Node& n, float* out) {
        const auto& q = n.geo;
        return rt_conv2d(ctx(), n.in[0].buf->data(), n.in[1].buf->data(), n.in.size() > 2 ? n.in[2].buf->data() : nullptr, q[0], q[1], q[2], q[3],
                         q[4], (int)q[5], (int)q[6], (int)q[7], (int)q[8], (int)q[9], (int)q[10], out);
      });
    }
    Storage y = alloc(ys);
    check(rt_conv2d(ctx(), x.ptr(), w.ptr(), bias ? bias->ptr() : nullptr, (int64_t)x.shape[0], (int64_t)x.shape[1],
                    (int64_t)x.shape[2], (int64_t)x.shape[3], (int64_t)w.shape[0], (int)w.shape[2], (int)w.shape[3],
                    (int)s.first, (int)s.second, (int)p.first, (int)p.second, y.ptr()));
    return y;
  }
  static std::tuple<Storage, Storage, std::optional<Storage>> conv2d_backward(const Storage& x, const Storage& w,
                                                                              const Storage& g, Pair s, Pair p,
                                                                              bool need_x = true, bool need_w = true,
                                                                              bool need_b = true) {
    conv_shapes(x, w, "conv2d_backward");
    size_t ho = (x.shape[2] + 2 * p.first - w.shape[2]) / s.first + 1, wo = (x.shape[3] + 2 * p.second - w.shape[3]) / s.second + 1;
    Shape gs{x.shape[0], w.shape[0], ho, wo};
    if (g.shape != gs) throw Error::shape_mismatch(gs, g.shape);
    Storage dx = need_x ? alloc(x.shape) : Storage{nullptr, x.shape};
    Storage dw = need_w ? alloc(w.shape) : Storage{nullptr, w.shape};
    Storage db = need_b ? alloc(Shape{w.shape[0]}) : Storage{nullptr, Shape{w.shape[0]}};
    check(rt_conv2d_backward(ctx(), x.ptr(), w.ptr(), g.ptr(), (int64_t)x.shape[0], (int64_t)x.shape[1], (int64_t)x.shape[2],
                             (int64_t)x.shape[3], (int64_t)w.shape[0], (int)w.shape[2], (int)w.shape[3], (int)s.first,
                             (int)s.second, (int)p.first, (int)p.second, dx.ptr(), dw.ptr(), db.ptr()));
    return {std::move(dx), std::move(dw), std::optional<Storage>(std::move(db))};
  }
  // max_pool2d(relu(conv2d(x, w) + bias), 2x2, stride 2) without keeping the convolution output: {pooled values, indices}
  static std::pair<Storage, Storage> conv2d_relu_max_pool2x2(const Storage& x, const Storage& w, const Storage* bias, Pair s, Pair p) {
    conv_shapes(x, w, "conv2d_relu_max_pool2x2");
    if (x.shape[1] != w.shape[1]) throw Error::invalid_op("conv2d_relu_max_pool2x2: input channels != weight channels");
    if (bias && bias->numel() != w.shape[0]) throw Error::invalid_op("conv2d_relu_max_pool2x2: bias shape mismatch");
    size_t ho = (x.shape[2] + 2 * p.first - w.shape[2]) / s.first + 1, wo = (x.shape[3] + 2 * p.second - w.shape[3]) / s.second + 1;
    if ((ho & 1) || (wo & 1)) throw Error::invalid_op("conv2d_relu_max_pool2x2: the convolution output must have even extents");
    Storage y = alloc(Shape{x.shape[0], w.shape[0], ho / 2, wo / 2}), idx = alloc(Shape{x.shape[0], w.shape[0], ho / 2, wo / 2});
    check(rt_conv2d_relu_max_pool2x2(ctx(), x.ptr(), w.ptr(), bias ? bias->ptr() : nullptr, (int64_t)x.shape[0], (int64_t)x.shape[1],
                                     (int64_t)x.shape[2], (int64_t)x.shape[3], (int64_t)w.shape[0], (int)w.shape[2], (int)w.shape[3],
                                     (int)s.first, (int)s.second, (int)p.first, (int)p.second, y.ptr(), idx.ptr()));
    return {std::move(y), std::move(idx)};
  }
  // Its backward: the gradient of the convolution output from the pooled output and the indices, then conv2d_backward.
  static std::tuple<Storage, Storage, std::optional<Storage>> conv2d_relu_max_pool2x2_backward(
      const Storage& x, const Storage& w, const Storage& y, const Storage& idx, const Storage& g, Pair s, Pair p, bool need_x, bool need_w,
      bool need_b) {
    if (g.shape != y.shape) throw Error::shape_mismatch(y.shape, g.shape);
    Storage dconv = alloc(Shape{y.shape[0], y.shape[1], y.shape[2] * 2, y.shape[3] * 2});
    check(rt_relu_max_pool2x2_backward_from_output(ctx(), y.ptr(), g.ptr(), idx.ptr(), (int64_t)y.shape[0], (int64_t)y.shape[1],
                                                   (int64_t)y.shape[2] * 2, (int64_t)y.shape[3] * 2, dconv.ptr()));
    return conv2d_backward(x, w, dconv, s, p, need_x, need_w, need_b);
  }
  static Storage conv2d_transpose(const Storage& x, const Storage& w, const Storage* bias, Pair s, Pair p) {
    if (x.shape.size() != 4) throw Error(ErrorKind::ShapeError, "Expected 4D input tensor for conv2d_transpose");
    if (w.shape.size() != 4) throw Error(ErrorKind::ShapeError, "Expected 4D weights tensor for conv2d_transpose");
    if (x.shape[1] != w.shape[0]) throw Error::shape_mismatch(Shape{x.shape[0], w.shape[0], x.shape[2], x.shape[3]}, x.shape);
    if (bias && (bias->shape.size() != 1 || bias->shape[0] != w.shape[1])) throw Error::shape_mismatch(Shape{w.shape[1]}, bias->shape);
    size_t oh = (x.shape[2] - 1) * s.first + w.shape[2] - 2 * p.first, ow = (x.shape[3] - 1) * s.second + w.shape[3] - 2 * p.second;
    Storage y = alloc(Shape{x.shape[0], w.shape[1], oh, ow});
    check(rt_conv2d_transpose(ctx(), x.ptr(), w.ptr(), bias ? bias->ptr() : nullptr, (int64_t)x.shape[0], (int64_t)x.shape[1],
                              (int64_t)x.shape[2], (int64_t)x.shape[3], (int64_t)w.shape[1], (int)w.shape[2], (int)w.shape[3],
                              (int)s.first, (int)s.second, (int)p.first, (int)p.second, y.ptr()));
    return y;
  }
  static std::tuple<Storage, Storage, std::optional<Storage>> conv2d_transpose_backward(const Storage& x, const Storage& w,
                                                                                        const Storage& g, Pair s, Pair p,
                                                                                        bool need_x = true, bool need_w = true,
                                                                                        bool need_b = true) {
    if (x.shape.size() != 4 || w.shape.size() != 4 || g.shape.size() != 4)
      throw Error(ErrorKind::ShapeError, "Expected 4D tensors for conv2d_transpose_backward");
    if (x.shape[1] != w.shape[0]) throw Error::shape_mismatch(Shape{x.shape[0], w.shape[0], x.shape[2], x.shape[3]}, x.shape);
    if (g.shape[1] != w.shape[1]) throw Error::shape_mismatch(Shape{x.shape[0], w.shape[1], g.shape[2], g.shape[3]}, g.shape);
    size_t oh = (x.shape[2] - 1) * s.first + w.shape[2] - 2 * p.first, ow = (x.shape[3] - 1) * s.second + w.shape[3] - 2 * p.second;
    if (g.shape[2] != oh || g.shape[3] != ow || g.shape[0] != x.shape[0])
      throw Error::shape_mismatch(Shape{x.shape[0], w.shape[1], oh, ow}, g.shape);
    Storage dx = need_x ? alloc(x.shape) : Storage{nullptr, x.shape};
    Storage dw = need_w ? alloc(w.shape) : Storage{nullptr, w.shape};
    Storage db = need_b ? alloc(Shape{w.shape[1]}) : Storage{nullptr, Shape{w.shape[1]}};
    check(rt_conv2d_transpose_backward(ctx(), x.ptr(), w.ptr(), g.ptr(), (int64_t)x.shape[0], (int64_t)x.shape[1],
                                       (int64_t)x.shape[2], (int64_t)x.shape[3], (int64_t)w.shape[1], (int)w.shape[2],
                                       (int)w.shape[3], (int)s.first, (int)s.second, (int)p.first, (int)p.second, dx.ptr(),
                                       dw.ptr(), db.ptr()));
    return {std::move(dx), std::move(dw), std::optional<Storage>(std::move(db))};
  }
  static std::pair<Storage, Storage> max_pool2d(const Storage& x, Pair k, Pair s, Pair p) {
    if (x.shape.size() != 4) throw Error::invalid_op("max_pool2d expects 4D input (NCHW)");
    size_t ho = (x.shape[2] + 2 * p.first - k.first) / s.first + 1, wo = (x.shape[3] + 2 * p.second - k.second) / s.second + 1;
    Shape os{x.shape[0], x.shape[1], ho, wo};
    if (const lazy::Node* act = x.buf ? x.buf->node.get() : nullptr; lazy::is_op(act, lazy::Kind::Unary, RT_F_RELU) && act->shape == x.shape) {
      // relu in front of the pooling, its result not in memory: both in one kernel, with the convolution below it where that has one
      const lazy::Input pre = act->in[0];
      const lazy::Node* cv = lazy::tagged(pre, lazy::Tag::Conv);
      Storage y = alloc(os), idx = alloc(os);
      const bool halves = k == Pair{2, 2} && s == Pair{2, 2} && p == Pair{0, 0} && x.shape[2] % 2 == 0 && x.shape[3] % 2 == 0;
      if (cv && halves && pre.buf->readers.size() == 1) {
        const auto& q = cv->geo;
        const float *px = cv->in[0].buf->data(), *pw = cv->in[1].buf->data(), *pb = cv->in.size() > 2 ? cv->in[2].buf->data() : nullptr;
        check(rt_conv2d_relu_max_pool2x2(ctx(), px, pw, pb, q[0], q[1], q[2], q[3], q[4], (int)q[5], (int)q[6], (int)q[7], (int)q[8], (int)q[9],
                                         (int)q[10], y.ptr(), idx.ptr()));
      } else {
        check(rt_relu_max_pool2d(ctx(), pre.buf->data(), (int64_t)x.shape[0], (int64_t)x.shape[1], (int64_t)x.shape[2], (int64_t)x.shape[3],
                                 (int)k.first, (int)k.second, (int)s.first, (int)s.second, (int)p.first, (int)p.second, y.ptr(), idx.ptr()));
      }
      return {std::move(y), std::move(idx)};
    }
    Storage y = alloc(os), idx = alloc(os);
    check(rt_max_pool2d(ctx(), x.ptr(), (int64_t)x.shape[0], (int64_t)x.shape[1], (int64_t)x.shape[2], (int64_t)x.shape[3],
                        (int)k.first, (int)k.second, (int)s.first, (int)s.second, (int)p.first, (int)p.second, y.ptr(),
                        idx.ptr()));
    return {std::move(y), std::move(idx)};
  }
  static Storage max_pool2d_backward(const OpB& o, const Storage& g) {
    if (o.inputs.size() < 2) throw Error::invalid_op("max_pool2d_backward requires at least 2 inputs (input and indices)");
    if (o.op_type.kind != OpType::MaxPool2D) throw Error::internal("Expected MaxPool2d op type for max_pool2d_backward");
    Shape is = o.inputs[0].shape();
    const Storage& idx = o.inputs[1].data();
    if (g.numel() != idx.numel()) throw Error::shape_mismatch(idx.shape, g.shape);
    Pair k = o.op_type.kernel_size, s = o.op_type.stride, p = o.op_type.padding;
    const bool halves = k == Pair{2, 2} && s == Pair{2, 2} && p == Pair{0, 0} && is[2] % 2 == 0 && is[3] % 2 == 0;
    if (deferrable(is) && g.numel() > 0) {
      std::vector<lazy::Input> in{input(g), input(idx)};
      const Storage& x = o.inputs[0].data();
      if (halves && o.cached_outputs && lazy::is_op(x.buf->node.get(), lazy::Kind::Unary, RT_F_RELU)) in.push_back(input(*o.cached_outputs));
      std::vector<int64_t> q{(int64_t)is[0], (int64_t)is[1], (int64_t)is[2], (int64_t)is[3], (int64_t)k.first, (int64_t)k.second,
                             (int64_t)s.first, (int64_t)s.second, (int64_t)p.first, (int64_t)p.second, (int64_t)x.buf->id};
      return lz_opaque(lazy::Tag::PoolGrad, std::move(q), std::move(in), is, [](lazy::Node& n, float* out) {
        const auto& q = n.geo;
        return rt_max_pool2d_backward(ctx(), n.in[0].buf->data(), n.in[1].buf->data(), q[0], q[1], q[2], q[3], (int)q[4], (int)q[5], (int)q[6],
                                      (int)q[7], (int)q[8], (int)q[9], out);
      });
    }
    Storage dx = alloc(is);
    check(rt_max_pool2d_backward(ctx(), g.ptr(), idx.ptr(), (int64_t)is[0], (int64_t)is[1], (int64_t)is[2], (int64_t)is[3],
                                 (int)k.first, (int)k.second, (int)s.first, (int)s.second, (int)p.first, (int)p.second,
                                 dx.ptr()));
    return dx;
  }

  // ---- fused forward ops (no counterpart in the reference; ops::fused_* in autograd.hpp) -------------------------
  static std::pair<Storage, Storage> relu_max_pool2d(const Storage& x, Pair k, Pair s, Pair p) {
    if (x.shape.size() != 4) throw Error::invalid_op("relu_max_pool2d expects 4D input (NCHW)");
    size_t ho = (x.shape[2] + 2 * p.first - k.first) / s.first + 1, wo = (x.shape[3] + 2 * p.second - k.second) / s.second + 1;
    Shape os{x.shape[0], x.shape[1], ho, wo};
    Storage y = alloc(os), idx = alloc(os);
    check(rt_relu_max_pool2d(ctx(), x.ptr(), (int64_t)x.shape[0], (int64_t)x.shape[1], (int64_t)x.shape[2], (int64_t)x.shape[3],
                             (int)k.first, (int)k.second, (int)s.first, (int)s.second, (int)p.first, (int)p.second, y.ptr(),
                             idx.ptr()));
    return {std::move(y), std::move(idx)};
  }
  static Storage relu_max_pool2d_backward(const OpB& o, const Storage& g) {
    if (o.inputs.size() < 2) throw Error::invalid_op("relu_max_pool2d_backward requires the input and the indices");
    const Storage& x = o.inputs[0].data();
    const Storage& idx = o.inputs[1].data();
    if (g.numel() != idx.numel()) throw Error::shape_mismatch(idx.shape, g.shape);
    Shape is = x.shape;
    Pair k = o.op_type.kernel_size, s = o.op_type.stride, p = o.op_type.padding;
    Storage dx = alloc(is);
    check(rt_relu_max_pool2d_backward(ctx(), x.ptr(), g.ptr(), idx.ptr(), (int64_t)is[0], (int64_t)is[1], (int64_t)is[2],
                                      (int64_t)is[3], (int)k.first, (int)k.second, (int)s.first, (int)s.second, (int)p.first,
                                      (int)p.second, dx.ptr()));
    return dx;
  }
  static Storage softmax_nll(const Storage& logits, const Storage& targets) {
    // deferred, unless it is a size to be refused at once: its gradient, asked for first, brings the loss with it
    if (deferrable(logits.shape) && logits.shape[1] <= 4096 && logits.shape[0] <= ((size_t)1 << 24))
      return lz_opaque(lazy::Tag::FusedLoss, {}, {input(logits), input(targets)}, Shape{}, [](lazy::Node& n, float* out) {
        const float *x = n.in[0].buf->data(), *t = n.in[1].buf->data();
        return rt_softmax_cross_entropy(ctx(), x, t, (int64_t)n.in[0].shape[0], (int64_t)n.in[0].shape[1], out);
      });
    Storage loss = alloc(Shape{});
    check(rt_softmax_cross_entropy(ctx(), logits.ptr(), targets.ptr(), (int64_t)logits.shape[0], (int64_t)logits.shape[1],
                                   loss.ptr()));
    return loss;
  }
  static std::pair<Storage, Storage> softmax_nll_backward(const OpB& o, const Storage& g) {
    const Storage& logits = o.inputs[0].data();
    const Storage& targets = o.inputs[1].data();
    if (g.numel() != 1) throw Error::shape_mismatch(Shape{}, g.shape);
    const bool need_l = o.inputs[0].requires_grad(), need_t = o.inputs[1].requires_grad();
    Storage dl = need_l ? alloc(logits.shape) : unused_grad(logits.shape);
    Storage dt = need_t ? alloc(targets.shape) : unused_grad(targets.shape);
    if (need_l && !need_t && logits.buf) {
      const float *x = logits.ptr(), *t = targets.ptr(), *gp = g.ptr();
      for (DeviceBuffer* r : logits.buf->readers) {
        if (!r->node || r->node->tag != lazy::Tag::FusedLoss || r->node->in[0].buf != logits.buf || r->node->in[1].buf != targets.buf) continue;
        auto loss = r->shared_from_this();
        lazy::Block out(loss->ctx, loss->numel);
        const int64_t rows = (int64_t)logits.shape[0];
        check(rt_softmax_nll_with_grad(ctx(), x, t, rows, (int64_t)logits.shape[1], -1.f, (float)rows, gp, 0.f, out.ptr, dl.ptr()));
        out.to(loss.get());
        return {std::move(dl), std::move(dt)};
      }
    }
    check(rt_softmax_cross_entropy_backward(ctx(), logits.ptr(), targets.ptr(), g.ptr(), (int64_t)logits.shape[0],
                                            (int64_t)logits.shape[1], need_l ? dl.ptr() : nullptr, need_t ? dt.ptr() : nullptr));
    return {std::move(dl), std::move(dt)};
  }

  // Column block i of the [batch, 4 * hidden] gate pre-activations, activated; and a gradient put back into its block.
  static Storage gate(const Storage& gates, const Shape& s, size_t i, uint8_t act) {
    return lz_unary(act, lz_box(lazy::Kind::Slice, gates, s, Shape{0, i * s[1]}));
  }
  // What the forward pass has kept of a cell, unless the gates have been changed since.
  static bool keeps(const OpB& o, const Storage& gates) {
    return o.cached_outputs && o.cached_outputs->buf && !o.cached_outputs->buf->saved.empty() && o.cached_outputs->buf->made_from == gates.buf->id &&
           (!gates.buf->escaped || lazy::capturing());
  }
  static Storage saved_gate(const OpB& o, size_t k, const Storage& gates, const Shape& s, size_t i, uint8_t act) {
    return keeps(o, gates) ? Storage{o.cached_outputs->buf->saved[k], s} : gate(gates, s, i, act);
  }
  static Storage to_gate(const Storage& g, const Shape& gates, size_t i) { return lz_box(lazy::Kind::Pad, g, gates, Shape{0, i * g.shape[1]}); }
  static Storage lstm_cell_c(const Storage& gates, const Storage& c_prev) {
    if (deferrable(gates.shape) && deferrable(c_prev.shape)) {  // joins the ops around it in one launch
      const Shape& s = c_prev.shape;
      const Storage i = gate(gates, s, 0, RT_F_SIGMOID), f = gate(gates, s, 1, RT_F_SIGMOID), gg = gate(gates, s, 2, RT_F_TANH);
      Storage c = lz_binary(RT_F_ADD, lz_mul(f, c_prev), lz_mul(i, gg), s);
      c.buf->made_from = gates.buf->id;
      c.buf->saved = {i.buf, f.buf, gg.buf};
      return c;
    }
    Storage c = alloc(c_prev.shape);
    check(rt_lstm_cell_c(ctx(), gates.ptr(), c_prev.ptr(), (int64_t)c_prev.shape[0], (int64_t)c_prev.shape[1], c.ptr()));
    return c;
  }
  static std::pair<Storage, Storage> lstm_cell_c_backward(const OpB& o, const Storage& g) {
    const Storage& gates = o.inputs[0].data();
    const Storage& c_prev = o.inputs[1].data();
    if (g.shape != c_prev.shape) throw Error::shape_mismatch(c_prev.shape, g.shape);
    const bool ng = o.inputs[0].requires_grad(), nc = o.inputs[1].requires_grad();
    if (deferrable(gates.shape) && deferrable(g.shape)) {
      const Shape &s = g.shape, &gs = gates.shape;
      const Storage i = saved_gate(o, 0, gates, s, 0, RT_F_SIGMOID), f = saved_gate(o, 1, gates, s, 1, RT_F_SIGMOID),
                    gg = saved_gate(o, 2, gates, s, 2, RT_F_TANH);
      Storage dgates = unused_grad(gs), dprev = unused_grad(s);
      if (ng) {
        const Storage di = to_gate(lz_mul(lz_mul(g, gg), lz_unary(RT_F_LOGISTIC_SLOPE, i)), gs, 0);
        const Storage df = to_gate(lz_mul(lz_mul(g, c_prev), lz_unary(RT_F_LOGISTIC_SLOPE, f)), gs, 1);
        const Storage dg = to_gate(lz_mul(lz_mul(g, i), lz_unary(RT_F_ONE_MINUS_SQUARE, gg)), gs, 2);
        dgates = lz_binary(RT_F_ADD, lz_binary(RT_F_ADD, di, df, gs), dg, gs);
      }
      if (nc) dprev = lz_mul(g, f);
      return {std::move(dgates), std::move(dprev)};
    }
    Storage dg = ng ? alloc(gates.shape) : unused_grad(gates.shape);
    Storage dc = nc ? alloc(c_prev.shape) : unused_grad(c_prev.shape);
    check(rt_lstm_cell_c_backward(ctx(), gates.ptr(), c_prev.ptr(), g.ptr(), (int64_t)c_prev.shape[0], (int64_t)c_prev.shape[1],
                                  ng ? dg.ptr() : nullptr, nc ? dc.ptr() : nullptr));
    return {std::move(dg), std::move(dc)};
  }
  static Storage lstm_cell_h(const Storage& gates, const Storage& c) {
    if (deferrable(gates.shape) && deferrable(c.shape)) {
      const Storage og = gate(gates, c.shape, 3, RT_F_SIGMOID), th = lz_unary(RT_F_TANH, c);
      Storage h = lz_mul(og, th);
      h.buf->made_from = gates.buf->id;
      h.buf->saved = {og.buf, th.buf};
      return h;
    }
    Storage h = alloc(c.shape);
    check(rt_lstm_cell_h(ctx(), gates.ptr(), c.ptr(), (int64_t)c.shape[0], (int64_t)c.shape[1], h.ptr()));
    return h;
  }
  static std::pair<Storage, Storage> lstm_cell_h_backward(const OpB& o, const Storage& g) {
    const Storage& gates = o.inputs[0].data();
    const Storage& c = o.inputs[1].data();
    if (g.shape != c.shape) throw Error::shape_mismatch(c.shape, g.shape);
    const bool ng = o.inputs[0].requires_grad(), nc = o.inputs[1].requires_grad();
    if (deferrable(gates.shape) && deferrable(g.shape)) {
      const Storage og = saved_gate(o, 0, gates, c.shape, 3, RT_F_SIGMOID);
      const bool kept = keeps(o, gates) && o.cached_outputs->buf->saved[1]->made_from == c.buf->id && (!c.buf->escaped || lazy::capturing());
      const Storage th = kept ? Storage{o.cached_outputs->buf->saved[1], c.shape} : lz_unary(RT_F_TANH, c);
      Storage dgates = ng ? to_gate(lz_mul(lz_mul(g, th), lz_unary(RT_F_LOGISTIC_SLOPE, og)), gates.shape, 3) : unused_grad(gates.shape);
      Storage dc = nc ? lz_mul(lz_mul(g, og), lz_unary(RT_F_ONE_MINUS_SQUARE, th)) : unused_grad(c.shape);
      return {std::move(dgates), std::move(dc)};
    }
    Storage dg = ng ? alloc(gates.shape) : unused_grad(gates.shape);
    Storage dc = nc ? alloc(c.shape) : unused_grad(c.shape);
    check(rt_lstm_cell_h_backward(ctx(), gates.ptr(), c.ptr(), g.ptr(), (int64_t)c.shape[0], (int64_t)c.shape[1],
                                  ng ? dg.ptr() : nullptr, nc ? dc.ptr() : nullptr));
    return {std::move(dg), std::move(dc)};
  }

  // The recurrence in one kernel.  Kept for the gradient: the activated gates, the cell states and their tangents.
  static Storage lstm_sequence(const Storage& x, const Storage& w, const Storage& b, size_t steps) {
    const int64_t rows = (int64_t)x.shape[0], V = (int64_t)x.shape[1], H = (int64_t)w.shape[1] / 4;
    const float *px = x.ptr(), *pw = w.ptr(), *pb = b.ptr();
    Storage h = alloc({x.shape[0], (size_t)H}), saved = alloc({6 * x.shape[0], (size_t)H});
    lazy::Block pre(ctx(), (size_t)(rows * 4 * H));
    if (V > 0) {
      check(rt_gemm_bias_act(ctx(), rows, 4 * H, V, px, V, pw, 4 * H, pb, RT_ACT_NONE, pre.ptr, 4 * H));
    } else {
      const int64_t bs[2] = {1, 4 * H}, os[2] = {rows, 4 * H};
      check(rt_broadcast_to(ctx(), pb, bs, 2, os, 2, pre.ptr));
    }
    check(rt_lstm_sequence(ctx(), pre.ptr, pw + V * 4 * H, 4 * H, nullptr, nullptr, (int64_t)steps, rows / (int64_t)steps, H, saved.ptr(), h.ptr()));
    h.buf->saved = {saved.buf};
    return h;
  }
  // From the gradient of the states: that of the gates [rows, 4H], of the weights and of the input.
  struct SequenceGradients {
    Storage dgates, dw, dx;
  };
  static SequenceGradients sequence_gradients(const float* saved, const float* x, int64_t features, const float* h, const float* w, const float* dh,
                                              int64_t steps, int64_t batch, int64_t H, bool need_w, bool need_x) {
    const int64_t rows = steps * batch, V = features, G = 4 * H;
    SequenceGradients r{alloc({(size_t)rows, (size_t)G}), {}, {}};
    const float* dz = r.dgates.ptr();
    check(rt_lstm_sequence_backward(ctx(), saved, w + V * G, G, nullptr, dh, steps, batch, H, r.dgates.ptr(), nullptr, nullptr));
    if (need_x) {
      r.dx = alloc({(size_t)rows, (size_t)V});
      if (V > 0) check(rt_gemm(ctx(), 0, 1, rows, V, G, dz, G, w, G, r.dx.ptr(), V, 0));
    }
    if (need_w) {
      r.dw = alloc({(size_t)(V + H), (size_t)G});
      float *of_x = r.dw.ptr(), *of_h = of_x + V * G;
      if (V > 0) check(rt_gemm(ctx(), 1, 0, V, G, rows, x, V, dz, G, of_x, G, 0));
      // every timestep but the first multiplies the weights with the state before it
      if (steps > 1) check(rt_gemm(ctx(), 1, 0, H, G, rows - batch, h, H, dz + batch * G, G, of_h, G, 0));
      else check(rt_fill(ctx(), of_h, 0.f, H * G));
    }
    return r;
  }
  static std::vector<Storage> lstm_sequence_backward(const OpB& o, const Storage& g, size_t steps) {
    const Storage &x = o.inputs[0].data(), &w = o.inputs[1].data(), &h = *o.cached_outputs;
    if (g.shape != h.shape) throw Error::shape_mismatch(h.shape, g.shape);
    const int64_t rows = (int64_t)x.shape[0], H = (int64_t)w.shape[1] / 4;
    const float *saved = h.buf->saved[0]->data(), *pw = w.ptr(), *px = x.ptr(), *pg = g.ptr(), *states = h.ptr();
    const bool written = h.buf->escaped && !lazy::capturing();  // perhaps, since: h = o * tanh(c) once more
    lazy::Block again(ctx(), written ? (size_t)(rows * H) : 1);
    if (written) {
      const int64_t n[1] = {rows * H};
      check(rt_binary(ctx(), RT_MUL, saved + 3 * rows * H, n, 1, saved + 5 * rows * H, n, 1, again.ptr));
      states = again.ptr;
    }
    SequenceGradients r = sequence_gradients(saved, px, (int64_t)x.shape[1], states, pw, pg, (int64_t)steps, rows / (int64_t)steps, H,
                                             o.inputs[1].requires_grad(), o.inputs[0].requires_grad());
    std::vector<Storage> out{unused_grad(x.shape), unused_grad(w.shape), unused_grad(o.inputs[2].shape())};
    if (r.dx.buf) out[0] = std::move(r.dx);
    if (r.dw.buf) out[1] = std::move(r.dw);
    if (o.inputs[2].requires_grad()) out[2] = unbroadcast(r.dgates, o.inputs[2].shape());
    return out;
  }

  // ---- sequences on the tape (Tensor::backward) ----------------------------------------------------------------------------------
  // An LSTM that was written op by op and computed as one (lazy::rewrite_recurrence) goes backward as one, too: its nodes take no part in the
  // walk, and once everything else is done the gradients of all its states go through rt_lstm_sequence_backward.  Its weights and bias are
  // leaves and its inputs take no gradient, so nothing but leaves waits for it; nobody but the tape holds its intermediate tensors, whose
  // own gradients are therefore not missed.
  using T = Tensor<B200Backend>;
  struct TapeSequence {
    std::vector<T> h;
    T w, b;
    std::vector<size_t> members;
  };
  static bool is_plain(const T& t) { return !t.inner->op && !t.requires_grad(); }
  struct TapeCell {
    const T *h, *c, *h_prev, *c_prev, *w, *b;
    std::vector<const T*> inner;  // everything between: used once each, z four times
    const T* z;
  };
  static const T* input_of(const T& t, OpType::Kind kind, size_t inputs = 1) {
    const auto& op = t.inner->op;
    return op && op->op_type.kind == kind && op->inputs.size() == inputs ? op->inputs.data() : nullptr;
  }
  static const T* tape_gate(const T& t, OpType::Kind act, size_t block, TapeCell* q) {
    const T* s = input_of(t, act);
    const T* z = s ? input_of(*s, OpType::Slice) : nullptr;
    if (!z || t.shape().size() != 2) return nullptr;
    const size_t B = t.shape()[0], H = t.shape()[1];
    const auto& r = s->inner->op->op_type.ranges;
    if (z->shape() != Shape{B, 4 * H} || r.size() != 2 || r[0].start != 0 || r[0].end != B || r[1].start != block * H || r[1].end != (block + 1) * H) return nullptr;
    q->inner.push_back(&t);
    q->inner.push_back(s);
    return z;
  }
  static bool tape_cell(const T& h, TapeCell* out) {
    const T* m = input_of(h, OpType::Mul, 2);
    if (!m) return false;
    const Shape s = h.shape();
    for (int k = 0; k < 2; ++k) {
      TapeCell q{};
      const T* z = tape_gate(m[k], OpType::Sigmoid, 3, &q);
      const T* c = z && m[1 - k].shape() == s ? input_of(m[1 - k], OpType::Tanh) : nullptr;
      const T* sum = c ? input_of(*c, OpType::Add, 2) : nullptr;
      if (!sum) continue;
      q.inner.push_back(&m[1 - k]);
      for (int e = 0; e < 8; ++e) {
        TapeCell p = q;
        const T &fc = sum[e & 1], &ig = sum[1 - (e & 1)];
        const T *u = input_of(fc, OpType::Mul, 2), *v = input_of(ig, OpType::Mul, 2);
        if (!u || !v || fc.shape() != s || ig.shape() != s) continue;
        const T &f = u[e >> 1 & 1], &before = u[1 - (e >> 1 & 1)], &i = v[e >> 2], &g = v[1 - (e >> 2)];
        if (before.shape() != s) continue;
        const T *zf = tape_gate(f, OpType::Sigmoid, 1, &p), *zi = tape_gate(i, OpType::Sigmoid, 0, &p), *zg = tape_gate(g, OpType::Tanh, 2, &p);
        if (!zf || !zi || !zg || zf->id() != z->id() || zi->id() != z->id() || zg->id() != z->id()) continue;
        const T* zs = input_of(*z, OpType::Add, 2);
        if (!zs) return false;
        for (int w = 0; w < 2; ++w) {
          const T* mm = input_of(zs[w], OpType::Matmul, 2);
          if (!mm) continue;
          const T* cat = input_of(mm[0], OpType::Concat, 2);
          if (cat ? *mm[0].inner->op->op_type.axis != 1 : !is_plain(mm[0])) continue;  // the first timestep's takes no gradient
          const T* bias = &zs[1 - w];
          p.inner.push_back(&zs[w]);
          if (cat) p.inner.push_back(&mm[0]);
          p.inner.push_back(&fc);
          p.inner.push_back(&ig);
          if (const T* b0 = input_of(*bias, OpType::Broadcast)) {
            p.inner.push_back(bias);
            bias = b0;
          }
          if (bias->inner->op || mm[1].inner->op || bias->shape() != Shape{4 * s[1]}) return false;
          if (cat && (cat[0].requires_grad() || cat[1].shape() != s)) return false;
          p.h = &h; p.c = c; p.z = z; p.h_prev = cat ? &cat[1] : nullptr; p.c_prev = &before; p.w = &mm[1]; p.b = bias;
          *out = p;
          return true;
        }
      }
    }
    return false;
  }
  static std::vector<TapeSequence> sequences(const std::vector<T>& nodes) {
    std::vector<TapeSequence> found;
    if (!lazy::capturing()) return found;
    std::unordered_map<size_t, long> uses;
    std::unordered_map<size_t, TapeCell> next;  // by the id of the state before
    for (const T& n : nodes)
      if (n.inner->op)
        for (const T& i : n.inner->op->inputs) ++uses[i.id()];
    std::vector<TapeCell> firsts;
    for (const T& n : nodes) {
      TapeCell q;
      if (!tape_cell(n, &q)) continue;
      if (!q.h_prev || is_plain(*q.h_prev)) {
        if (is_plain(*q.c_prev)) firsts.push_back(q);
      } else if (!next.emplace(q.h_prev->id(), q).second) {
        return {};  // a state that two cells go on from
      }
    }
    auto only = [&](const T& t, long n) { return uses[t.id()] == n && t.inner.use_count() == n + 1 && !t.inner->grad; };  // + 1: `nodes`
    for (const TapeCell& first : firsts) {
      TapeSequence s;
      bool ok = true;
      for (const TapeCell* q = &first; q;) {
        auto it = next.find(q->h->id());
        const TapeCell* after = it == next.end() ? nullptr : &it->second;
        if (after && (after->c_prev->id() != q->c->id() || after->w->id() != q->w->id() || after->b->id() != q->b->id())) after = nullptr;
        for (const T* t : q->inner) ok = ok && only(*t, 1);
        ok = ok && only(*q->z, 4) && only(*q->c, after ? 2 : 1) && q->h->inner.use_count() == uses[q->h->id()] + 1 && !q->h->inner->grad;
        s.h.push_back(*q->h);
        for (const T* t : q->inner) s.members.push_back(t->id());
        for (const T* t : {q->h, q->c, q->z}) s.members.push_back(t->id());
        s.w = *q->w;
        s.b = *q->b;
        q = after;
      }
      if (s.h.size() < 2) continue;
      s.h.back().data().ptr();  // computes the sequence, which the walk needs in any case
      if (!ok) continue;
      const auto& seq = s.h[0].data().buf->sequence;
      ok = seq && seq->steps == (int64_t)s.h.size() && seq->w == s.w.data().buf;
      for (size_t t = 0; t < s.h.size() && ok; ++t) ok = s.h[t].data().buf->sequence == seq && s.h[t].data().buf->timestep == (int64_t)t;
      if (ok) found.push_back(std::move(s));
    }
    return found;
  }
  static void sequence_backward(const TapeSequence& s) {
    const std::shared_ptr<Recurrence> q = s.h[0].data().buf->sequence;
    const int64_t n = q->batch * q->hidden;
    lazy::Block dh(ctx(), (size_t)(q->steps * n));
    for (int64_t t = 0; t < q->steps;) {
      float* out = dh.ptr + t * n;
      const auto& g = s.h[t].grad();
      auto product = [&](int64_t i) -> const lazy::Node* {  // the gradient is a product that nobody else has asked for
        if (i >= q->steps || !s.h[i].grad() || !s.h[i].grad()->buf) return nullptr;
        const DeviceBuffer* b = s.h[i].grad()->buf.get();
        return b->node && b->node->tag == lazy::Tag::MatmulNT && b->readers.empty() ? b->node.get() : nullptr;
      };
      if (const lazy::Node* p = product(t)) {  // and those after it, as long as their operands follow in memory
        const int64_t m = (int64_t)p->in[0].shape[0], cols = (int64_t)p->in[0].shape[1], k = (int64_t)p->in[1].shape[0];
        const float* first = p->in[0].buf->data();
        int64_t count = 1;
        for (const lazy::Node* r; (r = product(t + count)) && r->in[1].buf == p->in[1].buf && r->in[0].shape == p->in[0].shape &&
                                  r->in[0].buf->data() == first + count * m * cols;)
          ++count;
        check(rt_gemm(ctx(), 0, 1, count * m, k, cols, first, cols, p->in[1].buf->data(), cols, out, k, 0));
        t += count;
      } else {
        if (g) check(rt_memcpy_d2d(ctx(), out, g->ptr(), sizeof(float) * (size_t)n));
        else check(rt_fill(ctx(), out, 0.f, n));
        ++t;
      }
    }
    SequenceGradients r = sequence_gradients(q->saved->ptr, q->x_rows, q->features, q->h->ptr, q->w->ptr, dh.ptr, q->steps, q->batch, q->hidden,
                                             s.w.requires_grad(), false);
    if (r.dw.buf) s.w.add_grad(std::move(r.dw));
    if (s.b.requires_grad()) s.b.add_grad(unbroadcast(r.dgates, s.b.shape()));
  }

  // One launch for all parameters of an optimizer step.  kind as rt_optimizer_step_multi; s1 / s2: the optimizer's states.
  static void step_all(int kind, const std::vector<Storage*>& ps, const std::vector<Storage>& gs, const std::vector<Storage*>& s1,
                       const std::vector<Storage*>& s2, float lr, float b1, float b2, float eps, float momentum, size_t t) {
    if (kind == 1 && t == 0) throw Error::internal("Adam step called with t=0");
    std::vector<float*> p, a, b;
    std::vector<const float*> g;
    std::vector<int64_t> n;
    auto launch = [&] {
      if (!p.empty())
        check(rt_optimizer_step_multi(ctx(), kind, (int)p.size(), p.data(), g.data(), a.data(), b.data(), n.data(), lr, b1, b2, eps, momentum,
                                      (int64_t)t, 1.f, 0, 0.f, 0.f));
      p.clear(); a.clear(); b.clear(); g.clear(); n.clear();
    };
    for (size_t i = 0; i < ps.size(); ++i) {
      if (ps[i]->shape != gs[i].shape) throw Error::shape_mismatch(ps[i]->shape, gs[i].shape);
      if (ps[i]->numel() == 0) continue;
      g.push_back(gs[i].ptr());
      if (std::find(p.begin(), p.end(), ps[i]->buf->ptr) != p.end()) launch();  // a parameter listed twice is updated twice, in order
      make_unique(*ps[i]);
      p.push_back(ps[i]->ptr());
      if (kind != 0) {
        make_unique(*s1[i]);
        a.push_back(s1[i]->ptr());
      } else {
        a.push_back(nullptr);
      }
      if (kind == 1) {
        make_unique(*s2[i]);
        b.push_back(s2[i]->ptr());
      } else {
        b.push_back(nullptr);
      }
      n.push_back((int64_t)ps[i]->numel());
    }
    launch();
  }

  // ---- optimizer steps (mod.rs:18-36, 256-272) ---------------------------------------------------
  static void sgd_step(Storage& w, const Storage& dw, float lr) {
    if (w.shape != dw.shape) throw Error::shape_mismatch(w.shape, dw.shape);
    make_unique(w);
    check(rt_sgd_step(ctx(), w.ptr(), dw.ptr(), (int64_t)w.numel(), lr));
  }
  static void momentum_sgd_step(Storage& p, const Storage& g, Storage& vel, float lr, float mu) {
    if (p.shape != vel.shape) throw Error::shape_mismatch(p.shape, vel.shape);
    if (p.shape != g.shape) throw Error::shape_mismatch(p.shape, g.shape);
    make_unique(p);
    make_unique(vel);
    check(rt_momentum_sgd_step(ctx(), p.ptr(), g.ptr(), vel.ptr(), (int64_t)p.numel(), lr, mu));
  }
  static void adagrad_step(Storage& p, const Storage& g, Storage& acc, float lr, float eps) {
    if (p.shape != g.shape) throw Error::shape_mismatch(p.shape, g.shape);
    if (p.shape != acc.shape) throw Error::shape_mismatch(p.shape, acc.shape);
    make_unique(p);
    make_unique(acc);
    check(rt_adagrad_step(ctx(), p.ptr(), g.ptr(), acc.ptr(), (int64_t)p.numel(), lr, eps));
  }
  static void adam_step(Storage& p, const Storage& g, Storage& m, Storage& v, float lr, float b1, float b2, float eps,
                        size_t t) {
    if (p.shape != g.shape) throw Error::shape_mismatch(p.shape, g.shape);
    if (p.shape != m.shape) throw Error::shape_mismatch(p.shape, m.shape);
    if (p.shape != v.shape) throw Error::shape_mismatch(p.shape, v.shape);
    if (t == 0) throw Error::internal("Adam step called with t=0");
    make_unique(p);
    make_unique(m);
    make_unique(v);
    check(rt_adam_step(ctx(), p.ptr(), g.ptr(), m.ptr(), v.ptr(), (int64_t)p.numel(), lr, b1, b2, eps, (int64_t)t));
  }
};

}  // namespace rt
