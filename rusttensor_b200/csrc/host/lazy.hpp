// Deferred elementwise ops of the CUDA backend.
//
// A model written op by op asks for one small kernel after another, and inside a CUDA graph as well as outside of it every
// kernel costs 1.3 - 2 us and a pass over memory however little it computes.  The backend therefore only notes down what an
// elementwise op (arithmetic, activations and their gradients, broadcasting, slicing, padding, concatenation) is to compute:
// the result's buffer holds an expression (Node) over its operands' buffers.  The first use that needs the values - a product,
// a reduction, an optimizer step, a copy to the host, a device pointer - evaluates the expression together with all the
// unevaluated ones below it in ONE launch of the interpreting kernel (rt_fused_elementwise).
//
// Rules that keep this invisible:
//  * Buffers are immutable once produced.  What does change one in place (optimizer steps, update_from_host, accumulating
//    kernels) first evaluates every expression that reads it (flush_readers).
//  * A buffer whose address has been handed out may be written behind the engine's back, so expressions that read it are
//    evaluated on the spot - except inside a graph capture, where the whole step is recorded anyway.
//  * A slice of whole rows points into its base's block only inside a capture, where nothing outside the engine sees either of them
//    before the step is recorded; what a step leaves behind gets a block of its own (B200Backend::own).  Elsewhere the address of one
//    of the two may be handed out and written through, and a slice would keep its base's memory.  Results that a capture computes as one
//    matrix (place) are rows of a block that no tensor has as a whole: they stay there, where every replay writes them.
//  * A capture starts with nothing unevaluated (flush_all), so that it records exactly the step's own work, and rth_sync leaves
//    nothing unevaluated either.
//  * Depth is bounded: a result whose expression has become kMaxDepth ops deep is evaluated at once.  The timesteps of a recurrence in a
//    capture, which wait for the last one, are evaluated from the first one on where they do not become one sequence.
//
// What is written to memory besides the asked-for result: intermediate results that somebody else still refers to, when the
// tensor is small (a launch later on would cost more than the store), or when recomputing them would be expensive.
#pragma once
#include <algorithm>
#include <cstring>
#include <functional>
#include <memory>
#include <unordered_set>
#include <vector>

#include "../../../include/rt_b200.h"
#include "autograd.hpp"

namespace rt {

struct DeviceBuffer;
void lazy_evaluate(DeviceBuffer* b);

namespace lazy {

struct Input {
  std::shared_ptr<DeviceBuffer> buf;
  Shape shape;
};
enum class Kind : uint8_t { Const, Unary, BinaryImm, Binary, Broadcast, Slice, Pad, Concat, Opaque };
// Opaque: computed by a kernel of its own.  Deferred only because what it feeds may take a kernel that does both.
// Tag::RowGrad (the gradient of a logsumexp) is a Binary with a kernel of its own besides (`run`, from in[0] and in[2]): an expression in compiled
// programs that carry a reduction, memory in all others, which the interpreter would run.
enum class Tag : uint8_t { None, Matmul, Conv, LogSoftmax, Reduce, PoolGrad, SumProducts, SumRows, FusedLoss, NllGrad, MatmulNT, RowGrad };

struct Node {
  Kind kind;
  uint8_t op = 0;
  bool swap = false;  // BinaryImm: the immediate is the left operand
  float imm = 0.f;
  int depth = 1;
  int weight = 0;     // cost of evaluating it from its evaluated inputs, in simple ops
  Shape shape;
  Shape starts;       // Slice, Pad: the box's origin; Concat: {axis}
  std::vector<Input> in;
  // Opaque, RowGrad
  Tag tag = Tag::None;
  std::vector<int64_t> geo;  // its parameters, as its tag has them
  std::function<void(Node&, DeviceBuffer*)> run;  // computes the buffer (sets ptr)
  bool waits() const { return tag == Tag::Matmul && !geo.empty(); }  // the product of a recurrence's timestep, for the last one
};

constexpr int kMaxDepth = 200;
constexpr size_t kSmall = (size_t)1 << 20;    // elements up to which shared intermediate results are always written
constexpr int kRecompute = 16;              // weight from which they are written whatever the size
constexpr int kDuplicate = 2;               // most weight that is repeated for every element of a broadcast
constexpr int kMaxChain = 512;              // depth of a sum of scalars (the losses of a sequence)

// What evaluating an expression costs now, up to `limit`; products and the like count as evaluated, which they will be by then.
int current_weight(const Node& n, int limit);

}  // namespace lazy

// An LSTM over a sequence that was written op by op and has been computed as one (lazy::rewrite_recurrence).
struct Recurrence {
  std::shared_ptr<DeviceBuffer> saved, h, x, w;  // six planes and the states [steps * batch, hidden]; inputs; weights
  const float* x_rows = nullptr;                 // [steps * batch, features]
  int64_t steps = 0, batch = 0, hidden = 0, features = 0;
};

struct DeviceBuffer : std::enable_shared_from_this<DeviceBuffer> {
  rt_ctx* ctx;
  float* ptr;
  size_t numel;
  bool escaped = false;
  std::shared_ptr<DeviceBuffer> owner;  // set: ptr points into this buffer's block (contiguous rows of it)
  bool apart = false;        // with an owner: these rows of its block are this buffer's alone, and no tensor is the whole block
  uint64_t id = next_id();   // of the values: another one after every change in place
  uint64_t made_from = 0;    // id of the operand's values, for results from which their gradient follows
  std::shared_ptr<Recurrence> sequence;  // set: the state after timestep `timestep` of it
  int64_t timestep = 0;
  std::vector<std::shared_ptr<DeviceBuffer>> saved;  // intermediate results of a fused op that its gradient uses
  std::unique_ptr<lazy::Node> node;    // what to compute; null once the values are in memory
  std::vector<DeviceBuffer*> readers;  // unevaluated buffers whose expression takes this one as an input
  DeviceBuffer *prev = nullptr, *next = nullptr;  // list of all unevaluated buffers

  static uint64_t next_id() {
    static uint64_t n = 0;
    return ++n;
  }
  static DeviceBuffer*& head() {
    static DeviceBuffer* h = nullptr;
    return h;
  }
  // How many products of timesteps wait for their last one; how many gradients of rows are pending.
  static size_t& waiting() {
    static size_t n = 0;
    return n;
  }
  static size_t& row_gradients() {
    static size_t n = 0;
    return n;
  }
  DeviceBuffer(rt_ctx* c, float* p, size_t n) : ctx(c), ptr(p), numel(n) {}
  DeviceBuffer(rt_ctx* c, std::unique_ptr<lazy::Node> nd, size_t n) : ctx(c), ptr(nullptr), numel(n), node(std::move(nd)) {
    for (auto& i : node->in) i.buf->readers.push_back(this);
    if (node->waits()) ++waiting();
    if (node->tag == lazy::Tag::RowGrad) ++row_gradients();
    next = head();
    if (next) next->prev = this;
    head() = this;
  }
  DeviceBuffer(const DeviceBuffer&) = delete;
  DeviceBuffer& operator=(const DeviceBuffer&) = delete;
  ~DeviceBuffer() {
    drop_node();
    if (ptr && !owner) rt_free(ctx, ptr);
  }
  void drop_node() {
    if (!node) return;
    std::unique_ptr<lazy::Node> gone = std::move(node);
    if (prev) prev->next = next;
    else head() = next;
    if (next) next->prev = prev;
    prev = next = nullptr;
    // The operands are let go of one after another, not each within the one that reads it: an expression may be as deep as a sequence is long.
    static auto& dying = *new std::vector<std::shared_ptr<DeviceBuffer>>;  // used until the last buffer goes, at exit
    static bool busy = false;
    if (gone->waits()) --waiting();
    if (gone->tag == lazy::Tag::RowGrad) --row_gradients();
    for (auto& i : gone->in) {
      auto& r = i.buf->readers;
      for (size_t k = r.size(); k-- > 0;)
        if (r[k] == this) {
          r[k] = r.back();
          r.pop_back();
          break;
        }
      dying.push_back(std::move(i.buf));
    }
    if (busy) return;
    busy = true;
    while (!dying.empty()) {
      const std::shared_ptr<DeviceBuffer> b = std::move(dying.back());
      dying.pop_back();
    }
    busy = false;
  }
  // Whether the values are also those of another buffer (a slice's, of its base).
  bool shares_rows() const { return owner && !apart; }
  float* data() {
    if (node) lazy_evaluate(this);
    return ptr;
  }
  void flush_readers() {
    while (!readers.empty()) lazy_evaluate(readers.back());
  }
};

namespace lazy {

int op_weight(uint8_t op);
inline int current_weight(const Node& n, int limit) {
  if (n.kind == Kind::Opaque) return 0;
  int w = n.kind == Kind::Unary || n.kind == Kind::Binary || n.kind == Kind::BinaryImm ? op_weight(n.op) : 0;
  for (auto& i : n.in) {
    if (w > limit) break;
    if (i.buf->node) w += current_weight(*i.buf->node, limit - w);
  }
  return w;
}

inline bool& capturing() {
  static bool c = false;
  return c;
}
// Off: every op runs at once by its own kernel, as tensors of 2^31 and more elements always do (rth_set_deferred_ops).
inline bool& deferring() {
  static bool d = true;
  return d;
}
inline void flush_all() {
  while (DeviceBuffer::head()) lazy_evaluate(DeviceBuffer::head());
}

inline int op_weight(uint8_t op) {
  switch (op) {
    case RT_F_EXP: case RT_F_LN: case RT_F_SIN: case RT_F_COS: case RT_F_TAN: case RT_F_TANH: case RT_F_SIGMOID: case RT_F_SOFTPLUS:
    case RT_F_ELU: case RT_F_ELU_SLOPE: case RT_F_POWF: return 4;
    case RT_F_DIV: case RT_F_RECIP: case RT_F_SQRT: case RT_F_HALF_RSQRT: case RT_F_RECIP_SQUARE: return 3;
    default: return 1;
  }
}

// ---- from an expression to a program -----------------------------------------------------------------------------------------
constexpr int kMaxRawDims = 8;

// How a tensor's coordinates follow from the iteration coordinates: dimension j = (map[j] < 0 ? 0 : iteration[map[j]]) + off[j].
struct View {
  int nd = 0;
  int8_t map[kMaxRawDims];
  int64_t off[kMaxRawDims];
  int region = RT_FUSED_NONE;
  bool operator==(const View& o) const {
    if (nd != o.nd || region != o.region) return false;
    for (int j = 0; j < nd; ++j)
      if (map[j] != o.map[j] || off[j] != o.off[j]) return false;
    return true;
  }
};

// While it lives, expressions are being walked over: an evaluation is under way, or a program is being built.  What is evaluated meanwhile lies
// below them; reductions over the same values, which do not, are taken along only where nothing is being walked (they would disappear from under
// whoever walks).
struct Walk {
  static int& depth() {
    static int n = 0;
    return n;
  }
  Walk() { ++depth(); }
  ~Walk() { --depth(); }
  Walk(const Walk&) = delete;
};

class Compiler {
 public:
  // Builds the program of `root`; false: it does not fit (the caller evaluates some inputs first and tries again).
  bool build(DeviceBuffer* root, rt_fused_program* p, std::vector<DeviceBuffer*>* stored) {
    const Walk walk;
    const Node& n = *root->node;
    nd_ = (int)n.shape.size();
    if (nd_ > kMaxRawDims) return false;
    for (int d = 0; d < nd_; ++d) shape_[d] = (int64_t)n.shape[d];
    if (nd_ == 0) {
      nd_ = 1;
      shape_[0] = 1;
    }
    numel_ = root->numel;
    View id;
    id.nd = (int)n.shape.size();
    for (int j = 0; j < id.nd; ++j) {
      id.map[j] = (int8_t)j;
      id.off[j] = 0;
    }
    views_.push_back(id);
    root_ = root;
    root_shape_ = n.shape;
    const int r = node_value(root, 0);
    if (r < 0) return false;
    outputs_.push_back({r, root});
    std::pair<int, DeviceBuffer*> sum{-1, nullptr};
    if (look_for_sums_ && nd_ == 2) sum = waiting_sum();
    if (!root->node) return false;
    for (auto& c : stored_) {
      if ((int)outputs_.size() + (sum.second ? 1 : 0) == RT_FUSED_MAX_OUTPUTS) break;
      if (c.second->node && wanted_later(c.second)) outputs_.push_back({c.first, c.second});  // not evaluated meanwhile, as part of some other program
    }
    if (sum.second) {
      sums_ = (int)outputs_.size();
      outputs_.push_back(sum);
    }
    if (!collapse(p)) return false;
    for (int pre = std::min<int>((int)operands_.size(), RT_FUSED_PRELOAD); pre >= 0; --pre)
      if (emit(p, pre)) {
        for (auto& o : outputs_) stored->push_back(o.second);
        return true;
      }
    return false;
  }
  const std::vector<std::pair<int, DeviceBuffer*>>& outputs() const { return outputs_; }
  // The dimensions stay those of the root (two), for a reduction over one of them; with_sums: for pending column sums, if there are any.
  void keep_rows(bool with_sums) {
    keep_rows_ = true;
    look_for_sums_ = with_sums;
  }
  // Among the outputs, the pending column sums of a term that shares values with the root (its buffer in the outputs is the sums'); -1: none.
  int sums() const { return sums_; }

 private:
  struct Value {
    uint8_t op;       // RT_F_*; RT_F_LOAD: operand `a`; RT_F_REG: the immediate
    bool swap;
    int a, b;         // value numbers; b < 0: none, or the immediate for a binary op
    int region;       // RT_F_SELECT: a inside, b (or the immediate) outside
    float imm;
  };
  struct Operand {
    std::shared_ptr<DeviceBuffer> buf;  // stays allocated until the launch
    const float* ptr;
    int64_t stride[kMaxRawDims];
    int region;
  };
  struct Box {
    int64_t lo[kMaxRawDims], hi[kMaxRawDims];
  };
  struct Memo {
    DeviceBuffer* b;
    uint64_t id;  // b's: what is evaluated on the way may free a buffer that has been walked over
    int view, value;
    bool of(const DeviceBuffer* x, int v) const { return b == x && id == x->id && view == v; }
  };
  DeviceBuffer* root_ = nullptr;
  Shape root_shape_;
  int nd_ = 0;
  int64_t shape_[kMaxRawDims];
  size_t numel_ = 0;
  std::vector<View> views_;
  std::vector<Value> values_;
  std::vector<Operand> operands_;
  std::vector<Box> regions_;
  std::vector<Memo> memo_;
  std::vector<std::pair<int, DeviceBuffer*>> stored_, outputs_;

  bool keep_rows_ = false, look_for_sums_ = false;
  int sums_ = -1;
  // A bias that is broadcast over the rows gets the column sums of a product of something that is computed here anyway: the term's value
  // and the buffer of the sums.
  std::pair<int, DeviceBuffer*> waiting_sum() {
    const std::pair<int, DeviceBuffer*> none{-1, nullptr};
    for (DeviceBuffer* x = DeviceBuffer::head(); x; x = x->next) {  // what was walked over and is still pending
      if (std::none_of(memo_.begin(), memo_.end(), [&](const Memo& m) { return m.of(x, 0); })) continue;
      for (DeviceBuffer* r : x->readers) {
        if (!r->node || r->node->kind == Kind::Opaque || r->node->shape != root_shape_ || r->readers.size() != 1) continue;
        DeviceBuffer* s = r->readers[0];
        if (!s->node || s->node->tag != Tag::SumRows || s->node->geo[0] >= 0 || s->node->in[0].shape != root_shape_ || (int64_t)s->numel != shape_[1]) continue;
        const std::weak_ptr<DeviceBuffer> term = r->weak_from_this(), sum = s->weak_from_this();
        const int v = node_value(r, 0);
        // what the term needs besides may have been evaluated on the way, and with it the term or the root
        if (v < 0 || is_imm(v) || sum.expired() || !s->node || term.expired() || !r->node || !root_->node) return none;
        return {v, s};
      }
    }
    return none;
  }
  // In a capture a large intermediate result whose readers are all part of this program is left to whoever asks for it after all (the tape holds
  // every tensor's gradient): writing it would cost as much as the program.
  bool wanted_later(DeviceBuffer* b) const {
    if (!capturing() || b->numel <= kSmall) return true;
    for (DeviceBuffer* r : b->readers) {
      bool here = false;
      for (auto& m : memo_) here = here || m.of(r, 0);
      if (!here) return true;
    }
    return false;
  }

  int view_id(const View& v) {
    for (size_t i = 0; i < views_.size(); ++i)
      if (views_[i] == v) return (int)i;
    views_.push_back(v);
    return (int)views_.size() - 1;
  }
  int add(uint8_t op, int a, int b, float imm, bool swap = false, int region = RT_FUSED_NONE) {
    for (size_t i = values_.size(); i-- > 0;) {
      const Value& v = values_[i];
      if (v.op == op && v.a == a && v.b == b && v.swap == swap && v.region == region && std::memcmp(&v.imm, &imm, sizeof(float)) == 0)
        return (int)i;
    }
    if (values_.size() >= RT_FUSED_MAX_CODE) return -1;
    values_.push_back({op, swap, a, b, region, imm});
    return (int)values_.size() - 1;
  }
  bool is_imm(int v) const { return values_[v].op == RT_F_REG; }

  int region_id(const Box& b) {
    for (size_t i = 0; i < regions_.size(); ++i) {
      bool same = true;
      for (int d = 0; d < nd_; ++d) same = same && regions_[i].lo[d] == b.lo[d] && regions_[i].hi[d] == b.hi[d];
      if (same) return (int)i;
    }
    if (regions_.size() >= RT_FUSED_MAX_REGIONS) return -1;
    regions_.push_back(b);
    return (int)regions_.size() - 1;
  }

  // Maps a view of a node onto one of its inputs (right-aligned dimensions; extent 1 stretches).
  View child_view(const View& v, const Shape& node, const Shape& child) const {
    View c;
    c.nd = (int)child.size();
    c.region = v.region;
    const int lead = (int)node.size() - c.nd;
    for (int j = 0; j < c.nd; ++j) {
      if (child[j] == 1 && node[j + lead] != 1) {
        c.map[j] = -1;
        c.off[j] = 0;
      } else {
        c.map[j] = v.map[j + lead];
        c.off[j] = v.off[j + lead];
      }
    }
    return c;
  }
  // Restricts a view to the box [start, start + extent) of its tensor and moves the origin there.  -1: no room for the region;
  // false in `any`: nothing of the box is seen.
  int box_view(const View& v, const Shape& starts, const Shape& extent, View* out, bool* any) {
    Box b;
    for (int d = 0; d < nd_; ++d) {
      b.lo[d] = v.region == RT_FUSED_NONE ? 0 : regions_[v.region].lo[d];
      b.hi[d] = v.region == RT_FUSED_NONE ? shape_[d] : regions_[v.region].hi[d];
    }
    *out = v;
    *any = true;
    for (int j = 0; j < v.nd; ++j) {
      const int64_t s = (int64_t)starts[j], n = (int64_t)extent[j];
      out->off[j] = v.off[j] - s;
      if (v.map[j] < 0) {
        if (v.off[j] < s || v.off[j] >= s + n) *any = false;
        continue;
      }
      const int d = v.map[j];
      b.lo[d] = std::max(b.lo[d], s - v.off[j]);
      b.hi[d] = std::min(b.hi[d], s + n - v.off[j]);
      if (b.lo[d] >= b.hi[d]) *any = false;
    }
    if (!*any) return RT_FUSED_NONE;
    bool full = true;
    for (int d = 0; d < nd_; ++d) full = full && b.lo[d] <= 0 && b.hi[d] >= shape_[d];
    if (full) return out->region = RT_FUSED_NONE;
    const int r = region_id(b);
    if (r < 0) return -1;
    return out->region = r;
  }

  // The view of a tensor as seen by an expression of the same values whose shape differs in extents of 1 only.
  static bool squeezed_view(const View& v, const Shape& from, const Shape& to, View* w) {
    w->nd = (int)to.size();
    w->region = v.region;
    size_t i = 0;
    for (size_t j = 0; j < to.size(); ++j) {
      w->map[j] = -1;
      w->off[j] = 0;
      if (to[j] == 1) continue;
      while (i < from.size() && from[i] == 1) ++i;
      if (i == from.size() || from[i] != to[j]) return false;
      w->map[j] = v.map[i];
      w->off[j] = v.off[i];
      ++i;
    }
    while (i < from.size() && from[i] == 1) ++i;
    return i == from.size();
  }

  int leaf(const Input& in, const View& v) {
    Operand o;
    for (int d = 0; d < kMaxRawDims; ++d) o.stride[d] = 0;
    int64_t stride = 1, off = 0;
    for (int j = v.nd - 1; j >= 0; --j) {
      off += v.off[j] * stride;
      if (v.map[j] >= 0 && shape_[v.map[j]] != 1) o.stride[v.map[j]] += stride;
      stride *= (int64_t)in.shape[j];
    }
    if (stride >= (1ll << 31)) return -1;
    o.buf = in.buf;
    o.ptr = in.buf->ptr + off;
    o.region = v.region;
    for (size_t k = 0; k < operands_.size(); ++k) {
      bool same = operands_[k].ptr == o.ptr && operands_[k].region == o.region;
      for (int d = 0; d < nd_; ++d) same = same && operands_[k].stride[d] == o.stride[d];
      if (same) return add(RT_F_LOAD, (int)k, -1, 0.f);
    }
    if (operands_.size() >= RT_FUSED_MAX_OPERANDS) return -1;
    operands_.push_back(o);
    return add(RT_F_LOAD, (int)operands_.size() - 1, -1, 0.f);
  }

  int input_value(const Input& in, const View& v) {
    if (in.buf->node && in.buf->node->kind != Kind::Opaque && in.buf->node->shape != in.shape) {
      if (in.buf->node->kind == Kind::Const) return add(RT_F_REG, -1, -1, in.buf->node->imm);
      View w;
      if (in.buf->node->weight <= kDuplicate && squeezed_view(v, in.shape, in.buf->node->shape, &w)) return node_value(in.buf.get(), view_id(w));
      lazy_evaluate(in.buf.get());  // its own dimensions do not match the iteration's
    }
    if (in.buf->node && in.buf->node->kind != Kind::Const && in.buf->node->kind != Kind::Opaque && in.buf->node->weight > kDuplicate) {
      // an expensive expression under a broadcast would be evaluated over and over
      for (int d = 0; d < nd_; ++d) {
        if (shape_[d] == 1) continue;
        bool seen = false;
        for (int j = 0; j < v.nd; ++j) seen = seen || v.map[j] == d;
        if (!seen) {
          lazy_evaluate(in.buf.get());
          break;
        }
      }
    }
    if (in.buf->node && in.buf->node->kind == Kind::Opaque) lazy_evaluate(in.buf.get());
    // seen through a window (not over its own full shape), costly, and part of several expressions: once, into memory
    if (in.buf->node && in.buf->readers.size() >= 2 && !(v == views_[0] && in.shape == root_shape_) && current_weight(*in.buf->node, 4) > 3)
      lazy_evaluate(in.buf.get());
    if (!in.buf->node) return leaf(in, v);
    return node_value(in.buf.get(), view_id(v));
  }

  int node_value(DeviceBuffer* b, int vid) {
    for (auto& m : memo_)
      if (m.of(b, vid)) return m.value;
    const int r = make_value(b, vid);
    if (r >= 0) {
      memo_.push_back({b, b->id, vid, r});
      if (vid == 0 && b != root_ && b->node->shape == root_shape_ && values_[r].op != RT_F_LOAD && values_[r].op != RT_F_REG && worth_storing(b))
        stored_.push_back({r, b});
    }
    return r;
  }
  static bool worth_storing(DeviceBuffer* b) {
    const Node& n = *b->node;
    if (n.kind == Kind::Const || n.kind == Kind::Broadcast || n.kind == Kind::Slice) return false;
    // whoever is not an unevaluated expression: tensors, recorded ops, callers
    const long outside = b->weak_from_this().use_count() - (long)b->readers.size();
    if (outside <= 0) return false;
    return b->numel <= kSmall || n.weight >= kRecompute;
  }

  int make_value(DeviceBuffer* b, int vid) {
    const Node& n = *b->node;
    const View v = views_[vid];  // a copy: views_ grows below
    switch (n.kind) {
      case Kind::Const: return add(RT_F_REG, -1, -1, n.imm);
      case Kind::Unary: {
        const int a = input_value(n.in[0], child_view(v, n.shape, n.in[0].shape));
        return a < 0 ? -1 : add(n.op, a, -1, n.imm);
      }
      case Kind::BinaryImm: {
        const int a = input_value(n.in[0], child_view(v, n.shape, n.in[0].shape));
        return a < 0 ? -1 : add(n.op, a, -1, n.imm, n.swap);
      }
      case Kind::Broadcast: return input_value(n.in[0], child_view(v, n.shape, n.in[0].shape));
      case Kind::Binary: {
        int a, c;
        const View va = child_view(v, n.shape, n.in[0].shape), vb = child_view(v, n.shape, n.in[1].shape);
        auto cost = [](const Input& i) { return i.buf->node ? 1 + current_weight(*i.buf->node, 64) : 0; };
        if (cost(n.in[1]) > cost(n.in[0])) {  // the larger side first: fewer values are alive at a time
          c = input_value(n.in[1], vb);
          a = c < 0 ? -1 : input_value(n.in[0], va);
        } else {
          a = input_value(n.in[0], va);
          c = a < 0 ? -1 : input_value(n.in[1], vb);
        }
        if (a < 0 || c < 0) return -1;
        if (is_imm(c)) return add(n.op, a, -1, values_[c].imm);
        if (is_imm(a)) return add(n.op, c, -1, values_[a].imm, true);
        return add(n.op, a, c, 0.f);
      }
      case Kind::Slice: {
        settle_shared(n.in[0]);
        View c = v;
        for (int j = 0; j < v.nd; ++j) c.off[j] += (int64_t)n.starts[j];
        return input_value(n.in[0], c);
      }
      case Kind::Pad: return boxed(n.in[0], v, n.starts, -1);
      case Kind::Concat: {
        Shape starts(n.shape.size(), 0);
        int r = -1;
        for (auto& piece : n.in) {
          settle_shared(piece);
          r = boxed(piece, v, starts, r);
          if (r < 0) return -1;
          starts[n.starts[0]] += piece.shape[n.starts[0]];
        }
        return r;
      }
      case Kind::Opaque: break;
    }
    return -1;
  }
  // A costly result that others use too and that is seen here only through a window: it is written to memory now, because the
  // program around the window cannot write it and whoever else asks would compute it again.
  static void settle_shared(const Input& in) {
    DeviceBuffer* b = in.buf.get();
    if (b->node && b->weak_from_this().use_count() > (long)b->readers.size() && current_weight(*b->node, 4) > 3) lazy_evaluate(b);
  }
  // The value of `in` placed at `starts`, and `other` (0 when negative) elsewhere.
  int boxed(const Input& in, const View& v, const Shape& starts, int other) {
    View c;
    bool any;
    const int r = box_view(v, starts, in.shape, &c, &any);
    if (r < 0) return -1;
    if (!any) return other < 0 ? add(RT_F_REG, -1, -1, 0.f) : other;
    const int a = input_value(in, c);
    if (a < 0 || r == RT_FUSED_NONE) return a;
    if (other < 0 && values_[a].op == RT_F_LOAD && operands_[values_[a].a].region == r) return a;  // 0 outside already
    if (other < 0 || is_imm(other)) return add(RT_F_SELECT, a, -1, other < 0 ? 0.f : values_[other].imm, false, r);
    return add(RT_F_SELECT, a, other, 0.f, false, r);
  }

  // Merges neighbouring dimensions that every operand walks as one and writes shape, operands and regions.
  bool collapse(rt_fused_program* p) {
    int nd = 0;
    int keep[kMaxRawDims];
    int64_t shape[kMaxRawDims];
    std::vector<Operand> ops = operands_;
    std::vector<Box> boxes = regions_;
    for (int d = 0; d < nd_; ++d) {
      if (!keep_rows_ && shape_[d] == 1 && !(d == nd_ - 1 && nd == 0)) {
        bool trivial = true;
        for (auto& b : boxes) trivial = trivial && b.lo[d] <= 0 && b.hi[d] >= 1;
        if (trivial) continue;
      }
      bool merge = nd > 0 && !keep_rows_;
      if (merge) {
        const int q = keep[nd - 1];
        for (auto& o : ops) merge = merge && o.stride[q] == o.stride[d] * shape_[d];
        for (auto& b : boxes) merge = merge && b.lo[d] <= 0 && b.hi[d] >= shape_[d];
        if (merge) {
          for (auto& o : ops) o.stride[q] = o.stride[d];
          for (auto& b : boxes) {
            b.lo[q] *= shape_[d];
            b.hi[q] *= shape_[d];
          }
          shape[nd - 1] *= shape_[d];
          continue;
        }
      }
      keep[nd] = d;
      shape[nd++] = shape_[d];
    }
    if (nd == 0) {
      keep[0] = nd_ - 1;
      shape[0] = 1;
      nd = 1;
    }
    if (nd > RT_FUSED_MAX_DIMS) return false;
    p->nd = nd;
    for (int i = 0; i < nd; ++i) p->shape[i] = (int32_t)shape[i];
    p->n_operands = (int)ops.size();
    for (size_t k = 0; k < ops.size(); ++k) {
      p->operand[k].ptr = ops[k].ptr;
      p->operand[k].region = ops[k].region;
      for (int i = 0; i < RT_FUSED_MAX_DIMS; ++i) p->operand[k].stride[i] = i < nd ? (int32_t)ops[k].stride[keep[i]] : 0;
    }
    p->n_regions = (int)boxes.size();
    for (size_t k = 0; k < boxes.size(); ++k)
      for (int i = 0; i < RT_FUSED_MAX_DIMS; ++i) {
        p->region[k].lo[i] = i < nd ? (int32_t)boxes[k].lo[keep[i]] : 0;
        p->region[k].hi[i] = i < nd ? (int32_t)boxes[k].hi[keep[i]] : 1;
      }
    return true;
  }

  // ---- instructions and registers: one accumulator, a value goes to a register when the accumulator is overwritten before its
  // last use (the instruction that produced it then also writes the register) -------------------------------------------------
  struct Emitter {
    rt_fused_program* p;
    const std::vector<Value>& values;
    std::vector<int> where, left;  // register of a value or -1; uses that are still to come
    int acc = -1;
    unsigned free_regs = (1u << RT_FUSED_REGS) - 1;
    bool ok = true;

    int take() {
      for (int r = 0; r < RT_FUSED_REGS; ++r)
        if (free_regs & (1u << r)) {
          free_regs &= ~(1u << r);
          return r;
        }
      return -1;
    }
    void keep_acc() {  // gives the accumulator's value a register
      if (acc < 0 || where[acc] >= 0) return;
      const int r = take();
      if (r < 0) {
        ok = ok && values[acc].op == RT_F_LOAD;  // an operand can be loaded again
        return;
      }
      p->code[p->n_code - 1].dst = (uint8_t)r;
      where[acc] = r;
    }
    void put(uint8_t op, uint8_t src, uint8_t swap, float imm, int value) {
      if (value != acc && acc >= 0 && left[acc] > 0) keep_acc();
      if (p->n_code >= RT_FUSED_MAX_CODE) ok = false;
      if (!ok) return;
      p->code[p->n_code++] = {op, src, RT_FUSED_NONE, swap, imm};
      acc = value;
    }
    void release(int v) {
      if (left[v] == 0 && where[v] >= 0) {
        free_regs |= 1u << where[v];
        where[v] = -1;
      }
    }
    void to_acc(int v) {
      if (acc == v || !ok) return;
      if (where[v] >= 0) put(RT_F_REG, (uint8_t)where[v], 0, 0.f, v);
      else if (values[v].op == RT_F_REG) put(RT_F_REG, RT_FUSED_IMM, 0, values[v].imm, v);
      else if (values[v].op == RT_F_LOAD) put(RT_F_LOAD, (uint8_t)values[v].a, 0, 0.f, v);
      else ok = false;
    }
    void to_register(int v) {
      if (where[v] >= 0 || !ok) return;
      to_acc(v);
      keep_acc();
      if (where[v] < 0) ok = false;
    }
  };

  bool emit(rt_fused_program* p, int preload) {
    Emitter e{p, values_, std::vector<int>(values_.size(), -1), std::vector<int>(values_.size(), 0)};
    p->n_code = 0;
    p->n_preload = preload;
    std::vector<char> live(values_.size(), 0);
    for (auto& o : outputs_) live[o.first] = 1;
    for (int v = (int)values_.size() - 1; v >= 0; --v) {
      if (!live[v]) continue;
      const Value& x = values_[v];
      if (x.op == RT_F_LOAD || x.op == RT_F_REG) continue;
      live[x.a] = 1;
      e.left[x.a]++;
      if (x.b >= 0) {
        live[x.b] = 1;
        e.left[x.b]++;
      }
    }
    for (size_t v = 0; v < values_.size(); ++v)
      if (live[v] && values_[v].op == RT_F_LOAD && values_[v].a < preload) {
        e.where[v] = values_[v].a;
        e.free_regs &= ~(1u << values_[v].a);
      }
    auto store = [&](int v) {
      for (size_t k = 0; k < outputs_.size(); ++k)
        if (outputs_[k].first == v) e.put(RT_F_OUT, (uint8_t)k, 0, 0.f, v);
    };
    for (int v = 0; v < (int)values_.size() && e.ok; ++v) {
      const Value& x = values_[v];
      if (!live[v] || x.op == RT_F_LOAD || x.op == RT_F_REG) continue;
      uint8_t src = RT_FUSED_IMM, swap = x.swap ? 1 : 0;
      if (x.op == RT_F_SELECT) {
        if (x.b >= 0) e.to_register(x.b);
        e.to_acc(x.a);
        if (!e.ok) return false;
        if (x.b >= 0) src = (uint8_t)e.where[x.b];
        swap = (uint8_t)x.region;
      } else if (x.b < 0) {
        e.to_acc(x.a);
      } else if (x.a == x.b) {
        e.to_register(x.a);
        e.to_acc(x.a);
        if (!e.ok) return false;
        src = (uint8_t)e.where[x.a];
      } else {
        if (e.acc == x.b && e.where[x.a] >= 0) {
          swap ^= 1;
        } else if (!(e.acc == x.a && e.where[x.b] >= 0)) {
          if (e.where[x.a] >= 0 && e.where[x.b] < 0) {
            e.to_acc(x.b);
            swap ^= 1;
          } else {
            e.to_register(x.b);
            e.to_acc(x.a);
          }
        }
        if (!e.ok) return false;
        src = (uint8_t)e.where[e.acc == x.a ? x.b : x.a];
      }
      if (!e.ok) return false;
      --e.left[x.a];
      if (x.b >= 0) --e.left[x.b];
      e.put(x.op, src, swap, x.imm, v);  // may give the old accumulator a register: `src` is still taken here
      e.release(x.a);
      if (x.b >= 0) e.release(x.b);
      store(v);
    }
    for (size_t v = 0; v < values_.size() && e.ok; ++v)
      if (live[v] && (values_[v].op == RT_F_LOAD || values_[v].op == RT_F_REG)) {
        bool out = false;
        for (auto& o : outputs_) out = out || o.first == (int)v;
        if (!out) continue;
        e.to_acc((int)v);
        store((int)v);
      }
    p->n_outputs = (int)outputs_.size();
    return e.ok;
  }
};

inline void check(rt_ctx* ctx, rt_status st) {
  if (st != RT_OK) throw Error((ErrorKind)st, rt_last_error(ctx));
}
// A new block for a result; given back unless it becomes a buffer's.
struct Block {
  rt_ctx* ctx;
  float* ptr = nullptr;
  Block(rt_ctx* c, size_t numel) : ctx(c) {
    void* p = nullptr;
    check(ctx, rt_malloc(ctx, sizeof(float) * std::max<size_t>(numel, 1), &p));
    ptr = (float*)p;
  }
  Block(Block&& o) noexcept : ctx(o.ctx), ptr(std::exchange(o.ptr, nullptr)) {}
  Block& operator=(Block&&) = delete;
  ~Block() {
    if (ptr) rt_free(ctx, ptr);
  }
  float* release() { return std::exchange(ptr, nullptr); }
  void to(DeviceBuffer* b) {
    b->ptr = release();
    b->drop_node();
  }
};
inline int unary_entry(uint8_t op) {  // the stand-alone kernel of an op, or -1
  switch (op) {
    case RT_F_RELU: return RT_RELU;
    case RT_F_EXP: return RT_EXP;
    case RT_F_LN: return RT_LN;
    case RT_F_SIN: return RT_SIN;
    case RT_F_COS: return RT_COS;
    case RT_F_TAN: return RT_TAN;
    case RT_F_TANH: return RT_TANH;
    case RT_F_SIGMOID: return RT_SIGMOID;
    case RT_F_SOFTPLUS: return RT_SOFTPLUS;
    case RT_F_SQRT: return RT_SQRT;
    case RT_F_ABS: return RT_ABS;
    case RT_F_SQUARE: return RT_SQUARE;
    case RT_F_ELU: return RT_ELU;
    default: return -1;
  }
}
inline int binary_entry(uint8_t op) {
  static_assert(RT_F_LE - RT_F_ADD == RT_LESS_EQUAL - RT_ADD && RT_F_EQ - RT_F_ADD == RT_EQUAL - RT_ADD && RT_F_MAX - RT_F_ADD == RT_MAXIMUM - RT_ADD,
                "binary ops are listed in the same order");
  return op >= RT_F_ADD && op <= RT_F_LE ? op - RT_F_ADD + RT_ADD : -1;
}
inline std::vector<int64_t> dims64(const Shape& s) { return std::vector<int64_t>(s.begin(), s.end()); }

// One op by its stand-alone kernel, its inputs in memory.  False: the op has none.
inline bool evaluate_alone(DeviceBuffer* b) {
  const Node& n = *b->node;
  rt_ctx* c = b->ctx;
  const int u = n.kind == Kind::Unary ? unary_entry(n.op) : -1, bi = n.kind == Kind::Binary ? binary_entry(n.op) : -1;
  if ((n.kind == Kind::Unary && u < 0) || (n.kind == Kind::Binary && bi < 0) || n.kind == Kind::BinaryImm) return false;
  Block block(c, b->numel);
  float* out = block.ptr;
  auto nd = dims64(n.shape);
  rt_status st = RT_OK;
  auto place = [&](const Input& in, const std::vector<int64_t>& starts) {
    auto id = dims64(in.shape);
    if (st == RT_OK && shape_numel(in.shape) > 0)
      st = rt_slice_assign(c, out, nd.data(), (int)nd.size(), starts.data(), in.buf->data(), id.data());
  };
  switch (n.kind) {
    case Kind::Const: st = rt_fill(c, out, n.imm, (int64_t)b->numel); break;
    case Kind::Unary: st = rt_unary(c, u, n.in[0].buf->data(), out, (int64_t)b->numel, n.imm, 0.f); break;
    case Kind::Binary: {
      auto as = dims64(n.in[0].shape), bs = dims64(n.in[1].shape);
      st = rt_binary(c, bi, n.in[0].buf->data(), as.data(), (int)as.size(), n.in[1].buf->data(), bs.data(), (int)bs.size(), out);
      break;
    }
    case Kind::Broadcast: {
      auto xs = dims64(n.in[0].shape);
      st = rt_broadcast_to(c, n.in[0].buf->data(), xs.data(), (int)xs.size(), nd.data(), (int)nd.size(), out);
      break;
    }
    case Kind::Slice: {
      auto xs = dims64(n.in[0].shape), s0 = dims64(n.starts);
      st = rt_slice(c, n.in[0].buf->data(), xs.data(), (int)xs.size(), s0.data(), nd.data(), out);
      break;
    }
    case Kind::Pad:
      st = rt_fill(c, out, 0.f, (int64_t)b->numel);
      place(n.in[0], dims64(n.starts));
      break;
    case Kind::Concat: {
      std::vector<int64_t> s0(n.shape.size(), 0);
      for (auto& piece : n.in) {
        place(piece, s0);
        s0[n.starts[0]] += (int64_t)piece.shape[n.starts[0]];
      }
      break;
    }
    default: break;
  }
  check(c, st);
  block.to(b);
  return true;
}

// ---- combinations that one kernel computes ---------------------------------------------------------------------------------
inline Node* pending(const Input& i) { return i.buf->node.get(); }
inline Node* tagged(const Input& i, Tag t) { return pending(i) && i.buf->node->tag == t ? i.buf->node.get() : nullptr; }
inline bool is_op(const Node* n, Kind k, uint8_t op) { return n && n->kind == k && n->op == op; }

// n = other * constant: the other factor, and the constant in `c`
inline const Input* times_constant(const Node* n, float* c) {
  if (is_op(n, Kind::BinaryImm, RT_F_MUL)) {
    *c = n->imm;
    return &n->in[0];
  }
  if (is_op(n, Kind::Binary, RT_F_MUL))
    for (int i = 0; i < 2; ++i)
      if (pending(n->in[i]) && n->in[i].buf->node->kind == Kind::Const && n->in[1 - i].shape == n->shape) {
        *c = n->in[i].buf->node->imm;
        return &n->in[1 - i];
      }
  return nullptr;
}

// Several results computed as one matrix, in a capture: each is rows of the common block, and the only one to be so.
inline std::shared_ptr<DeviceBuffer> common_block(rt_ctx* ctx, size_t numel) {
  Block block(ctx, numel);
  auto b = std::make_shared<DeviceBuffer>(ctx, block.ptr, numel);
  block.release();
  return b;
}
inline void place(DeviceBuffer* b, const std::shared_ptr<DeviceBuffer>& block, size_t offset) {
  b->ptr = block->ptr + offset;
  b->owner = block;
  b->apart = true;
  b->drop_node();
}

// ---- LSTM cells written op by op ---------------------------------------------------------------------------------------------
//   z = concat(x_t, h_prev) w + b;  i, f, g, o = the column blocks of z, activated;  c = f c_prev + i g;  h = o tanh(c)
// A capture records a whole step, so the product of such a cell need not be computed when it is asked for: matmul leaves it pending as long
// as every cell below it is of this form and the states before the first are zeros, and whoever asks for a state then gets the sequence from
// rt_lstm_sequence, every timestep at once.
struct Cell {
  std::shared_ptr<DeviceBuffer> h, c, i, f, g, o, tc, product;
  Input z, xh, h_prev, c_prev, w, bias;
};
inline const Input* unary_of(const Input& x, uint8_t op) {
  return pending(x) && pending(x)->kind == Kind::Unary && pending(x)->op == op && pending(x)->shape == x.shape ? &pending(x)->in[0] : nullptr;
}
// x = act(columns block * H .. of z)
inline const Input* gate_of(const Input& x, uint8_t act, size_t block) {
  const Input* s = unary_of(x, act);
  const Node* n = s ? pending(*s) : nullptr;
  if (!n || n->kind != Kind::Slice || n->shape != x.shape || s->shape != x.shape || x.shape.size() != 2) return nullptr;
  if (n->starts != Shape{0, block * x.shape[1]} || n->in[0].shape != Shape{x.shape[0], 4 * x.shape[1]}) return nullptr;
  return &n->in[0];
}
inline bool match_cell(DeviceBuffer* b, Cell* q) {
  const Node* n = b->node.get();
  if (!is_op(n, Kind::Binary, RT_F_MUL) || n->shape.size() != 2) return false;
  const Shape& s = n->shape;
  for (int k = 0; k < 2; ++k) {
    const Input &o = n->in[k], &tc = n->in[1 - k];
    const Input *zo = o.shape == s ? gate_of(o, RT_F_SIGMOID, 3) : nullptr, *c = zo && tc.shape == s ? unary_of(tc, RT_F_TANH) : nullptr;
    if (!c || c->shape != s || !is_op(pending(*c), Kind::Binary, RT_F_ADD)) continue;
    for (int a = 0; a < 2; ++a) {
      const Input &fc = pending(*c)->in[a], &ig = pending(*c)->in[1 - a];
      if (fc.shape != s || ig.shape != s || !is_op(pending(fc), Kind::Binary, RT_F_MUL) || !is_op(pending(ig), Kind::Binary, RT_F_MUL)) continue;
      for (int e = 0; e < 4; ++e) {
        const Input &f = pending(fc)->in[e & 1], &before = pending(fc)->in[1 - (e & 1)], &i = pending(ig)->in[e >> 1], &g = pending(ig)->in[1 - (e >> 1)];
        if (f.shape != s || before.shape != s || i.shape != s || g.shape != s) continue;
        const Input *zf = gate_of(f, RT_F_SIGMOID, 1), *zi = gate_of(i, RT_F_SIGMOID, 0), *zg = gate_of(g, RT_F_TANH, 2);
        if (!zf || !zi || !zg || zf->buf != zo->buf || zi->buf != zo->buf || zg->buf != zo->buf) continue;
        const Node* z = pending(*zo);
        if (!is_op(z, Kind::Binary, RT_F_ADD) || z->shape != zo->shape) return false;
        for (int p = 0; p < 2; ++p) {
          const Node* m = tagged(z->in[p], Tag::Matmul);
          Input bias = z->in[1 - p];
          if (!m || m->geo.empty() || m->shape != z->shape || z->in[p].shape != m->shape) continue;
          if (pending(bias) && pending(bias)->kind == Kind::Broadcast && pending(bias)->shape == bias.shape) bias = Input(pending(bias)->in[0]);
          if (bias.shape.empty() || bias.shape.back() != m->shape[1] || shape_numel(bias.shape) != m->shape[1] || bias.buf->node) continue;
          const Node* cat = pending(m->in[0]);
          if (!cat || cat->kind != Kind::Concat || cat->in.size() != 2) return false;
          *q = Cell{b->shared_from_this(), c->buf, i.buf, f.buf, g.buf, o.buf, tc.buf, z->in[p].buf, *zo, m->in[0], cat->in[1], before, m->in[1], bias};
          return true;
        }
      }
    }
  }
  return false;
}
inline bool is_zero(const Input& x) { return pending(x) && pending(x)->kind == Kind::Const && pending(x)->imm == 0.f; }
// The rows of a matrix in memory that a cell's input is.
inline bool rows_of(const Input& x, Input* base, int64_t* first) {
  const Node* n = pending(x);
  if (!n || n->kind != Kind::Slice || n->shape != x.shape || n->in[0].shape.size() != 2 || n->in[0].buf->node) return false;
  if (n->starts[1] != 0 || n->in[0].shape[1] != x.shape[1]) return false;
  *base = n->in[0];
  *first = (int64_t)n->starts[0];
  return true;
}
// The timestep, counted from 1, whose product a * w would be in a sequence whose cells are all pending; 0: none.
inline int64_t timestep_of(const Input& a, const Input& w) {
  const Node* cat = pending(a);
  if (!capturing() || !cat || cat->kind != Kind::Concat || cat->in.size() != 2 || cat->starts[0] != 1 || a.shape != cat->shape || a.shape.size() != 2) return 0;
  if (w.shape.size() != 2 || w.shape[0] != a.shape[1] || w.buf->node) return 0;
  const Input &x = cat->in[0], &h = cat->in[1];
  Input base;
  int64_t first;
  if (h.shape.size() != 2 || w.shape[1] != 4 * h.shape[1] || !rows_of(x, &base, &first)) return 0;
  if (is_zero(h)) return 1;
  Cell q;
  if (!h.buf->node || !match_cell(h.buf.get(), &q) || q.w.buf != w.buf) return 0;
  Input before;
  int64_t at;
  if (!rows_of(pending(q.xh)->in[0], &before, &at) || before.buf != base.buf || at + (int64_t)x.shape[0] != first || q.h_prev.shape != h.shape) return 0;
  const int64_t t = pending(Input{q.product, {}})->geo[0];
  if (t == 1 ? !is_zero(q.c_prev) : !q.c_prev.buf->node) return 0;
  if (t > 1) {  // the cell state must be that of the cell whose h this one takes
    Cell r;
    if (!match_cell(q.h_prev.buf.get(), &r) || r.c != q.c_prev.buf || r.bias.buf != q.bias.buf) return 0;
  }
  q.c->node->depth = 1;  // like the products: the sequence is evaluated from its first timestep on, however long it is
  return t + 1;
}
// The states of the cells, the first first, each by itself: what becomes of a recurrence that is not a sequence (any more, since somebody has
// asked for something within it).  Whether b is among what has been evaluated.
inline bool evaluate_in_order(const std::vector<Cell>& cells, DeviceBuffer* b) {
  for (const Cell& q : cells)
    if (q.h.get() != b) lazy_evaluate(q.h.get());
  return !b->node;
}
// The states of such cells that the expression b reads, the last first, which brings the others along.  Walking through them would be as deep as the
// recurrence is long: a cell state reads the one before.
inline void settle_states(DeviceBuffer* b) {
  if (!capturing() || DeviceBuffer::waiting() == 0) return;
  std::vector<std::pair<int64_t, std::shared_ptr<DeviceBuffer>>> states;
  std::unordered_set<const DeviceBuffer*> seen;
  std::vector<const Node*> open{b->node.get()};
  while (!open.empty()) {
    const Node* n = open.back();
    open.pop_back();
    for (const Input& i : n->in) {
      const Node* m = pending(i);
      Cell q;
      if (!m || !seen.insert(i.buf.get()).second) continue;
      if (match_cell(i.buf.get(), &q)) states.push_back({q.product->node->geo[0], i.buf});
      else if (m->kind != Kind::Opaque || m->waits()) open.push_back(m);
    }
  }
  std::stable_sort(states.begin(), states.end(), [](auto& x, auto& y) { return x.first > y.first; });
  for (auto& s : states) lazy_evaluate(s.second.get());
}
inline bool rewrite_recurrence(DeviceBuffer* b) {
  if (!capturing() || !is_op(b->node.get(), Kind::Binary, RT_F_MUL)) return false;
  std::vector<Cell> cells;  // the last first
  bool whole = false;
  for (DeviceBuffer* at = b; !whole;) {
    Cell q;
    if (!at->node || !match_cell(at, &q)) break;
    if (!cells.empty() && (cells.back().c_prev.buf != q.c || cells.back().w.buf != q.w.buf || cells.back().bias.buf != q.bias.buf)) break;
    at = q.h_prev.buf.get();
    cells.push_back(std::move(q));
    whole = is_zero(cells.back().h_prev) && is_zero(cells.back().c_prev);
  }
  std::reverse(cells.begin(), cells.end());
  if (!whole) return !cells.empty() && evaluate_in_order(cells, b);
  auto seq = std::make_shared<Recurrence>();
  const Input& w = cells[0].w;
  Input x;
  int64_t first = 0;
  for (size_t t = 0; t < cells.size(); ++t) {  // as timestep_of has found them, unless a timestep's inputs have been asked for
    Input base;
    int64_t at = 0;
    const bool rows = rows_of(pending(cells[t].xh)->in[0], &base, &at);
    if (rows && t == 0) {
      x = base;
      first = at;
    }
    if (!rows || base.buf != x.buf || at != first + (int64_t)(t * cells[0].h_prev.shape[0])) {
      if (t == 0) return evaluate_in_order(cells, b);
      lazy_evaluate(cells[t - 1].h.get());  // those before it are a sequence
      return evaluate_in_order(cells, b);
    }
  }
  seq->steps = (int64_t)cells.size();
  seq->batch = (int64_t)cells[0].h_prev.shape[0];
  seq->hidden = (int64_t)cells[0].h_prev.shape[1];
  seq->features = (int64_t)x.shape[1];
  const int64_t rows = seq->steps * seq->batch, H = seq->hidden, n = seq->batch * H;
  seq->x = x.buf;
  seq->w = w.buf;
  seq->x_rows = x.buf->ptr + first * seq->features;
  seq->saved = common_block(b->ctx, (size_t)(6 * rows * H));
  seq->h = common_block(b->ctx, (size_t)(rows * H));
  Block pre(b->ctx, (size_t)(rows * 4 * H));
  check(b->ctx, rt_gemm_bias_act(b->ctx, rows, 4 * H, seq->features, seq->x_rows, seq->features, w.buf->ptr, 4 * H, cells[0].bias.buf->ptr, RT_ACT_NONE,
                                 pre.ptr, 4 * H));
  check(b->ctx, rt_lstm_sequence(b->ctx, pre.ptr, w.buf->ptr + seq->features * 4 * H, 4 * H, nullptr, nullptr, seq->steps, seq->batch, H, seq->saved->ptr,
                                 seq->h->ptr));
  for (size_t t = 0; t < cells.size(); ++t) {
    Cell& q = cells[t];
    DeviceBuffer* planes[6] = {q.i.get(), q.f.get(), q.g.get(), q.o.get(), q.c.get(), q.tc.get()};
    for (int k = 0; k < 6; ++k) place(planes[k], seq->saved, (size_t)(k * rows * H + (int64_t)t * n));
    place(q.h.get(), seq->h, (size_t)((int64_t)t * n));
    q.h->sequence = seq;
    q.h->timestep = (int64_t)t;
  }
  return true;
}

// act(a * b + bias), act one of none, relu, tanh, sigmoid: bias and activation in the product's epilogue.  Products of one shape
// with the same b (a layer applied to every timestep) whose left operands are all there are computed in one launch.
struct Linear {
  DeviceBuffer* out;
  Input a, b, bias;  // bias.buf null: none
  int act;
  bool waits;  // of a recurrence's timestep: those after it need its result
};
inline bool match_linear(DeviceBuffer* out, Linear* l) {
  const Node* n = out->node.get();
  l->out = out;
  l->act = RT_ACT_NONE;
  if (n->tag == Tag::Matmul) {
    l->a = n->in[0];
    l->b = n->in[1];
    l->bias = Input{};
    l->waits = n->waits();
    return true;
  }
  const Node* sum = n;
  if (n->kind == Kind::Unary && (n->op == RT_F_RELU || n->op == RT_F_TANH || n->op == RT_F_SIGMOID)) {
    l->act = n->op == RT_F_RELU ? RT_ACT_RELU : (n->op == RT_F_TANH ? RT_ACT_TANH : RT_ACT_SIGMOID);
    sum = pending(n->in[0]);
    if (!sum || n->in[0].shape != sum->shape) return false;
  }
  if (!is_op(sum, Kind::Binary, RT_F_ADD)) return false;
  for (int i = 0; i < 2; ++i) {
    const Node* m = tagged(sum->in[i], Tag::Matmul);
    if (!m || sum->in[i].buf->readers.size() != 1 || m->shape != sum->shape || sum->in[i].shape != m->shape) continue;
    Input bias = sum->in[1 - i];
    if (pending(bias) && pending(bias)->kind == Kind::Broadcast && pending(bias)->shape == bias.shape) bias = Input(pending(bias)->in[0]);
    if (bias.shape.empty() || bias.shape.back() != m->shape[1] || shape_numel(bias.shape) != m->shape[1]) continue;
    l->a = m->in[0];
    l->b = m->in[1];
    l->bias = bias;
    l->waits = m->waits();
    return true;
  }
  return false;
}
// The expression around a product that is computed with it: the product itself, its sum with a bias, the activation of that.
inline DeviceBuffer* epilogue_of(DeviceBuffer* product, int act, bool bias) {
  if (!bias) return product;
  if (product->readers.size() != 1) return nullptr;
  DeviceBuffer* sum = product->readers[0];
  if (act == RT_ACT_NONE) return sum;
  return sum->readers.size() == 1 ? sum->readers[0] : nullptr;
}
inline bool rewrite_linear(DeviceBuffer* b) {
  Linear first{};
  if (!match_linear(b, &first)) return false;
  std::vector<Linear> all{first};
  const float *pa = first.a.buf->data(), *pb = first.b.buf->data(), *bias = first.bias.buf ? first.bias.buf->data() : nullptr;
  std::vector<DeviceBuffer*> others;
  if (!first.waits) others = first.b.buf->readers;
  for (DeviceBuffer* r : others) {
    if (all.size() == 256) break;
    if (!r->node || r->node->tag != Tag::Matmul || r->node->in[1].buf != first.b.buf || r->node->in[0].buf->node) continue;
    DeviceBuffer* e = epilogue_of(r, first.act, bias != nullptr);
    Linear l;
    // a product of a matrix with itself reads it twice
    if (!e || std::any_of(all.begin(), all.end(), [e](const Linear& x) { return x.out == e; }) || !match_linear(e, &l)) continue;
    if (l.act != first.act || l.b.buf != first.b.buf || l.a.shape != first.a.shape || l.b.shape != first.b.shape || l.bias.buf != first.bias.buf) continue;
    all.push_back(l);
  }
  const int64_t rows = (int64_t)first.a.shape[0], k = (int64_t)first.a.shape[1], cols = (int64_t)first.b.shape[1];
  if (capturing() && all.size() > 1) {  // left operands that follow one another in memory (the states of a sequence) are one
    std::sort(all.begin(), all.end(), [](const Linear& x, const Linear& y) { return x.a.buf->ptr < y.a.buf->ptr; });
    bool together = true;
    for (size_t i = 1; i < all.size(); ++i) together = together && all[i].a.buf->ptr == all[i - 1].a.buf->ptr + rows * k;
    if (together && (int64_t)all.size() * rows * std::max(cols, k) < (int64_t(1) << 31)) {
      const auto block = common_block(b->ctx, all.size() * (size_t)(rows * cols));
      std::vector<std::shared_ptr<DeviceBuffer>> outs;
      for (auto& l : all) outs.push_back(l.out->shared_from_this());
      check(b->ctx, rt_gemm_bias_act(b->ctx, (int64_t)all.size() * rows, cols, k, all[0].a.buf->ptr, k, pb, cols, bias, first.act, block->ptr, cols));
      for (size_t i = 0; i < outs.size(); ++i) place(outs[i].get(), block, i * (size_t)(rows * cols));
      return true;
    }
  }
  std::vector<std::shared_ptr<DeviceBuffer>> keep;
  for (auto& l : all) keep.push_back(l.out->shared_from_this());
  std::vector<const float*> as;
  std::vector<float*> outs;
  std::vector<Block> blocks;
  for (auto& l : all) {
    as.push_back(l.a.buf->data());
    blocks.emplace_back(b->ctx, l.out->numel);
    outs.push_back(blocks.back().ptr);
  }
  rt_status st;
  if (all.size() > 1) st = rt_gemm_bias_act_list(b->ctx, (int)all.size(), as.data(), outs.data(), rows, cols, k, pb, bias, first.act);
  else st = rt_gemm_bias_act(b->ctx, rows, cols, k, pa, k, pb, cols, bias, first.act, outs[0], cols);
  check(b->ctx, st);
  for (size_t i = 0; i < all.size(); ++i) blocks[i].to(all[i].out);
  return true;
}

// constant * [mean or sum over rows] of [constant *] sum over classes of log_softmax(x) * y: a classification loss.
struct Loss {
  const Input *logits, *targets;
  int64_t rows, classes;
  float scale, divisor;
  bool same_kind(const Loss& o) const { return rows == o.rows && classes == o.classes && scale == o.scale && divisor == o.divisor; }
};
inline bool match_loss(DeviceBuffer* b, Loss* l) {
  float scale = 1.f, c = 1.f;
  const Node* n = b->node.get();
  if (const Input* f = times_constant(n, &c)) {
    if (!tagged(*f, Tag::Reduce) || f->buf->readers.size() != 1) return false;
    scale *= c;
    n = pending(*f);
  }
  if (n->tag != Tag::Reduce || n->geo[1] >= 0) return false;  // over all elements
  const bool mean = n->geo[0] == RT_RED_MEAN;
  const Input* rows_of = &n->in[0];
  if (pending(*rows_of))
    if (const Input* f = times_constant(pending(*rows_of), &c)) {
      scale *= c;
      rows_of = f;
    }
  const Node* per_row = tagged(*rows_of, Tag::Reduce);
  if (!per_row || per_row->geo[0] != RT_RED_SUM || per_row->geo[1] != 1 || per_row->in[0].shape.size() != 2) return false;
  const Node* prod = pending(per_row->in[0]);
  if (!is_op(prod, Kind::Binary, RT_F_MUL) || prod->shape != per_row->in[0].shape) return false;
  for (int i = 0; i < 2; ++i) {
    const Node* ls = tagged(prod->in[i], Tag::LogSoftmax);
    if (!ls || ls->geo[0] != 1 || ls->shape != prod->shape || prod->in[1 - i].shape != prod->shape) continue;
    const int64_t rows = (int64_t)ls->shape[0], classes = (int64_t)ls->shape[1];
    if (classes > 4096 || rows > (1 << 22)) return false;
    *l = Loss{&ls->in[0], &prod->in[1 - i], rows, classes, scale, mean ? (float)rows : 1.f};
    return true;
  }
  return false;
}
inline bool rewrite_loss(DeviceBuffer* b) {
  Loss l;
  if (!match_loss(b, &l)) return false;
  const Input logits = *l.logits, targets = *l.targets;  // kept through the evaluations
  const float *x = logits.buf->data(), *y = targets.buf->data();
  Block out(b->ctx, b->numel);
  check(b->ctx, rt_softmax_nll_scaled(b->ctx, x, y, l.rows, l.classes, l.scale, l.divisor, out.ptr));
  out.to(b);
  return true;
}

// The unevaluated classification loss that log_softmax of `logits` leads to, if nothing else reads any step of it.
inline DeviceBuffer* loss_over(DeviceBuffer* logits, DeviceBuffer* targets, Loss* l) {
  for (DeviceBuffer* r : logits->readers) {
    if (!r->node || r->node->tag != Tag::LogSoftmax) continue;
    DeviceBuffer* root = nullptr;
    for (DeviceBuffer* b = r; b->readers.size() == 1;) {
      b = b->readers[0];
      if (b->node && match_loss(b, l)) root = b;
    }
    if (root && root->readers.empty() && match_loss(root, l) && l->logits->buf.get() == logits && l->targets->buf.get() == targets) return root;
  }
  return nullptr;
}

// Gradients of classification losses of one kind (Tag::NllGrad), in a capture: those whose rows follow one another in one launch.
inline bool rewrite_nll_grad(DeviceBuffer* b) {
  if (b->node->tag != Tag::NllGrad || !capturing()) return false;
  const int64_t rows = b->node->geo[0], classes = b->node->geo[1], n = rows * classes;
  std::vector<std::shared_ptr<DeviceBuffer>> all;
  const std::vector<int64_t> geo = b->node->geo;
  for (DeviceBuffer* p = DeviceBuffer::head(); p; p = p->next)
    if (p->node->tag == Tag::NllGrad && p->node->geo == geo && !p->node->in[0].buf->node) all.push_back(p->shared_from_this());
  for (auto& p : all) p->node->in[1].buf->data();
  std::sort(all.begin(), all.end(), [](auto& x, auto& y) { return x->node->in[0].buf->ptr < y->node->in[0].buf->ptr; });
  size_t lo = 0, at = 0;
  while (at < all.size() && all[at].get() != b) ++at;
  if (at == all.size()) return false;
  auto follows = [&](size_t i) {
    return all[i]->node->in[0].buf->ptr == all[i - 1]->node->in[0].buf->ptr + n && all[i]->node->in[1].buf->ptr == all[i - 1]->node->in[1].buf->ptr + n;
  };
  size_t hi = lo = at;
  while (lo > 0 && follows(lo)) --lo;
  while (hi + 1 < all.size() && follows(hi + 1)) ++hi;
  const size_t count = hi - lo + 1;
  if (count < 2 || (int64_t)count * rows > (1 << 22)) return false;
  float c;
  std::memcpy(&c, &geo[2], sizeof(float));
  const auto block = common_block(b->ctx, count * (size_t)n);
  check(b->ctx, rt_softmax_nll_scaled_backward(b->ctx, all[lo]->node->in[0].buf->ptr, all[lo]->node->in[1].buf->ptr, (int64_t)count * rows, classes, c,
                                               block->ptr));
  for (size_t i = 0; i < count; ++i) place(all[lo + i].get(), block, i * (size_t)n);
  return true;
}

// max_pool2d's gradient masked by the relu in front of the pooling: one pass.
inline bool rewrite_pool(DeviceBuffer* b) {
  const Node* n = b->node.get();
  if (!is_op(n, Kind::Binary, RT_F_MUL)) return false;
  for (int i = 0; i < 2; ++i) {
    const Node* pg = tagged(n->in[i], Tag::PoolGrad);
    const Node* st = pending(n->in[1 - i]);
    if (!pg || !is_op(st, Kind::Unary, RT_F_STEP) || pg->shape != n->shape || st->shape != n->shape || n->in[i].shape != n->shape) continue;
    if (n->in[i].buf->readers.size() != 1 || pg->in.size() != 3) continue;  // in: g, idx, pooled relu output
    if (pg->geo[10] != (int64_t)st->in[0].buf->id) continue;                // the relu's output is what was pooled
    const auto& q = pg->geo;
    const float *y = pg->in[2].buf->data(), *g = pg->in[0].buf->data(), *idx = pg->in[1].buf->data();
    Block out(b->ctx, b->numel);
    check(b->ctx, rt_relu_max_pool2x2_backward_from_output(b->ctx, y, g, idx, q[0], q[1], q[2], q[3], out.ptr));
    out.to(b);
    return true;
  }
  return false;
}
// A sum of scalars, among them several classification losses of one shape: the losses of a sequence, computed in one launch.
inline bool rewrite_loss_sum(DeviceBuffer* b) {
  if (b->numel != 1 || !is_op(b->node.get(), Kind::Binary, RT_F_ADD)) return false;
  std::vector<Input> leaves;  // keeps the operands alive
  std::vector<const Node*> open{b->node.get()};
  for (size_t i = 0; i < open.size(); ++i)
    for (auto& in : open[i]->in) {
      const Node* n = pending(in);
      // a partial sum that nobody else uses belongs to this sum
      if (is_op(n, Kind::Binary, RT_F_ADD) && in.buf->numel == 1 && in.buf->readers.size() == 1) open.push_back(n);
      else leaves.push_back(in);
    }
  std::vector<Loss> losses;
  std::vector<Input> rest;
  for (auto& l : leaves) {
    Loss x;
    if (pending(l) && match_loss(l.buf.get(), &x) && (losses.empty() || x.same_kind(losses[0])) && losses.size() < 256) losses.push_back(x);
    else rest.push_back(l);
  }
  if (losses.size() < 2 || rest.size() > 16) return false;
  std::vector<const float*> xs, ys, more;
  std::vector<Input> keep;
  for (auto& l : losses) {
    keep.push_back(*l.logits);
    keep.push_back(*l.targets);
  }
  const Loss first = losses[0];
  for (size_t i = 0; i < keep.size(); i += 2) {
    xs.push_back(keep[i].buf->data());
    ys.push_back(keep[i + 1].buf->data());
  }
  for (auto& r : rest) more.push_back(r.buf->data());
  Block out(b->ctx, 1);
  check(b->ctx, rt_softmax_nll_list(b->ctx, (int)xs.size(), xs.data(), ys.data(), first.rows, first.classes, first.scale, first.divisor,
                                    (int)more.size(), more.data(), out.ptr));
  out.to(b);
  return true;
}
// Rows of a tensor that is in memory, inside a capture: no copy, the result points into it.
inline bool rewrite_rows(DeviceBuffer* b) {
  const Node* n = b->node.get();
  if (n->kind != Kind::Slice || !capturing()) return false;
  const Input& base = n->in[0];
  if (base.buf->node && base.buf->node->kind != Kind::Opaque) return false;
  size_t d = 0;
  while (d < n->shape.size() && n->shape[d] == 1) ++d;  // leading extents of 1, then one free extent, then whole ones
  for (size_t j = d + 1; j < n->shape.size(); ++j)
    if (n->shape[j] != base.shape[j]) return false;
  int64_t off = 0;
  for (size_t j = 0; j < n->shape.size(); ++j) off = off * (int64_t)base.shape[j] + (int64_t)n->starts[j];
  std::shared_ptr<DeviceBuffer> root = base.buf;
  const float* p = root->data();
  while (root->shares_rows()) root = root->owner;
  b->ptr = const_cast<float*>(p) + off;
  b->owner = root;
  b->drop_node();
  return true;
}
inline bool rewrite(DeviceBuffer* b) {
  if (b->node->kind == Kind::Const) return false;
  return rewrite_rows(b) || rewrite_recurrence(b) || rewrite_linear(b) || rewrite_nll_grad(b) || rewrite_loss(b) || rewrite_loss_sum(b) || rewrite_pool(b);
}

// Whether column sums over an expression of b's shape are pending.
inline bool column_sum_waits(DeviceBuffer* b) {
  for (DeviceBuffer* p = DeviceBuffer::head(); p; p = p->next)
    if (p->node->tag == Tag::SumRows && p->node->geo[0] < 0 && p->node->in[0].shape == b->node->shape && pending(p->node->in[0]) &&
        pending(p->node->in[0])->kind != Kind::Opaque && p->node->in[0].buf.get() != b)
      return true;
  return false;
}
// A program with a reduction of one of its outputs: column sums of output c.sums(), or with `lse` the logsumexp of the rows.  False: it has not been
// launched (there is no kernel for such a one, or b has been evaluated while it was built), and no memory has been taken for it.
inline bool evaluate_reduced(DeviceBuffer* b, Compiler& c, float* lse) {
  rt_fused_program p;
  std::vector<DeviceBuffer*> outs;
  if (!c.build(b, &p, &outs) || (c.sums() < 0) != (lse != nullptr)) return false;
  const rt_status known = rt_fused_reduction_known(b->ctx, &p, c.sums());
  if (known == RT_ERR_UNIMPLEMENTED) return false;
  check(b->ctx, known);
  std::vector<Block> blocks;
  for (size_t k = 0; k < outs.size(); ++k) {
    blocks.emplace_back(b->ctx, outs[k]->numel);
    p.out[k] = blocks.back().ptr;
  }
  check(b->ctx, lse ? rt_fused_logsumexp(b->ctx, &p, lse) : rt_fused_column_sums(b->ctx, &p, c.sums(), p.out[c.sums()]));
  std::vector<std::shared_ptr<DeviceBuffer>> keep;
  for (auto* o : outs) keep.push_back(o->shared_from_this());
  for (size_t k = 0; k < outs.size(); ++k) blocks[k].to(outs[k]);
  return true;
}
// Whether a program of the expression b can be one of those: building it to be told otherwise costs as much as building the one that is launched
// (3 us of a small model's training step on the host).
inline bool may_be_reduced(DeviceBuffer* b, int which) {
  uint64_t ops = 0;
  std::vector<const DeviceBuffer*> open{b}, seen{b};
  while (!open.empty()) {
    const Node& n = *open.back()->node;
    open.pop_back();
    if (n.kind == Kind::Unary || n.kind == Kind::BinaryImm || n.kind == Kind::Binary) ops |= uint64_t(1) << n.op;
    for (const Input& i : n.in) {
      const DeviceBuffer* x = i.buf.get();
      if (!x->node || x->node->kind == Kind::Opaque || std::find(seen.begin(), seen.end(), x) != seen.end()) continue;
      if (seen.size() == RT_FUSED_MAX_CODE) return false;  // no program is as long
      seen.push_back(x);
      open.push_back(x);
    }
  }
  return rt_fused_reduction_possible(b->ctx, which, ops) == RT_OK;
}
// An expression over [rows, columns] together with the pending column sums of a term that it shares values with.  True: b is evaluated.
inline bool evaluate_with_sums(DeviceBuffer* b) {
  if (Walk::depth() > 1 || b->node->shape.size() != 2 || b->numel == 0 || !column_sum_waits(b) || !may_be_reduced(b, 0)) return false;
  Compiler c;
  c.keep_rows(true);
  return evaluate_reduced(b, c, nullptr) || !b->node;
}
// The gradients of rows that the expression b reads, each by its own kernel: no compiled program without a reduction has one.  (Interpreted within
// the rest, tanh(x + b) of [4096, 4096] with its logsumexp and gradients 194 us, 164 this way; the same with the sine and exponential of the
// elementwise workload and x * x 672 and 560.)
inline void settle_row_gradients(DeviceBuffer* b) {
  if (DeviceBuffer::row_gradients() == 0) return;
  std::vector<std::shared_ptr<DeviceBuffer>> found;
  std::unordered_set<const DeviceBuffer*> seen;
  std::vector<const Node*> open{b->node.get()};
  while (!open.empty()) {
    const Node* n = open.back();
    open.pop_back();
    for (const Input& i : n->in) {
      const Node* m = pending(i);
      if (!m || m->kind == Kind::Opaque || !seen.insert(i.buf.get()).second) continue;
      if (m->tag == Tag::RowGrad) found.push_back(i.buf);
      else open.push_back(m);
    }
  }
  for (auto& f : found) lazy_evaluate(f.get());
}
// The rows of an expression and their logsumexp.  True only if `out` has been computed; b may have been evaluated without it.
inline bool evaluate_with_logsumexp(DeviceBuffer* b, float* out) {
  if (Walk::depth() > 0 || !b->node || b->node->kind == Kind::Opaque || b->node->kind == Kind::Const || b->node->shape.size() != 2 || b->numel == 0) return false;
  if (!may_be_reduced(b, -1)) return false;
  std::shared_ptr<DeviceBuffer> guard = b->shared_from_this();
  Compiler c;
  c.keep_rows(false);
  return evaluate_reduced(b, c, out);
}

}  // namespace lazy

inline void lazy_evaluate(DeviceBuffer* b) {
  using namespace lazy;
  if (!b->node) return;
  std::shared_ptr<DeviceBuffer> guard = b->shared_from_this();
  const Walk walk;
  if (rewrite(b)) return;
  if (b->node->kind == Kind::Opaque || b->node->tag == Tag::RowGrad) {
    b->node->run(*b->node, b);
    b->drop_node();
    return;
  }
  settle_states(b);
  if (!b->node) return;
  const bool lone = (b->node->kind == Kind::Unary || b->node->kind == Kind::Binary) &&
                    std::all_of(b->node->in.begin(), b->node->in.end(), [](const Input& i) { return !i.buf->node; });
  if ((lone || b->node->kind == Kind::Const) && evaluate_alone(b)) return;
  if (evaluate_with_sums(b)) return;
  settle_row_gradients(b);
  if (!b->node) return;
  for (int attempt = 0; attempt < 2; ++attempt) {
    rt_fused_program p;
    Compiler c;
    std::vector<DeviceBuffer*> outs;
    if (c.build(b, &p, &outs)) {
      std::vector<Block> blocks;
      for (size_t k = 0; k < outs.size(); ++k) {
        blocks.emplace_back(b->ctx, b->numel);
        p.out[k] = blocks.back().ptr;
      }
      check(b->ctx, rt_fused_elementwise(b->ctx, &p));
      std::vector<std::shared_ptr<DeviceBuffer>> keep;
      for (auto* o : outs) keep.push_back(o->shared_from_this());
      for (size_t k = 0; k < outs.size(); ++k) blocks[k].to(outs[k]);
      return;
    }
    // too long, or more dimensions than the kernel walks: evaluate what lies below first
    for (auto& i : b->node->in) i.buf->data();
  }
  if (!evaluate_alone(b)) throw Error::internal("an elementwise op could not be evaluated");
}

}  // namespace rt
