// PyTorch side of the launch path in C++: argument checks, output allocation, the stream lookup and the autograd chain of
// the convolution and of the spherical harmonics.  A small convolution takes a few microseconds on the GPU; the same
// chain in Python costs some two hundred per forward and backward.
//
// The C-ABI library stays the product: this module only calls its entry points (resolved at load time from the path
// Python passes, so that both use the same build) and has no kernels of its own.
//
// Autograd.  F(x, y, w, g) is linear in every operand; ConvForward is dF/dg, ConvBackward the other three first
// derivatives, ConvDouble the derivatives of ConvBackward, and everything beyond is made of ConvPartial, the derivative
// of F with respect to one operand, whose own derivatives are again ConvPartial.  Which gradients are worth computing is
// asked from the running graph task (needs_input_grad).
#include <dlfcn.h>

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <algorithm>
#include <array>
#include <memory>
#include <mutex>
#include <optional>
#include <utility>

#include "../../include/luna_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// ---- the library ------------------------------------------------------------------------------------------------------
struct Api {
  decltype(&luna_last_error) last_error = nullptr;
  decltype(&luna_uvu_plan_destroy) plan_destroy = nullptr;
  decltype(&luna_uvu_plan_query) plan_query = nullptr;
  decltype(&luna_uvu_conv_scratch_bytes) scratch_bytes = nullptr;
  decltype(&luna_uvu_conv_fwd) fwd = nullptr;
  decltype(&luna_uvu_conv_bwd) bwd = nullptr, bwd_add_gw = nullptr;
  decltype(&luna_uvu_conv_dbl_bwd) dbl_bwd = nullptr;
  decltype(&luna_graph_scratch_bytes) graph_scratch_bytes = nullptr;
  decltype(&luna_graph_build_all) graph_build_all = nullptr;
  decltype(&luna_sh_fwd) sh_fwd = nullptr;
  decltype(&luna_sh_bwd) sh_bwd = nullptr;
  decltype(&luna_sh_dbl_bwd) sh_dbl_bwd = nullptr;
} api;

template <typename F>
void resolve(void* library, const char* name, F& function) {
  function = reinterpret_cast<F>(dlsym(library, name));
  TORCH_CHECK(function != nullptr, "symbol ", name, " is missing from the library");
}

void load(const std::string& path) {
  void* library = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(library != nullptr, "cannot load ", path, ": ", dlerror());
  resolve(library, "luna_last_error", api.last_error);
  resolve(library, "luna_uvu_plan_destroy", api.plan_destroy);
  resolve(library, "luna_uvu_plan_query", api.plan_query);
  resolve(library, "luna_uvu_conv_scratch_bytes", api.scratch_bytes);
  resolve(library, "luna_uvu_conv_fwd", api.fwd);
  resolve(library, "luna_uvu_conv_bwd", api.bwd);
  resolve(library, "luna_uvu_conv_bwd_add_gw", api.bwd_add_gw);
  resolve(library, "luna_uvu_conv_dbl_bwd", api.dbl_bwd);
  resolve(library, "luna_graph_scratch_bytes", api.graph_scratch_bytes);
  resolve(library, "luna_graph_build_all", api.graph_build_all);
  resolve(library, "luna_sh_fwd", api.sh_fwd);
  resolve(library, "luna_sh_bwd", api.sh_bwd);
  resolve(library, "luna_sh_dbl_bwd", api.sh_dbl_bwd);
}

// A failed status as the exception Python raises for it.
void check(int status) {
  if (C10_LIKELY(status == LUNA_OK)) return;
  const char* text = api.last_error();
  switch (status) {
    case LUNA_ERR_INVALID_ARGUMENT:
    case LUNA_ERR_MISALIGNED:
      TORCH_CHECK_VALUE(false, text);
    case LUNA_ERR_UNSUPPORTED:
      TORCH_CHECK_NOT_IMPLEMENTED(false, text);
    default:
      TORCH_CHECK(false, text, " (status ", status, ")");
  }
}

// ---- handles kept by Python and by autograd nodes -----------------------------------------------------------------------
struct Op : torch::CustomClassHolder {
  luna_uvu_plan* plan;
  int64_t X, Y, O, W;
  at::ScalarType dtype;
  Op(int64_t handle, int64_t x, int64_t y, int64_t o, int64_t w, bool f64)
      : plan(reinterpret_cast<luna_uvu_plan*>(handle)), X(x), Y(y), O(o), W(w), dtype(f64 ? at::kDouble : at::kFloat) {}
  ~Op() override { api.plan_destroy(plan); }
};

struct Graph : torch::CustomClassHolder {
  std::array<Tensor, 5> tables;  // src, dst, dst_rowptr, src_rowptr, edge_ids_by_src
  luna_graph native{};
  Graph(std::array<Tensor, 5> t, int64_t nodes, int64_t source_rows) : tables(std::move(t)) {
    native.num_nodes = nodes;
    native.num_src_nodes = source_rows;
    native.num_edges = tables[0].numel();
    native.src = tables[0].data_ptr<int32_t>();
    native.dst = tables[1].data_ptr<int32_t>();
    native.dst_rowptr = tables[2].data_ptr<int32_t>();
    native.src_rowptr = tables[3].data_ptr<int32_t>();
    native.edge_ids_by_src = tables[4].data_ptr<int32_t>();
  }
};

using OpPtr = c10::intrusive_ptr<Op>;
using GraphPtr = c10::intrusive_ptr<Graph>;

template <typename H>
void keep(AutogradContext* ctx, const char* name, const c10::intrusive_ptr<H>& holder) {
  ctx->saved_data[name] = c10::IValue::make_capsule(holder);
}
template <typename H>
c10::intrusive_ptr<H> kept(AutogradContext* ctx, const char* name) {
  return c10::static_intrusive_pointer_cast<H>(ctx->saved_data[name].toCapsule());
}

// ---- launch wrappers ----------------------------------------------------------------------------------------------------
// Contiguous and 16-byte aligned (the staged kernels move 16-byte pieces of rows).
Tensor prepared(const Tensor& t) {
  if (!t.defined()) return t;
  Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 ? c.clone() : c;
}

// The kernels compute values only.  An operand of forward-mode AD does not have to require grad, so it can reach a launch
// without passing an autograd function; its tangent would be dropped, which reads as a derivative of zero.
void refuse_tangents(std::initializer_list<const Tensor*> tensors) {
  for (const Tensor* t : tensors)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(0).defined(),
                                "forward-mode automatic differentiation is not provided");
}

void check_operand(const Op& op, const Tensor& x, const Tensor& t, const char* name, int64_t rows, int64_t columns) {
  if (!t.defined()) return;
  TORCH_CHECK_TYPE(t.scalar_type() == op.dtype, name, " must be ", op.dtype == at::kDouble ? "torch.float64" : "torch.float32",
                   ", got ", t.scalar_type());
  TORCH_CHECK_VALUE(t.device() == x.device(), "features, weights and graph must share one CUDA device");
  TORCH_CHECK_VALUE(t.dim() == 2 && t.size(0) == rows && t.size(1) == columns, name, " must have shape (", rows, ", ",
                    columns, "), got ", t.sizes());
}

void check_operands(const Op& op, const Graph& graph, const Tensor& x, const Tensor& y, const Tensor& w, const Tensor& g) {
  refuse_tangents({&x, &y, &w, &g});
  TORCH_CHECK(x.is_cuda(), "CUDA is required for SO3 LunaTP.");
  check_operand(op, x, x, "x", graph.native.num_src_nodes, op.X);
  check_operand(op, x, y, "edge_attr", graph.native.num_edges, op.Y);
  check_operand(op, x, w, "weight", graph.native.num_edges, op.W);
  check_operand(op, x, g, "grad_out", graph.native.num_nodes, op.O);
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
void* pointer(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

Tensor scratch_for(const Op& op, const Graph& graph, const Tensor& like, int64_t* bytes) {
  *bytes = 0;
  if (!api.plan_query(op.plan, LUNA_PLAN_NEEDS_SCRATCH)) return Tensor();
  *bytes = api.scratch_bytes(op.plan, graph.native.num_nodes, graph.native.num_edges);
  return *bytes > 0 ? at::empty({*bytes}, like.options().dtype(at::kByte)) : Tensor();
}

Tensor run_forward(const Op& op, const Graph& graph, const Tensor& x_, const Tensor& y_, const Tensor& w_) {
  check_operands(op, graph, x_, y_, w_, Tensor());
  const c10::cuda::CUDAGuard guard(x_.device());
  const Tensor x = prepared(x_), y = prepared(y_), w = prepared(w_);
  Tensor out = at::empty({graph.native.num_nodes, op.O}, x.options());
  check(api.fwd(op.plan, &graph.native, x.data_ptr(), y.data_ptr(), w.data_ptr(), out.data_ptr(), stream_of(x)));
  return out;
}

enum : int { kX = 1, kY = 2, kW = 4, kG = 8 };

// The first derivatives named in `mask`; the others stay undefined.  gw, if given, is added to and becomes the third.
std::array<Tensor, 3> run_backward(const Op& op, const Graph& graph, const Tensor& x_, const Tensor& y_, const Tensor& w_,
                                   const Tensor& g_, int mask, const Tensor& gw = Tensor()) {
  std::array<Tensor, 3> out;
  if (!mask) return out;
  check_operands(op, graph, x_, y_, w_, g_);
  const c10::cuda::CUDAGuard guard(x_.device());
  const Tensor x = prepared(x_), y = prepared(y_), w = prepared(w_), g = prepared(g_);
  const Tensor* like[3] = {&x, &y, &w};
  const bool empty = graph.native.num_edges == 0 || graph.native.num_nodes == 0;
  for (int s = 0; s < 3; ++s)
    if (mask >> s & 1) out[s] = s == 2 && gw.defined() ? gw : (empty ? at::zeros_like(*like[s]) : at::empty_like(*like[s]));
  if (empty) return out;
  int64_t bytes = 0;
  const Tensor scratch = scratch_for(op, graph, x, &bytes);
  const auto entry = gw.defined() ? api.bwd_add_gw : api.bwd;
  check(entry(op.plan, &graph.native, x.data_ptr(), y.data_ptr(), w.data_ptr(), g.data_ptr(), pointer(out[0]),
                pointer(out[1]), pointer(out[2]), pointer(scratch), bytes, stream_of(x)));
  return out;
}

// The second derivatives named in `mask` (x, y, w, g) for the cotangents rx, ry, rw, each of which may be undefined.
std::array<Tensor, 4> run_double(const Op& op, const Graph& graph, const Tensor& x_, const Tensor& y_, const Tensor& w_,
                                 const Tensor& g_, const Tensor& rx_, const Tensor& ry_, const Tensor& rw_, int mask) {
  std::array<Tensor, 4> out;
  if (!mask) return out;
  refuse_tangents({&rx_, &ry_, &rw_});
  check_operands(op, graph, x_, y_, w_, g_);
  check_operand(op, x_, rx_, "rx", graph.native.num_src_nodes, op.X);
  check_operand(op, x_, ry_, "ry", graph.native.num_edges, op.Y);
  check_operand(op, x_, rw_, "rw", graph.native.num_edges, op.W);
  const c10::cuda::CUDAGuard guard(x_.device());
  const Tensor x = prepared(x_), y = prepared(y_), w = prepared(w_), g = prepared(g_), rx = prepared(rx_),
               ry = prepared(ry_), rw = prepared(rw_);
  const Tensor* like[4] = {&x, &y, &w, &g};
  const bool empty = graph.native.num_edges == 0 || graph.native.num_nodes == 0;
  for (int s = 0; s < 4; ++s)
    if (mask >> s & 1) out[s] = empty ? at::zeros_like(*like[s]) : at::empty_like(*like[s]);
  if (empty) return out;
  int64_t bytes = 0;
  const Tensor scratch = scratch_for(op, graph, x, &bytes);
  check(api.dbl_bwd(op.plan, &graph.native, x.data_ptr(), y.data_ptr(), w.data_ptr(), g.data_ptr(), pointer(rx), pointer(ry),
                    pointer(rw), pointer(out[0]), pointer(out[1]), pointer(out[2]), pointer(out[3]), pointer(scratch), bytes,
                    stream_of(x)));
  return out;
}

// ---- the autograd chain of the convolution --------------------------------------------------------------------------------
template <size_t N>
variable_list only(const std::array<Tensor, N>& tensors, int mask) {
  variable_list list;
  for (size_t s = 0; s < N; ++s)
    if (mask >> s & 1) list.push_back(tensors[s]);
  return list;
}
// The reverse: a list that holds the entries of `mask` only.
template <size_t N>
std::array<Tensor, N> spread(const variable_list& list, int mask) {
  std::array<Tensor, N> tensors;
  size_t next = 0;
  for (size_t s = 0; s < N; ++s)
    if (mask >> s & 1) tensors[s] = list[next++];
  return tensors;
}
Tensor contiguous(const Tensor& t) { return t.defined() ? t.contiguous() : t; }

// Energy training differentiates the weights once, force training twice: the gradients of both orders meet at the weights, and
// the engine adds two tensors of the weights' size, three more passes over memory beside the two that wrote them.  So the second
// order's graph names the weights through a node of its own (SecondOrderWeights), and if both that one and the first order's node,
// ConvForward, run in a task, the first order's kernel adds to the second order's gradient in place.  Which of the two comes first is
// the engine's choice unless the energy is nonlinear in the output: the second order leaves its gradient for the first, or the first
// leaves its operands for the second.  Neither node sees anything else of the other: ConvForward has one output, and runs when
// something reaches that.
// FP64 force step, degrees (2, 3, 3), 128 channels, 1.05 M edges (18 GB of weights): 33.6 -> 27.4 ms; FP32, (2, 2, 2),
// 32 channels, 0.2 M edges (295 MB): 936 -> 818 us.  Energy and forces in one loss, the energy linear in the output: FP64, 0.4 M edges
// 11.5 -> 8.9 ms; FP32, 0.2 M edges 610 -> 514 us.
//
// Not where a hook sees what one of the nodes returns, or where a graph of the gradient is wanted: there the engine adds them.
using NodePtr = std::shared_ptr<torch::autograd::Node>;

// Whether the running task runs a node, or has.
bool in_running_task(const NodePtr& node) {
  const auto* reached = torch::autograd::get_current_graph_task_nodes_in_graph();
  const auto* wanted = torch::autograd::get_current_graph_task_exec_info();
  if (!node || !reached || !wanted || reached->count(node.get()) == 0) return false;
  if (wanted->empty()) return true;
  const auto info = wanted->find(node.get());
  return info != wanted->end() && info->second.should_execute();
}

// The last tasks that something was done in.  Their numbers rise; of those before the ones kept anything may be true.
struct RecentTasks {
  std::array<int64_t, 8> tasks{-1, -1, -1, -1, -1, -1, -1, -1};
  size_t next = 0;
  int64_t forgotten = -1;
  void add(int64_t task) {
    forgotten = std::max(forgotten, tasks[next]);
    tasks[next] = task;
    next = (next + 1) % tasks.size();
  }
  bool may_have(int64_t task) const {
    return task <= forgotten || std::find(tasks.begin(), tasks.end(), task) != tasks.end();
  }
};

// Where the two nodes leave things for each other.  What a task that failed has left stays until the graph goes, and later tasks
// leave nothing.
struct WeightGradient : torch::CustomClassHolder {
  struct Operands {
    Tensor x, y, w, g;
    OpPtr op;
    GraphPtr graph;
  };

  explicit WeightGradient(const NodePtr& node) : first(node) {}
  void second_order_is(const NodePtr& node) {
    const std::lock_guard<std::mutex> lock(mutex);
    second = node;
  }

  // By the first order's node when it runs: what the second order has left for it in this task, if anything.
  Tensor first_runs() {
    const int64_t running = torch::autograd::get_current_graph_task_id();
    const std::lock_guard<std::mutex> lock(mutex);
    first_ran.add(running);
    return gradient_task == running ? std::exchange(gradient, Tensor()) : Tensor();
  }
  // Whether its operands were left for the second order's node, which runs later in this task.
  bool leave_operands(const Operands& all) {
    const std::lock_guard<std::mutex> lock(mutex);
    const NodePtr node = second.lock();
    const int64_t running = torch::autograd::get_current_graph_task_id();
    if (running < 0 || operands || second_ran.may_have(running) || !quiet(node) || !in_running_task(node)) return false;
    operands = all;
    operands_task = running;
    operands_for = node;
    return true;
  }
  // By a second order's node when it runs.
  std::optional<Operands> second_runs() {
    const int64_t running = torch::autograd::get_current_graph_task_id();
    const std::lock_guard<std::mutex> lock(mutex);
    second_ran.add(running);
    if (!operands || operands_task != running || operands_for.lock() != torch::autograd::get_current_node()) return std::nullopt;
    return std::exchange(operands, std::nullopt);
  }
  bool leave_gradient(const Tensor& w_gradient) {
    const std::lock_guard<std::mutex> lock(mutex);
    const int64_t running = torch::autograd::get_current_graph_task_id();
    const NodePtr node = first.lock();
    if (running < 0 || gradient.defined() || first_ran.may_have(running) || !quiet(node) || !in_running_task(node)) return false;
    gradient = w_gradient;
    gradient_task = running;
    return true;
  }

 private:
  // Whether no hook sees what the running node returns, nor what the other one does.
  static bool quiet(const NodePtr& other) {
    const NodePtr running = torch::autograd::get_current_node();
    return running && other && running->post_hooks().empty() && other->post_hooks().empty();
  }

  std::mutex mutex;  // tasks of several threads may run through one graph
  const std::weak_ptr<torch::autograd::Node> first;
  std::weak_ptr<torch::autograd::Node> second;  // the last one made
  std::weak_ptr<torch::autograd::Node> operands_for;
  RecentTasks first_ran, second_ran;
  Tensor gradient;
  std::optional<Operands> operands;
  int64_t gradient_task = -1, operands_task = -1;
};

// Whether nobody else can see the second order's gradient, so that a kernel may add to it.
bool only_ours(const Tensor& t) {
  return t.defined() && t.use_count() == 1 && t.has_storage() && t.storage().use_count() == 1 && !t.requires_grad() &&
         t.layout() == at::kStrided && t.is_contiguous() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}
// The first order's gradients, that of the weights added to the second order's if there is one.
std::array<Tensor, 3> first_on_second(const WeightGradient::Operands& all, int mask, const Tensor& second) {
  const bool ours = mask & kW && only_ours(second);
  auto d = run_backward(*all.op, *all.graph, all.x, all.y, all.w, all.g, mask, ours ? second : Tensor());
  if (second.defined() && !ours) d[2] = d[2].defined() ? d[2] + second : second;
  return d;
}

struct SecondOrderWeights : Function<SecondOrderWeights> {
  static Tensor forward(AutogradContext* ctx, const Tensor& w, const c10::intrusive_ptr<WeightGradient>& sum) {
    ctx->set_materialize_grads(false);
    keep(ctx, "sum", sum);
    return w.detach();
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    if (at::GradMode::is_enabled()) return {grads[0], Tensor()};
    const auto sum = kept<WeightGradient>(ctx, "sum");
    if (const auto operands = sum->second_runs()) return {first_on_second(*operands, kW, grads[0])[2], Tensor()};
    if (grads[0].defined() && sum->leave_gradient(grads[0])) return {Tensor(), Tensor()};
    return {grads[0], Tensor()};
  }
};

// dF/d(operand `slot`), slots 0..3 = x, y, w, g; a, b, c: the other three operands in that order.  The kernels take all four
// operands and look at the shape of the free slot's only: `free` lends it (none for g).
struct ConvPartial : Function<ConvPartial> {
  static Tensor forward(AutogradContext* ctx, const Tensor& a, const Tensor& b, const Tensor& c,
                        const std::optional<Tensor>& free, int64_t slot, const OpPtr& op, const GraphPtr& graph) {
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({a, b, c});
    ctx->saved_data["slot"] = slot;
    keep(ctx, "op", op);
    keep(ctx, "graph", graph);
    const auto all = operands({a, b, c}, slot, free ? *free : Tensor());
    if (slot == 3) return run_forward(*op, *graph, all[0], all[1], all[2]);
    return run_backward(*op, *graph, all[0], all[1], all[2], all[3], 1 << slot)[slot];
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list out(7);
    if (!grads[0].defined()) return out;
    const auto saved = ctx->get_saved_variables();
    const int64_t slot = ctx->saved_data["slot"].toInt();
    const auto op = kept<Op>(ctx, "op");
    const auto graph = kept<Graph>(ctx, "graph");
    // <r, dF/ds(a, b, c)> = F with r in slot s: the gradient of another operand is its partial at the rest
    const auto full = operands({saved[0], saved[1], saved[2]}, slot, grads[0].contiguous());
    for (int64_t other = 0, position = 0; other < 4; ++other) {
      if (other == slot) continue;
      if (ctx->needs_input_grad(position)) out[position] = of(full, other, op, graph);
      ++position;
    }
    return out;
  }
  static std::array<Tensor, 4> operands(const std::array<Tensor, 3>& others, int64_t slot, const Tensor& free) {
    std::array<Tensor, 4> full;
    for (int64_t s = 0, next = 0; s < 4; ++s) full[s] = s == slot ? free : others[next++];
    return full;
  }
  static Tensor of(const std::array<Tensor, 4>& full, int64_t slot, const OpPtr& op, const GraphPtr& graph) {
    std::array<Tensor, 3> others;
    for (int64_t s = 0, next = 0; s < 4; ++s)
      if (s != slot) others[next++] = full[s];
    // without history: nothing depends on its values
    const std::optional<Tensor> free = slot == 3 ? std::nullopt : std::optional<Tensor>(full[slot].detach());
    return apply(others[0], others[1], others[2], free, slot, op, graph);
  }
};

struct ConvDouble : Function<ConvDouble> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& y, const Tensor& w, const Tensor& g,
                               const std::optional<Tensor>& rx, const std::optional<Tensor>& ry,
                               const std::optional<Tensor>& rw, int64_t mask, const OpPtr& op, const GraphPtr& graph) {
    const Tensor none;
    const Tensor &tx = rx ? *rx : none, &ty = ry ? *ry : none, &tw = rw ? *rw : none;
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({x, y, w, g, tx, ty, tw});
    ctx->saved_data["mask"] = mask;
    keep(ctx, "op", op);
    keep(ctx, "graph", graph);
    return only(run_double(*op, *graph, x, y, w, g, tx, ty, tw, static_cast<int>(mask)), static_cast<int>(mask));
  }
  // The outputs contracted with their cotangents b are a sum of F with three of its operands replaced; the gradient of
  // a tensor is the sum of the partials over the terms it appears in.
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list out(10);
    const auto saved = ctx->get_saved_variables();
    const auto op = kept<Op>(ctx, "op");
    const auto graph = kept<Graph>(ctx, "graph");
    const auto b = spread<4>(grads, static_cast<int>(ctx->saved_data["mask"].toInt()));
    // tensors by number: 0..6 = x, y, w, g, rx, ry, rw (saved), 7..10 = bx, by, bw, bg
    std::array<Tensor, 11> t;
    for (int s = 0; s < 7; ++s) t[s] = saved[s];
    for (int s = 0; s < 4; ++s) t[7 + s] = contiguous(b[s]);
    static constexpr int terms[9][4] = {{7, 5, 2, 3}, {7, 1, 6, 3}, {4, 8, 2, 3}, {0, 8, 6, 3}, {4, 1, 9, 3},
                                        {0, 5, 9, 3}, {4, 1, 2, 10}, {0, 5, 2, 10}, {0, 1, 6, 10}};
    for (int v = 0, edge = 0; v < 7; ++v) {
      if (!t[v].defined()) continue;  // a missing tangent has no edge
      if (!ctx->needs_input_grad(edge++)) continue;
      Tensor sum;
      for (const auto& term : terms) {
        bool whole = true;
        int slot = -1;
        for (int s = 0; s < 4; ++s) {
          whole = whole && t[term[s]].defined();
          if (term[s] == v) slot = s;
        }
        if (!whole || slot < 0) continue;
        const Tensor part = ConvPartial::of({t[term[0]], t[term[1]], t[term[2]], t[term[3]]}, slot, op, graph);
        sum = sum.defined() ? sum + part : part;
      }
      out[v] = sum;
    }
    return out;
  }
};

struct ConvBackward : Function<ConvBackward> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& y, const Tensor& w, const Tensor& g,
                               int64_t mask, const OpPtr& op, const GraphPtr& graph) {
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({x, y, w, g});
    ctx->saved_data["mask"] = mask;
    keep(ctx, "op", op);
    keep(ctx, "graph", graph);
    return only(run_backward(*op, *graph, x, y, w, g, static_cast<int>(mask)), static_cast<int>(mask));
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list out(7);
    const auto r = spread<3>(grads, static_cast<int>(ctx->saved_data["mask"].toInt()));
    if (!r[0].defined() && !r[1].defined() && !r[2].defined()) return out;
    int mask = 0;
    for (int s = 0; s < 4; ++s) mask |= ctx->needs_input_grad(s) ? 1 << s : 0;
    if (!mask) return out;
    const auto saved = ctx->get_saved_variables();
    const auto op = kept<Op>(ctx, "op");
    const auto graph = kept<Graph>(ctx, "graph");
    std::array<Tensor, 4> h;
    if (at::GradMode::is_enabled()) {
      auto optional = [](const Tensor& t) { return t.defined() ? std::optional<Tensor>(t.contiguous()) : std::nullopt; };
      h = spread<4>(ConvDouble::apply(saved[0], saved[1], saved[2], saved[3], optional(r[0]), optional(r[1]),
                                      optional(r[2]), static_cast<int64_t>(mask), op, graph),
                    mask);
    } else {
      h = run_double(*op, *graph, saved[0], saved[1], saved[2], saved[3], r[0], r[1], r[2], mask);
    }
    for (int s = 0; s < 4; ++s) out[s] = h[s];
    return out;
  }
};

// Below this size of the weights the engine's sum, 15 us for 32 MiB, is not worth a node.
constexpr int64_t kSecondOrderBytes = 32 << 20;

struct ConvForward : Function<ConvForward> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& y, const Tensor& w, const OpPtr& op,
                        const GraphPtr& graph) {
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({x, y, w});
    keep(ctx, "op", op);
    keep(ctx, "graph", graph);
    return run_forward(*op, *graph, x, y, w);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list out(5);
    auto sum = ctx->saved_data.count("sum") ? kept<WeightGradient>(ctx, "sum") : c10::intrusive_ptr<WeightGradient>();
    const Tensor second = sum ? sum->first_runs() : Tensor();
    int mask = 0;
    for (int s = 0; s < 3; ++s) mask |= ctx->needs_input_grad(s) ? 1 << s : 0;
    if (!grads[0].defined() || !mask) {
      out[2] = second;
      return out;
    }
    const auto saved = ctx->get_saved_variables();
    const auto op = kept<Op>(ctx, "op");
    const auto graph = kept<Graph>(ctx, "graph");
    const Tensor g = grads[0].contiguous();
    std::array<Tensor, 3> d;
    if (at::GradMode::is_enabled()) {
      Tensor w = saved[2];
      if (w.requires_grad() && static_cast<int64_t>(w.nbytes()) >= kSecondOrderBytes) {
        if (!sum) {
          sum = c10::make_intrusive<WeightGradient>(torch::autograd::get_current_node());
          keep(ctx, "sum", sum);
        }
        w = SecondOrderWeights::apply(w, sum);
        sum->second_order_is(w.grad_fn());
      }
      d = spread<3>(ConvBackward::apply(saved[0], saved[1], w, g, static_cast<int64_t>(mask), op, graph), mask);
    } else {
      const WeightGradient::Operands all{saved[0], saved[1], saved[2], g, op, graph};
      if (sum && mask & kW && !second.defined() && sum->leave_operands(all)) mask &= ~kW;
      d = first_on_second(all, mask, second);
    }
    for (int s = 0; s < 3; ++s) out[s] = d[s];
    return out;
  }
};

bool tracked(std::initializer_list<const Tensor*> tensors) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : tensors)
    if (t->requires_grad()) return true;
  return false;
}

Tensor conv(const OpPtr& op, const GraphPtr& graph, const Tensor& x, const Tensor& y, const Tensor& w) {
  pybind11::gil_scoped_release release;
  return tracked({&x, &y, &w}) ? ConvForward::apply(x, y, w, op, graph) : run_forward(*op, *graph, x, y, w);
}

// ---- graph tables ---------------------------------------------------------------------------------------------------------
// Every table of a graph with nodes and edges: src, dst, dst_rowptr, src_rowptr, edge_ids_by_src, edge_ids_by_dst,
// node_order, source_node_order, node_tiers and the five of the segments; nothing if an index is out of range or dst is
// not ascending.  src, dst: contiguous, int32 or int64, on one CUDA device, of one length.
std::vector<Tensor> graph_tables(const Tensor& src, const Tensor& dst, int64_t nodes, int64_t source_rows) {
  pybind11::gil_scoped_release release;
  const c10::cuda::CUDAGuard guard(src.device());
  const int64_t edges = src.numel();
  const auto options = src.options().dtype(at::kInt);
  auto table = [&](int64_t entries) { return at::empty({entries}, options); };
  const int64_t room = source_rows + edges / 32;  // a segment per row at least, and one per 32 edges at most beyond that
  Tensor by_src = table(edges), by_dst = table(edges), src_out = table(edges), dst_out = table(edges);
  Tensor dst_rowptr = table(nodes + 1), src_rowptr = table(source_rows + 1), order = table(nodes);
  Tensor source_order = table(source_rows), tiers = table(3), seg_rowptr = table(source_rows + 1);
  Tensor seg_nodes = table(room), seg_begin = table(room), seg_end = table(room), seg_order = table(room);
  const int64_t bytes = api.graph_scratch_bytes(std::max(nodes, source_rows), edges);
  const Tensor scratch = at::empty({bytes}, options.dtype(at::kByte));
  auto ints = [](const Tensor& t) { return t.data_ptr<int32_t>(); };
  const luna_graph_out out{ints(src_out), ints(dst_out), ints(dst_rowptr), ints(src_rowptr),
                           ints(by_src),  ints(order),   ints(source_order)};
  const luna_graph_pieces pieces{ints(by_dst),  ints(tiers),      ints(seg_nodes), ints(seg_begin),
                                 ints(seg_end), ints(seg_rowptr), ints(seg_order)};
  int bad = 0;
  int64_t segments = 0;
  check(api.graph_build_all(src.data_ptr(), dst.data_ptr(), src.scalar_type() == at::kLong ? 64 : 32, nodes, source_rows,
                            edges, &out, &pieces, &bad, &segments, scratch.data_ptr(), bytes, stream_of(src)));
  if (bad) return {};
  auto cut = [&](const Tensor& t) { return t.narrow(0, 0, segments); };
  return {src_out, dst_out, dst_rowptr, src_rowptr, by_src, by_dst, order, source_order, tiers,
          cut(seg_nodes), cut(seg_begin), cut(seg_end), seg_rowptr, cut(seg_order)};
}

// ---- spherical harmonics --------------------------------------------------------------------------------------------------
struct Harmonics : torch::CustomClassHolder {
  luna_sh_desc desc{};
  int64_t columns;
  bool constant;
  Harmonics(const std::vector<int64_t>& degrees, bool normalize, int64_t normalization, int64_t out_dim, bool f64)
      : columns(out_dim), constant(true) {
    TORCH_CHECK_NOT_IMPLEMENTED(degrees.size() <= 32, "at most 32 degree entries are supported");
    desc.dtype = f64 ? LUNA_F64 : LUNA_F32;
    desc.num_degrees = static_cast<int32_t>(degrees.size());
    for (size_t i = 0; i < degrees.size(); ++i) {
      desc.degrees[i] = static_cast<int32_t>(degrees[i]);
      constant = constant && degrees[i] == 0;
    }
    desc.normalize = normalize;
    desc.normalization = static_cast<int32_t>(normalization);
  }
};
using HarmonicsPtr = c10::intrusive_ptr<Harmonics>;

Tensor rows_of(const Tensor& t) { return t.reshape({-1, t.size(-1)}).contiguous(); }

void check_vectors(const Harmonics& h, const Tensor& v) {
  TORCH_CHECK(v.is_cuda(), "CUDA is required for spherical harmonics in this library");
  TORCH_CHECK_TYPE(v.scalar_type() == (h.desc.dtype == LUNA_F64 ? at::kDouble : at::kFloat),
                   "spherical harmonics require float32 or float64 input");
  TORCH_CHECK_VALUE(v.dim() > 0 && v.size(-1) == 3, "SphericalHarmonics input must have shape (...,3)");
}

Tensor sh_forward(const Harmonics& h, const Tensor& v) {
  if (!h.constant) refuse_tangents({&v});  // the values of degree 0 alone have no derivative
  check_vectors(h, v);
  const c10::cuda::CUDAGuard guard(v.device());
  const Tensor flat = rows_of(v);
  auto shape = v.sizes().vec();
  shape.back() = h.columns;
  Tensor out = at::empty(shape, v.options());
  check(api.sh_fwd(&h.desc, flat.data_ptr(), out.data_ptr(), flat.size(0), stream_of(v)));
  return out;
}

Tensor sh_backward(const Harmonics& h, const Tensor& v, const Tensor& g) {
  refuse_tangents({&v, &g});
  check_vectors(h, v);
  const c10::cuda::CUDAGuard guard(v.device());
  const Tensor flat = rows_of(v), cotangents = rows_of(g);
  Tensor dv = at::empty(v.sizes(), v.options());
  check(api.sh_bwd(&h.desc, flat.data_ptr(), cotangents.data_ptr(), dv.data_ptr(), flat.size(0), stream_of(v)));
  return dv;
}

std::array<Tensor, 2> sh_double(const Harmonics& h, const Tensor& v, const Tensor& g, const Tensor& r, int mask) {
  refuse_tangents({&v, &g, &r});
  check_vectors(h, v);
  const c10::cuda::CUDAGuard guard(v.device());
  const Tensor flat = rows_of(v), cotangents = rows_of(g), tangents = rows_of(r);
  std::array<Tensor, 2> out;
  if (mask & 1) out[0] = at::empty(v.sizes(), v.options());
  if (mask & 2) out[1] = at::empty(g.sizes(), g.options());
  check(api.sh_dbl_bwd(&h.desc, flat.data_ptr(), cotangents.data_ptr(), tangents.data_ptr(), pointer(out[0]),
                       pointer(out[1]), flat.size(0), stream_of(v)));
  return out;
}

struct ShDouble : Function<ShDouble> {
  static variable_list forward(AutogradContext* ctx, const Tensor& v, const Tensor& g, const Tensor& r,
                               const HarmonicsPtr& h) {
    ctx->set_materialize_grads(false);
    return only(sh_double(*h, v, g, r, 3), 3);
  }
  static variable_list backward(AutogradContext*, const variable_list& grads) {
    TORCH_CHECK_NOT_IMPLEMENTED(!grads[0].defined() && !grads[1].defined(),
                                "third-order derivatives of the spherical harmonics are not provided");
    return variable_list(4);
  }
};

struct ShBackward : Function<ShBackward> {
  static Tensor forward(AutogradContext* ctx, const Tensor& v, const Tensor& g, const HarmonicsPtr& h) {
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({v, g});
    keep(ctx, "op", h);
    return sh_backward(*h, v, g);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list out(3);
    if (!grads[0].defined()) return out;
    const auto saved = ctx->get_saved_variables();
    const auto h = kept<Harmonics>(ctx, "op");
    const int mask = (ctx->needs_input_grad(0) ? 1 : 0) | (ctx->needs_input_grad(1) ? 2 : 0);
    if (!mask) return out;
    if (at::GradMode::is_enabled()) {
      const auto d = ShDouble::apply(saved[0], saved[1], grads[0], h);
      if (mask & 1) out[0] = d[0];
      if (mask & 2) out[1] = d[1];
    } else {
      const auto d = sh_double(*h, saved[0], saved[1], grads[0], mask);
      out[0] = d[0];
      out[1] = d[1];
    }
    return out;
  }
};

struct ShForward : Function<ShForward> {
  static Tensor forward(AutogradContext* ctx, const Tensor& v, const HarmonicsPtr& h) {
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({v});
    keep(ctx, "op", h);
    return sh_forward(*h, v);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list out(2);
    const auto h = kept<Harmonics>(ctx, "op");
    if (!grads[0].defined() || h->constant || !ctx->needs_input_grad(0)) return out;
    const auto saved = ctx->get_saved_variables();
    out[0] = at::GradMode::is_enabled() ? ShBackward::apply(saved[0], grads[0], h) : sh_backward(*h, saved[0], grads[0]);
    return out;
  }
};

Tensor harmonics(const HarmonicsPtr& h, const Tensor& v) {
  pybind11::gil_scoped_release release;
  return !h->constant && tracked({&v}) ? ShForward::apply(v, h) : sh_forward(*h, v);
}

}  // namespace

PYBIND11_MODULE(luna_torch, m) {
  m.def("load", torch::wrap_pybind_function(load));
  py::class_<Op, OpPtr>(m, "Op").def(py::init<int64_t, int64_t, int64_t, int64_t, int64_t, bool>());
  py::class_<Graph, GraphPtr>(m, "Graph").def(py::init<std::array<Tensor, 5>, int64_t, int64_t>());
  py::class_<Harmonics, HarmonicsPtr>(m, "Harmonics")
      .def(py::init<const std::vector<int64_t>&, bool, int64_t, int64_t, bool>());
  m.def("graph_tables", torch::wrap_pybind_function(graph_tables));
  m.def("conv", torch::wrap_pybind_function(conv));
  m.def("harmonics", torch::wrap_pybind_function(harmonics));
}
