// Autograd nodes of the operators that opake_b200/ops/nodes.py defines.
//
// Why native: under vmap(grad(...)) torch handles a Python autograd.Function in Python at every transform level (about 600 us for
// one forward and backward through an elementwise function), an operator with an autograd kernel of its own in the dispatcher.
// The kernels here are the same two boxed functions for every operator: `differentiable` records a node that keeps inputs and
// outputs and calls the operator of the backward pass, `terminal` lets nothing differentiate through one.
#include <ATen/core/dispatch/Dispatcher.h>
#include <torch/csrc/autograd/VariableTypeUtils.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/library.h>
#include <torch/python.h>

#include <map>
#include <mutex>
#include <shared_mutex>

namespace {

using at::Tensor;
using c10::IValue;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

enum Source { GRAD = 0, INPUT = 1, OUTPUT = 2 };

struct Rule {
  std::optional<c10::OperatorHandle> backward;
  std::vector<std::pair<int, int>> args;      // arguments of the backward operator: (Source, index)
  std::vector<int> grads;                     // per input of the forward operator: result of the backward operator, -1 none, -2 no tensor
  std::vector<bool> differentiable;           // per output
  std::string message;                        // `terminal`: what an attempt to differentiate says
};
std::shared_mutex g_lock;
std::map<std::string, std::shared_ptr<const Rule>>& rules() {
  static auto* all = new std::map<std::string, std::shared_ptr<const Rule>>;      // for the life of the process
  return *all;
}
std::shared_ptr<const Rule> rule_of(const c10::OperatorHandle& op) {
  std::shared_lock<std::shared_mutex> hold(g_lock);
  auto it = rules().find(op.operator_name().name);
  TORCH_CHECK(it != rules().end(), "no autograd rule for ", op.operator_name().name);
  return it->second;
}

struct Backward : public Node {
  std::shared_ptr<const Rule> rule;
  std::vector<SavedVariable> saved;           // the tensors among rule->args, in order
  std::vector<bool> is_output;
  std::vector<IValue> constants;              // the arguments that are not gradients, in order; None stands for a tensor
  std::string label;
  bool released = false;

  variable_list apply(variable_list&& grads) override {
    std::unique_lock<std::mutex> hold(mutex_);
    TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
    torch::jit::Stack stack;
    size_t next = 0, constant = 0;
    for (const auto& [source, index] : rule->args) {
      if (source == GRAD) {
        // an output that the loss does not use: zeros, as a Python function is given
        stack.emplace_back(grads[index].defined() ? grads[index] : input_metadata(index).zeros_like());
      } else if (constants[constant].isNone()) {
        stack.emplace_back(saved[next].unpack(is_output[next] ? shared_from_this() : nullptr));
        ++next;
        ++constant;
      } else {
        stack.emplace_back(constants[constant++]);
      }
    }
    hold.unlock();                            // the call below takes Python's lock
    rule->backward->callBoxed(stack);
    variable_list by_edge;
    for (const int result : rule->grads)
      if (result != -2) by_edge.push_back(result >= 0 && task_should_compute_output(by_edge.size()) ? stack[result].toTensor() : Tensor());
    return by_edge;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> hold(mutex_);
    for (auto& s : saved) s.reset_data();
    released = true;
  }
  std::string name() const override { return label; }
};

struct Terminal : public Node {
  std::string message, label;
  variable_list apply(variable_list&&) override { TORCH_CHECK_NOT_IMPLEMENTED(false, message); }
  std::string name() const override { return label; }
};

bool wants_grad(at::ArrayRef<IValue> args) {
  if (!c10::GradMode::is_enabled()) return false;
  for (const auto& a : args)
    if (a.isTensor() && a.toTensor().requires_grad()) return true;
  return false;
}
void no_forward_mode(const c10::OperatorHandle& op, at::ArrayRef<IValue> args) {
  for (const auto& a : args)
    TORCH_CHECK_NOT_IMPLEMENTED(!(a.isTensor() && torch::autograd::isFwGradDefined(a.toTensor())), op.operator_name().name,
                                " has no forward-mode derivative");
}
template <class N>
std::shared_ptr<N> make_node(const c10::OperatorHandle& op, at::ArrayRef<IValue> args) {
  auto node = std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
  torch::autograd::edge_list edges;
  for (const auto& a : args)
    if (a.isTensor()) edges.push_back(torch::autograd::impl::gradient_edge(a.toTensor()));
  node->set_next_edges(std::move(edges));
  node->label = op.operator_name().name + "Backward";
  return node;
}

void differentiable(const c10::OperatorHandle& op, c10::DispatchKeySet keys, torch::jit::Stack* stack) {
  const size_t n_in = op.schema().arguments().size(), n_out = op.schema().returns().size();
  const auto rule = rule_of(op);
  std::vector<IValue> in(stack->end() - n_in, stack->end());
  no_forward_mode(op, in);
  std::shared_ptr<Backward> node;
  if (wants_grad(in)) {
    node = make_node<Backward>(op, in);
    node->rule = rule;
  }
  {
    at::AutoDispatchBelowADInplaceOrView below;
    op.redispatchBoxed(keys & c10::after_autograd_keyset, stack);
  }
  if (!node) return;
  const auto out = at::ArrayRef<IValue>(*stack).slice(stack->size() - n_out, n_out);
  for (size_t i = 0; i < n_out; ++i)
    if (rule->differentiable[i]) torch::autograd::set_history(out[i].toTensor(), node);
  for (const auto& [source, index] : rule->args) {
    if (source == GRAD) continue;
    const IValue& v = source == INPUT ? in[index] : out[index];
    if (v.isTensor()) {
      const bool own = source == OUTPUT && rule->differentiable[index];
      node->saved.emplace_back(v.toTensor(), own);
      node->is_output.push_back(own);
      node->constants.emplace_back();
    } else {
      node->constants.push_back(v);
    }
  }
}

void terminal(const c10::OperatorHandle& op, c10::DispatchKeySet keys, torch::jit::Stack* stack) {
  const size_t n_in = op.schema().arguments().size(), n_out = op.schema().returns().size();
  std::vector<IValue> in(stack->end() - n_in, stack->end());
  no_forward_mode(op, in);
  const bool wants = wants_grad(in);
  {
    at::AutoDispatchBelowADInplaceOrView below;
    op.redispatchBoxed(keys & c10::after_autograd_keyset, stack);
  }
  if (!wants) return;
  auto node = make_node<Terminal>(op, in);
  node->message = rule_of(op)->message;
  for (size_t i = stack->size() - n_out; i < stack->size(); ++i) {
    const Tensor& t = (*stack)[i].toTensor();
    if (at::isFloatingType(t.scalar_type())) torch::autograd::set_history(t, node);
  }
}

c10::OperatorHandle find(const std::string& name) { return c10::Dispatcher::singleton().findSchemaOrThrow(name.c_str(), ""); }
void install(const std::string& name, std::shared_ptr<const Rule> rule, torch::CppFunction&& kernel) {
  static auto* libraries = new std::vector<std::unique_ptr<torch::Library>>;       // for the life of the process
  {
    std::unique_lock<std::shared_mutex> hold(g_lock);
    rules()[name] = std::move(rule);
  }
  const auto colon = name.find("::");
  auto lib = std::make_unique<torch::Library>(torch::Library::IMPL, name.substr(0, colon), std::make_optional(c10::DispatchKey::Autograd),
                                              __FILE__, __LINE__);
  lib->impl(name.substr(colon + 2).c_str(), std::move(kernel));
  libraries->push_back(std::move(lib));
}

void register_differentiable(const std::string& name, const std::string& backward, std::vector<std::pair<int, int>> args,
                             std::vector<int> grads, std::vector<bool> outputs) {
  auto rule = std::make_shared<Rule>();
  const auto fwd = find(name);
  rule->backward = find(backward);
  TORCH_CHECK(grads.size() == fwd.schema().arguments().size() && outputs.size() == fwd.schema().returns().size() &&
                  args.size() == rule->backward->schema().arguments().size(),
              "autograd rule of ", name, " does not fit the schemas");
  for (size_t i = 0; i < grads.size(); ++i) {
    const bool tensor = fwd.schema().arguments()[i].type()->kind() == c10::TypeKind::TensorType;
    TORCH_CHECK(tensor || grads[i] < 0, "argument ", i, " of ", name, " is not a tensor");
    if (!tensor) grads[i] = -2;
  }
  rule->args = std::move(args);
  rule->grads = std::move(grads);
  rule->differentiable = std::move(outputs);
  install(name, rule, torch::CppFunction::makeFromBoxedFunction<&differentiable>());
}
void register_terminal(const std::string& name, const std::string& message) {
  auto rule = std::make_shared<Rule>();
  rule->message = message;
  find(name);
  install(name, rule, torch::CppFunction::makeFromBoxedFunction<&terminal>());
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("register_differentiable", &register_differentiable);
  m.def("register_terminal", &register_terminal);
}
