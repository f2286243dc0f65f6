// Helpers of the native host path and the base of its backward nodes.
#pragma once

#include <ATen/TracerMode.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>

#include <memory>
#include <mutex>
#include <vector>

#include "host_common.h"

namespace kda_host {

using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

inline bool is_io(const Tensor& t) { return t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kFloat; }
inline int dt(const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? KDA_DTYPE_BF16 : KDA_DTYPE_F32; }
inline int wflag(const Tensor& x, const Tensor& w) {
    return (w.scalar_type() == at::kFloat && x.scalar_type() != at::kFloat) ? KDA_WEIGHT_F32 : 0;
}
inline bool on(const Tensor& t, const Tensor& like) { return t.is_cuda() && t.device() == like.device(); }
inline Tensor dense(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
inline Tensor dense_as(const Tensor& t, at::ScalarType type) { return t.scalar_type() == type ? dense(t) : t.to(type).contiguous(); }

// A torch.jit trace records dispatched operators and Python autograd functions, not these calls: inside one the entries
// answer None, and the Python side makes the call through an autograd function (ops.traced) that the tracer can see.
inline bool tracing() { return at::tracer::impl::is_dispatch_enabled(); }

// The nodes below are reverse-mode only: a dual tensor's tangent is refused, not dropped.
inline void refuse_tangent(const Tensor& t) {
    TORCH_CHECK_NOT_IMPLEMENTED(!t.defined() || !t._fw_grad(0).defined(), "KDA operators have no forward-mode derivative");
}
inline void refuse_tangent(const OptTensor& t) {
    if (has(t)) refuse_tangent(*t);
}
inline void refuse_tangent(const std::vector<Tensor>& ts) {
    for (const auto& t : ts) refuse_tangent(t);
}
template <class... Ts>
void refuse_tangents(const Ts&... ts) {
    (refuse_tangent(ts), ...);
}

// A backward node: saved inputs, released with the graph.  Derived classes hold their sizes as plain fields.
struct HostNode : public Node {
    std::vector<SavedVariable> saved;
    void keep(const Tensor& t) { saved.emplace_back(t, false); }
    Tensor get(size_t i) { return saved[i].unpack(); }
    void release_variables() override {
        std::lock_guard<std::mutex> lk(mutex_);
        for (auto& s : saved) s.reset_data();
    }
};

template <class N>
std::shared_ptr<N> make_node() {
    return std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
}

}  // namespace kda_host
