// The native host path of the Python surface (kda.py): input checks, allocation, autograd bookkeeping and the C-ABI
// calls of one operator in one call from Python.
//
// At the sizes a training step or a decode loop runs, the kernels of an operator take 2 - 80 us each, so the host's share
// decides: through ctypes, torch.autograd.Function and torch.empty in Python the forward and backward of
// convolutions -> chunk_kda_norm at B2 T4096 H3 D128 cost 620 us of host time against 290 us of kernels.  Here a backward
// is a C++ node that the engine runs without the interpreter, allocations go straight to the caching allocator, and a
// forward is one pybind call.
//
// Every entry checks that its inputs are the plain valid case and otherwise returns None without having done anything;
// kda.py then runs its Python checks, which name the mistake.  Results, error texts and defaults are kda.py's.

#include <torch/extension.h>

#include <atomic>
#include <tuple>

#include "host_node.h"

namespace kda_host {

// ------------------------------------------------------------------------------------------------ device status
namespace {
constexpr int kDevices = 64;
std::mutex status_mu;
std::atomic<int32_t*> status_words{nullptr};      // page-locked int32 [kDevices], one per device, never freed
std::atomic<bool> registered[kDevices];
}  // namespace

void watch_status(int device) {
    if (device < 0 || device >= kDevices) return;
    if (!registered[device].load(std::memory_order_acquire)) {
        // page-locked memory cannot be had during a stream capture; such a call goes unwatched, the next one registers
        if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return;
        std::lock_guard<std::mutex> lk(status_mu);
        if (status_words.load() == nullptr) {
            static Tensor* keep = new Tensor(at::zeros({kDevices}, at::TensorOptions().dtype(at::kInt).pinned_memory(true)));
            status_words.store(keep->data_ptr<int32_t>());
        }
        must(kda_set_status_mirror(device, status_words.load() + device), "kda_set_status_mirror");
        registered[device].store(true, std::memory_order_release);
    }
    int32_t* word = status_words.load(std::memory_order_relaxed) + device;
    if (__atomic_load_n(word, __ATOMIC_ACQUIRE) == 0) return;
    const int32_t bad = __atomic_exchange_n(word, 0, __ATOMIC_ACQ_REL);
    if (bad == 0) return;
    const int rc = kda_status_word_code(bad);
    TORCH_CHECK(false, "an earlier KDA call on cuda:", device, " reported device status ", bad, ": ", kda_error_string(rc), " (", rc,
                "); its results are undefined");
}

namespace {

// ------------------------------------------------------------------------------------------------ chunked operator
struct Dims {
    int64_t B, T, H, K, V, N;
};

// The plain valid case of chunk_kda's inputs (raw: kda's, whose activations must be bf16 and whose gate is raw).
bool chunk_dims(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const OptTensor& h0, const OptTensor& cu,
                Dims& d) {
    if (tracing() || q.dim() != 4 || v.dim() != 4 || beta.dim() != 3 || !q.is_cuda()) return false;
    if (k.sizes() != q.sizes() || g.sizes() != q.sizes() || v.sizes().slice(0, 3) != q.sizes().slice(0, 3) || beta.sizes() != q.sizes().slice(0, 3))
        return false;
    d = Dims{q.size(0), q.size(1), q.size(2), q.size(3), v.size(3), q.size(0)};
    if (d.K > KDA_MAX_DIM || d.V > KDA_MAX_DIM || d.B * d.T >= (int64_t(1) << 31)) return false;
    if (!is_io(q) || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) return false;
    if (!is_io(g) || beta.scalar_type() != g.scalar_type()) return false;
    if (!on(k, q) || !on(v, q) || !on(g, q) || !on(beta, q)) return false;
    if (has(cu)) {
        if (d.B != 1 || cu->dim() != 1 || cu->numel() < 2 || cu->scalar_type() != at::kInt || !on(*cu, q)) return false;
        d.N = cu->numel() - 1;
    }
    if (has(h0)) {
        const int64_t want[4] = {d.N, d.H, d.V, d.K};
        if (h0->sizes() != at::IntArrayRef(want, 4) || h0->scalar_type() != at::kFloat || !on(*h0, q)) return false;
    }
    return true;
}

bool tc_shape(const Tensor& q, const Dims& d) { return q.scalar_type() == at::kBFloat16 && d.K == 128 && d.V == 128; }

KdaChunkShape chunk_shape(const Tensor& q, const Tensor& g, const Dims& d, bool packed, double scale, bool l2norm, int lane, bool forward_only) {
    KdaChunkShape sh;
    sh.n_seq = (int32_t)d.N;
    sh.seq_len = packed ? 0 : (int32_t)d.T;
    sh.tokens = (int32_t)(d.B * d.T);
    sh.heads = (int32_t)d.H;
    sh.key_dim = (int32_t)d.K;
    sh.value_dim = (int32_t)d.V;
    sh.io_dtype = dt(q);
    sh.gate_dtype = dt(g);
    sh.lane = lane;
    sh.l2norm = l2norm ? 1 : 0;
    sh.scale = (float)scale;
    sh.forward_only = forward_only ? 1 : 0;
    return sh;
}

struct ChunkGrads {
    Tensor dq, dk, dv, dg, db, dh0;
};

ChunkGrads run_chunk_bwd(const KdaChunkShape& sh, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta,
                         const Tensor& cu, const Tensor& d_o, const Tensor& dfs, const Tensor& ws, bool want_dh0) {
    ChunkGrads r{empty_as(q), empty_as(k), empty_as(v), empty_as(g), empty_as(beta), Tensor()};
    if (want_dh0) r.dh0 = empty({sh.n_seq, sh.heads, sh.value_dim, sh.key_dim}, at::kFloat, q);
    Tensor scr = bytes(kda_chunk_bwd_scratch_bytes(&sh), q);
    must(kda_chunk_bwd(&sh, q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(),
                        cu.defined() ? cu.data_ptr<int32_t>() : nullptr, d_o.data_ptr(), dfs.defined() ? dfs.data_ptr<float>() : nullptr,
                        ws.data_ptr(), (size_t)ws.numel(), scr.data_ptr(), (size_t)scr.numel(), r.dq.data_ptr(), r.dk.data_ptr(),
                        r.dv.data_ptr(), r.dg.data_ptr(), r.db.data_ptr(), want_dh0 ? r.dh0.data_ptr<float>() : nullptr, stream_of(q)),
          "kda_chunk_bwd");
    return r;
}

// Backward of chunk_kda: the gradients of (q, k, v, g, beta, h0) from the cotangents of (o, final state).  The workspace
// rides with the saved tensors: it lives exactly as long as the graph does.  A backward of the tensor-core lane writes its
// own panels there (adjoint states, dZ, the split scan's maps) and nothing the forward left for it, so a second one through
// a retained graph finds all it reads.
struct ChunkNode : public HostNode {
    KdaChunkShape sh;
    Tensor cu;
    bool has_h0 = false;
    std::string name() const override { return "ChunkKDABackward"; }
    variable_list apply(variable_list&& grads) override {
        std::vector<Tensor> t;
        {
            std::lock_guard<std::mutex> lk(mutex_);
            for (size_t i = 0; i < saved.size(); ++i) t.push_back(get(i));
        }
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor &q = t[0], &k = t[1], &v = t[2], &g = t[3], &beta = t[4], &ws = t[5];
        c10::cuda::CUDAGuard guard(q.device());
        watch_status(q.device().index());
        const Tensor d_o = grads[0].defined() ? aligned(dense(grads[0])) : at::zeros_like(v);
        const Tensor dfs = grads[1].defined() ? aligned(dense_as(grads[1], at::kFloat)) : Tensor();
        ChunkGrads r = run_chunk_bwd(sh, q, k, v, g, beta, cu, d_o, dfs, ws, has_h0);
        return {r.dq, r.dk, r.dv, r.dg, r.db, r.dh0};
    }
};

struct ChunkOut {
    Tensor o;
    OptTensor fs;
};

ChunkOut run_chunk(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& g_, const Tensor& beta_, const OptTensor& h0_,
                   bool want_final, const OptTensor& cu_, double scale, bool l2norm, int lane, const Dims& d) {
    refuse_tangents(q_, k_, v_, g_, beta_, h0_);
    const bool tracked = torch::autograd::compute_requires_grad(q_, k_, v_, g_, beta_, has(h0_) ? *h0_ : Tensor());
    c10::cuda::CUDAGuard guard(q_.device());
    watch_status(q_.device().index());
    Tensor q, k, v, g, beta, h0, cu, ws;
    KdaChunkShape sh;
    ChunkOut out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        q = aligned(dense(q_)), k = aligned(dense(k_)), v = aligned(dense(v_)), g = aligned(dense(g_)), beta = dense(beta_);
        if (has(h0_)) h0 = aligned(dense(*h0_));
        if (has(cu_)) cu = dense(*cu_);
        sh = chunk_shape(q, g, d, cu.defined(), scale, l2norm, lane, !tracked);
        out.o = empty(v.sizes(), v.scalar_type(), q);
        if (want_final) out.fs = empty({d.N, d.H, d.V, d.K}, at::kFloat, q);
        ws = bytes(kda_chunk_workspace_bytes(&sh), q);
    }
    must(kda_chunk_fwd(&sh, q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(), h0.defined() ? h0.data_ptr<float>() : nullptr,
                        cu.defined() ? cu.data_ptr<int32_t>() : nullptr, out.o.data_ptr(), want_final ? out.fs->data_ptr<float>() : nullptr,
                        ws.data_ptr(), (size_t)ws.numel(), stream_of(q)),
          "kda_chunk_fwd");
    if (tracked) {
        auto node = make_node<ChunkNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(q_, k_, v_, g_, beta_, has(h0_) ? *h0_ : Tensor()));
        node->sh = sh;
        node->cu = cu;
        node->has_h0 = h0.defined();
        for (const Tensor* t : {&q, &k, &v, &g, &beta, &ws}) node->keep(*t);
        torch::autograd::set_history(out.o, node);
        torch::autograd::set_history(want_final ? *out.fs : Tensor(), node);
    }
    return out;
}

using ChunkResult = c10::optional<std::tuple<Tensor, OptTensor>>;

// lane: 0 float32, 1 tensor cores, -1 whichever fits
ChunkResult chunk_kda(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const OptTensor& h0,
                      bool want_final, const OptTensor& cu, c10::optional<double> scale, bool l2norm, int lane) {
    Dims d;
    if (!chunk_dims(q, k, v, g, beta, h0, cu, d)) return c10::nullopt;
    const bool tc = tc_shape(q, d);
    if (lane == KDA_LANE_TC && !tc) return c10::nullopt;
    if (lane < 0) lane = tc ? KDA_LANE_TC : KDA_LANE_FP32;
    const double sc = scale.has_value() ? *scale : 1.0 / std::sqrt((double)d.K);
    ChunkOut r = run_chunk(q, k, v, g, beta, h0, want_final, cu, sc, l2norm, lane, d);
    return std::make_tuple(r.o, r.fs);
}

// Backward of chunk_kda_norm: the norm's backward, then the chunk's.
struct ChunkNormNode : public HostNode {
    KdaChunkShape sh;
    Tensor cu;
    bool has_h0 = false;
    at::ScalarType wtype = at::kFloat;
    std::string name() const override { return "ChunkKDANormBackward"; }
    variable_list apply(variable_list&& grads) override {
        std::vector<Tensor> t;
        {
            std::lock_guard<std::mutex> lk(mutex_);
            for (size_t i = 0; i < saved.size(); ++i) t.push_back(get(i));
        }
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor &q = t[0], &k = t[1], &v = t[2], &g = t[3], &beta = t[4], &ws = t[5], &o = t[6], &gate = t[7], &w32 = t[8], &inv = t[9];
        c10::cuda::CUDAGuard guard(q.device());
        watch_status(q.device().index());
        const Tensor dy = grads[0].defined() ? aligned(dense_as(grads[0], o.scalar_type())) : at::zeros_like(o);
        const Tensor dfs = grads[1].defined() ? aligned(dense_as(grads[1], at::kFloat)) : Tensor();
        const int64_t D = o.size(3), rows = o.numel() / D;
        Tensor d_o = empty_as(o), dgate = empty_as(gate), dw = empty({D}, at::kFloat, o);
        Tensor nscr = bytes(kda_rmsnorm_gate_bwd_scratch_bytes(rows, (int32_t)D), o);
        must(kda_rmsnorm_gate_bwd(rows, (int32_t)D, dt(o), o.data_ptr(), gate.data_ptr(), w32.data_ptr<float>(), inv.data_ptr<float>(),
                                   dy.data_ptr(), d_o.data_ptr(), dgate.data_ptr(), dw.data_ptr<float>(), nscr.data_ptr(), (size_t)nscr.numel(),
                                   stream_of(o)),
              "kda_rmsnorm_gate_bwd");
        ChunkGrads r = run_chunk_bwd(sh, q, k, v, g, beta, cu, d_o, dfs, ws, has_h0);
        return {r.dq, r.dk, r.dv, r.dg, r.db, dgate, wtype == at::kFloat ? dw : dw.to(wtype), r.dh0};
    }
};

ChunkResult chunk_kda_norm(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& g_, const Tensor& beta_, const Tensor& gate_,
                           const Tensor& nw_, double eps, const OptTensor& h0_, bool want_final, const OptTensor& cu_,
                           c10::optional<double> scale, bool l2norm) {
    Dims d;
    if (!chunk_dims(q_, k_, v_, g_, beta_, h0_, cu_, d) || !tc_shape(q_, d)) return c10::nullopt;
    if (gate_.sizes() != v_.sizes() || nw_.dim() != 1 || nw_.numel() != d.V || !on(gate_, q_) || !on(nw_, q_)) return c10::nullopt;
    const double sc = scale.has_value() ? *scale : 1.0 / std::sqrt((double)d.K);
    refuse_tangents(q_, k_, v_, g_, beta_, gate_, nw_, h0_);
    const bool tracked = torch::autograd::compute_requires_grad(q_, k_, v_, g_, beta_, gate_, nw_, has(h0_) ? *h0_ : Tensor());
    c10::cuda::CUDAGuard guard(q_.device());
    watch_status(q_.device().index());
    Tensor q, k, v, g, beta, h0, cu, o, y, inv, ws, gate, w32;
    OptTensor fs;
    KdaChunkShape sh;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        q = aligned(dense(q_)), k = aligned(dense(k_)), v = aligned(dense(v_)), g = aligned(dense(g_)), beta = dense(beta_);
        if (has(h0_)) h0 = aligned(dense(*h0_));
        if (has(cu_)) cu = dense(*cu_);
        sh = chunk_shape(q, g, d, cu.defined(), sc, l2norm, KDA_LANE_TC, !tracked);
        gate = aligned(dense_as(gate_, v.scalar_type()));
        w32 = aligned(dense_as(nw_, at::kFloat));
        o = empty(v.sizes(), v.scalar_type(), q);
        y = empty(v.sizes(), v.scalar_type(), q);
        inv = empty({d.B * d.T * d.H}, at::kFloat, q);
        if (want_final) fs = empty({d.N, d.H, d.V, d.K}, at::kFloat, q);
        ws = bytes(kda_chunk_workspace_bytes(&sh), q);
    }
    must(kda_chunk_fwd_norm(&sh, q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(),
                             h0.defined() ? h0.data_ptr<float>() : nullptr, cu.defined() ? cu.data_ptr<int32_t>() : nullptr, o.data_ptr(),
                             want_final ? fs->data_ptr<float>() : nullptr, ws.data_ptr(), (size_t)ws.numel(), gate.data_ptr(),
                             w32.data_ptr<float>(), (float)eps, y.data_ptr(), inv.data_ptr<float>(), stream_of(q)),
          "kda_chunk_fwd_norm");
    if (tracked) {
        auto node = make_node<ChunkNormNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(q_, k_, v_, g_, beta_, gate_, nw_, has(h0_) ? *h0_ : Tensor()));
        node->sh = sh;
        node->cu = cu;
        node->has_h0 = h0.defined();
        node->wtype = nw_.scalar_type();
        for (const Tensor* t : {&q, &k, &v, &g, &beta, &ws, &o, &gate, &w32, &inv}) node->keep(*t);
        torch::autograd::set_history(y, node);
        torch::autograd::set_history(want_final ? *fs : Tensor(), node);
    }
    return std::make_tuple(y, fs);
}

// ------------------------------------------------------------------------------------------------ gate activations
struct GateNode : public HostNode {
    double lb = 0;
    at::ScalarType atype = at::kFloat, btype = at::kFloat;
    std::vector<int64_t> bias_shape;
    std::string name() const override { return "KDAGateBackward"; }
    variable_list apply(variable_list&& grads) override {
        std::vector<Tensor> t;
        {
            std::lock_guard<std::mutex> lk(mutex_);
            for (size_t i = 0; i < saved.size(); ++i) t.push_back(get(i));
        }
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor &raw = t[0], &bl = t[1], &A = t[2], &bias = t[3];
        c10::cuda::CUDAGuard guard(raw.device());
        const int64_t B = raw.size(0), T = raw.size(1), H = raw.size(2), K = raw.size(3);
        const Tensor dg = grads[0].defined() ? dense_as(grads[0], at::kFloat) : at::zeros({B, T, H, K}, raw.options().dtype(at::kFloat));
        const Tensor db = grads[1].defined() ? dense_as(grads[1], at::kFloat) : at::zeros({B, T, H}, raw.options().dtype(at::kFloat));
        Tensor d_raw = empty_as(raw), d_bl = empty_as(bl), dA = empty({H}, at::kFloat, raw), dbias = empty({H * K}, at::kFloat, raw);
        Tensor scr = bytes(kda_gate_bwd_scratch_bytes((int32_t)(B * T), (int32_t)H, (int32_t)K), raw);
        must(kda_gate_bwd((int32_t)(B * T), (int32_t)H, (int32_t)K, dt(raw), raw.data_ptr(), bl.data_ptr(), A.data_ptr<float>(),
                           bias.data_ptr<float>(), (float)lb, dg.data_ptr<float>(), db.data_ptr<float>(), d_raw.data_ptr(), d_bl.data_ptr(),
                           dA.data_ptr<float>(), dbias.data_ptr<float>(), scr.data_ptr(), (size_t)scr.numel(), stream_of(raw)),
              "kda_gate_bwd");
        return {d_raw, d_bl, atype == at::kFloat ? dA : dA.to(atype), (btype == at::kFloat ? dbias : dbias.to(btype)).view(bias_shape)};
    }
};

using TensorPair = c10::optional<std::tuple<Tensor, Tensor>>;

// (raw gate, beta logits, A_log, dt_bias) -> (g, beta) in float32
TensorPair gate(const Tensor& raw_, const Tensor& bl_, const Tensor& A_, const Tensor& bias_, double lb) {
    if (tracing() || raw_.dim() != 4 || bl_.dim() != 3 || bl_.sizes() != raw_.sizes().slice(0, 3) || !raw_.is_cuda() || !on(bl_, raw_) || !on(A_, raw_) ||
        !on(bias_, raw_) || !is_io(raw_))
        return c10::nullopt;
    const int64_t B = raw_.size(0), T = raw_.size(1), H = raw_.size(2), K = raw_.size(3);
    if (A_.numel() != H || bias_.numel() != H * K || B * T >= (int64_t(1) << 31)) return c10::nullopt;
    refuse_tangents(raw_, bl_, A_, bias_);
    const bool tracked = torch::autograd::compute_requires_grad(raw_, bl_, A_, bias_);
    c10::cuda::CUDAGuard guard(raw_.device());
    Tensor g, beta, raw, bl, A, bias;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        raw = dense(raw_);
        bl = dense_as(bl_, raw.scalar_type());
        A = dense_as(A_, at::kFloat);
        bias = dense_as(bias_, at::kFloat);
        g = empty({B, T, H, K}, at::kFloat, raw);
        beta = empty({B, T, H}, at::kFloat, raw);
    }
    must(kda_gate_fwd((int32_t)(B * T), (int32_t)H, (int32_t)K, dt(raw), raw.data_ptr(), bl.data_ptr(), A.data_ptr<float>(),
                       bias.data_ptr<float>(), (float)lb, g.data_ptr<float>(), beta.data_ptr<float>(), stream_of(raw)),
          "kda_gate_fwd");
    if (tracked) {
        auto node = make_node<GateNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(raw_, bl_, A_, bias_));
        node->lb = lb;
        node->atype = A_.scalar_type();
        node->btype = bias_.scalar_type();
        node->bias_shape = bias_.sizes().vec();
        for (const Tensor* t : {&raw, &bl, &A, &bias}) node->keep(*t);
        torch::autograd::set_history(g, node);
        torch::autograd::set_history(beta, node);
    }
    return std::make_tuple(g, beta);
}

// ------------------------------------------------------------------------------------------------ decode
TensorPair decode_step(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& g_, const Tensor& beta_, const Tensor& state,
                       double scale, bool l2norm, const OptTensor& out_state) {
    if (q_.dim() < 2 || v_.dim() < 2 || !q_.is_cuda() || !on(k_, q_) || !on(v_, q_) || !on(g_, q_) || !on(beta_, q_) || !on(state, q_)) return c10::nullopt;
    if (!is_io(q_) || !is_io(g_) || k_.scalar_type() != q_.scalar_type() || v_.scalar_type() != q_.scalar_type()) return c10::nullopt;
    const int64_t H = q_.size(-2), K = q_.size(-1), V = v_.size(-1);
    if (H == 0 || K == 0 || V == 0) return c10::nullopt;
    const int64_t n = q_.numel() / (H * K);
    const int64_t want[4] = {n, H, V, K};
    if (k_.numel() != q_.numel() || g_.numel() != q_.numel() || v_.numel() != n * H * V || beta_.numel() != n * H) return c10::nullopt;
    if (state.scalar_type() != at::kFloat || !state.is_contiguous() || state.sizes() != at::IntArrayRef(want, 4)) return c10::nullopt;
    if (has(out_state) && (out_state->scalar_type() != at::kFloat || !out_state->is_contiguous() || out_state->sizes() != state.sizes() || !on(*out_state, q_)))
        return c10::nullopt;
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor q = dense(q_), k = dense(k_), v = dense(v_), g = dense(g_);
    const Tensor beta = dense_as(beta_, g.scalar_type());
    c10::cuda::CUDAGuard guard(q.device());
    Tensor new_state = has(out_state) ? *out_state : empty_as(state), o = empty_as(v);
    must(kda_decode_step((int32_t)n, (int32_t)H, (int32_t)K, (int32_t)V, dt(q), dt(g), l2norm ? 1 : 0, (float)scale, q.data_ptr(), k.data_ptr(),
                          v.data_ptr(), g.data_ptr(), beta.data_ptr(), state.data_ptr<float>(), new_state.data_ptr<float>(), o.data_ptr(),
                          stream_of(q)),
          "kda_decode_step");
    return std::make_tuple(o, new_state);
}

// ------------------------------------------------------------------------------------------------ raw-input operator
ChunkResult kda_raw(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& raw, const Tensor& bl, const Tensor& A_log, const Tensor& dt_bias,
                    const OptTensor& h0, bool want_final, double lb, c10::optional<double> scale, const OptTensor& cu, int lane) {
    Dims d;
    if (!chunk_dims(q, k, v, raw, bl, h0, cu, d)) return c10::nullopt;
    if (q.scalar_type() != at::kBFloat16 || raw.scalar_type() != at::kBFloat16 || bl.scalar_type() != at::kBFloat16) return c10::nullopt;
    if (A_log.scalar_type() != at::kFloat || dt_bias.scalar_type() != at::kFloat || A_log.dim() != 1 || A_log.size(0) != d.H ||
        dt_bias.numel() != d.H * d.K || !(lb >= -5.0 && lb < 0.0))
        return c10::nullopt;
    const bool tc = tc_shape(q, d);
    if (lane == KDA_LANE_TC && !tc) return c10::nullopt;
    if (lane < 0) lane = tc ? KDA_LANE_TC : KDA_LANE_FP32;
    TensorPair gb = gate(raw, bl, A_log, dt_bias, lb);
    if (!gb.has_value()) return c10::nullopt;
    const double sc = scale.has_value() ? *scale : 1.0 / std::sqrt((double)d.K);
    ChunkOut r = run_chunk(q, k, v, std::get<0>(*gb), std::get<1>(*gb), h0, want_final, cu, sc, true, lane, d);
    return std::make_tuple(r.o, r.fs);
}

// ------------------------------------------------------------------------------------------------ short convolution
// weight of a convolution as the fast kernels take it: [C, W] dense and 16-byte aligned, float32 or the activations' type
Tensor conv_weight(const Tensor& w, const Tensor& x) {
    return aligned(w.scalar_type() == at::kFloat ? dense(w) : dense_as(w, x.scalar_type()));
}

Tensor grad_like(const Tensor& dw, at::ScalarType type, const std::vector<int64_t>& shape) {
    return (type == at::kFloat ? dw : dw.to(type)).view(shape);
}

void run_conv_bwd(const Tensor& x, const Tensor& w, const Tensor& s0, const Tensor& dy, const Tensor& dfin, bool silu, Tensor& dx, Tensor& dw, Tensor& dinit) {
    const int32_t B = (int32_t)x.size(0), T = (int32_t)x.size(1), C = (int32_t)x.size(2), W = (int32_t)(w.numel() / x.size(2));
    dx = empty_as(x);
    dw = empty({C, W}, at::kFloat, x);
    if (s0.defined()) dinit = empty_as(s0);
    Tensor scr = bytes(kda_conv_bwd_scratch_bytes(B, T, C, W), x);
    must(kda_conv_bwd(B, T, C, W, dt(x) | wflag(x, w), silu ? 1 : 0, x.data_ptr(), w.data_ptr(), s0.defined() ? s0.data_ptr() : nullptr, dy.data_ptr(),
                       dfin.defined() ? dfin.data_ptr() : nullptr, dx.data_ptr(), dw.data_ptr<float>(), s0.defined() ? dinit.data_ptr() : nullptr,
                       scr.data_ptr(), (size_t)scr.numel(), stream_of(x)),
          "kda_conv_bwd");
}

struct ConvNode : public HostNode {
    at::ScalarType wtype = at::kFloat;
    std::vector<int64_t> wshape;
    bool has_s0 = false, silu = true;
    std::string name() const override { return "ShortConvolutionBackward"; }
    variable_list apply(variable_list&& grads) override {
        Tensor x, w, s0;
        {
            std::lock_guard<std::mutex> lk(mutex_);
            x = get(0);
            w = get(1);
            if (has_s0) s0 = get(2);
        }
        at::AutoDispatchBelowADInplaceOrView below;
        c10::cuda::CUDAGuard guard(x.device());
        const Tensor dy = grads[0].defined() ? dense_as(grads[0], x.scalar_type()) : at::zeros_like(x);
        const Tensor dfin = grads[1].defined() ? dense_as(grads[1], x.scalar_type()) : Tensor();
        Tensor dx, dw, dinit;
        run_conv_bwd(x, w, s0, dy, dfin, silu, dx, dw, dinit);
        return {dx, grad_like(dw, wtype, wshape), dinit};
    }
};

// x [B,T,C], weight [C,1,W] or [C,W], state [B,C,W] or none
ChunkResult conv(const Tensor& x_, const Tensor& w_, const OptTensor& s0_, bool want_final, bool silu) {
    if (tracing() || x_.dim() != 3 || !x_.is_cuda() || !is_io(x_) || !on(w_, x_) || w_.dim() < 2 || w_.size(0) != x_.size(2) || w_.numel() == 0 || x_.numel() == 0)
        return c10::nullopt;
    const int64_t B = x_.size(0), T = x_.size(1), C = x_.size(2), W = w_.numel() / C;
    const int64_t want[3] = {B, C, W};
    if (B * T >= (int64_t(1) << 31) || C >= (int64_t(1) << 31)) return c10::nullopt;
    if (has(s0_) && (s0_->sizes() != at::IntArrayRef(want, 3) || !on(*s0_, x_))) return c10::nullopt;
    refuse_tangents(x_, w_, s0_);
    const bool tracked = torch::autograd::compute_requires_grad(x_, w_, has(s0_) ? *s0_ : Tensor());
    c10::cuda::CUDAGuard guard(x_.device());
    Tensor x, w, s0, y;
    OptTensor fin;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        x = dense(x_);
        w = conv_weight(w_, x);
        if (has(s0_)) s0 = dense_as(s0_->detach(), x.scalar_type());
        y = empty_as(x);
        if (want_final) fin = empty({B, C, W}, x.scalar_type(), x);
    }
    must(kda_conv_fwd((int32_t)B, (int32_t)T, (int32_t)C, (int32_t)W, dt(x) | wflag(x, w), silu ? 1 : 0, x.data_ptr(), w.data_ptr(),
                       s0.defined() ? s0.data_ptr() : nullptr, y.data_ptr(), want_final ? fin->data_ptr() : nullptr, stream_of(x)),
          "kda_conv_fwd");
    if (tracked) {
        auto node = make_node<ConvNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(x_, w_, has(s0_) ? *s0_ : Tensor()));
        node->wtype = w_.scalar_type();
        node->wshape = w_.sizes().vec();
        node->has_s0 = s0.defined();
        node->silu = silu;
        node->keep(x);
        node->keep(w);
        if (s0.defined()) node->keep(s0);
        torch::autograd::set_history(y, node);
        torch::autograd::set_history(want_final ? *fin : Tensor(), node);
    }
    return std::make_tuple(y, fin);
}

// n same-shaped convolutions without carried-in or carried-out windows: one launch each way
struct ConvMultiNode : public HostNode {
    size_t n = 0;
    bool silu = true;
    std::vector<at::ScalarType> wtypes;
    std::vector<std::vector<int64_t>> wshapes;
    std::string name() const override { return "ShortConvolutionsBackward"; }
    variable_list apply(variable_list&& grads) override {
        std::vector<Tensor> t;
        {
            std::lock_guard<std::mutex> lk(mutex_);
            for (size_t i = 0; i < saved.size(); ++i) t.push_back(get(i));
        }
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor& x0 = t[0];
        c10::cuda::CUDAGuard guard(x0.device());
        const int32_t B = (int32_t)x0.size(0), T = (int32_t)x0.size(1), C = (int32_t)x0.size(2), W = (int32_t)(t[n].numel() / C);
        std::vector<Tensor> dys(n), dxs(n), dws(n);
        const void *xp[4], *wp[4], *gp[4];
        void* dp[4];
        float* wg[4];
        Tensor dw_all = empty({(int64_t)n, C, W}, at::kFloat, x0);
        for (size_t i = 0; i < n; ++i) {
            dys[i] = grads[i].defined() ? dense_as(grads[i], x0.scalar_type()) : at::zeros_like(t[i]);
            dxs[i] = empty_as(t[i]);
            dws[i] = dw_all.select(0, (int64_t)i);
            xp[i] = t[i].data_ptr();
            wp[i] = t[n + i].data_ptr();
            gp[i] = dys[i].data_ptr();
            dp[i] = dxs[i].data_ptr();
            wg[i] = dws[i].data_ptr<float>();
        }
        Tensor scr = bytes(kda_conv_bwd_multi_scratch_bytes((int32_t)n, B, T, C, W), x0);
        const int rc = kda_conv_bwd_multi((int32_t)n, B, T, C, W, dt(x0) | wflag(x0, t[n]), silu ? 1 : 0, xp, wp, gp, dp, wg, scr.data_ptr(), (size_t)scr.numel(),
                                          stream_of(x0));
        if (rc == KDA_ERR_UNSUPPORTED) {      // e.g. a cotangent that is not 16-byte aligned
            for (size_t i = 0; i < n; ++i) {
                Tensor none;
                run_conv_bwd(t[i], t[n + i], Tensor(), dys[i], Tensor(), silu, dxs[i], dws[i], none);
            }
        } else {
            must(rc, "kda_conv_bwd_multi");
        }
        variable_list out(dxs.begin(), dxs.end());
        for (size_t i = 0; i < n; ++i) out.push_back(grad_like(dws[i], wtypes[i], wshapes[i]));
        return out;
    }
};

c10::optional<std::vector<Tensor>> conv_multi(const std::vector<Tensor>& xs_, const std::vector<Tensor>& ws_, bool silu) {
    const size_t n = xs_.size();
    if (tracing() || n < 1 || n > 4 || ws_.size() != n) return c10::nullopt;
    const Tensor& x0 = xs_[0];
    if (x0.dim() != 3 || !x0.is_cuda() || !is_io(x0) || x0.numel() == 0) return c10::nullopt;
    for (size_t i = 0; i < n; ++i)
        if (xs_[i].sizes() != x0.sizes() || xs_[i].scalar_type() != x0.scalar_type() || !on(xs_[i], x0) || ws_[i].sizes() != ws_[0].sizes() ||
            !on(ws_[i], x0) || ws_[i].scalar_type() != ws_[0].scalar_type() || ws_[i].dim() < 2 || ws_[i].size(0) != x0.size(2))
            return c10::nullopt;
    const int64_t B = x0.size(0), T = x0.size(1), C = x0.size(2), W = ws_[0].numel() / C;
    if (W == 0 || B * T >= (int64_t(1) << 31)) return c10::nullopt;
    refuse_tangents(xs_, ws_);
    bool tracked = false;
    for (size_t i = 0; i < n; ++i) tracked = tracked || torch::autograd::compute_requires_grad(xs_[i], ws_[i]);
    c10::cuda::CUDAGuard guard(x0.device());
    std::vector<Tensor> xs(n), ws(n), ys(n);
    const void *xp[4], *wp[4];
    void* yp[4];
    {
        at::AutoDispatchBelowADInplaceOrView below;
        for (size_t i = 0; i < n; ++i) {
            xs[i] = dense(xs_[i]);
            ws[i] = conv_weight(ws_[i], xs[i]);
            ys[i] = empty_as(xs[i]);
            xp[i] = xs[i].data_ptr();
            wp[i] = ws[i].data_ptr();
            yp[i] = ys[i].data_ptr();
        }
    }
    const int rc = kda_conv_fwd_multi((int32_t)n, (int32_t)B, (int32_t)T, (int32_t)C, (int32_t)W, dt(xs[0]) | wflag(xs[0], ws[0]), silu ? 1 : 0, xp, wp, yp,
                                      stream_of(x0));
    if (rc == KDA_ERR_UNSUPPORTED) return c10::nullopt;      // the caller runs them one by one
    must(rc, "kda_conv_fwd_multi");
    if (tracked) {
        auto node = make_node<ConvMultiNode>();
        torch::autograd::edge_list edges;
        for (const auto& t : xs_) edges.push_back(torch::autograd::impl::gradient_edge(t));
        for (const auto& t : ws_) edges.push_back(torch::autograd::impl::gradient_edge(t));
        node->set_next_edges(std::move(edges));
        node->n = n;
        node->silu = silu;
        for (const auto& t : xs) node->keep(t);
        for (size_t i = 0; i < n; ++i) {
            node->keep(ws[i]);
            node->wtypes.push_back(ws_[i].scalar_type());
            node->wshapes.push_back(ws_[i].sizes().vec());
        }
        for (const auto& y : ys) torch::autograd::set_history(y, node);
    }
    return ys;
}

// ------------------------------------------------------------------------------------------------ gated RMSNorm
struct NormNode : public HostNode {
    at::ScalarType wtype = at::kFloat;
    std::string name() const override { return "RMSNormGatedBackward"; }
    variable_list apply(variable_list&& grads) override {
        Tensor x, gate, w, inv;
        {
            std::lock_guard<std::mutex> lk(mutex_);
            x = get(0);
            gate = get(1);
            w = get(2);
            inv = get(3);
        }
        at::AutoDispatchBelowADInplaceOrView below;
        c10::cuda::CUDAGuard guard(x.device());
        const Tensor dy = dense_as(grads[0], x.scalar_type());
        const int64_t D = x.size(-1), rows = x.numel() / D;
        Tensor dx = empty_as(x), dgate = empty_as(gate), dw = empty({D}, at::kFloat, x);
        Tensor scr = bytes(kda_rmsnorm_gate_bwd_scratch_bytes(rows, (int32_t)D), x);
        must(kda_rmsnorm_gate_bwd(rows, (int32_t)D, dt(x), x.data_ptr(), gate.data_ptr(), w.data_ptr<float>(), inv.data_ptr<float>(), dy.data_ptr(),
                                   dx.data_ptr(), dgate.data_ptr(), dw.data_ptr<float>(), scr.data_ptr(), (size_t)scr.numel(), stream_of(x)),
              "kda_rmsnorm_gate_bwd");
        return {dx, dgate, wtype == at::kFloat ? dw : dw.to(wtype)};
    }
};

OptTensor rmsnorm(const Tensor& x_, const Tensor& gate_, const Tensor& w_, double eps) {
    if (tracing() || x_.dim() < 1 || x_.numel() == 0 || !x_.is_cuda() || !is_io(x_) || !on(gate_, x_) || !on(w_, x_) || gate_.sizes() != x_.sizes()) return c10::nullopt;
    const int64_t D = x_.size(-1), rows = x_.numel() / D;
    if (w_.numel() != D) return c10::nullopt;
    refuse_tangents(x_, gate_, w_);
    const bool tracked = torch::autograd::compute_requires_grad(x_, gate_, w_);
    c10::cuda::CUDAGuard guard(x_.device());
    Tensor x, gate, w, y, inv;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        x = dense(x_);
        gate = dense_as(gate_, x.scalar_type());
        w = dense_as(w_, at::kFloat);
        y = empty_as(x);
        inv = empty({rows}, at::kFloat, x);
    }
    must(kda_rmsnorm_gate_fwd(rows, (int32_t)D, dt(x), (float)eps, x.data_ptr(), gate.data_ptr(), w.data_ptr<float>(), y.data_ptr(),
                               inv.data_ptr<float>(), stream_of(x)),
          "kda_rmsnorm_gate_fwd");
    if (tracked) {
        auto node = make_node<NormNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(x_, gate_, w_));
        node->wtype = w_.scalar_type();
        for (const Tensor* t : {&x, &gate, &w, &inv}) node->keep(*t);
        torch::autograd::set_history(y, node);
    }
    return y;
}

}  // namespace
}  // namespace kda_host

namespace kda_host {
void bind_layer(pybind11::module_& m);      // kda_layer.cpp
}

PYBIND11_MODULE(libkda_b200_torch, m) {
    namespace py = pybind11;
    using namespace kda_host;
    using nogil = py::call_guard<py::gil_scoped_release>;
    m.def("watch_status", &watch_status, nogil());
    m.def("chunk_kda", &chunk_kda, nogil());
    m.def("chunk_kda_norm", &chunk_kda_norm, nogil());
    m.def("kda_raw", &kda_raw, nogil());
    m.def("gate", &gate, nogil());
    m.def("decode_step", &decode_step, nogil());
    m.def("conv", &conv, nogil());
    m.def("conv_multi", &conv_multi, nogil());
    m.def("rmsnorm", &rmsnorm, nogil());
    bind_layer(m);
}
