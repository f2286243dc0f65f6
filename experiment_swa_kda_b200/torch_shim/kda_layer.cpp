// KimiDeltaAttention as one call each way (head width 128, bf16 activations).
//
// The module's stages one by one cost 65 launches forward and backward at width 768: a cast per weight, a GEMM per
// projection, a GEMM and an addition per input gradient.  Here the six projections of the layer's input are ONE GEMM on
// the weights packed side by side (their casts are one launch), the kernels behind it read and write their slices of the
// projection in place, and the backward forms the gradient of the input as one GEMM over all six and the six weight
// gradients as another, both accumulated in float32.  Columns of the projection P [tokens][n]:
//     q | k | v | output gate (hidden each) | f_a (128) | b (heads) | zero padding to a multiple of 8
// B2 T2045 width 768, forward and backward: 1,141 -> see DESIGN; 65 -> 27 launches.

#include <torch/extension.h>

#include <cmath>
#include <tuple>

#include <ATen/autocast_mode.h>

#include "host_node.h"

namespace kda_host {
namespace {

constexpr int64_t kHead = 128;

// positions in the parameter list
enum { kQ, kK, kV, kG, kFa, kB, kFb, kO, kCq, kCk, kCv, kAlog, kDt, kNorm, kParams };

struct Sizes {
    int64_t B, T, H, M, hid, n, pad, W;      // M = B * T tokens, n = columns of P
    int64_t fa() const { return 4 * hid; }
    int64_t b() const { return 4 * hid + kHead; }
};

// all weights of the layer's products in bf16: rows of P's matrix, then f_b, then the output projection
struct Packed {
    Tensor all, p, fb, o;
};

Packed pack_weights(const std::vector<Tensor>& w, const Sizes& z) {
    const int64_t h = z.hid;
    Packed r;
    r.all = empty({(z.n + kHead + h) * h}, at::kBFloat16, w[kQ]);
    const void* src[9] = {w[kQ].data_ptr(), w[kK].data_ptr(), w[kV].data_ptr(), w[kG].data_ptr(), w[kFa].data_ptr(),
                          w[kB].data_ptr(), nullptr, w[kFb].data_ptr(), w[kO].data_ptr()};
    const int64_t elems[9] = {h * h, h * h, h * h, h * h, kHead * h, z.H * h, z.pad * h, h * kHead, h * h};
    must(kda_pack_bf16(9, dt(w[kQ]), src, elems, r.all.data_ptr(), stream_of(w[kQ])), "kda_pack_bf16");
    r.p = r.all.narrow(0, 0, z.n * h).view({z.n, h});
    r.fb = r.all.narrow(0, z.n * h, h * kHead).view({h, kHead});
    r.o = r.all.narrow(0, (z.n + kHead) * h, h * h).view({h, h});
    return r;
}

char* at_col(const Tensor& p, int64_t col) { return static_cast<char*>(p.data_ptr()) + 2 * col; }

KdaChunkShape layer_shape(const Sizes& z, bool forward_only) {
    KdaChunkShape sh;
    sh.n_seq = (int32_t)z.B;
    sh.seq_len = (int32_t)z.T;
    sh.tokens = (int32_t)z.M;
    sh.heads = (int32_t)z.H;
    sh.key_dim = sh.value_dim = (int32_t)kHead;
    sh.io_dtype = KDA_DTYPE_BF16;
    sh.gate_dtype = KDA_DTYPE_F32;
    sh.lane = KDA_LANE_TC;
    sh.l2norm = 1;
    sh.scale = (float)(1.0 / std::sqrt((double)kHead));
    sh.forward_only = forward_only ? 1 : 0;
    return sh;
}

// weight gradient dY^T X: float32 straight from the accumulators when the parameter is float32
Tensor weight_grad(const Tensor& dy, const Tensor& x, at::ScalarType type) {
    return type == at::kFloat ? at::mm(dy.t(), x, at::kFloat) : at::mm(dy.t(), x);
}

struct LayerNode : public HostNode {
    Sizes z;
    double lb = 0;
    at::ScalarType wtype = at::kFloat, ntype = at::kFloat;
    at::ScalarType ctype = at::kFloat, stype[3] = {at::kFloat, at::kFloat, at::kFloat};
    std::vector<int64_t> cshape[3], dt_shape;
    bool has_state = false;
    std::string name() const override { return "KimiDeltaAttentionBackward"; }
    // saved: x, conv weights, A_log, dt_bias, norm weight | pack, P, raw, g, beta, q, k, v, ws, o, inv, mixed | windows
    enum { sX, sCq, sCk, sCv, sA, sDt, sN, sPack, sP, sRaw, sG, sBeta, sQ, sK, sV, sWs, sO, sInv, sMixed, sWq, sWk, sWv };

    variable_list apply(variable_list&& grads) override {
        std::vector<Tensor> t;
        {
            std::lock_guard<std::mutex> lk(mutex_);
            for (size_t i = 0; i < saved.size(); ++i) t.push_back(get(i));
        }
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor& x = t[sX];
        c10::cuda::CUDAGuard guard(x.device());
        watch_status(x.device().index());
        void* st = stream_of(x);
        const int64_t h = z.hid, M = z.M, H = z.H;
        variable_list out(15 + (has_state ? 4 : 0));
        auto want = [&](size_t i) { return task_should_compute_output(i); };
        const Tensor P = t[sP], x2 = x.view({M, h});
        const Tensor wp = t[sPack].narrow(0, 0, z.n * h).view({z.n, h}), wfb = t[sPack].narrow(0, z.n * h, h * kHead).view({h, kHead}),
                     wo = t[sPack].narrow(0, (z.n + kHead) * h, h * h).view({h, h});

        const Tensor dy = grads[0].defined() ? dense_as(grads[0], at::kBFloat16).view({M, h}) : at::zeros({M, h}, x.options());
        if (want(1 + kO)) out[1 + kO] = weight_grad(dy, t[sMixed].view({M, h}), wtype);
        const Tensor d_mixed = at::mm(dy, wo);

        // gated norm: its gate and the gate's gradient are slices of P and dP
        Tensor dP = empty({M, z.n}, at::kBFloat16, x);
        Tensor d_o = empty_as(t[sO]), dnw = empty({kHead}, at::kFloat, x);
        Tensor nscr = bytes(kda_rmsnorm_gate_bwd_scratch_bytes(M * H, (int32_t)kHead), x);
        must(kda_rmsnorm_gate_bwd_rows(M * H, KDA_DTYPE_BF16, (int32_t)H, (int32_t)z.n, t[sO].data_ptr(), at_col(P, 3 * h),
                                       t[sN].data_ptr<float>(), t[sInv].data_ptr<float>(), d_mixed.data_ptr(), d_o.data_ptr(), at_col(dP, 3 * h),
                                       dnw.data_ptr<float>(), nscr.data_ptr(), (size_t)nscr.numel(), st),
             "kda_rmsnorm_gate_bwd_rows");
        out[1 + kNorm] = ntype == at::kFloat ? dnw : dnw.to(ntype);

        // chunked operator
        const KdaChunkShape sh = layer_shape(z, false);
        const Tensor dmem = grads[1].defined() ? dense_as(grads[1], at::kFloat) : Tensor();
        Tensor dqkv = empty({3, M, h}, at::kBFloat16, x), dg = empty_as(t[sG]), db = empty_as(t[sBeta]), dh0;
        if (has_state) dh0 = empty({z.B, H, kHead, kHead}, at::kFloat, x);
        char* d3 = static_cast<char*>(dqkv.data_ptr());
        Tensor scr = bytes(kda_chunk_bwd_scratch_bytes(&sh), x);
        must(kda_chunk_bwd(&sh, t[sQ].data_ptr(), t[sK].data_ptr(), t[sV].data_ptr(), t[sG].data_ptr(), t[sBeta].data_ptr(), nullptr, d_o.data_ptr(),
                           dmem.defined() ? dmem.data_ptr<float>() : nullptr, t[sWs].data_ptr(), (size_t)t[sWs].numel(), scr.data_ptr(),
                           (size_t)scr.numel(), d3, d3 + 2 * M * h, d3 + 4 * M * h, dg.data_ptr(), db.data_ptr(),
                           has_state ? dh0.data_ptr<float>() : nullptr, st),
             "kda_chunk_bwd");

        // gate activations, then the low-rank gate projection
        Tensor d_raw = empty_as(t[sRaw]), dA = empty({H}, at::kFloat, x), dbias = empty({h}, at::kFloat, x);
        Tensor gscr = bytes(kda_gate_bwd_scratch_bytes((int32_t)M, (int32_t)H, (int32_t)kHead), x);
        must(kda_gate_bwd_rows((int32_t)M, (int32_t)H, (int32_t)kHead, KDA_DTYPE_BF16, t[sRaw].data_ptr(), at_col(P, z.b()), (int32_t)z.n,
                               (int32_t)z.pad, t[sA].data_ptr<float>(), t[sDt].data_ptr<float>(), (float)lb, dg.data_ptr<float>(),
                               db.data_ptr<float>(), d_raw.data_ptr(), at_col(dP, z.b()), dA.data_ptr<float>(), dbias.data_ptr<float>(),
                               gscr.data_ptr(), (size_t)gscr.numel(), st),
             "kda_gate_bwd_rows");
        out[1 + kAlog] = dA;
        out[1 + kDt] = dbias.view(dt_shape);
        if (want(1 + kFb)) out[1 + kFb] = weight_grad(d_raw, P.narrow(1, z.fa(), kHead), wtype);
        Tensor dfa = dP.narrow(1, z.fa(), kHead);
        at::mm_out(dfa, d_raw, wfb);

        // convolutions
        Tensor dcw = empty({3, h, z.W}, at::kFloat, x);
        const bool windows = has_state || grads[2].defined() || grads[3].defined() || grads[4].defined();
        if (!windows) {
            const void *xp[3], *wpt[3], *gp[3];
            void* dp[3];
            float* wg[3];
            for (int i = 0; i < 3; ++i) {
                xp[i] = at_col(P, i * h);
                wpt[i] = t[sCq + i].data_ptr();
                gp[i] = d3 + 2 * i * M * h;
                dp[i] = at_col(dP, i * h);
                wg[i] = dcw.data_ptr<float>() + i * h * z.W;
            }
            Tensor cscr = bytes(kda_conv_bwd_multi_scratch_bytes(3, (int32_t)z.B, (int32_t)z.T, (int32_t)h, (int32_t)z.W), x);
            must(kda_conv_bwd_rows(3, (int32_t)z.B, (int32_t)z.T, (int32_t)h, (int32_t)z.W, KDA_DTYPE_BF16 | wflag(x, t[sCq]), 1, xp, (int32_t)z.n,
                                   wpt, gp, dp, wg, cscr.data_ptr(), (size_t)cscr.numel(), st),
                 "kda_conv_bwd_rows");
        } else {      // windows carried in or out: the general kernel, on dense copies
            for (int i = 0; i < 3; ++i) {
                const Tensor xc = P.narrow(1, i * h, h).contiguous();
                const Tensor dfin = grads[2 + i].defined() ? dense_as(grads[2 + i], at::kBFloat16) : Tensor();
                Tensor dx = empty({M, h}, at::kBFloat16, x), dinit;
                if (has_state) dinit = empty({z.B, h, z.W}, at::kBFloat16, x);
                Tensor cscr = bytes(kda_conv_bwd_scratch_bytes((int32_t)z.B, (int32_t)z.T, (int32_t)h, (int32_t)z.W), x);
                must(kda_conv_bwd((int32_t)z.B, (int32_t)z.T, (int32_t)h, (int32_t)z.W, KDA_DTYPE_BF16 | wflag(x, t[sCq]), 1, xc.data_ptr(),
                                  t[sCq + i].data_ptr(), has_state ? t[sWq + i].data_ptr() : nullptr, d3 + 2 * i * M * h,
                                  dfin.defined() ? dfin.data_ptr() : nullptr, dx.data_ptr(), dcw.data_ptr<float>() + i * h * z.W,
                                  has_state ? dinit.data_ptr() : nullptr, cscr.data_ptr(), (size_t)cscr.numel(), st),
                     "kda_conv_bwd");
                dP.narrow(1, i * h, h).copy_(dx);
                if (has_state) out[16 + i] = stype[i] == at::kBFloat16 ? dinit : dinit.to(stype[i]);
            }
            if (has_state) out[15] = dh0;
        }
        for (int i = 0; i < 3; ++i) {
            const Tensor d = dcw.select(0, i);
            out[1 + kCq + i] = (ctype == at::kFloat ? d : d.to(ctype)).view(cshape[i]);
        }

        // the input and the six weights of P
        if (want(0)) out[0] = at::mm(dP, wp).view(x.sizes());
        bool any = false;
        for (int i = kQ; i <= kB; ++i) any = any || want(1 + i);
        if (any) {
            const Tensor dW = weight_grad(dP, x2, wtype);
            for (int i = kQ; i <= kG; ++i) out[1 + i] = dW.narrow(0, i * h, h);
            out[1 + kFa] = dW.narrow(0, z.fa(), kHead);
            out[1 + kB] = dW.narrow(0, z.b(), H);
        }
        return out;
    }
};

// ------------------------------------------------------------------------------------------------ forward
// The plain case: bf16 input, 128-wide heads, weights of one type (float32 masters or bf16), everything dense on one GPU.
bool layer_sizes(const Tensor& x, const std::vector<Tensor>& w, int64_t heads, const std::vector<Tensor>& state, Sizes& z) {
    if (w.size() != kParams || x.dim() != 3 || !x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.numel() == 0 || heads < 1) return false;
    z.B = x.size(0), z.T = x.size(1), z.H = heads, z.M = z.B * z.T, z.hid = heads * kHead;
    z.pad = (8 - heads % 8) % 8;
    z.n = 4 * z.hid + kHead + heads + z.pad;
    const int64_t h = z.hid;
    if (x.size(2) != h || z.M * z.n >= (int64_t(1) << 40) || z.M >= (int64_t(1) << 31) / 2) return false;
    const at::ScalarType wt = w[kQ].scalar_type(), ct = w[kCq].scalar_type();
    if ((wt != at::kFloat && wt != at::kBFloat16) || (ct != at::kFloat && ct != at::kBFloat16)) return false;
    auto is = [&](const Tensor& t, int64_t r, int64_t c, at::ScalarType type) {
        return t.dim() == 2 && t.size(0) == r && t.size(1) == c && t.scalar_type() == type && t.is_contiguous() && on(t, x) &&
               reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
    };
    for (int i : {kQ, kK, kV, kG, kO})
        if (!is(w[i], h, h, wt)) return false;
    if (!is(w[kFa], kHead, h, wt) || !is(w[kFb], h, kHead, wt) || !is(w[kB], heads, h, wt)) return false;
    z.W = w[kCq].dim() == 3 ? w[kCq].size(2) : 0;
    if (z.W < 1 || z.W > 4) return false;
    for (int i : {kCq, kCk, kCv})
        if (w[i].dim() != 3 || w[i].size(0) != h || w[i].size(1) != 1 || w[i].size(2) != z.W || w[i].scalar_type() != ct || !w[i].is_contiguous() || !on(w[i], x))
            return false;
    if (w[kAlog].dim() != 1 || w[kAlog].size(0) != heads || w[kDt].numel() != h || w[kNorm].dim() != 1 || w[kNorm].size(0) != kHead) return false;
    for (int i : {kAlog, kDt})
        if (w[i].scalar_type() != at::kFloat || !w[i].is_contiguous() || !on(w[i], x)) return false;
    if (!on(w[kNorm], x)) return false;
    if (!state.empty()) {
        const int64_t mem[4] = {z.B, heads, kHead, kHead}, win[3] = {z.B, h, z.W};
        if (state.size() != 4 || state[0].sizes() != at::IntArrayRef(mem, 4) || state[0].scalar_type() != at::kFloat || !on(state[0], x)) return false;
        for (int i = 1; i < 4; ++i)
            if (state[i].sizes() != at::IntArrayRef(win, 3) || !on(state[i], x)) return false;
    }
    return !at::autocast::is_autocast_enabled(at::kCUDA);
}

using LayerResult = c10::optional<std::vector<c10::optional<Tensor>>>;

// x [B,T,hidden], the parameters in the order above, state {memory, q, k, v windows} or empty
// -> {y, memory, q, k, v windows} (the last four only when want_state)
LayerResult layer(const Tensor& x_, const std::vector<Tensor>& w, int64_t heads, double eps, double lb, const std::vector<Tensor>& state,
                  bool want_state, bool fuse_conv) {
    Sizes z;
    if (!layer_sizes(x_, w, heads, state, z) || !(lb >= -5.0 && lb < 0.0)) return c10::nullopt;
    bool tracked = torch::autograd::compute_requires_grad(x_);
    for (const auto& t : w) tracked = tracked || torch::autograd::compute_requires_grad(t);
    for (const auto& t : state) tracked = tracked || torch::autograd::compute_requires_grad(t);
    fuse_conv = fuse_conv && !tracked && state.empty() && z.W == 4;
    c10::cuda::CUDAGuard guard(x_.device());
    watch_status(x_.device().index());
    void* st = stream_of(x_);
    const int64_t h = z.hid, M = z.M;
    Tensor x, P, raw, g, beta, qkv, o, mixed, inv, nw, y, ws, mem, win[3], cache[3], h0;
    Packed pk;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        x = dense(x_);
        pk = pack_weights(w, z);
        nw = dense_as(w[kNorm], at::kFloat);
        P = at::mm(x.view({M, h}), pk.p.t());
        raw = at::mm(P.narrow(1, z.fa(), kHead), pk.fb.t());
        if (!fuse_conv) qkv = empty({3, M, h}, at::kBFloat16, x);
        g = empty({M, h}, at::kFloat, x);
        beta = empty({M, heads}, at::kFloat, x);
        mixed = empty({M, h}, at::kBFloat16, x);
        if (tracked) {
            o = empty({z.B, z.T, heads, kHead}, at::kBFloat16, x);
            inv = empty({M * heads}, at::kFloat, x);
        }
        if (want_state) {
            mem = empty({z.B, heads, kHead, kHead}, at::kFloat, x);
            for (auto& t : win) t = empty({z.B, h, z.W}, at::kBFloat16, x);
        }
        if (!state.empty()) {
            h0 = dense(state[0]);
            for (int i = 0; i < 3; ++i) cache[i] = dense_as(state[1 + i], at::kBFloat16);
        }
    }
    // convolutions on their slices of P: one launch; a call that carries windows issues them one by one
    char* q3 = fuse_conv ? nullptr : static_cast<char*>(qkv.data_ptr());
    if (!fuse_conv) {
        const void *xp[3], *wp[3], *cp[3];
        void *yp[3], *fp[3];
        for (int i = 0; i < 3; ++i) {
            xp[i] = at_col(P, i * h);
            wp[i] = w[kCq + i].data_ptr();
            yp[i] = q3 + 2 * i * M * h;
            cp[i] = cache[i].defined() ? cache[i].data_ptr() : nullptr;
            fp[i] = want_state ? win[i].data_ptr() : nullptr;
        }
        const int io = KDA_DTYPE_BF16 | wflag(x, w[kCq]), step = (want_state || !state.empty()) ? 1 : 3;
        for (int i = 0; i < 3; i += step)
            must(kda_conv_fwd_rows(step, (int32_t)z.B, (int32_t)z.T, (int32_t)h, (int32_t)z.W, io, 1, xp + i, (int32_t)z.n, wp + i, cp + i, yp + i, fp + i, st),
                 "kda_conv_fwd_rows");
    }
    must(kda_gate_fwd_rows((int32_t)M, (int32_t)heads, (int32_t)kHead, KDA_DTYPE_BF16, raw.data_ptr(), at_col(P, z.b()), (int32_t)z.n,
                           w[kAlog].data_ptr<float>(), w[kDt].data_ptr<float>(), (float)lb, g.data_ptr<float>(), beta.data_ptr<float>(), st),
         "kda_gate_fwd_rows");
    const KdaChunkShape sh = layer_shape(z, !tracked);
    ws = bytes(kda_chunk_workspace_bytes(&sh), x);
    KdaChunkExtras ex = {};
    ex.gate = at_col(P, 3 * h);
    ex.gate_ld = z.n;
    ex.norm_weight = nw.data_ptr<float>();
    ex.eps = (float)eps;
    ex.y = mixed.data_ptr();
    ex.inv_rms = tracked ? inv.data_ptr<float>() : nullptr;
    const void *qp = q3, *kp = q3 ? q3 + 2 * M * h : nullptr, *vp = q3 ? q3 + 4 * M * h : nullptr;
    if (fuse_conv) {
        qp = at_col(P, 0), kp = at_col(P, h), vp = at_col(P, 2 * h);
        for (int i = 0; i < 3; ++i) ex.conv_weight[i] = w[kCq + i].data_ptr();
        ex.conv_width = 4;
        ex.conv_weight_dtype = dt(w[kCq]);
        ex.x_ld = z.n;
    }
    must(kda_chunk_fwd_ex(&sh, &ex, qp, kp, vp, g.data_ptr(), beta.data_ptr(), h0.defined() ? h0.data_ptr<float>() : nullptr, nullptr,
                          tracked ? o.data_ptr() : nullptr, want_state ? mem.data_ptr<float>() : nullptr, ws.data_ptr(), (size_t)ws.numel(), st),
         "kda_chunk_fwd_ex");
    {
        at::AutoDispatchBelowADInplaceOrView below;
        y = at::mm(mixed, pk.o.t()).view({z.B, z.T, h});
        if (fuse_conv && want_state) {      // windows of the convolutions' inputs: the last W rows, zeros before the first
            const int64_t keep = std::min<int64_t>(z.T, z.W);
            for (int i = 0; i < 3; ++i) {
                const Tensor tail = P.view({z.B, z.T, z.n}).narrow(1, z.T - keep, keep).narrow(2, i * h, h).transpose(1, 2);
                if (keep < z.W) win[i].zero_();
                win[i].narrow(2, z.W - keep, keep).copy_(tail);
            }
        }
    }
    if (tracked) {
        auto node = make_node<LayerNode>();
        torch::autograd::edge_list edges;
        edges.push_back(torch::autograd::impl::gradient_edge(x_));
        for (const auto& t : w) edges.push_back(torch::autograd::impl::gradient_edge(t));
        for (const auto& t : state) edges.push_back(torch::autograd::impl::gradient_edge(t));
        node->set_next_edges(std::move(edges));
        node->z = z;
        node->lb = lb;
        node->wtype = w[kQ].scalar_type();
        node->ntype = w[kNorm].scalar_type();
        node->ctype = w[kCq].scalar_type();
        for (int i = 0; i < 3; ++i) {
            node->cshape[i] = w[kCq + i].sizes().vec();
            if (!state.empty()) node->stype[i] = state[1 + i].scalar_type();
        }
        node->dt_shape = w[kDt].sizes().vec();
        node->has_state = !state.empty();
        const Tensor q = qkv.select(0, 0), k = qkv.select(0, 1), v = qkv.select(0, 2);
        for (const Tensor* t : std::initializer_list<const Tensor*>{&x, &w[kCq], &w[kCk], &w[kCv], &w[kAlog], &w[kDt], &nw, &pk.all, &P, &raw, &g, &beta, &q, &k,
                                                                    &v, &ws, &o, &inv, &mixed})
            node->keep(*t);
        if (!state.empty())
            for (auto& t : cache) node->keep(t);
        torch::autograd::set_history(y, node);
        torch::autograd::set_history(mem, node);
        for (auto& t : win) torch::autograd::set_history(t, node);
    }
    if (!want_state) return std::vector<c10::optional<Tensor>>{y};
    return std::vector<c10::optional<Tensor>>{y, mem, win[0], win[1], win[2]};
}

}  // namespace

void bind_layer(pybind11::module_& m) {
    namespace py = pybind11;
    using nogil = py::call_guard<py::gil_scoped_release>;
    m.def("layer", &layer, nogil());
}

}  // namespace kda_host
