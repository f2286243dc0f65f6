// KimiDeltaAttention as one call each way (head width 128, bf16 activations).
//
// The module's stages one by one cost 65 launches forward and backward at width 768: a cast per weight, a GEMM per
// projection, a GEMM and an addition per input gradient.  Here the six projections of the layer's input are ONE GEMM on
// the weights packed side by side (their casts are one launch), the kernels behind it read and write their slices of the
// projection in place, and the backward forms the gradient of the input as one GEMM over all six and the six weight
// gradients as another, both accumulated in float32.  Columns of the projection P [tokens][n]:
//     q | k | v | output gate (hidden each) | f_a (128) | b (heads) | zero padding to a multiple of 8
// B2 T2045 width 768, forward and backward: 1,141 us and 65 launches -> 406 us and 27.

#include <torch/extension.h>

#include <cmath>
#include <tuple>

#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <cublas_v2.h>

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

char* at_col(char* p, int64_t col) { return p + 2 * col; }

// all weights of the layer's products in bf16: rows of P's matrix, then f_b, then the output projection
size_t packed_bytes(const Sizes& z) { return 2 * (size_t)((z.n + kHead + z.hid) * z.hid); }
char* packed_fb(char* pack, const Sizes& z) { return pack + 2 * z.n * z.hid; }
char* packed_o(char* pack, const Sizes& z) { return pack + 2 * (z.n + kHead) * z.hid; }

void pack_weights(const std::vector<Tensor>& w, const Sizes& z, char* pack, void* st) {
    const int64_t h = z.hid;
    const void* src[9] = {w[kQ].data_ptr(), w[kK].data_ptr(), w[kV].data_ptr(), w[kG].data_ptr(), w[kFa].data_ptr(),
                          w[kB].data_ptr(), nullptr, w[kFb].data_ptr(), w[kO].data_ptr()};
    const int64_t elems[9] = {h * h, h * h, h * h, h * h, kHead * h, z.H * h, z.pad * h, h * kHead, h * h};
    must(kda_pack_bf16(9, dt(w[kQ]), src, elems, pack, st), "kda_pack_bf16");
}

// cuBLAS wants a context on the calling thread; an engine thread that has made no runtime call yet has none
void bind_context(int device) {
    thread_local int bound = -1;
    if (bound == device) return;
    TORCH_CHECK(cudaSetDevice(device) == cudaSuccess, "cudaSetDevice failed");
    bound = device;
}

// torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction, as torch's own products take it; its third setting (no
// split of k either) has no cuBLAS equivalent, and such a layer runs its modules.
cublasMath_t product_math() {
    return at::globalContext().allowBF16ReductionCuBLAS() == at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK
               ? CUBLAS_DEFAULT_MATH
               : CUBLAS_MATH_DISALLOW_REDUCED_PRECISION_REDUCTION;
}

// Row-major products with row strides, bf16 operands and float32 accumulation.  cuBLAS directly: at::mm spends as long in
// dispatch and views as the call itself takes, and these operands are slices.
void gemm(cublasOperation_t ta, cublasOperation_t tb, int64_t m, int64_t n, int64_t k, const void* a, int64_t lda, const void* b, int64_t ldb,
          void* c, int64_t ldc, at::ScalarType ctype) {
    const float one = 1.f, zero = 0.f;
    const cublasHandle_t handle = at::cuda::getCurrentCUDABlasHandle();      // in the default mode, in which it goes back
    const cublasMath_t math = product_math();
    if (math != CUBLAS_DEFAULT_MATH) cublasSetMathMode(handle, math);
    const cublasStatus_t rc = cublasGemmEx(handle, ta, tb, (int)m, (int)n, (int)k, &one, a, CUDA_R_16BF, (int)lda, b,
                                           CUDA_R_16BF, (int)ldb, &zero, c, ctype == at::kFloat ? CUDA_R_32F : CUDA_R_16BF, (int)ldc,
                                           CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT_TENSOR_OP);
    if (math != CUBLAS_DEFAULT_MATH) cublasSetMathMode(handle, CUBLAS_DEFAULT_MATH);
    TORCH_CHECK(rc == CUBLAS_STATUS_SUCCESS, "cublasGemmEx failed (", (int)rc, ")");
}
// y [m][n] = x [m][k] w^T, w [n][k]
void linear(const void* x, int64_t ldx, const void* w, int64_t ldw, void* y, int64_t ldy, int64_t m, int64_t n, int64_t k) {
    gemm(CUBLAS_OP_T, CUBLAS_OP_N, n, m, k, w, ldw, x, ldx, y, ldy, at::kBFloat16);
}
// dx [m][k] = dy [m][n] w
void linear_dx(const void* dy, int64_t ldy, const void* w, int64_t ldw, void* dx, int64_t ldx, int64_t m, int64_t n, int64_t k) {
    gemm(CUBLAS_OP_N, CUBLAS_OP_N, k, m, n, w, ldw, dy, ldy, dx, ldx, at::kBFloat16);
}
// dw [n][k] = dy^T x, in float32 straight from the accumulators when the parameter is float32
Tensor linear_dw(const void* dy, int64_t ldy, const void* x, int64_t ldx, int64_t m, int64_t n, int64_t k, at::ScalarType type, const Tensor& like) {
    Tensor dw = empty({n, k}, type, like);
    gemm(CUBLAS_OP_N, CUBLAS_OP_T, k, n, m, x, ldx, dy, ldy, dw.data_ptr(), k, type);
    return dw;
}

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

// What a forward keeps for its backward, one allocation
struct Kept {
    Slab slab;
    size_t pack, P, raw, g, beta, q, k, v, ws, o, inv, mixed, ws_bytes;
    Kept(const Sizes& z, const KdaChunkShape& sh, bool tracked, bool with_pack, bool with_qkv) {
        const size_t act = 2 * (size_t)(z.M * z.hid);
        pack = slab.take(with_pack ? packed_bytes(z) : 0);
        P = slab.take(2 * (size_t)(z.M * z.n));
        raw = slab.take(act);
        g = slab.take(2 * act);
        beta = slab.take(4 * (size_t)(z.M * z.H));
        q = slab.take(with_qkv ? act : 0);
        k = slab.take(with_qkv ? act : 0);
        v = slab.take(with_qkv ? act : 0);
        mixed = slab.take(act);
        o = slab.take(tracked ? act : 0);
        inv = slab.take(tracked ? 4 * (size_t)(z.M * z.H) : 0);
        ws_bytes = kda_chunk_workspace_bytes(&sh);
        ws = slab.take(ws_bytes);
    }
};

struct LayerNode : public HostNode {
    Sizes z;
    double lb = 0;
    at::ScalarType wtype = at::kFloat, ntype = at::kFloat;
    at::ScalarType ctype = at::kFloat, stype[3] = {at::kFloat, at::kFloat, at::kFloat};
    std::vector<int64_t> cshape[3], dt_shape;
    bool has_state = false;
    std::string name() const override { return "KimiDeltaAttentionBackward"; }
    // saved: x, conv weights, A_log, dt_bias, norm weight, the forward's slab | windows
    enum { sX, sCq, sCk, sCv, sA, sDt, sN, sKept, sWq, sWk, sWv };

    variable_list apply(variable_list&& grads) override {
        std::vector<Tensor> t;
        {
            std::lock_guard<std::mutex> lk(mutex_);
            for (size_t i = 0; i < saved.size(); ++i) t.push_back(get(i));
        }
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor& x = t[sX];
        c10::cuda::CUDAGuard guard(x.device());
        bind_context(x.device().index());
        watch_status(x.device().index());
        void* st = stream_of(x);
        const int64_t h = z.hid, M = z.M, H = z.H, n = z.n;
        const size_t act = 2 * (size_t)(M * h);
        variable_list out(15 + (has_state ? 4 : 0));
        auto want = [&](size_t i) { return task_should_compute_output(i); };
        const KdaChunkShape sh = layer_shape(z, false);
        const Kept kept(z, sh, true, true, true);
        char* base = static_cast<char*>(t[sKept].data_ptr());
        char *pack = base + kept.pack, *P = base + kept.P;

        Slab tmp;      // the backward's temporaries
        const size_t t_dmix = tmp.take(act), t_dP = tmp.take(2 * (size_t)(M * n)), t_do = tmp.take(act), t_dq = tmp.take(3 * act),
                     t_dg = tmp.take(2 * act), t_db = tmp.take(4 * (size_t)(M * H)), t_draw = tmp.take(act);
        const size_t nb_norm = kda_rmsnorm_gate_bwd_scratch_bytes(M * H, (int32_t)kHead), nb_chunk = std::max<size_t>(kda_chunk_bwd_scratch_bytes(&sh), 256),
                     nb_gate = kda_gate_bwd_scratch_bytes((int32_t)M, (int32_t)H, (int32_t)kHead),
                     nb_conv = kda_conv_bwd_multi_scratch_bytes(3, (int32_t)z.B, (int32_t)z.T, (int32_t)h, (int32_t)z.W);
        const size_t t_scr = tmp.take(std::max(std::max(nb_norm, nb_chunk), std::max(nb_gate, nb_conv)));      // one after the other on one stream
        tmp.make(x);
        char *dmix = tmp.at(t_dmix), *dP = tmp.at(t_dP), *dq = tmp.at(t_dq), *draw = tmp.at(t_draw), *scr = tmp.at(t_scr);
        Tensor small = empty({kHead + H + h + 3 * h * z.W}, at::kFloat, x);      // gradients of the vectors and the taps
        float *dnw = small.data_ptr<float>(), *dA = dnw + kHead, *dbias = dA + H, *dcw = dbias + h;

        const Tensor dy = grads[0].defined() ? aligned(dense_as(grads[0], at::kBFloat16)) : at::zeros({M, h}, x.options());
        if (want(1 + kO)) out[1 + kO] = linear_dw(dy.data_ptr(), h, base + kept.mixed, h, M, h, h, wtype, x);
        linear_dx(dy.data_ptr(), h, packed_o(pack, z), h, dmix, h, M, h, h);

        // gated norm: its gate and the gate's gradient are slices of P and dP
        must(kda_rmsnorm_gate_bwd_rows(M * H, KDA_DTYPE_BF16, (int32_t)H, (int32_t)n, base + kept.o, at_col(P, 3 * h), t[sN].data_ptr<float>(),
                                       reinterpret_cast<float*>(base + kept.inv), dmix, tmp.at(t_do), at_col(dP, 3 * h), dnw, scr, nb_norm, st),
             "kda_rmsnorm_gate_bwd_rows");
        const Tensor g_nw = small.narrow(0, 0, kHead);
        out[1 + kNorm] = ntype == at::kFloat ? g_nw : g_nw.to(ntype);

        // chunked operator
        const Tensor dmem = grads[1].defined() ? aligned(dense_as(grads[1], at::kFloat)) : Tensor();
        Tensor dh0;
        if (has_state) dh0 = empty({z.B, H, kHead, kHead}, at::kFloat, x);
        must(kda_chunk_bwd(&sh, base + kept.q, base + kept.k, base + kept.v, base + kept.g, base + kept.beta, nullptr, tmp.at(t_do),
                           dmem.defined() ? dmem.data_ptr<float>() : nullptr, base + kept.ws, kept.ws_bytes, scr, nb_chunk, dq, dq + act, dq + 2 * act,
                           tmp.at(t_dg), tmp.at(t_db), has_state ? dh0.data_ptr<float>() : nullptr, st),
             "kda_chunk_bwd");

        // gate activations, then the low-rank gate projection
        must(kda_gate_bwd_rows((int32_t)M, (int32_t)H, (int32_t)kHead, KDA_DTYPE_BF16, base + kept.raw, at_col(P, z.b()), (int32_t)n, (int32_t)z.pad,
                               t[sA].data_ptr<float>(), t[sDt].data_ptr<float>(), (float)lb, tmp.f32(t_dg), tmp.f32(t_db), draw, at_col(dP, z.b()), dA,
                               dbias, scr, nb_gate, st),
             "kda_gate_bwd_rows");
        out[1 + kAlog] = small.narrow(0, kHead, H);
        out[1 + kDt] = small.narrow(0, kHead + H, h).view(dt_shape);
        if (want(1 + kFb)) out[1 + kFb] = linear_dw(draw, h, at_col(P, z.fa()), n, M, h, kHead, wtype, x);
        linear_dx(draw, h, packed_fb(pack, z), kHead, at_col(dP, z.fa()), n, M, h, kHead);

        // convolutions
        const int io = KDA_DTYPE_BF16 | wflag(x, t[sCq]);
        const bool windows = has_state || grads[2].defined() || grads[3].defined() || grads[4].defined();
        if (!windows) {
            const void *xp[3], *wpt[3], *gp[3];
            void* dp[3];
            float* wg[3];
            for (int i = 0; i < 3; ++i) {
                xp[i] = at_col(P, i * h);
                wpt[i] = t[sCq + i].data_ptr();
                gp[i] = dq + i * act;
                dp[i] = at_col(dP, i * h);
                wg[i] = dcw + i * h * z.W;
            }
            must(kda_conv_bwd_rows(3, (int32_t)z.B, (int32_t)z.T, (int32_t)h, (int32_t)z.W, io, 1, xp, (int32_t)n, wpt, gp, dp, wg, scr, nb_conv, st),
                 "kda_conv_bwd_rows");
        } else {      // windows carried in or out: the general kernel, on dense copies
            const size_t row = 2 * h;
            Tensor xc = empty({M, h}, at::kBFloat16, x), dx = empty({M, h}, at::kBFloat16, x);
            auto copy_rows = [&](void* dst, size_t dld, const void* src, size_t sld) {
                TORCH_CHECK(cudaMemcpy2DAsync(dst, dld, src, sld, row, (size_t)M, cudaMemcpyDeviceToDevice, (cudaStream_t)st) == cudaSuccess,
                            "copying a slice of the projection failed");
            };
            for (int i = 0; i < 3; ++i) {
                copy_rows(xc.data_ptr(), row, at_col(P, i * h), 2 * n);
                const Tensor dfin = grads[2 + i].defined() ? dense_as(grads[2 + i], at::kBFloat16) : Tensor();
                Tensor dinit;
                if (has_state) dinit = empty({z.B, h, z.W}, at::kBFloat16, x);
                must(kda_conv_bwd((int32_t)z.B, (int32_t)z.T, (int32_t)h, (int32_t)z.W, io, 1, xc.data_ptr(), t[sCq + i].data_ptr(),
                                  has_state ? t[sWq + i].data_ptr() : nullptr, dq + i * act, dfin.defined() ? dfin.data_ptr() : nullptr,
                                  dx.data_ptr(), dcw + i * h * z.W, has_state ? dinit.data_ptr() : nullptr, scr, nb_conv, st),
                     "kda_conv_bwd");
                copy_rows(at_col(dP, i * h), 2 * n, dx.data_ptr(), row);
                if (has_state) out[16 + i] = stype[i] == at::kBFloat16 ? dinit : dinit.to(stype[i]);
            }
            if (has_state) out[15] = dh0;
        }
        for (int i = 0; i < 3; ++i) {
            const Tensor d = small.narrow(0, kHead + H + h + i * h * z.W, h * z.W);
            out[1 + kCq + i] = (ctype == at::kFloat ? d : d.to(ctype)).view(cshape[i]);
        }

        // the input and the six weights of P
        if (want(0)) {
            out[0] = empty_as(x);
            linear_dx(dP, n, pack, h, out[0].data_ptr(), h, M, n, h);
        }
        bool any = false;
        for (int i = kQ; i <= kB; ++i) any = any || want(1 + i);
        if (any) {
            const Tensor dW = linear_dw(dP, n, x.data_ptr(), h, M, n, h, wtype, x);
            for (int i = kQ; i <= kG; ++i) out[1 + i] = dW.narrow(0, i * h, h);
            out[1 + kFa] = dW.narrow(0, z.fa(), kHead);
            out[1 + kB] = dW.narrow(0, z.b(), H);
        }
        return out;
    }
};

// ------------------------------------------------------------------------------------------------ forward
// The plain case: bf16 input, 128-wide heads, weights of one type (float32 masters or bf16), everything dense on one GPU.
// A call that passes must not be declined by a kernel any more: what the kernels need aligned is tested here (the
// projections, read as they are) or copied where it is not (the input, the vectors, the taps, the incoming memory), and
// the convolutions' grid limits are tested by fits_grid.
bool layer_sizes(const Tensor& x, const std::vector<Tensor>& w, int64_t heads, const std::vector<Tensor>& state, Sizes& z) {
    if (tracing() || w.size() != kParams || x.dim() != 3 || !x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.numel() == 0 || heads < 1) return false;
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
    return !at::autocast::is_autocast_enabled(at::kCUDA) &&
           at::globalContext().allowBF16ReductionCuBLAS() != at::CuBLASReductionOption::DisallowReducedPrecisionDisallowSplitK;
}

// kda_conv_*_rows: `items` convolutions share a launch whose grid has items x batch and 64-token tiles as its y and z
bool fits_grid(const Sizes& z, int64_t items) { return z.B * items <= 65535 && (z.T + 63) / 64 <= 65535; }

// Rows that one launch of the rows product takes.  A no-grad layer of 16 heads, on the device with a cold L2: 76 us at 8 rows, 80
// at 32 and 94 at 64, through the packed matrix 84, 84 and 88; with 3 heads 54, 57 and 59 against 57.  A token of more
// sequences runs module by module (16 heads, by the host: 83 us at 64 sequences, 292 at 65).
constexpr int64_t kFewRows = 64;

// products of at most kFewRows rows with `count` consecutive weights of the list, straight from the parameters
void few_rows(const std::vector<Tensor>& w, int first, int count, const Sizes& z, const void* x, int64_t ldx, int64_t k, char* out, int64_t ldo,
              const KdaTokenConv* conv, void* st, int32_t flags = 0) {
    const void* wp[6];
    int32_t rows[6];
    for (int i = 0; i < count; ++i) {
        wp[i] = w[first + i].data_ptr();
        rows[i] = (int32_t)w[first + i].size(0);
    }
    must(kda_rows_linear((int32_t)z.M, (int32_t)k, count, dt(w[first]) | flags, x, ldx, wp, rows, out, ldo, conv, st), "kda_rows_linear");
}

using LayerResult = c10::optional<std::vector<c10::optional<Tensor>>>;

// x [B,T,hidden], the parameters in the order above, state {memory, q, k, v windows} or empty
// -> {y, memory, q, k, v windows} (the last four only when want_state)
LayerResult layer(const Tensor& x_, const std::vector<Tensor>& w, int64_t heads, double eps, double lb, const std::vector<Tensor>& state,
                  bool want_state, bool fuse_conv) {
    Sizes z;
    if (!layer_sizes(x_, w, heads, state, z) || !(lb >= -5.0 && lb < 0.0)) return c10::nullopt;
    refuse_tangents(x_, w, state);
    bool tracked = torch::autograd::compute_requires_grad(x_);
    for (const auto& t : w) tracked = tracked || torch::autograd::compute_requires_grad(t);
    for (const auto& t : state) tracked = tracked || torch::autograd::compute_requires_grad(t);
    // One launch for the three convolutions (8,191 x 2,048: 3 x 25 us one by one, 49 at once).  Below 1,024 rows a call that carries
    // windows still issues them one by one, not for speed (77 rows of 384: 72 us, 62 at once): the form with the convolutions inside
    // the forward kernel is defined, and tested, as this one without those three launches.
    const int conv_step = (want_state || !state.empty()) && (z.M < 1024 || !fits_grid(z, 3)) ? 1 : 3;
    if (!fits_grid(z, tracked ? 3 : conv_step)) return c10::nullopt;
    fuse_conv = fuse_conv && !tracked && state.empty() && z.W == 4;
    // without a backward, up to 64 rows go straight to the float32 masters (kda_rows_linear): nothing to pack
    const bool few = !tracked && z.M <= kFewRows;
    c10::cuda::CUDAGuard guard(x_.device());
    watch_status(x_.device().index());
    void* st = stream_of(x_);
    const int64_t h = z.hid, M = z.M, n = z.n;
    const KdaChunkShape sh = layer_shape(z, !tracked);
    Kept kept(z, sh, tracked, !few, !fuse_conv);
    Tensor x, nw, dt_bias, y, mem, win[3], cache[3], h0, taps[3];
    {
        at::AutoDispatchBelowADInplaceOrView below;
        x = aligned(dense(x_));
        nw = aligned(dense_as(w[kNorm], at::kFloat));
        dt_bias = aligned(w[kDt]);
        for (int i = 0; i < 3; ++i) taps[i] = aligned(w[kCq + i]);
        kept.slab.make(x);
        y = empty({z.B, z.T, h}, at::kBFloat16, x);
        if (want_state) {
            mem = empty({z.B, heads, kHead, kHead}, at::kFloat, x);
            for (auto& t : win) t = empty({z.B, h, z.W}, at::kBFloat16, x);
        }
        if (!state.empty()) {
            h0 = aligned(dense(state[0]));
            for (int i = 0; i < 3; ++i) cache[i] = dense_as(state[1 + i], at::kBFloat16);
        }
    }
    const Slab& sl = kept.slab;
    char *P = sl.at(kept.P), *raw = sl.at(kept.raw), *pack = sl.at(kept.pack);
    if (few) {
        few_rows(w, kQ, 6, z, x.data_ptr(), h, h, P, n, nullptr, st);
        few_rows(w, kFb, 1, z, at_col(P, z.fa()), n, kHead, raw, h, nullptr, st, KDA_BEHIND_OWN_LAUNCH);
    } else {
        pack_weights(w, z, pack, st);
        linear(x.data_ptr(), h, pack, h, P, n, M, n, h);
        linear(at_col(P, z.fa()), n, packed_fb(pack, z), kHead, raw, h, M, h, kHead);
    }
    // convolutions on their slices of P
    const char* qkv[3] = {sl.at(kept.q), sl.at(kept.k), sl.at(kept.v)};
    if (!fuse_conv) {
        const void *xp[3], *wp[3], *cp[3];
        void *yp[3], *fp[3];
        for (int i = 0; i < 3; ++i) {
            xp[i] = at_col(P, i * h);
            wp[i] = taps[i].data_ptr();
            yp[i] = const_cast<char*>(qkv[i]);
            cp[i] = cache[i].defined() ? cache[i].data_ptr() : nullptr;
            fp[i] = want_state ? win[i].data_ptr() : nullptr;
        }
        const int io = KDA_DTYPE_BF16 | wflag(x, w[kCq]);
        for (int i = 0; i < 3; i += conv_step)
            must(kda_conv_fwd_rows(conv_step, (int32_t)z.B, (int32_t)z.T, (int32_t)h, (int32_t)z.W, i > 0 ? io | KDA_BESIDE_OWN_LAUNCH : io, 1, xp + i, (int32_t)n, wp + i,
                                   cp + i, yp + i, fp + i, st),
                 "kda_conv_fwd_rows");
    }
    // beside the convolutions: neither needs the other
    must(kda_gate_fwd_rows((int32_t)M, (int32_t)heads, (int32_t)kHead, fuse_conv ? KDA_DTYPE_BF16 : KDA_DTYPE_BF16 | KDA_BESIDE_OWN_LAUNCH, raw, at_col(P, z.b()), (int32_t)n, w[kAlog].data_ptr<float>(),
                           dt_bias.data_ptr<float>(), (float)lb, sl.f32(kept.g), sl.f32(kept.beta), st),
         "kda_gate_fwd_rows");
    KdaChunkExtras ex = {};
    ex.gate = at_col(P, 3 * h);
    ex.gate_ld = n;
    ex.norm_weight = nw.data_ptr<float>();
    ex.eps = (float)eps;
    ex.y = sl.at(kept.mixed);
    ex.inv_rms = tracked ? sl.f32(kept.inv) : nullptr;
    if (fuse_conv) {
        for (int i = 0; i < 3; ++i) {
            qkv[i] = at_col(P, i * h);
            ex.conv_weight[i] = taps[i].data_ptr();
        }
        ex.conv_width = 4;
        ex.conv_weight_dtype = dt(w[kCq]);
        ex.x_ld = n;
    }
    must(kda_chunk_fwd_ex(&sh, &ex, qkv[0], qkv[1], qkv[2], sl.at(kept.g), sl.at(kept.beta), h0.defined() ? h0.data_ptr<float>() : nullptr, nullptr,
                          tracked ? sl.at(kept.o) : nullptr, want_state ? mem.data_ptr<float>() : nullptr, sl.at(kept.ws), kept.ws_bytes, st),
         "kda_chunk_fwd_ex");
    if (few) few_rows(w, kO, 1, z, sl.at(kept.mixed), h, h, static_cast<char*>(y.data_ptr()), h, nullptr, st);
    else linear(sl.at(kept.mixed), h, packed_o(pack, z), h, y.data_ptr(), h, M, h, h);
    if (fuse_conv && want_state) {      // windows of the convolutions' inputs: the last W rows, zeros before the first
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor Pt = at::from_blob(P, {z.B, z.T, n}, x.options());
        const int64_t keep = std::min<int64_t>(z.T, z.W);
        for (int i = 0; i < 3; ++i) {
            if (keep < z.W) win[i].zero_();
            win[i].narrow(2, z.W - keep, keep).copy_(Pt.narrow(1, z.T - keep, keep).narrow(2, i * h, h).transpose(1, 2));
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
        const Tensor all = kept.slab.tensor();
        for (const Tensor* t : std::initializer_list<const Tensor*>{&x, &taps[0], &taps[1], &taps[2], &w[kAlog], &dt_bias, &nw, &all}) node->keep(*t);
        if (!state.empty())
            for (auto& t : cache) node->keep(t);
        torch::autograd::set_history(y, node);
        torch::autograd::set_history(mem, node);
        for (auto& t : win) torch::autograd::set_history(t, node);
    }
    if (!want_state) return std::vector<c10::optional<Tensor>>{y};
    return std::vector<c10::optional<Tensor>>{y, mem, win[0], win[1], win[2]};
}

// ------------------------------------------------------------------------------------------------ one token
// x [B,1,hidden] with B <= 64, no gradients.  in_place: three launches, the state tensors (windows bf16, dense) are
// rewritten -> {y}; otherwise six, into new tensors -> {y, memory, q, k, v windows}.  Both give the same bits.
LayerResult token(const Tensor& x_, const std::vector<Tensor>& w, int64_t heads, double eps, double lb, const std::vector<Tensor>& state, bool in_place) {
    Sizes z;
    if (state.size() != 4 || !layer_sizes(x_, w, heads, state, z) || z.T != 1 || z.M > kFewRows || !(lb >= -5.0 && lb < 0.0)) return c10::nullopt;
    if (!in_place) refuse_tangents(x_, w, state);
    // updated where it lies: bf16 windows, and a memory whose rows are read and written in 16-byte pieces
    if (in_place)
        for (int i = 0; i < 4; ++i)
            if (!state[i].is_contiguous() || (i > 0 ? state[i].scalar_type() != at::kBFloat16 : reinterpret_cast<uintptr_t>(state[i].data_ptr()) % 16 != 0))
                return c10::nullopt;
    at::AutoDispatchBelowADInplaceOrView below;
    c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = aligned(dense(x_)), nw = aligned(dense_as(w[kNorm], at::kFloat));
    void* st = stream_of(x);
    const int64_t h = z.hid, M = z.M, n = z.n;
    const size_t act = 2 * (size_t)(M * h);
    Slab tmp;
    const size_t oP = tmp.take(2 * (size_t)(M * n)), oq = tmp.take(3 * act), omix = tmp.take(act), oraw = tmp.take(in_place ? 0 : act),
                 oo = tmp.take(in_place ? 0 : act), oinv = tmp.take(in_place ? 0 : 4 * (size_t)(M * heads));
    tmp.make(x);
    Tensor y = empty({z.B, 1, h}, at::kBFloat16, x);
    char *P = tmp.at(oP), *q = tmp.at(oq), *mixed = tmp.at(omix);
    const float scale = (float)(1.0 / std::sqrt((double)kHead));
    std::vector<c10::optional<Tensor>> out{y};
    if (in_place) {
        KdaTokenConv cv = {};
        for (int i = 0; i < 3; ++i) {
            cv.weight[i] = w[kCq + i].data_ptr();
            cv.cache[i] = state[1 + i].data_ptr();
        }
        cv.act = q;
        cv.width = (int32_t)z.W;
        cv.weight_dtype = dt(w[kCq]);
        few_rows(w, kQ, 6, z, x.data_ptr(), h, h, P, n, &cv, st);
        must(kda_token_mix((int32_t)M, (int32_t)heads, scale, q, q + act, q + 2 * act, at_col(P, z.fa()), at_col(P, z.b()), at_col(P, 3 * h), n,
                           w[kFb].data_ptr(), dt(w[kFb]) | KDA_BEHIND_OWN_LAUNCH, w[kAlog].data_ptr<float>(), w[kDt].data_ptr<float>(), (float)lb, nw.data_ptr<float>(),
                           (float)eps, state[0].data_ptr<float>(), state[0].data_ptr<float>(), mixed, st),
             "kda_token_mix");
    } else {
        const Tensor mem_in = aligned(dense(state[0])), mem = empty_as(mem_in);
        out.push_back(mem);
        const void *xp[3], *wp[3], *cp[3];
        void *yp[3], *fp[3];
        Tensor cache[3], taps[3];
        for (int i = 0; i < 3; ++i) {
            taps[i] = aligned(w[kCq + i]);
            cache[i] = dense_as(state[1 + i], at::kBFloat16);
            const Tensor win = empty_as(cache[i]);
            out.push_back(win);
            xp[i] = at_col(P, i * h);
            wp[i] = taps[i].data_ptr();
            yp[i] = q + i * act;
            cp[i] = cache[i].data_ptr();
            fp[i] = win.data_ptr();
        }
        few_rows(w, kQ, 6, z, x.data_ptr(), h, h, P, n, nullptr, st);
        must(kda_conv_fwd_rows(3, (int32_t)z.B, 1, (int32_t)h, (int32_t)z.W, KDA_DTYPE_BF16 | wflag(x, w[kCq]), 1, xp, (int32_t)n, wp, cp, yp, fp, st),
             "kda_conv_fwd_rows");
        must(kda_narrow_linear((int32_t)M, (int32_t)h, dt(w[kFb]), at_col(P, z.fa()), n, w[kFb].data_ptr(), tmp.at(oraw), st), "kda_narrow_linear");
        must(kda_decode_step_raw_rows((int32_t)M, (int32_t)heads, (int32_t)kHead, (int32_t)kHead, KDA_DTYPE_BF16, scale, q, q + act, q + 2 * act,
                                      tmp.at(oraw), at_col(P, z.b()), n, w[kAlog].data_ptr<float>(), w[kDt].data_ptr<float>(), (float)lb,
                                      mem_in.data_ptr<float>(), mem.data_ptr<float>(), tmp.at(oo), st),
             "kda_decode_step_raw_rows");
        must(kda_rmsnorm_gate_fwd_rows(M * heads, KDA_DTYPE_BF16, (int32_t)heads, (int32_t)n, (float)eps, tmp.at(oo), at_col(P, 3 * h),
                                       nw.data_ptr<float>(), mixed, tmp.f32(oinv), st),
             "kda_rmsnorm_gate_fwd_rows");
    }
    few_rows(w, kO, 1, z, mixed, h, h, static_cast<char*>(y.data_ptr()), h, nullptr, st, in_place ? KDA_BEHIND_OWN_LAUNCH : 0);
    return out;
}

// The layer's parameters in the order above, or None when a submodule is not the plain one the class built.  A token is three
// launches, and these few dozen lookups as Python statements took as long as two of them.  plain: ((name, class), ...), the
// norm last; types: what a parameter's type may be.
pybind11::object plain_weights(const pybind11::dict& modules, const pybind11::dict& own, const pybind11::tuple& plain, const pybind11::tuple& types) {
    namespace py = pybind11;
    static PyObject* const hooks[4] = {PyUnicode_InternFromString("_forward_hooks"), PyUnicode_InternFromString("_forward_pre_hooks"),
                                       PyUnicode_InternFromString("_backward_hooks"), PyUnicode_InternFromString("_backward_pre_hooks")};
    static PyObject *const s_forward = PyUnicode_InternFromString("forward"), *const s_params = PyUnicode_InternFromString("_parameters"),
                    *const s_bias = PyUnicode_InternFromString("bias"), *const s_weight = PyUnicode_InternFromString("weight"),
                    *const s_A = PyUnicode_InternFromString("A_log"), *const s_dt = PyUnicode_InternFromString("dt_bias");
    py::list out;
    bool ok = true;
    auto add = [&](PyObject* w) {
        if (w != nullptr && (reinterpret_cast<PyObject*>(Py_TYPE(w)) == types[0].ptr() || reinterpret_cast<PyObject*>(Py_TYPE(w)) == types[1].ptr()))
            out.append(py::handle(w));
        else ok = false;
    };
    const py::ssize_t n = PyTuple_GET_SIZE(plain.ptr());
    for (py::ssize_t i = 0; i < n && ok; ++i) {
        if (i == n - 1) {
            add(PyDict_GetItem(own.ptr(), s_A));
            add(PyDict_GetItem(own.ptr(), s_dt));
        }
        PyObject* const item = PyTuple_GET_ITEM(plain.ptr(), i);
        PyObject* const m = PyDict_GetItem(modules.ptr(), PyTuple_GET_ITEM(item, 0));
        if (m == nullptr || reinterpret_cast<PyObject*>(Py_TYPE(m)) != PyTuple_GET_ITEM(item, 1)) return py::none();
        const py::object d = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(m, nullptr));
        if (!d) throw py::error_already_set();
        for (PyObject* h : hooks) {
            PyObject* const v = PyDict_GetItem(d.ptr(), h);
            if (v == nullptr || PyObject_Size(v) != 0) return py::none();
        }
        PyObject* const params = PyDict_GetItem(d.ptr(), s_params);
        if (params == nullptr || !PyDict_Check(params) || PyDict_GetItem(d.ptr(), s_forward) != nullptr) return py::none();
        PyObject* const bias = PyDict_GetItem(params, s_bias);
        if (bias != nullptr && bias != Py_None) return py::none();
        add(PyDict_GetItem(params, s_weight));
    }
    return ok ? py::object(out) : py::none();
}

}  // namespace

void bind_layer(pybind11::module_& m) {
    namespace py = pybind11;
    using nogil = py::call_guard<py::gil_scoped_release>;
    m.def("layer", &layer, nogil());
    m.def("token", &token, nogil());
    m.def("plain_weights", &plain_weights);
    m.def("product_math", [] { return (int)product_math(); });      // the mode the layer's products would run in now
}

}  // namespace kda_host
