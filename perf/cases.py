"""The work this package is used for, as cases a timing program can run: decoding, prefill and training through the
layer, the operators on activated inputs, the registered `torch.ops.nanochat_kda.*` operators and the bandwidth
modules on their own.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call: inputs, modules, decode state
    run(state)          one pass through the public entry points; returns every output
    work(case)          bytes and floating-point operations a pass cannot do without
    tolerance(case)     how far another correct implementation of the same precision may be off
"""

import math
import random

import torch

import experiment_swa_kda_b200 as m

DEVICE = "cuda:0"
HEAD = 128          # head width of every layer case (the width the reference trains with)
WIDTH = 4           # taps of the short convolutions


def listed():
    return [
        # one new token of one conversation through a layer of the reference's 384-wide model: the latency of serving
        {"name": "token_b1_h3", "kind": "token", "batch": 1, "heads": 3},
        # one new token of a serving batch through a 2048-wide layer
        {"name": "token_b32_h16", "kind": "token", "batch": 32, "heads": 16},
        # the decode operator alone at the large serving batch: 256 MiB of float32 state read and 256 MiB written
        {"name": "step_b256_h16", "kind": "step", "batch": 256, "heads": 16, "dim": 128, "dtype": "bf16"},
        # a short prompt (ragged last chunk) through a layer, without gradients, keeping the decode state
        {"name": "prefill_t77_h3", "kind": "prefill", "batch": 1, "seq": 77, "heads": 3},
        # a long prompt through a 2048-wide layer
        {"name": "prefill_t8191_h16", "kind": "prefill", "batch": 1, "seq": 8191, "heads": 16},
        # the float32 verification shape: operator forward and backward with the final state
        {"name": "chunk_f32_t256_d64", "kind": "chunk", "batch": 1, "seq": 256, "heads": 2, "dim": 64, "dtype": "f32", "docs": 0, "state": False},
        # 64-wide heads in bf16, an odd length, states carried in and out (truncated back-propagation through time)
        {"name": "chunk_bf16_t2047_d64", "kind": "chunk", "batch": 2, "seq": 2047, "heads": 6, "dim": 64, "dtype": "bf16", "docs": 0, "state": True},
        # packed documents, 16 heads, an initial state for every document: the large training batch
        {"name": "packed_t65536_h16", "kind": "chunk", "batch": 1, "seq": 65536, "heads": 16, "dim": 128, "dtype": "bf16", "docs": 22, "state": True},
        # convolutions -> chunked operator -> gated norm, forward and backward: the benchmark's training step
        {"name": "chain_b2_t4096_h3", "kind": "chain", "batch": 2, "seq": 4096, "heads": 3},
        # the same mixer the way the reference's model calls it: the registered operators under its own autograd functions
        {"name": "ops_b2_t4096_h3", "kind": "ops", "batch": 2, "seq": 4096, "heads": 3},
        # a training step of the whole layer, projections and every parameter gradient included, at an odd length
        {"name": "layer_b2_t2045_h6", "kind": "layer", "batch": 2, "seq": 2045, "heads": 6},
        # the bandwidth modules on their own at a size that does not fit in L2: convolution and gated norm, both directions
        {"name": "pointwise_t65536_c2048", "kind": "pointwise", "batch": 1, "seq": 65536, "heads": 16},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(("token", "step", "prefill", "chunk", "chunk", "general", "chain", "ops", "layer", "pointwise"))
    heads = rng.choice((1, 2, 3, 4, 6, 8, 12, 16))
    if kind == "token":
        return {"kind": kind, "batch": _log_int(rng, 1, 64), "heads": heads}
    if kind == "step":
        return {"kind": kind, "batch": _log_int(rng, 1, 256), "heads": heads, "dim": rng.choice((64, 128, 128)),
                "dtype": rng.choice(("bf16", "bf16", "f32"))}
    if kind == "general":
        # every head width and type that is not bf16 at width 128
        dtype = rng.choice(("f32", "bf16"))
        dim = rng.choice((32, 64, 128)) if dtype == "f32" else rng.choice((32, 64, 96))
        heads, batch = min(heads, 8), rng.randint(1, 3)
        most = min(4096, 2 * 2047 * 6 * 64 * 64 // (batch * heads * max(dim, 64) ** 2))
        return {"kind": "chunk", "batch": batch, "seq": _log_int(rng, 32, most), "heads": heads, "dim": dim, "dtype": dtype, "docs": 0,
                "state": rng.random() < 0.5}
    if kind == "chunk":
        if rng.random() < 0.5:
            seq = _log_int(rng, 512, 65536)
            return {"kind": kind, "batch": 1, "seq": seq, "heads": heads, "dim": 128, "dtype": "bf16",
                    "docs": rng.randint(2, max(2, min(48, seq // 256))), "state": rng.random() < 0.5}
        return {"kind": kind, "batch": rng.randint(1, 4), "seq": _log_int(rng, 48, 8192), "heads": heads, "dim": 128, "dtype": "bf16", "docs": 0,
                "state": rng.random() < 0.5}
    batch = rng.randint(1, 4)
    if kind == "prefill":
        return {"kind": kind, "batch": batch, "seq": _log_int(rng, 16, 8192 // batch), "heads": heads}
    if kind == "pointwise":
        return {"kind": kind, "batch": batch, "seq": _log_int(rng, 64, 65536 // batch), "heads": heads}
    return {"kind": kind, "batch": batch, "seq": _log_int(rng, 64, 49152 // (batch * heads)), "heads": heads}


# ----------------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------------
class _Source:
    """Seeded inputs of the benchmark's distributions, drawn on the device."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEVICE).manual_seed(seed)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.gen, device=DEVICE)

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, generator=self.gen, device=DEVICE) * (hi - lo) + lo

    def unit(self, *shape):
        t = self.normal(*shape)
        return t / t.norm(dim=-1, keepdim=True)

    def decay(self, *shape):
        return (-torch.nn.functional.softplus(self.normal(*shape)) * 0.1).clamp(-5, 0)

    def beta(self, *shape):
        return torch.sigmoid(self.normal(*shape))


def _lengths(docs, total, seed):
    """`docs` document lengths in the proportions of uniform draws from [256, 8192], summing to `total`."""
    rng = random.Random(seed)
    w = [rng.uniform(256, 8192) for _ in range(docs)]
    out = [int(x / sum(w) * total) for x in w]
    out[-1] += total - sum(out)
    return out


def _layer(src, heads):
    """A layer with float32 master weights in the reference's initial scale and a spread of decay rates."""
    hidden = heads * HEAD
    layer = m.KimiDeltaAttention(hidden_size=hidden, num_heads=heads, head_dim=HEAD, conv_size=WIDTH, norm_eps=1e-6).to(DEVICE)
    with torch.no_grad():
        for name, p in layer.named_parameters():
            if name == "A_log":
                p.copy_(0.3 * src.normal(*p.shape))
            elif name == "dt_bias":
                p.copy_(src.uniform(-6.0, 0.0, *p.shape))
            elif name == "o_norm.weight":
                p.copy_(src.uniform(0.5, 1.5, *p.shape))
            elif "conv1d" in name:
                bound = WIDTH ** -0.5
                p.copy_(src.uniform(-bound, bound, *p.shape))
            else:
                bound = (3.0 / p.shape[1]) ** 0.5
                p.copy_(src.uniform(-bound, bound, *p.shape))
    return layer


def _chain_inputs(case, src):
    B, T, H = case["batch"], case["seq"], case["heads"]
    bf = torch.bfloat16
    bound = WIDTH ** -0.5
    return {
        "x": [src.normal(B, T, H * HEAD).to(bf).requires_grad_(True) for _ in range(3)],
        "gate": src.normal(B, T, H, HEAD).to(bf).requires_grad_(True),
        "probe": src.normal(B, T, H, HEAD).to(bf),
        "conv_w": [src.uniform(-bound, bound, H * HEAD, WIDTH) for _ in range(3)],
        "norm_w": src.uniform(0.5, 1.5, HEAD),
    }


def _conv(weight):
    conv = m.ShortConvolution(weight.shape[0], weight.shape[1]).to(DEVICE)
    with torch.no_grad():
        conv.weight.copy_(weight.unsqueeze(1))
    return conv


def _norm(weight):
    norm = m.RMSNormGated(weight.shape[0], eps=1e-6).to(DEVICE)
    with torch.no_grad():
        norm.weight.copy_(weight)
    return norm


def _operator_functions():
    """Autograd functions that save the operator inputs and the forward output and call the registered operators, as the
    reference's mixer does."""
    from experiment_swa_kda_b200 import nanochat_ops
    nanochat_ops.register()
    ops = torch.ops.nanochat_kda

    class Conv(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x, w):
            y, _ = ops.causal_convolution_forward(x, w, None, False)
            ctx.save_for_backward(x, w, y)
            return y

        @staticmethod
        def backward(ctx, dy):
            x, w, y = ctx.saved_tensors
            dx, dw, _ = ops.causal_convolution_backward(x, w, None, y, None, dy, None)
            return dx, dw

    class Chunk(torch.autograd.Function):
        @staticmethod
        def forward(ctx, q, k, v, raw, bl, A_log, dt_bias, scale):
            o, _ = ops.chunk_forward(q, k, v, raw, bl, A_log, dt_bias, None, False, -5.0, scale)
            ctx.scale = scale
            ctx.save_for_backward(q, k, v, raw, bl, A_log, dt_bias, o)
            return o

        @staticmethod
        def backward(ctx, do):
            q, k, v, raw, bl, A_log, dt_bias, o = ctx.saved_tensors
            g = ops.chunk_backward(q, k, v, raw, bl, A_log, dt_bias, None, o, None, do, None, -5.0, ctx.scale)
            return (*g[:7], None)

    class Norm(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x, gate, w, eps):
            y, inv = ops.rmsnorm_gate_forward(x, gate, w, eps)
            ctx.eps = eps
            ctx.save_for_backward(x, gate, w, inv)
            return y

        @staticmethod
        def backward(ctx, dy):
            x, gate, w, inv = ctx.saved_tensors
            return (*ops.rmsnorm_gate_backward(x, gate, w, inv, dy, ctx.eps), None)

    return Conv, Chunk, Norm


def prepare(case, seed):
    src, kind = _Source(seed), case["kind"]
    bf = torch.bfloat16
    H = case["heads"]
    s = {"case": dict(case)}
    if kind == "token":
        s["layer"] = _layer(src, H)
        s["x"] = src.normal(case["batch"], 1, H * HEAD).to(bf)
        st = m.KDAState.zeros(case["batch"], H, HEAD, WIDTH, DEVICE)
        st.memory.copy_(0.02 * src.normal(*st.memory.shape))
        for c in (st.q_conv, st.k_conv, st.v_conv):
            c.copy_(src.normal(*c.shape))
        s["decode"] = st
    elif kind == "step":
        B, D, dt = case["batch"], case["dim"], bf if case["dtype"] == "bf16" else torch.float32
        s["in"] = [src.unit(B, 1, H, D).to(dt), src.unit(B, 1, H, D).to(dt), src.normal(B, 1, H, D).to(dt), src.decay(B, 1, H, D).to(dt),
                   src.beta(B, 1, H).to(dt)]
        s["state"] = 0.02 * src.normal(B, H, D, D)
    elif kind in ("prefill", "layer"):
        s["layer"] = _layer(src, H)
        s["x"] = src.normal(case["batch"], case["seq"], H * HEAD).to(bf)
        if kind == "layer":
            s["x"].requires_grad_(True)
            s["leaves"] = [s["x"]] + [p for _, p in s["layer"].named_parameters()]
            s["probe"] = src.normal(*s["x"].shape).to(bf)
    elif kind == "chunk":
        B, T, D, dt = case["batch"], case["seq"], case["dim"], bf if case["dtype"] == "bf16" else torch.float32
        x = [src.unit(B, T, H, D).to(dt), src.unit(B, T, H, D).to(dt), src.normal(B, T, H, D).to(dt), src.decay(B, T, H, D).to(dt),
             src.beta(B, T, H).to(dt)]
        s["in"] = [t.requires_grad_(True) for t in x]
        n = B
        s["cu"] = None
        if case["docs"]:
            ends = [0]
            for length in _lengths(case["docs"], T, seed):
                ends.append(ends[-1] + length)
            s["cu"], n = torch.tensor(ends, dtype=torch.int32, device=DEVICE), case["docs"]
        s["h0"] = (0.02 * src.normal(n, H, D, D)).requires_grad_(True) if case["state"] else None
        s["probe"] = src.normal(B, T, H, D).to(dt)
        s["probe_state"] = src.normal(n, H, D, D)
    elif kind == "chain":
        s.update(_chain_inputs(case, src))
        B, T = case["batch"], case["seq"]
        s["g"] = src.decay(B, T, H, HEAD).to(bf).requires_grad_(True)
        s["beta"] = src.beta(B, T, H).to(bf).requires_grad_(True)
        s["convs"], s["norm"] = [_conv(w) for w in s["conv_w"]], _norm(s["norm_w"])
        s["leaves"] = [*s["x"], s["g"], s["beta"], s["gate"], *[c.weight for c in s["convs"]], s["norm"].weight]
    elif kind == "ops":
        s.update(_chain_inputs(case, src))
        B, T = case["batch"], case["seq"]
        s["functions"] = _operator_functions()
        p = (src.decay(B, T, H, HEAD) / -5.0).clamp(1e-4, 1 - 1e-4)
        s["raw"] = (torch.log(p) - torch.log1p(-p)).to(bf).requires_grad_(True)
        s["bl"] = src.normal(B, T, H).to(bf).requires_grad_(True)
        s["A_log"] = (0.1 * src.normal(H)).requires_grad_(True)
        s["dt_bias"] = (0.1 * src.normal(H * HEAD)).requires_grad_(True)
        s["w"] = [w.to(bf).requires_grad_(True) for w in s["conv_w"]]
        s["nw"] = s["norm_w"].clone().requires_grad_(True)
        s["leaves"] = [*s["x"], s["raw"], s["bl"], s["gate"], *s["w"], s["nw"], s["A_log"], s["dt_bias"]]
    else:
        B, T = case["batch"], case["seq"]
        bound = WIDTH ** -0.5
        s["conv"] = _conv(src.uniform(-bound, bound, H * HEAD, WIDTH))
        s["norm"] = _norm(src.uniform(0.5, 1.5, HEAD))
        s["x"] = src.normal(B, T, H * HEAD).to(bf).requires_grad_(True)
        s["o"], s["gate"] = (src.normal(B, T, H, HEAD).to(bf).requires_grad_(True) for _ in range(2))
        s["dy"] = src.normal(B, T, H * HEAD).to(bf)
        s["dn"] = src.normal(B, T, H, HEAD).to(bf)
    return s


# ----------------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "token":
        st = s["decode"]
        y = s["layer"].decode_token(s["x"], st)
        return [y, st.memory, st.q_conv, st.k_conv, st.v_conv]
    if kind == "step":
        with torch.no_grad():
            return m.recurrent_kda_step(*s["in"], s["state"])
    if kind == "prefill":
        with torch.no_grad():
            y, st = s["layer"](s["x"], output_final_state=True)
        return [y, st.memory, st.q_conv, st.k_conv, st.v_conv]
    if kind == "layer":
        y, _ = s["layer"](s["x"])
        return [y, *torch.autograd.grad(y, s["leaves"], s["probe"])]
    if kind == "chunk":
        q, k, v, g, beta = s["in"]
        o, fs = m.chunk_kda(q, k, v, g, beta, initial_state=s["h0"], output_final_state=True, cu_seqlens=s["cu"])
        leaves = [*s["in"]] + ([s["h0"]] if s["h0"] is not None else [])
        if case["state"]:
            return [o, fs, *torch.autograd.grad((o, fs), leaves, (s["probe"], s["probe_state"]))]
        return [o, fs, *torch.autograd.grad(o, leaves, s["probe"])]
    shape4 = (case["batch"], case["seq"], case["heads"], HEAD)
    if kind == "chain":
        q, k, v = (t.view(shape4) for t in m.short_convolutions(s["convs"], s["x"]))
        y, _ = m.chunk_kda_norm(q, k, v, s["g"], s["beta"], s["gate"], s["norm"].weight, eps=1e-6)
        return [y, *torch.autograd.grad(y, s["leaves"], s["probe"])]
    if kind == "ops":
        conv, chunk, norm = s["functions"]
        q, k, v = (conv.apply(x, w).view(shape4) for x, w in zip(s["x"], s["w"]))
        o = chunk.apply(q, k, v, s["raw"], s["bl"], s["A_log"], s["dt_bias"], HEAD ** -0.5)
        y = norm.apply(o, s["gate"], s["nw"], 1e-6)
        return [y, *torch.autograd.grad(y, s["leaves"], s["probe"])]
    yc, _ = s["conv"](s["x"])
    yn = s["norm"](s["o"], s["gate"])
    leaves = [s["x"], s["conv"].weight, s["o"], s["gate"], s["norm"].weight]
    return [yc, yn, *torch.autograd.grad((yc, yn), leaves, (s["dy"], s["dn"]))]


# ----------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------
def _chunk_macs(dim, chunk=64):
    """Multiply-adds of the chunked forward per token and head, triangular products at triangular cost."""
    tri, stri = chunk * (chunk + 1) / 2, chunk * (chunk - 1) / 2
    total = (tri + stri) * dim + chunk ** 3 / 6 + 2 * tri * dim + 3 * chunk * dim * dim + tri * dim
    return total / chunk


def work(case):
    kind, B, H = case["kind"], case["batch"], case["heads"]
    D = case.get("dim", HEAD)
    io = 4 if case.get("dtype") == "f32" else 2
    hidden = H * D
    state = B * H * D * D * 4
    weights = 5 * hidden * hidden + 2 * hidden * HEAD + hidden * H        # q, k, v, gate, output; the low-rank decay gate; beta
    if kind == "step":
        return {"bytes": 2 * state + B * H * (5 * D + 1) * io, "flops": 7.0 * B * H * D * D}
    if kind == "token":
        return {"bytes": 2 * state + 4 * weights + 2 * 3 * B * hidden * WIDTH * 2 + 2 * B * hidden * 2,
                "flops": 2.0 * B * weights + 7.0 * B * H * D * D}
    T = case["seq"]
    n = B * T * hidden                     # elements of one activation tensor
    macs = B * T * H * _chunk_macs(D)
    if kind == "prefill":
        return {"bytes": 2 * n * 2 + 4 * weights + state, "flops": 2.0 * B * T * weights + 2.0 * macs}
    if kind == "layer":
        return {"bytes": 4 * n * 2 + 2 * 4 * weights, "flops": 3 * (2.0 * B * T * weights + 2.0 * macs)}
    if kind == "chunk":
        states = (case["docs"] or B) * H * D * D * 4
        moved = (2 if not case["state"] else 4) * states
        return {"bytes": 10 * n * io + 2 * B * T * H * io + moved, "flops": 3 * 2.0 * macs}
    if kind in ("chain", "ops"):
        # x_q, x_k, x_v, decay, gate, dy read; y and the five gradients written
        return {"bytes": 12 * n * 2, "flops": 3 * 2.0 * macs + 3 * 24.0 * n + 40.0 * n}
    # convolution: x, dy read, y, dx written; norm: x, gate, dy read, y, dx, dgate written
    return {"bytes": 10 * n * 2, "flops": 3 * 8.0 * n + 40.0 * n}


def tolerance(case):
    if case.get("dtype") == "f32":
        return {"rel": 1e-5}
    if case["kind"] in ("layer", "prefill", "ops"):
        return {"rel": 2e-2}               # bf16 products in series, and gate parameters that are sums of cancelling terms
    return {"rel": 1e-2}
