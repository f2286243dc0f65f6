"""GPU parity for the bandwidth kernels: convolution, gated RMSNorm, gate activations."""

import os

import numpy as np
import pytest
import torch

import kda_oracle as O

pytestmark = pytest.mark.gpu
D0 = "cuda:0"

CONV_TAGS = ["t9", "t9s", "t2s", "t4", "t70s", "t5w3"]


def _conv_mod(C, W, w):
    from experiment_swa_kda_b200 import ShortConvolution
    mod = ShortConvolution(C, W).to(D0)
    with torch.no_grad():
        mod.weight.copy_(w.unsqueeze(1))
    return mod


@pytest.mark.parametrize("tag", CONV_TAGS)
def test_conv_fp32_matches_reference_vectors(golden_dir, tag):
    z = np.load(os.path.join(golden_dir, "conv.npz"))
    g = lambda n: torch.from_numpy(z[f"{tag}_{n}"])
    x = g("x").to(D0).requires_grad_(True)
    w = g("w")
    has_state = f"{tag}_s0" in z.files
    s0 = g("s0").to(D0).requires_grad_(True) if has_state else None
    mod = _conv_mod(w.shape[0], w.shape[1], w.to(D0))
    y, fs = mod(x, s0, output_final_state=True)
    torch.testing.assert_close(y.cpu(), g("y"), atol=2e-6, rtol=1e-5)
    assert torch.equal(fs.cpu(), g("fs"))
    leaves = [x, mod.weight] + ([s0] if has_state else [])
    grads = torch.autograd.grad((y, fs), leaves, (g("cy").to(D0), g("cs").to(D0)))
    torch.testing.assert_close(grads[0].cpu(), g("dx"), atol=1e-5, rtol=1e-5)
    torch.testing.assert_close(grads[1].squeeze(1).cpu(), g("dw"), atol=1e-4, rtol=1e-5)
    if has_state:
        torch.testing.assert_close(grads[2].cpu(), g("ds0"), atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("B,T,C,state", [(2, 4096, 384, False), (2, 257, 384, True), (1, 3, 384, True), (3, 100, 20, True)])
def test_conv_bf16_matches_oracle(B, T, C, state):
    gen = torch.Generator().manual_seed(T + C)
    x = torch.randn(B, T, C, generator=gen).bfloat16()
    w = (torch.rand(C, 4, generator=gen) * 2 - 1) * (3 ** 0.5) * C ** -0.5
    s0 = torch.randn(B, C, 4, generator=gen).bfloat16() if state else None
    mod = _conv_mod(C, 4, w.to(D0))
    xd = x.to(D0).requires_grad_(True)
    sd = s0.to(D0).requires_grad_(True) if state else None
    y, fs = mod(xd, sd, output_final_state=True)
    xe = x.float().requires_grad_(True)
    we = w.bfloat16().float().requires_grad_(True)     # the module casts its weight to the activation dtype
    se = s0.float().requires_grad_(True) if state else None
    ye, fse = O.causal_conv(xe, we, initial_state=se)
    cy = torch.randn(ye.shape, generator=gen).bfloat16()
    cs = torch.randn(fse.shape, generator=gen).bfloat16()
    assert O.rel_l2(y.float(), ye) <= 1e-2 and torch.equal(fs.float().cpu(), fse.detach())
    leaves = [xd, mod.weight] + ([sd] if state else [])
    got = torch.autograd.grad((y, fs), leaves, (cy.to(D0), cs.to(D0)))
    want = torch.autograd.grad((ye, fse), [xe, we] + ([se] if state else []), (cy.float(), cs.float()))
    assert O.rel_l2(got[0].float(), want[0]) <= 1e-2
    assert O.rel_l2(got[1].squeeze(1).float(), want[1]) <= 1e-2
    if state:
        assert O.rel_l2(got[2].float(), want[2]) <= 1e-2


@pytest.mark.parametrize("B,T,C,dtype", [(2, 4096, 384, torch.bfloat16), (1, 100, 20, torch.bfloat16), (2, 67, 384, torch.float32),
                                         (3, 1, 64, torch.float32), (1, 5, 130, torch.bfloat16), (2, 129, 72, torch.float32),
                                         # bf16 with C % 128 == 0: small sizes stay on the tile kernel, large ones take the
                                         # streaming backward (32 and 64 tokens per thread run), all with ragged ends
                                         (1, 1, 128, torch.bfloat16), (2, 3, 256, torch.bfloat16), (3, 67, 128, torch.bfloat16),
                                         (2, 1031, 1024, torch.bfloat16), (2, 4099, 2048, torch.bfloat16),
                                         (1, 30001, 2048, torch.bfloat16)])
def test_conv_training_path_matches_oracle(B, T, C, dtype):
    """No carried-in window, no final state: the tiled forward / backward kernels (ragged T and C tails included)."""
    gen = torch.Generator().manual_seed(T * 7 + C)
    x = torch.randn(B, T, C, generator=gen).to(dtype)
    w = (torch.rand(C, 4, generator=gen) * 2 - 1) * (3 ** 0.5) * C ** -0.5
    mod = _conv_mod(C, 4, w.to(D0))
    xd = x.to(D0).requires_grad_(True)
    y, fs = mod(xd)
    assert fs is None
    xe = x.float().requires_grad_(True)
    we = (w.to(dtype).float() if dtype == torch.bfloat16 else w.clone()).requires_grad_(True)
    ye, _ = O.causal_conv(xe, we)
    cy = torch.randn(ye.shape, generator=gen).to(dtype)
    got = torch.autograd.grad(y, [xd, mod.weight], cy.to(D0))
    want = torch.autograd.grad(ye, [xe, we], cy.float())
    tol = 1e-2 if dtype == torch.bfloat16 else 1e-5
    assert O.rel_l2(y.float(), ye) <= tol
    assert O.rel_l2(got[0].float(), want[0]) <= tol
    assert O.rel_l2(got[1].squeeze(1).float(), want[1]) <= tol


def _forward_kernels(call):
    """Which forward convolution kernels a call launches: {"conv_fwd_stream_kernel"} or {"conv_fwd_kernel"}."""
    from experiment_swa_kda_b200 import _lib
    torch.cuda.synchronize()
    _lib.profile_report()
    _lib.profile(True)
    try:
        call()
    finally:
        _lib.profile(False)
    return {name for name in _lib.profile_report() if name.startswith("conv_fwd")}


# ends within a group of 8 rows, a run of 32, a block; sequences that fill their last block by half or more; every window width
@pytest.mark.parametrize("W,B,T,C", [(4, 1, 28423, 2048), (4, 1, 3549, 2048), (2, 1, 28417, 2048), (2, 222, 229, 128), (3, 111, 511, 1024), (4, 888, 133, 128),
                                     (1, 888, 161, 128), (4, 444, 197, 256)])
def test_streaming_convolution_equals_short_pieces(W, B, T, C):
    """Both kernels sum a window in the same order, so the long call equals calls on pieces of it to the bit."""
    gen = torch.Generator(device=D0).manual_seed(T + W)
    x = torch.randn(B, T, C, device=D0, generator=gen).bfloat16()
    mod = _conv_mod(C, W, torch.randn(C, W, device=D0, generator=gen))
    out = []
    with torch.no_grad():
        assert _forward_kernels(lambda: out.append(mod(x)[0])) == {"conv_fwd_stream_kernel"}
        for b in sorted({0, B // 2, B - 1}):
            for t0 in range(0, T, 2048):
                h = min(t0, W - 1)
                piece = x[b:b + 1, t0 - h:t0 + 2048].contiguous()
                assert _forward_kernels(lambda: out.append(mod(piece)[0])) == {"conv_fwd_kernel"}
                assert torch.equal(out[0][b, t0:t0 + 2048], out.pop()[0, h:])


# Either side of every line of the forward's dispatch: blocks of 256 tokens x 128 channels, how well a sequence fills its own, windows
# carried out
@pytest.mark.parametrize("n,B,T,C,W,windows,streams", [(3, 1, 1024, 2048, 4, False, False), (3, 1, 1281, 2048, 4, False, True), (1, 221, 256, 128, 4, False, False),
                                                       (1, 222, 205, 128, 4, False, True), (1, 222, 204, 128, 4, False, False), (1, 888, 128, 128, 4, False, True),
                                                       (1, 888, 127, 128, 4, False, False), (1, 887, 128, 128, 3, False, False), (1, 295, 256, 128, 4, True, False),
                                                       (1, 296, 256, 128, 4, True, True), (1, 221, 8, 128, 4, True, False), (1, 222, 8, 128, 4, True, True),
                                                       (1, 222, 9, 128, 4, True, False), (1, 1777, 1, 128, 4, True, False), (1, 1776, 1, 128, 4, True, True),
                                                       (1, 296, 8, 128, 4, False, False)])
def test_the_forward_kernel_by_size(n, B, T, C, W, windows, streams):
    import ctypes
    from experiment_swa_kda_b200 import _lib
    lib = _lib.load()
    xs, ws = [torch.randn(B, T, C, device=D0).bfloat16() for _ in range(n)], [torch.randn(C, W, device=D0) for _ in range(n)]
    ys, fins = [torch.empty_like(x) for x in xs], [torch.empty(B, C, W, device=D0, dtype=torch.bfloat16) for _ in range(n)]
    arr = lambda ts: ctypes.cast((ctypes.c_void_p * n)(*[t.data_ptr() for t in ts]), ctypes.c_void_p)
    a = [arr(ts) for ts in (xs, ws, ys, fins)]
    call = lambda: _lib.check(lib.kda_conv_fwd_rows(n, B, T, C, W, _lib.DTYPE_BF16 | 0x100, 1, a[0], C, a[1], None, a[2], a[3] if windows else None,
                                                    torch.cuda.current_stream().cuda_stream), "forward")
    assert _forward_kernels(call) == {"conv_fwd_stream_kernel" if streams else "conv_fwd_kernel"}


# 2,048 channels: 36 blocks of 64 tokens take the tile kernel, 37 the streaming one, both with ragged ends
@pytest.mark.parametrize("T", [36 * 64 - 1, 36 * 64 + 1])
def test_conv_backward_either_side_of_the_streaming_line(T):
    test_conv_training_path_matches_oracle(1, T, 2048, torch.bfloat16)


# the even, the odd (one channel a thread) and the final-state paths each end in the reduction that rounds
@pytest.mark.parametrize("B,T,C,W,state", [(2, 70, 384, 4, False), (1, 33, 17, 4, False), (2, 65, 24, 3, True), (1, 5, 8, 6, False)])
def test_bf16_weight_gradient_is_the_float32_one_rounded(B, T, C, W, state):
    from experiment_swa_kda_b200 import nanochat_ops
    nanochat_ops.register()
    ops = torch.ops.nanochat_kda
    gen = torch.Generator(device=D0).manual_seed(T + C)
    draw = lambda *n: torch.randn(*n, device=D0, generator=gen).bfloat16()
    x, dy, w = draw(B, T, C), draw(B, T, C), draw(C, W)
    s0, dfin = (draw(B, C, W), draw(B, C, W)) if state else (None, None)
    dx, dw, _ = ops.causal_convolution_backward(x, w, s0, x, None, dy, dfin)
    dx32, dw32, _ = ops.causal_convolution_backward(x, w.float(), s0, x, None, dy, dfin)
    assert dw.dtype == torch.bfloat16 and dw32.dtype == torch.float32
    assert torch.equal(dx, dx32) and torch.equal(dw, dw32.bfloat16())


@pytest.mark.parametrize("B,T,C,dtype", [(2, 300, 384, torch.bfloat16), (1, 67, 20, torch.float32)])
def test_short_convolutions_one_launch_equals_per_tensor_calls(B, T, C, dtype):
    """The batched q/k/v convolution entry points give bit-identical outputs and gradients to three separate calls."""
    gen = torch.Generator().manual_seed(T + C)
    mods = [_conv_mod(C, 4, ((torch.rand(C, 4, generator=gen) * 2 - 1) * 0.1).to(D0)) for _ in range(3)]
    xs = [torch.randn(B, T, C, generator=gen).to(dtype).to(D0).requires_grad_(True) for _ in range(3)]
    cys = [torch.randn(B, T, C, generator=gen).to(dtype).to(D0) for _ in range(3)]
    import experiment_swa_kda_b200 as M
    ys = M.short_convolutions(mods, xs)
    got = torch.autograd.grad(ys, xs + [m.weight for m in mods], cys)
    ys1 = [m(x)[0] for m, x in zip(mods, xs)]
    want = torch.autograd.grad(ys1, xs + [m.weight for m in mods], cys)
    for a, b in zip(ys, ys1):
        assert torch.equal(a, b)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_conv_full_sequence_equals_token_decode():
    gen = torch.Generator().manual_seed(99)
    x = torch.randn(2, 9, 8, generator=gen).to(D0)
    mod = _conv_mod(8, 4, torch.randn(8, 4, generator=gen).to(D0))
    with torch.no_grad():
        full, full_state = mod(x, output_final_state=True)
        state, pieces = None, []
        for t in range(9):
            y, state = mod(x[:, t:t + 1], state, output_final_state=True)
            pieces.append(y)
    torch.testing.assert_close(torch.cat(pieces, 1), full, atol=1e-6, rtol=1e-6)
    assert torch.equal(state, full_state)


@pytest.mark.parametrize("eps", [1e-5, 1e-6])
def test_rmsnorm_fp32_matches_reference_vectors(golden_dir, eps):
    from experiment_swa_kda_b200 import RMSNormGated
    z = np.load(os.path.join(golden_dir, "rmsnorm_gated.npz"))
    x = torch.from_numpy(z["x"]).to(D0).requires_grad_(True)
    gate = torch.from_numpy(z["gate"]).to(D0).requires_grad_(True)
    mod = RMSNormGated(16, eps=eps).to(D0)
    with torch.no_grad():
        mod.weight.copy_(torch.from_numpy(z["w"]))
    y = mod(x, gate)
    tag = f"eps{eps:g}"
    torch.testing.assert_close(y.cpu(), torch.from_numpy(z[f"{tag}_y"]), atol=1e-6, rtol=1e-5)
    got = torch.autograd.grad(y, (x, gate, mod.weight), torch.from_numpy(z[f"{tag}_cy"]).to(D0))
    for a, n in zip(got, ("dx", "dgate", "dw")):
        torch.testing.assert_close(a.cpu(), torch.from_numpy(z[f"{tag}_{n}"]), atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("rows,D,dtype", [(24576, 128, torch.bfloat16), (1000, 128, torch.float32), (77, 96, torch.bfloat16),
                                         (33, 256, torch.bfloat16)])
def test_rmsnorm_matches_oracle(rows, D, dtype):
    from experiment_swa_kda_b200 import RMSNormGated
    gen = torch.Generator().manual_seed(rows + D)
    x = torch.randn(rows, D, generator=gen).to(dtype)
    gate = torch.randn(rows, D, generator=gen).to(dtype)
    w = 1 + 0.1 * torch.randn(D, generator=gen)
    cy = torch.randn(rows, D, generator=gen).to(dtype)
    mod = RMSNormGated(D, eps=1e-6).to(D0)
    with torch.no_grad():
        mod.weight.copy_(w)
    xd, gd = x.to(D0).requires_grad_(True), gate.to(D0).requires_grad_(True)
    y = mod(xd, gd)
    got = torch.autograd.grad(y, (xd, gd, mod.weight), cy.to(D0))
    xe, ge, we = x.float().requires_grad_(True), gate.float().requires_grad_(True), w.clone().requires_grad_(True)
    ye = O.rmsnorm_gated(xe, ge, we, 1e-6)
    want = torch.autograd.grad(ye, (xe, ge, we), cy.float())
    tol = 1e-5 if dtype == torch.float32 else 1e-2
    assert O.rel_l2(y.float(), ye) <= tol
    for a, b in zip(got, want):
        assert O.rel_l2(a.float(), b) <= tol


def test_gate_matches_reference_vectors_and_gradients(golden_dir):
    from experiment_swa_kda_b200 import k3_decay_gate
    z = np.load(os.path.join(golden_dir, "gate.npz"))
    raw = torch.from_numpy(z["raw"]).float().to(D0).requires_grad_(True)
    A = torch.from_numpy(z["A_log"]).float().to(D0).requires_grad_(True)
    bias = torch.from_numpy(z["dt_bias"]).float().to(D0).requires_grad_(True)
    g = k3_decay_gate(raw, A, bias)
    torch.testing.assert_close(g.cpu().double(), torch.from_numpy(z["g"]), atol=2e-6, rtol=1e-5)
    g2 = k3_decay_gate(raw, A, bias, lower_bound=-2.0)
    torch.testing.assert_close(g2.cpu().double(), torch.from_numpy(z["g_lb2"]), atol=2e-6, rtol=1e-5)
    cot = torch.randn(g.shape, generator=torch.Generator().manual_seed(0)).to(D0)
    got = torch.autograd.grad(g, (raw, A, bias), cot)
    r64, A64, b64 = (t.detach().double().cpu().requires_grad_(True) for t in (raw, A, bias))
    want = torch.autograd.grad(O.decay_gate(r64, A64, b64), (r64, A64, b64), cot.double().cpu())
    for a, b in zip(got, want):
        torch.testing.assert_close(a.double().cpu(), b, atol=1e-5, rtol=1e-4)


# one quad of channels a thread up to 151,552 of them (296 rows of 2,048), two up to 303,104 (592), then four; rows narrower and wider
# than a block, row counts that four does not divide, fewer rows than that; beta logits in rows of their own and in wider ones
@pytest.mark.parametrize("tokens,H,K", [(1, 1, 4), (3, 2, 4), (5, 3, 12), (33, 3, 44), (296, 16, 128), (297, 16, 128), (592, 16, 128), (593, 16, 128),
                                        (4099, 3, 132), (200001, 1, 8), (70003, 8, 4)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gate_activations_at_every_width(tokens, H, K, dtype):
    from experiment_swa_kda_b200 import _lib
    lib = _lib.load()
    gen = torch.Generator(device=D0).manual_seed(tokens + K)
    raw = (3 * torch.randn(1, tokens, H, K, device=D0, generator=gen)).to(dtype)
    A_log, bias = 0.5 * torch.randn(H, device=D0, generator=gen), torch.randn(H * K, device=D0, generator=gen)
    want = O.decay_gate(raw.double(), A_log.double(), bias.double())
    for ld in (H, H + 3):
        logits = torch.randn(tokens, ld, device=D0, generator=gen).to(dtype)
        g, beta = torch.full((tokens * H * K + 8,), 9.0, device=D0), torch.full((tokens * H + 8,), 9.0, device=D0)
        _lib.check(lib.kda_gate_fwd_rows(tokens, H, K, _lib.DTYPE_BF16 if dtype == torch.bfloat16 else _lib.DTYPE_F32, raw.data_ptr(), logits.data_ptr(), ld,
                                         A_log.data_ptr(), bias.data_ptr(), -5.0, g.data_ptr(), beta.data_ptr(), torch.cuda.current_stream().cuda_stream), "gate")
        assert (g[-8:] == 9.0).all() and (beta[-8:] == 9.0).all()
        # float32 arithmetic on arguments of up to 60: their rounding, 2^-24 of them, times the slope's bound of 5 / 4
        torch.testing.assert_close(g[:-8].view_as(want).double(), want, atol=5e-6, rtol=1e-5)
        torch.testing.assert_close(beta[:-8].view(tokens, H).double(), torch.sigmoid(logits[:, :H].double()), atol=1e-6, rtol=1e-5)


def test_layer_forward_backward_finite_and_matches_composed_oracle():
    from experiment_swa_kda_b200 import KimiDeltaAttention
    torch.manual_seed(0)
    layer = KimiDeltaAttention(256, 2, 128, norm_eps=1e-6).to(D0)
    with torch.no_grad():
        layer.A_log.normal_(std=0.2)
        layer.dt_bias.normal_(std=0.3)
    x = torch.randn(2, 70, 256, device=D0, dtype=torch.bfloat16, requires_grad=True)
    y, st = layer(x, output_final_state=True)
    y.float().square().mean().backward()
    assert torch.isfinite(y).all() and torch.isfinite(x.grad).all()
    for n, p in layer.named_parameters():
        assert p.grad is not None and torch.isfinite(p.grad).all(), n
    # compose the same layer from the oracle pieces on the CPU, float32
    with torch.no_grad():
        P = {n: p.detach().float().cpu() for n, p in layer.named_parameters()}
        xc = x.detach().float().cpu()
        lin = lambda name, inp: inp @ P[name + ".weight"].bfloat16().float().t()
        q, _ = O.causal_conv(lin("q_proj", xc), P["q_conv1d.weight"].squeeze(1).bfloat16().float())
        k, _ = O.causal_conv(lin("k_proj", xc), P["k_conv1d.weight"].squeeze(1).bfloat16().float())
        v, _ = O.causal_conv(lin("v_proj", xc), P["v_conv1d.weight"].squeeze(1).bfloat16().float())
        sh = (2, 70, 2, 128)
        raw = lin("f_b_proj", lin("f_a_proj", xc)).reshape(sh)
        bl = lin("b_proj", xc)
        o, mem = O.kda_raw(q.reshape(sh), k.reshape(sh), v.reshape(sh), raw, bl, P["A_log"], P["dt_bias"])
        o = O.rmsnorm_gated(o, lin("g_proj", xc).reshape(sh), P["o_norm.weight"], 1e-6)
        ye = lin("o_proj", o.reshape(2, 70, 256))
    assert O.rel_l2(y.float(), ye) <= 3e-2      # several bf16 GEMMs in series
    assert O.rel_l2(st.memory, mem) <= 3e-2


# A weight that is a view into a flat parameter buffer (1, 2, 3 or 6 elements before it) allows no 16-byte loads: every
# entry point gives what it gives for an aligned copy.  Widths and types whose taps are read in 16-byte pieces otherwise; a
# carried window, none, and the channel counts of the pair (2), streaming (128) and one-channel kernels.
@pytest.mark.parametrize("B,T,C,W,dtype,wdtype", [(2, 70, 384, 4, torch.bfloat16, torch.float32), (1, 33, 130, 4, torch.bfloat16, torch.bfloat16),
                                                  (2, 65, 24, 4, torch.float32, torch.float32), (1, 9, 16, 8, torch.bfloat16, torch.bfloat16),
                                                  (1, 7, 5, 8, torch.float32, torch.float32), (1, 28423, 2048, 4, torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("state", [False, True])
@pytest.mark.parametrize("offset", [1, 6])
def test_convolution_weights_at_any_element_offset(B, T, C, W, dtype, wdtype, state, offset):
    from experiment_swa_kda_b200 import ops
    gen = torch.Generator(device=D0).manual_seed(T + C + offset)
    draw = lambda *n: torch.randn(*n, device=D0, generator=gen).to(dtype)
    x, dy = draw(B, T, C), draw(B, T, C)
    s0, dfin = (draw(B, C, W), draw(B, C, W)) if state else (None, None)
    w = torch.randn(C, W, device=D0, generator=gen).to(wdtype)
    flat = torch.empty(offset + C * W, device=D0, dtype=wdtype)
    view = flat[offset:].view(C, W).copy_(w)
    assert view.data_ptr() % 16 != 0 and w.data_ptr() % 16 == 0
    # the library itself: the one-channel kernels sum in the same order as the fast ones, up to the width of an fma
    tol = 1e-2 if dtype == torch.bfloat16 else 1e-5
    for a, b in zip((*ops.conv_fwd(x, view, s0, state), *ops.conv_bwd(x, view, s0, dy, dfin)),
                    (*ops.conv_fwd(x, w, s0, state), *ops.conv_bwd(x, w, s0, dy, dfin))):
        assert (a is None) == (b is None)
        if a is not None:
            assert O.rel_l2(a.float(), b.float()) <= tol
    # the operators: an aligned copy of the weight on the fast kernels, to the bit
    results = []
    for weight in (view, w):
        leaf = weight.detach().requires_grad_(True)
        assert leaf.data_ptr() == weight.data_ptr()
        xs = x.detach().clone().requires_grad_(True)
        y, fin = ops.conv(xs, leaf, s0, state)
        outs = [y, fin] if state else [y]
        results.append([*outs, *torch.autograd.grad(outs, [xs, leaf], [dy, dfin][:len(outs)])])
        if not state and W <= 4:
            ys = ops.ConvMultiFunction.apply(True, 2, xs, xs, leaf, leaf)
            results[-1] += [*ys, *torch.autograd.grad(ys, [xs, leaf], [dy, dy])]
    assert all(torch.equal(a, b) for a, b in zip(*results))


# either side of the line between the kernel of short runs and the streaming one (296 blocks of 256 tokens x 128 channels, three
# convolutions: 288 and 312 here), a last run of one token, several sequences, fewer tokens than the window holds
@pytest.mark.parametrize("B,T,C,W,streams", [(1, 3071, 1024, 4, False), (1, 3073, 1024, 4, True), (3, 1281, 768, 2, True), (1, 12801, 256, 3, True), (80, 2, 128, 4, True),
                                             (40, 1, 256, 4, True), (40, 8, 256, 3, True), (20, 3, 128, 4, False)])
def test_windows_carried_out_are_the_last_inputs(B, T, C, W, streams):
    import ctypes
    from experiment_swa_kda_b200 import _lib
    lib, n = _lib.load(), 3
    gen = torch.Generator(device=D0).manual_seed(T)
    xs = [torch.randn(B, T, C, device=D0, generator=gen).bfloat16() for _ in range(n)]
    ws = [torch.randn(C, W, device=D0, generator=gen) for _ in range(n)]
    arr = lambda ts: ctypes.cast((ctypes.c_void_p * n)(*[t.data_ptr() for t in ts]), ctypes.c_void_p)
    stream, io = torch.cuda.current_stream().cuda_stream, _lib.DTYPE_BF16 | 0x100

    def run(fins):
        ys = [torch.empty_like(x) for x in xs]
        _lib.check(lib.kda_conv_fwd_rows(n, B, T, C, W, io, 1, arr(xs), C, arr(ws), None, arr(ys), arr(fins) if fins else None, stream), "forward")
        return ys

    fins, got = [torch.full((B, C, W), 9.0, device=D0, dtype=torch.bfloat16) for _ in range(n)], []
    assert _forward_kernels(lambda: got.extend(run(fins))) == {"conv_fwd_stream_kernel" if streams else "conv_fwd_kernel"}
    assert all(torch.equal(a, b) for a, b in zip(got, run(None)))
    padded = [torch.nn.functional.pad(x, (0, 0, W, 0)) for x in xs]      # zeros before the first token
    assert all(torch.equal(f, x[:, T:].transpose(1, 2)) for f, x in zip(fins, padded))


# Three convolutions on slices of one wide matrix, as the layer keeps its projections, either side of every dispatch line:
# backward tile | ring (592 runs of 64 tokens x 128 channels: 65 and 66 tiles at 3 x 384), ring runs of 32 | 64 tokens (147 and 148
# tiles at 3 x 2,048), forward pair | streaming (222 blocks of 256 tokens x 128 channels: 192 and 240 at 3 x 2,048); ragged ends,
# several sequences.
@pytest.mark.parametrize("B,T,C,W", [(1, 4160, 384, 4), (1, 4161, 384, 4), (3, 1431, 384, 3), (1, 1024, 2048, 4), (1, 1027, 2048, 4), (1, 9408, 2048, 4),
                                     (1, 9409, 2048, 4), (2, 4801, 2048, 2), (2, 70, 130, 4)])
def test_convolutions_on_slices_equal_those_on_dense_copies(B, T, C, W):
    """The same kernels with another row stride: equal to the bit, with NaN in the columns that are not theirs and every column
    of the gradient's matrix outside the slices untouched."""
    import ctypes
    from experiment_swa_kda_b200 import _lib
    lib, n = _lib.load(), 3
    step = (C + 15) // 8 * 8                                # slices at 16-byte addresses, a few columns between them
    first, ld = [0, step, 2 * step], 4 * C + 144 + C % 8
    gen = torch.Generator(device=D0).manual_seed(T + C)
    dense = lambda *shape: torch.randn(*shape, device=D0, generator=gen).bfloat16()
    xs, dys = [dense(B * T, C) for _ in range(n)], [dense(B * T, C) for _ in range(n)]
    ws = [torch.randn(C, W, device=D0, generator=gen) for _ in range(n)]
    P = torch.full((B * T, ld), float("nan"), device=D0, dtype=torch.bfloat16)
    for f, x in zip(first, xs):
        P[:, f:f + C] = x
    arr = lambda ps: ctypes.cast((ctypes.c_void_p * n)(*ps), ctypes.c_void_p)
    ptrs = lambda ts: [t.data_ptr() for t in ts]
    at = lambda m: [m.data_ptr() + 2 * f for f in first]
    stream, io = torch.cuda.current_stream().cuda_stream, _lib.DTYPE_BF16 | 0x100
    scr = torch.empty(lib.kda_conv_bwd_multi_scratch_bytes(n, B, T, C, W), dtype=torch.uint8, device=D0)

    def run(x_at, x_ld, dx_at):
        ys, dws = [torch.empty_like(x) for x in xs], [torch.empty(C, W, device=D0) for _ in range(n)]
        _lib.check(lib.kda_conv_fwd_rows(n, B, T, C, W, io, 1, arr(x_at), x_ld, arr(ptrs(ws)), None, arr(ptrs(ys)), None, stream), "forward")
        _lib.check(lib.kda_conv_bwd_rows(n, B, T, C, W, io, 1, arr(x_at), x_ld, arr(ptrs(ws)), arr(ptrs(dys)), arr(dx_at), arr(ptrs(dws)),
                                         scr.data_ptr(), scr.numel(), stream), "backward")
        return [*ys, *dws]

    dxs, dP = [torch.empty_like(x) for x in xs], torch.full_like(P, 7.0)
    want, got = run(ptrs(xs), C, ptrs(dxs)), run(at(P), ld, at(dP))
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    outside = torch.ones(ld, dtype=torch.bool, device=D0)
    for f, dx in zip(first, dxs):
        assert torch.equal(dP[:, f:f + C], dx)
        outside[f:f + C] = False
    assert outside.any() and (dP[:, outside] == 7.0).all()
