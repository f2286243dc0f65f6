"""Autograd features around the operators, whose backwards are C++ nodes: what has no derivative here is refused, and a
program that traces or checkpoints a call gets what the call gives."""

import pytest
import torch
import torch.autograd.forward_ad as fw

pytestmark = pytest.mark.gpu
D0 = "cuda:0"


def _calls():
    """name -> (function of one tensor, that tensor)"""
    import experiment_swa_kda_b200 as m
    gen = torch.Generator().manual_seed(0)
    draw = lambda *n: torch.randn(*n, generator=gen).bfloat16().to(D0)
    q, k, v, raw, gate = (draw(2, 70, 2, 128) for _ in range(5))
    g, beta = -torch.rand(2, 70, 2, 128, generator=gen).to(D0), torch.rand(2, 70, 2, generator=gen).to(D0)
    A, bias, nw = torch.zeros(2, device=D0), torch.zeros(256, device=D0), torch.ones(128, device=D0)
    torch.manual_seed(0)
    conv, norm, layer = m.ShortConvolution(256, 4).to(D0), m.RMSNormGated(128).to(D0), m.KimiDeltaAttention(256, 2, 128).to(D0)
    x = draw(2, 70, 256)
    return {
        "chunk_kda": (lambda a: m.chunk_kda(a, k, v, g, beta)[0], q),
        "chunk_kda_f32": (lambda a: m.chunk_kda(a, k.float(), v.float(), g, beta)[0], q.float()),
        "chunk_kda_norm": (lambda a: m.chunk_kda_norm(a, k, v, g, beta, gate, nw)[0], q),
        "kda": (lambda a: m.kda(a, k, v, raw, beta.bfloat16(), A, bias)[0], q),
        "gate": (lambda a: m.k3_decay_gate(a, A, bias), raw),
        "conv": (lambda a: conv(a)[0], x),
        "convs": (lambda a: m.short_convolutions([conv, conv], [a, a])[0], x),
        "norm": (lambda a: norm(a, gate), q),
        "layer": (lambda a: layer(a)[0], x),
    }


NAMES = ["chunk_kda", "chunk_kda_f32", "chunk_kda_norm", "kda", "gate", "conv", "convs", "norm", "layer"]


@pytest.mark.parametrize("tracked", [False, True])
@pytest.mark.parametrize("name", NAMES)
def test_forward_mode_is_refused(name, tracked):
    call, a = _calls()[name]
    with fw.dual_level(), pytest.raises(RuntimeError, match="forward-mode|forward AD"):
        call(fw.make_dual(a.clone().requires_grad_(tracked), torch.ones_like(a)))
    call(a)      # outside of the level the same call runs


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("tracked", [False, True])
@pytest.mark.parametrize("name", NAMES)
def test_a_traced_call_follows_its_inputs(name, tracked):
    """torch.jit.trace of a call, run on other inputs, equals the call; so do its gradients."""
    call, a = _calls()[name]
    if name in ("conv", "convs", "norm", "layer"):      # parameters in a closure are constants that the tracer takes without gradients only
        for cell in call.__closure__:
            if isinstance(cell.cell_contents, torch.nn.Module):
                cell.cell_contents.requires_grad_(False)
    with torch.set_grad_enabled(tracked):
        other = (a * 0.5 + 1).to(a.dtype).requires_grad_(tracked)
        trace = torch.jit.trace(call, (a.clone().requires_grad_(tracked),), check_trace=False)
        got, want = trace(other), call(other)
        assert torch.equal(got, want)
        if tracked:
            dy = torch.randn(want.shape, generator=torch.Generator().manual_seed(1)).to(D0, want.dtype)
            assert torch.equal(*(torch.autograd.grad(o, other, dy)[0] for o in (got, want))) or name == "layer"
            for o in (got, want):
                assert o.requires_grad
    call(a)
