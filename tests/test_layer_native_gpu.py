"""The layer's native path against its modules run one by one (a forward hook on a projection sends a layer there).

Both round to bf16 between the stages and differ only in the order of float32 sums inside a product, which moves a bf16
value by at most one unit in the last place (2^-8 relative): the bound is 1e-2 relative L2 as for every bf16 operator
here, 2e-2 for gradients, which cross four such roundings in series."""

import pytest
import torch

import kda_oracle as O

pytestmark = pytest.mark.gpu
D0 = "cuda:0"


def _layer(heads, seed, wdtype=torch.float32):
    from experiment_swa_kda_b200 import KimiDeltaAttention
    torch.manual_seed(seed)
    layer = KimiDeltaAttention(heads * 128, heads, 128, norm_eps=1e-6).to(D0)
    with torch.no_grad():
        layer.A_log.normal_(std=0.2)
        layer.dt_bias.uniform_(-4, 0)
        for name, p in layer.named_parameters():
            if "proj" in name:
                p.data = p.data.to(wdtype)
    return layer


def _modules_one_by_one(layer):
    layer.q_proj.register_forward_hook(lambda *a: None)
    assert layer._plain_weights() is None
    return layer


def _state(batch, heads, gen):
    from experiment_swa_kda_b200 import KDAState
    st = KDAState.zeros(batch, heads, 128, 4, D0)
    st.memory.copy_(torch.randn(st.memory.shape, generator=gen) * 0.1)
    for c in (st.q_conv, st.k_conv, st.v_conv):
        c.copy_(torch.randn(c.shape, generator=gen))
    return st


# edges of the row tiles (8, 16, 32, 64), one row past the last, one-block and many-block decode launches
@pytest.mark.parametrize("batch,heads,wdtype", [(1, 1, torch.float32), (7, 3, torch.float32), (8, 2, torch.bfloat16), (9, 3, torch.float32),
                                                (17, 5, torch.bfloat16), (33, 5, torch.float32), (64, 3, torch.float32), (65, 2, torch.float32)])
def test_token_step_equals_the_modules(batch, heads, wdtype):
    gen = torch.Generator().manual_seed(batch + heads)
    layer = _layer(heads, 1, wdtype)
    x = torch.randn(batch, 1, heads * 128, generator=gen).bfloat16().to(D0)
    ours, theirs = _state(batch, heads, gen), None
    theirs = ours.clone()
    got = layer.decode_token(x, ours)
    want = _modules_one_by_one(layer).decode_token(x, theirs)
    assert O.rel_l2(got.float(), want.float()) <= 1e-2
    for a, b in ((ours.memory, theirs.memory), (ours.q_conv, theirs.q_conv), (ours.k_conv, theirs.k_conv), (ours.v_conv, theirs.v_conv)):
        assert O.rel_l2(a.float(), b.float()) <= 1e-2


# up to 64 rows straight from the parameters, more through the packed matrix; odd head counts pad the projection
@pytest.mark.parametrize("batch,T,heads,carried", [(1, 5, 1, False), (2, 32, 3, True), (1, 65, 3, True), (2, 130, 8, False)])
def test_prefill_equals_the_modules(batch, T, heads, carried):
    gen = torch.Generator().manual_seed(T)
    layer = _layer(heads, 2)
    x = torch.randn(batch, T, heads * 128, generator=gen).bfloat16().to(D0)
    state = _state(batch, heads, gen) if carried else None
    with torch.no_grad():
        y, st = layer(x, state=state, output_final_state=True)
        ye, se = _modules_one_by_one(layer)(x, state=state, output_final_state=True)
    for a, b in ((y, ye), (st.memory, se.memory), (st.q_conv, se.q_conv), (st.k_conv, se.k_conv), (st.v_conv, se.v_conv)):
        assert a.shape == b.shape and O.rel_l2(a.float(), b.float()) <= 1e-2


@pytest.mark.parametrize("batch,T,heads,carried,wdtype", [(1, 3, 1, False, torch.float32), (2, 67, 3, False, torch.float32),
                                                          (2, 70, 2, True, torch.float32), (1, 129, 8, False, torch.bfloat16)])
def test_training_step_equals_the_modules(batch, T, heads, carried, wdtype):
    from experiment_swa_kda_b200 import KDAState
    gen = torch.Generator().manual_seed(T + heads)
    layer = _layer(heads, 3, wdtype)
    x = torch.randn(batch, T, heads * 128, generator=gen).bfloat16().to(D0).requires_grad_(True)
    dy = torch.randn(batch, T, heads * 128, generator=gen).bfloat16().to(D0)
    init = _state(batch, heads, gen)
    names = [n for n, _ in layer.named_parameters()]
    results = []
    for _ in range(2):
        parts = [t.clone().requires_grad_(True) for t in (init.memory, init.q_conv, init.k_conv, init.v_conv)] if carried else []
        y, st = layer(x, state=KDAState(*parts) if carried else None, output_final_state=carried)
        outs = [y] + ([st.memory, st.q_conv, st.k_conv, st.v_conv] if carried else [])
        cots = [dy] + [torch.ones_like(t) * 0.1 for t in outs[1:]]
        results.append((outs, torch.autograd.grad(outs, [x, *layer.parameters(), *parts], cots)))
        _modules_one_by_one(layer)
    for a, b in zip(results[0][0], results[1][0]):
        assert O.rel_l2(a.float(), b.float()) <= 1e-2
    for n, a, b in zip(["x", *names, "memory", "q_conv", "k_conv", "v_conv"], results[0][1], results[1][1]):
        assert a.dtype == b.dtype and a.shape == b.shape, n
        if n in ("A_log", "dt_bias"):      # sums of cancelling terms: the reference's bar for gate parameters
            assert (a - b).abs().max() <= 5e-2 * b.abs().max() + 2e-2, n
        else:
            assert O.rel_l2(a.float(), b.float()) <= 2e-2, n
