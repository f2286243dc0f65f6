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


# up to 64 rows straight from the parameters, more through the packed matrix; odd head counts pad the projection; from 1,024 rows on
# the three convolutions in one launch, with windows carried in, out, and out of the streaming kernel
@pytest.mark.parametrize("batch,T,heads,carried", [(1, 5, 1, False), (2, 32, 3, True), (1, 65, 3, True), (2, 130, 8, False), (1, 1023, 3, True), (2, 512, 3, True),
                                                   (2, 601, 3, False), (4, 1100, 6, False), (520, 2, 1, True), (520, 2, 1, False)])
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


def _shifted(t):
    """The same values one element into a larger buffer: dense, at an address that allows no 16-byte access."""
    flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
    view = flat[1:].view(t.shape).copy_(t.detach())
    assert view.data_ptr() % 16 != 0
    return view


def _shifted_state(state):
    from experiment_swa_kda_b200 import KDAState
    return KDAState(*[_shifted(t) for t in (state.memory, state.q_conv, state.k_conv, state.v_conv)])


def _shift_vectors(layer):
    """dt_bias, the norm weight and the taps as a flat parameter buffer behind a 3-element A_log would hold them."""
    for p in (layer.dt_bias, layer.o_norm.weight, layer.q_conv1d.weight, layer.k_conv1d.weight, layer.v_conv1d.weight):
        p.data = _shifted(p.data)
    assert layer._plain_weights() is not None
    return layer


# few rows straight from the parameters and packed ones, with and without an incoming state; the convolutions in the kernel
@pytest.mark.parametrize("T,carried,fuse", [(5, False, False), (5, True, False), (70, True, False), (70, False, True)])
def test_prefill_with_tensors_at_odd_addresses(T, carried, fuse):
    gen = torch.Generator().manual_seed(T)
    layer, x, results = _layer(3, 2), torch.randn(2, T, 384, generator=gen).bfloat16().to(D0), []
    layer.fuse_prefill_conv = fuse
    state = _state(2, 3, gen) if carried else None
    for put in (False, True):
        if put:
            layer, x, state = _shift_vectors(layer), _shifted(x), _shifted_state(state) if carried else None
        with torch.no_grad():
            y, st = layer(x, state=state, output_final_state=True)
        results.append((y, st.memory, st.q_conv, st.k_conv, st.v_conv))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("carried", [False, True])
def test_training_step_with_tensors_at_odd_addresses(carried):
    from experiment_swa_kda_b200 import KDAState
    gen = torch.Generator().manual_seed(9)
    layer, x = _layer(3, 2), torch.randn(2, 70, 384, generator=gen).bfloat16().to(D0)
    dy, init, results = torch.randn(2, 70, 384, generator=gen).bfloat16().to(D0), _state(2, 3, gen), []
    for put in (lambda t: t.clone(), _shifted):
        if put is _shifted:
            _shift_vectors(layer)
        xs = put(x).requires_grad_(True)
        parts = [put(t).requires_grad_(True) for t in (init.memory, init.q_conv, init.k_conv, init.v_conv)] if carried else []
        y, st = layer(xs, state=KDAState(*parts) if carried else None, output_final_state=carried)
        outs = [y] + ([st.memory, st.q_conv, st.k_conv, st.v_conv] if carried else [])
        results.append([*outs, *torch.autograd.grad(outs, [xs, *layer.parameters(), *parts], [put(dy)] + [put(t.detach()) for t in outs[1:]])])
    assert all(torch.equal(a, b) for a, b in zip(*results))


def test_token_step_with_tensors_at_odd_addresses():
    """A memory at an odd address cannot be stepped by the fused kernel: the call is declined before anything has moved and
    runs module by module, so the windows advance once."""
    gen = torch.Generator().manual_seed(8)
    layer, x, state = _layer(3, 1), torch.randn(2, 1, 384, generator=gen).bfloat16().to(D0), _state(2, 3, gen)
    aligned, shifted = state.clone(), _shifted_state(state)
    want = layer.decode_token(x, aligned)
    with torch.no_grad():
        y, st = layer(_shifted(x), state=shifted, output_final_state=True, mode="project_recurrent")
    assert torch.equal(y, want) and torch.equal(st.memory, aligned.memory) and torch.equal(st.q_conv, aligned.q_conv)
    got = _shift_vectors(layer).decode_token(_shifted(x), shifted)
    assert O.rel_l2(got.float(), want.float()) <= 1e-2
    for a, b in ((shifted.memory, aligned.memory), (shifted.q_conv, aligned.q_conv), (shifted.k_conv, aligned.k_conv), (shifted.v_conv, aligned.v_conv)):
        assert O.rel_l2(a.float(), b.float()) <= 1e-2
    whole = aligned.clone()       # everything but the memory at odd addresses: the fused step, to the bit
    odd = _shifted_state(aligned)
    odd.memory = aligned.memory.clone()
    assert torch.equal(layer.decode_token(x, whole), layer.decode_token(_shifted(x), odd))
    assert torch.equal(whole.memory, odd.memory) and torch.equal(whole.v_conv, odd.v_conv)


# three convolutions of 21,845 sequences fill a grid; one more sequence runs module by module, forward and backward
@pytest.mark.parametrize("batch", [21845, 21846])
def test_more_sequences_than_the_batched_convolutions_grid_holds(batch):
    gen = torch.Generator().manual_seed(batch)
    layer = _layer(1, 4)
    x = torch.randn(batch, 1, 128, generator=gen).bfloat16().to(D0).requires_grad_(True)
    dy = torch.randn(batch, 1, 128, generator=gen).bfloat16().to(D0)
    results = []
    for _ in range(2):
        with torch.no_grad():
            y0, _ = layer(x)
        y, _ = layer(x)
        assert O.rel_l2(y0.float(), y.detach().float()) <= 1e-2
        results.append((y, *torch.autograd.grad(y, [x, layer.q_proj.weight, layer.v_conv1d.weight], dy)))
        _modules_one_by_one(layer)
    for a, b in zip(*results):
        assert O.rel_l2(a.detach().float(), b.detach().float()) <= 2e-2


def test_training_step_long_enough_for_the_streaming_convolutions():
    """2 x 1,100 tokens of 6 heads: 3 x 6 x 36 runs, past the line (592) from which slices of the projection are streamed."""
    test_training_step_equals_the_modules(2, 1100, 6, False, torch.float32)


@pytest.mark.parametrize("batch,T,heads", [(2, 512, 3), (2, 1100, 6)])
def test_training_step_whose_windows_go_through_one_launch(batch, T, heads):
    test_training_step_equals_the_modules(batch, T, heads, True, torch.float32)
