"""A token's three launches overlap: weights, state and the gate's weights are read while the launch before still runs, and at 149 to 266 and 445
to 532 states the blocks of four sequences form a cluster.  Many tokens in a row have to give the bits of the launches one by one."""

import pytest
import torch

pytestmark = pytest.mark.gpu
D0 = "cuda:0"


def _layer(heads, seed, dtype=torch.float32):
    import experiment_swa_kda_b200 as m
    torch.manual_seed(seed)
    layer = m.KimiDeltaAttention(hidden_size=heads * 128, num_heads=heads, head_dim=128, conv_size=4, norm_eps=1e-6).to(D0).eval()
    for name, p in layer.named_parameters():
        if name not in ("A_log", "dt_bias", "o_norm.weight"):
            p.data = p.data.to(dtype)
    with torch.no_grad():
        for p in layer.parameters():
            if p.dim() > 1:
                torch.nn.init.normal_(p, std=p.shape[-1] ** -0.5)
    return m, layer


# 32 warps a state up to 148 states; clusters of 16 (149 .. 266: 150, 156, 160, 264) and of 8 warps (445 .. 532: 448, 455, 465, 506, 512, 532) with 0,
# 1, 2 and 3 sequences over, and blocks over that fill the last cluster; 8 warps on their own, behind the projections (267 .. 444) and early (above 532)
@pytest.mark.parametrize("batch,heads,dtype", [(1, 1, torch.float32), (9, 16, torch.float32), (10, 16, torch.float32), (13, 12, torch.float32), (50, 3, torch.float32),
                                               (40, 4, torch.bfloat16), (44, 6, torch.float32), (7, 40, torch.float32), (37, 12, torch.float32), (28, 16, torch.float32),
                                               (35, 13, torch.float32), (31, 15, torch.bfloat16), (46, 11, torch.float32), (32, 16, torch.float32), (38, 14, torch.float32),
                                               (41, 13, torch.float32), (43, 14, torch.float32)])
def test_overlapping_launches_give_the_bits_of_separate_ones(batch, heads, dtype):
    m, layer = _layer(heads, batch, dtype)
    x = torch.randn(24, batch, 1, heads * 128, generator=torch.Generator().manual_seed(heads)).bfloat16().to(D0)
    a = m.KDAState.zeros(batch, heads, 128, 4, D0)
    a.memory.normal_(generator=torch.Generator(device=D0).manual_seed(1)).mul_(0.02)
    b = a.clone()
    with torch.no_grad():
        got = [layer.decode_token(t, a) for t in x]
        want = []
        for t in x:
            y, b = layer(t, state=b, output_final_state=True, mode="project_recurrent")
            want.append(y)
    assert all(torch.equal(p, q) for p, q in zip(got, want))
    assert torch.equal(a.memory, b.memory) and torch.equal(a.q_conv, b.q_conv) and torch.equal(a.v_conv, b.v_conv)


@pytest.mark.parametrize("batch,heads", [(2, 3), (13, 16)])
def test_overlapping_launches_in_a_graph(batch, heads):
    m, layer = _layer(heads, 5)
    xs = torch.randn(8, batch, 1, heads * 128, device=D0).bfloat16()
    eager, state = (m.KDAState.zeros(batch, heads, 128, 4, D0) for _ in range(2))
    x, stream, graph = xs[0].clone(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.no_grad():
        want = [layer.decode_token(t, eager) for t in xs]
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            layer.decode_token(x, state)
        torch.cuda.current_stream().wait_stream(stream)
        for t in (state.memory, state.q_conv, state.k_conv, state.v_conv):
            t.zero_()
        with torch.cuda.graph(graph):
            y = layer.decode_token(x, state)
        for t in (state.memory, state.q_conv, state.k_conv, state.v_conv):
            t.zero_()
        for t, w in zip(xs, want):
            x.copy_(t)
            graph.replay()
            assert torch.equal(y, w)
    assert torch.equal(state.memory, eager.memory)


@pytest.mark.parametrize("batch,tokens,heads", [(1, 77, 3), (3, 64, 8), (2, 1100, 6), (1, 20, 16)])
def test_launches_beside_one_another_give_the_bits_of_launches_one_by_one(batch, tokens, heads):
    """Convolutions, gate activations and the sums of partial gradients overlap inside a layer call; with events between the launches
    (launch accounting) they do not."""
    from experiment_swa_kda_b200 import _lib
    m, layer = _layer(heads, 9)
    xs = torch.randn(6, batch, tokens, heads * 128, generator=torch.Generator().manual_seed(2)).bfloat16().to(D0)
    leaves = list(layer.parameters())

    def passes():
        out = []
        for x in xs:
            with torch.no_grad():
                y, st = layer(x, output_final_state=True)
            out += [y, st.memory, st.q_conv, st.k_conv, st.v_conv]
            x = x.clone().requires_grad_(True)
            y, _ = layer(x)
            out += [y, *torch.autograd.grad(y, [x, *leaves], x.detach())]
        torch.cuda.synchronize()
        return out

    got = passes()
    _lib.load().kda_profile_enable(1)
    try:
        want = passes()
    finally:
        _lib.profile_report()
        _lib.load().kda_profile_enable(0)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
