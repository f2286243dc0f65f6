"""Recurrences that are walked by one kernel each way (tc_walk_kernel), at the sizes where its rings turn: two operand stages and state
tiles, three gate tiles, four slots of sums, two sets of output warps."""

import pytest
import torch

from oracle import kda_oracle as O
from test_tc_lane_gpu import D0, _kda_mod, _run_activated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [320, 321, 447, 577])
def test_walked_recurrences_against_the_oracle(tokens):
    _run_activated(O.make_inputs(2, tokens, 3, 128, 128, seed=600 + tokens, with_state=True))


@pytest.mark.parametrize("tokens", [64, 127, 128, 192, 193, 256, 321, 449, 837])
def test_norm_in_the_walk_equals_the_two_operators(tokens):
    """The two halves of a row meet between two blocks; same bits as the operator and the norm on their own, with and without a backward."""
    m = _kda_mod()
    d = {n: t.bfloat16().to(D0) for n, t in O.make_inputs(2, tokens, 3, 128, 128, seed=700 + tokens).items()}
    gen = torch.Generator().manual_seed(3)
    gate = torch.randn(2, tokens, 3, 128, generator=gen).bfloat16().to(D0)
    norm = m.RMSNormGated(128, eps=1e-6).to(D0)
    with torch.no_grad():
        norm.weight.copy_(1 + 0.1 * torch.randn(128, generator=gen))
    x = [d[n].requires_grad_(True) for n in ("q", "k", "v", "g", "beta")]
    o, s = m.chunk_kda(*x, output_final_state=True)
    want = norm(o, gate)
    y, sy = m.chunk_kda_norm(*x, gate, norm.weight, eps=1e-6, output_final_state=True)
    with torch.no_grad():
        z, sz = m.chunk_kda_norm(*x, gate, norm.weight, eps=1e-6, output_final_state=True)
    for got in ((y, sy), (z, sz)):
        assert torch.equal(got[0], want) and torch.equal(got[1], s)
    dy = torch.randn(want.shape, generator=gen).bfloat16().to(D0)
    for a, b in zip(torch.autograd.grad(want, x, dy), torch.autograd.grad(y, x, dy)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("tokens", [64 * 19 + 33, 64 * 100 + 5])      # four and eight segments
def test_walk_and_split_scans_agree(tokens):
    """Two recurrences of 19 or more whole chunks are split; with empty sequences beside them, which make the batch look like many short ones, they walk.
    Bounds as for split scans against single chains: bf16 operands of two groupings of the same products."""
    m = _kda_mod()
    d = O.make_inputs(1, tokens, 2, 128, 128, seed=91, with_state=True)
    gen = torch.Generator().manual_seed(4)
    do = torch.randn(1, tokens, 2, 128, generator=gen).bfloat16().to(D0)
    ds = torch.randn(1, 2, 128, 128, generator=gen).to(D0)
    res = []
    for empty in (0, 5):
        x = {n: (t.float() if n == "h0" else t.bfloat16()).to(D0) for n, t in d.items()}
        x["h0"] = torch.cat([x["h0"], torch.ones(empty, 2, 128, 128, device=D0)])
        x = {n: t.requires_grad_(True) for n, t in x.items()}
        cu = torch.tensor([0] + [tokens] * (empty + 1), dtype=torch.int32, device=D0)
        o, s = m.chunk_kda(x["q"], x["k"], x["v"], x["g"], x["beta"], initial_state=x["h0"], output_final_state=True, cu_seqlens=cu, lane="tc")
        assert torch.equal(s[1:], x["h0"][1:])
        grads = torch.autograd.grad((o, s), list(x.values()), (do, torch.cat([ds, torch.ones(empty, 2, 128, 128, device=D0)])))
        res.append([o, s[:1], *[g[:1] for g in grads]])
    assert not torch.equal(res[0][0], res[1][0])            # two kernels, not one
    for a, b in zip(*res):
        assert O.rel_l2(a.float(), b.float()) <= 6e-3
