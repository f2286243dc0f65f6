"""Recurrences that are walked by one kernel each way (tc_walk_kernel), at the sizes where its rings turn: two operand stages and state
tiles, three gate tiles, four slots of sums, two sets of output warps."""

import pytest
import torch

from oracle import kda_oracle as O
from test_tc_lane_gpu import BF16_TOL, D0, _kda_mod, _run_activated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [320, 321, 447, 577])
def test_walked_recurrences_against_the_oracle(tokens):
    _run_activated(O.make_inputs(2, tokens, 3, 128, 128, seed=600 + tokens, with_state=True))


@pytest.mark.parametrize("tokens", [64, 127, 128, 192, 193, 256, 321, 449, 837, 2112, 2137])      # the last two: split scans, in the chunk-output kernel
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
    from experiment_swa_kda_b200 import _lib
    _lib.load().kda_profile_enable(1)
    try:
        with torch.no_grad():
            z, sz = m.chunk_kda_norm(*x, gate, norm.weight, eps=1e-6, output_final_state=True)
        ran = _lib.profile_report()
    finally:
        _lib.load().kda_profile_enable(0)
    assert ("tc_chunk_out_kernel" if tokens > 2000 else "tc_walk_fwd_kernel") in ran
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
    for empty in (0, 8):
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


@pytest.mark.parametrize("tokens", [64, 37])
def test_a_small_initial_state_passes_through_a_walk(tokens):
    """The final state is linear in the initial one.  One 2^-7 as large as the values moves the token updates Z = U - W H by about their bf16
    rounding, so a walk that gave the state its rounded Z loses 0.35 and 0.21 of it.  What is left are bf16 W, E and H, each within
    2^-9 of itself, and what two roundings leave of Z, 2^-17 of it against the 2^-7: under 1e-2 together."""
    m = _kda_mod()
    d = {n: t.bfloat16().to(D0) for n, t in O.make_inputs(2, tokens, 12, 128, 128, seed=91).items()}
    h0 = 2.0 ** -7 * torch.randn(2, 12, 128, 128, generator=torch.Generator().manual_seed(6)).to(D0)
    x = [d[n] for n in ("q", "k", "v", "g", "beta")]
    states = [m.chunk_kda(*x, initial_state=h, output_final_state=True, lane="tc")[1].double() for h in (h0, torch.zeros_like(h0))]
    y = [t.double() for t in x]
    want = O.kda_recurrence(y[0], y[1], torch.zeros_like(y[2]), y[3], y[4], initial_state=h0.double(), compute_dtype=torch.float64)[1]
    assert O.rel_l2(states[0] - states[1], want) <= 1e-2


@pytest.mark.parametrize("tokens", [64 * 19 + 33, 64 * 36])
def test_a_walk_is_as_close_to_float64_as_split_scans(tokens):
    """Two recurrences are split, with empty sequences beside them they walk: outputs, final state and the gradients of values and initial state
    (the ones the recurrence alone makes) are no further from a float64 recurrence, 3 % for the luck of one draw aside."""
    m = _kda_mod()
    d = O.make_inputs(1, tokens, 2, 128, 128, seed=92, with_state=True)
    gen = torch.Generator().manual_seed(4)
    do = torch.randn(1, tokens, 2, 128, generator=gen).bfloat16().to(D0)
    ds = torch.randn(1, 2, 128, 128, generator=gen).to(D0)
    x = {n: (t.float() if n == "h0" else t.bfloat16()).to(D0) for n, t in d.items()}
    y = {n: t.double().requires_grad_(True) for n, t in x.items()}
    eo, es = O.kda_recurrence(y["q"], y["k"], y["v"], y["g"], y["beta"], initial_state=y["h0"], compute_dtype=torch.float64)
    want = [eo, es, *torch.autograd.grad((eo, es), [y["v"], y["h0"]], (do.double(), ds.double()))]
    errs = []
    for empty in (0, 5):
        x["h0"] = torch.cat([x["h0"][:1].detach(), torch.ones(empty, 2, 128, 128, device=D0)])
        z = {n: t.detach().requires_grad_(True) for n, t in x.items()}
        cu = torch.tensor([0] + [tokens] * (empty + 1), dtype=torch.int32, device=D0)
        o, s = m.chunk_kda(z["q"], z["k"], z["v"], z["g"], z["beta"], initial_state=z["h0"], output_final_state=True, cu_seqlens=cu, lane="tc")
        dv, dh = torch.autograd.grad((o, s), [z["v"], z["h0"]], (do, torch.cat([ds, torch.ones(empty, 2, 128, 128, device=D0)])))
        errs.append([O.rel_l2(a.double(), b.detach()) for a, b in zip((o, s[:1], dv, dh[:1]), want)])
    for split, walk in zip(*errs):
        assert walk <= 1.03 * split, errs


def test_an_infinite_value_spoils_its_own_column():
    m = _kda_mod()
    d = {n: t.bfloat16().to(D0) for n, t in O.make_inputs(2, 200, 12, 128, 128, seed=93).items()}
    states = []
    for infinite in (False, True):
        v = d["v"].clone()
        if infinite:
            v[1, 70, 3, 17] = float("inf")
        states.append(m.chunk_kda(d["q"], d["k"], v, d["g"], d["beta"], output_final_state=True, lane="tc")[1])
    assert not states[1][1, 3, 17].isfinite().any()
    states[1][1, 3, 17] = states[0][1, 3, 17]
    assert torch.equal(*states)


@pytest.mark.parametrize("batch,tokens,path", [(2, 200, "tc_walk_fwd_kernel"), (1, 64 * 36 + 9, "tc_chunk_out_kernel")])
def test_output_of_the_norms_forward_at_an_8_byte_address(batch, tokens, path):
    """kda_chunk_fwd_norm takes an o that starts on 8 bytes, by a walk as by split scans."""
    from experiment_swa_kda_b200 import _lib, ops
    lib, H = _lib.load(), 2
    d = {n: t.bfloat16().to(D0) for n, t in O.make_inputs(batch, tokens, H, 128, 128, seed=94).items()}
    gate, w = torch.randn_like(d["v"]), torch.ones(128, device=D0)
    sh = _lib.ChunkShape(batch, tokens, batch * tokens, H, 128, 128, _lib.DTYPE_BF16, _lib.DTYPE_BF16, _lib.LANE_TC, 1, 0.1)
    ws = torch.empty(lib.kda_chunk_workspace_bytes(sh), dtype=torch.uint8, device=D0)
    stream = torch.cuda.current_stream().cuda_stream
    results = []
    for shift in (0, 4):
        o = torch.zeros(d["v"].numel() + 8, dtype=torch.bfloat16, device=D0)
        y, inv = torch.zeros_like(d["v"]), torch.zeros(batch * tokens * H, device=D0)
        lib.kda_profile_enable(1)
        try:
            rc = lib.kda_chunk_fwd_norm(sh, *(d[n].data_ptr() for n in ("q", "k", "v", "g", "beta")), None, None, o.data_ptr() + 2 * shift, None,
                                        ws.data_ptr(), ws.numel(), gate.data_ptr(), w.data_ptr(), 1e-6, y.data_ptr(), inv.data_ptr(), stream)
            _lib.check(rc, "kda_chunk_fwd_norm")
            assert path in _lib.profile_report()
        finally:
            lib.kda_profile_enable(0)
        assert not o[:shift].any() and not o[shift + y.numel():].any()
        results.append([o[shift:shift + y.numel()], y, inv])
    assert all(torch.equal(a, b) and a.any() for a, b in zip(*results))


@pytest.mark.parametrize("lens,H,segments", [([64 * 20 + 5, 64 * 9, 64 * 16, 64 * 18 + 1], 4, 1),                                         # 16 recurrences, mean 15
                                             ([64 * 70 + 7, 30, 64 * 3 + 9, 0], 4, 4),                                                 # 16, mean 18
                                             ([64 * 50, 64 * 3 + 9, 64 * 19 + 63], 7, 1),                                              # 21, mean 24, three sequences
                                             ([64 * 60, 64 * 3 + 9, 64 * 19 + 63, 0, 5, 64 * 30, 64 * 9], 3, 4),                       # 21, mean 17, seven
                                             ([64, 64 * 110 + 7, 64 * 4 + 3, 0], 7, 1),                                                # 28, mean 28
                                             ([64 * 120 + 1, 64, 64 * 4 + 3, 5], 6, 1),                                                # 24, mean 31
                                             ([64 * 125 + 1, 64, 64 * 4 + 3, 5], 6, 2),                                                # 24, mean 32
                                             ([64 * 300 + 5, 30, 0], 1, 8), ([1, 64 * 200 + 63, 64 * 90, 0], 1, 4)])                   # 3, mean 100; 4, mean 72
def test_packed_batches_take_the_way_their_shape_says(lens, H, segments):
    """Which kernels run, and every output against the oracle: chains of very different lengths, segments of one chunk or none, empty sequences."""
    from experiment_swa_kda_b200 import _lib
    m = _kda_mod()
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    d = O.make_inputs(1, cu[-1], H, 128, 128, seed=500 + H, with_state=True, n_states=len(lens))
    x = {n: (t.float() if n == "h0" else t.bfloat16()).to(D0).requires_grad_(True) for n, t in d.items()}
    gen = torch.Generator().manual_seed(17)
    do, ds = torch.randn(d["v"].shape, generator=gen).bfloat16().to(D0), torch.randn(d["h0"].shape, generator=gen).to(D0)
    _lib.load().kda_profile_enable(1)
    try:
        o, s = m.chunk_kda(x["q"], x["k"], x["v"], x["g"], x["beta"], initial_state=x["h0"], output_final_state=True, lane="tc",
                           cu_seqlens=torch.tensor(cu, dtype=torch.int32, device=D0))
        got = [o, s, *torch.autograd.grad((o, s), list(x.values()), (do, ds))]
        ran = set(_lib.profile_report())
    finally:
        _lib.load().kda_profile_enable(0)
    walked = {"tc_walk_fwd_kernel", "tc_walk_bwd_kernel"}
    assert ran & walked == (walked if segments == 1 else set()) and ("tc_scan_fixup_kernel" in ran) == (segments > 1)
    # segments: 2 segments - 1 final states of 96 KB a recurrence, beside what each chunk-head has
    sh = _lib.ChunkShape(len(lens), 0, cu[-1], H, 128, 128, _lib.DTYPE_BF16, _lib.DTYPE_BF16, _lib.LANE_TC, 1, 0.1)
    panels = (cu[-1] // 64 + len(lens)) * H * (6 * 16384 + 3 * 8192 + 2 * 32768 + 512 + 768 + (0 if segments == 1 else 16384 + 2 * 32768))
    assert (_lib.load().kda_chunk_workspace_bytes(sh) - panels) // (len(lens) * H * 98304) == (0 if segments == 1 else 2 * segments - 1)
    y = {n: t.detach().float().requires_grad_(True) for n, t in x.items()}
    eo, es = O.kda_recurrence_varlen(y["q"], y["k"], y["v"], y["g"], y["beta"], cu, initial_state=y["h0"])
    for a, b in zip(got, (eo, es, *torch.autograd.grad((eo, es), list(y.values()), (do.float(), ds)))):
        assert O.rel_l2(a, b) <= BF16_TOL
