"""Packed batches with more sequences than one pass of the chunk table's block takes (512), with empty and one-token ones at the seams."""

import pytest
import torch

from oracle import kda_oracle as O

pytestmark = pytest.mark.gpu
D0 = "cuda:0"


def _batch(n_seq, seed):
    gen = torch.Generator().manual_seed(seed)
    lens = torch.randint(0, 12, (n_seq,), generator=gen)
    lens[torch.randint(0, n_seq, (8,), generator=gen)] = torch.tensor([64, 65, 128, 129, 63, 1, 200, 0])
    lens[510 if n_seq > 512 else 0] = 0 if n_seq > 1 else 130
    cu = torch.zeros(n_seq + 1, dtype=torch.int32)
    cu[1:] = lens.cumsum(0)
    return cu, O.make_inputs(1, int(cu[-1]), 1, 16, 16, seed=seed)


def _run(d, cu):
    import experiment_swa_kda_b200 as m
    x = [d[n].to(D0) for n in ("q", "k", "v", "g", "beta")]
    return [t.double().cpu() for t in m.chunk_kda(*x, cu_seqlens=cu.to(D0), output_final_state=True)]


@pytest.mark.parametrize("n_seq", [1, 31, 33, 511, 512, 513, 1025])
def test_every_sequence_finds_its_chunks(n_seq):
    cu, d = _batch(n_seq, 40 + n_seq)
    o, state = _run(d, cu)
    want, want_state = O.kda_recurrence_varlen(*(d[n].double() for n in ("q", "k", "v", "g", "beta")), cu_seqlens=cu, compute_dtype=torch.float64)
    # float32 arithmetic over sums of at most 64 terms a chunk: 1e-5 is the lane's bar everywhere
    assert O.rel_l2(o, want) < 1e-5 and O.rel_l2(state, want_state) < 1e-5


@pytest.mark.parametrize("at", [3, 511, 512, 700])
def test_a_wrong_segment_far_into_the_table_is_empty_and_the_others_stand(at):
    from experiment_swa_kda_b200 import ops
    cu, d = _batch(777, 5)
    o, _ = _run(d, cu)
    bad = cu.clone()
    bad[at] = int(cu[-1]) + 5          # segment at - 1 reaches past the tokens, segment at runs backwards
    got, _ = _run(d, bad)
    with pytest.raises(RuntimeError, match="cu_seqlens is inconsistent"):
        ops.poll_status(torch.device(D0))
    a, b = int(cu[at - 1]), int(cu[at + 1])
    assert torch.equal(got[:, :a], o[:, :a]) and torch.equal(got[:, b:], o[:, b:])
