"""Calls that move the same bytes and do the same sums in another shape take about the same time.

Each compares a shape that a dispatch or a walk over the work can serve badly with one that fills the chip, as the ratio of two
times taken in turn.  The bounds lie between what the shape costs by nature and what it cost when it was served badly; both figures
stand beside them."""

import pytest
import torch

pytestmark = pytest.mark.gpu

D0 = "cuda:0"


def _times(calls, launches):
    """Shortest device time of each call in us, `launches` calls from one graph, all of them in turn."""
    graphs = []
    for call in calls:
        call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(launches):
                call()
        graphs.append(graph)
    best = [float("inf")] * len(calls)
    for _ in range(8):
        for i, graph in enumerate(graphs):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            best[i] = min(best[i], a.elapsed_time(b) * 1e3 / launches)
    return best


def _gate(tokens, heads, key_dim):
    from experiment_swa_kda_b200 import _lib
    lib = _lib.load()
    raw = torch.randn(tokens, heads, key_dim, device=D0).bfloat16()
    logits = torch.randn(tokens, heads, device=D0).bfloat16()
    A_log, bias = torch.randn(heads, device=D0), torch.randn(heads * key_dim, device=D0)
    g, beta = torch.empty(tokens, heads, key_dim, device=D0), torch.empty(tokens, heads, device=D0)
    return lambda: _lib.check(lib.kda_gate_fwd(tokens, heads, key_dim, _lib.DTYPE_BF16, raw.data_ptr(), logits.data_ptr(), A_log.data_ptr(), bias.data_ptr(),
                                               -5.0, g.data_ptr(), beta.data_ptr(), torch.cuda.current_stream().cuda_stream), "gate")


# 1.7 by nature (as many beta logits as quads of channels), 13 with blocks of 128 columns of a row
def test_gate_activations_of_narrow_rows():
    narrow, wide = _times([_gate(1 << 21, 2, 4), _gate(1 << 17, 1, 128)], 10)
    assert narrow < 3 * wide

