"""Calls that move the same bytes and do the same sums in another shape take about the same time.

Each compares a shape that a dispatch or a walk over the work can serve badly with one that fills the chip, as the ratio of two
times taken in turn.  The bounds lie between what the shape costs by nature and what it cost when it was served badly; both figures
stand beside them."""

import ctypes

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


def _convolutions(n, B, T, C, windows):
    from experiment_swa_kda_b200 import _lib
    lib = _lib.load()
    xs, ws = [torch.randn(B, T, C, device=D0).bfloat16() for _ in range(n)], [torch.randn(C, 4, device=D0) for _ in range(n)]
    ys, fins = [torch.empty_like(x) for x in xs], [torch.empty(B, C, 4, device=D0, dtype=torch.bfloat16) for _ in range(n)]
    held = [(ctypes.c_void_p * n)(*[t.data_ptr() for t in ts]) for ts in (xs, ws, ys, fins)]
    a = [ctypes.cast(h, ctypes.c_void_p) for h in held]

    def call(keep=(xs, ws, ys, fins, held)):
        _lib.check(lib.kda_conv_fwd_rows(n, B, T, C, 4, _lib.DTYPE_BF16 | 0x100, 1, a[0], C, a[1], None, a[2], a[3] if windows else None,
                                         torch.cuda.current_stream().cuda_stream), "convolution")
    return call


# by nature 1.43 and 1.27 (halo rows and windows of every sequence); 1.91 and 1.59 with most warps of the streaming kernel without a run
@pytest.mark.parametrize("T,windows,bound", [(32, False, 1.67), (64, True, 1.43)])
def test_convolutions_of_short_sequences(T, windows, bound):
    short, long = _times([_convolutions(3, 8192 // T, T, 2048, windows), _convolutions(3, 1, 8192, 2048, windows)], 10)
    assert short < bound * long


def _backward(packed, n, length, heads, gates=torch.bfloat16):
    from experiment_swa_kda_b200 import _lib, ops
    B, T = (1, n * length) if packed else (n, length)
    gen = torch.Generator(device=D0).manual_seed(n)
    draw = lambda *s: torch.randn(*s, device=D0, generator=gen)
    q, k, v, do = (draw(B, T, heads, 128).bfloat16() for _ in range(4))
    g, beta = (-0.1 * draw(B, T, heads, 128).abs()).to(gates), torch.sigmoid(draw(B, T, heads)).to(gates)
    cu = torch.arange(0, n * length + 1, length, device=D0, dtype=torch.int32) if packed else None
    _, _, saved = ops.chunk_kda_fwd(q, k, v, g, beta, None, cu, 128 ** -0.5, True, False, lane=_lib.LANE_TC)
    return lambda: ops.chunk_kda_bwd(q, k, v, g, beta, cu, do, None, saved, False)


# A batch of ragged or short sequences has slots at the end of the chunk table that no sequence uses (here every second and every
# fourth).  1.08 and 1.03 by nature (the table's launch, the slots' blocks in the other kernels); 1.52 and 1.18 where the chunk-heads
# of the intra-chunk backward are dealt out to its blocks in advance
@pytest.mark.parametrize("n,length,bound", [(74, 64, 1.25), (37, 192, 1.1)])
def test_backward_of_packed_sequences_equals_a_fixed_batch(n, length, bound):
    packed, fixed = _times([_backward(True, n, length, 16), _backward(False, n, length, 16)], 4)
    assert packed < bound * fixed


# 1.14 to 1.16 by nature (twice the bytes, through the threads); 1.27 without the next chunk-head's rows on their way into L2
def test_backward_with_float32_gates():
    from experiment_swa_kda_b200 import _lib
    calls = [_backward(False, 22, 3000, 16, gates) for gates in (torch.float32, torch.bfloat16)]
    best = [float("inf")] * 2
    for _ in range(6):
        for i, call in enumerate(calls):
            call()
            torch.cuda.synchronize()
            _lib.profile_report()
            _lib.profile(True)
            try:
                for _ in range(4):
                    call()
            finally:
                _lib.profile(False)
            launches, ms = _lib.profile_report()["tc_intra_bwd_kernel"]
            best[i] = min(best[i], ms / launches)
    assert best[0] < 1.215 * best[1]
