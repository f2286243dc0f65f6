"""The scratch-free gated-RMSNorm backward (kda_rmsnorm_gate_bwd_static) against the regular entry point.

Meant for callers that cannot hand the library any scratch memory (fixed memory plans, plugins without an
allocator, paths that must not call cudaMalloc).  Called straight through the C ABI, twice in a row and from two
streams at once: a call's partial sums lie in its own dx until that is written.  Collected last on purpose.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ptr(t):
    return t.data_ptr()


@pytest.mark.parametrize("rows,dim,dtype", [(24576, 128, torch.bfloat16), (301, 256, torch.float32), (50, 96, torch.bfloat16)])
def test_static_scratch_backward_matches_regular_entry_point(rows, dim, dtype):
    from experiment_swa_kda_b200 import _lib
    lib = _lib.load()
    dev = torch.device("cuda:0")
    io = _lib.DTYPE_BF16 if dtype == torch.bfloat16 else _lib.DTYPE_F32
    stream = torch.cuda.current_stream(dev).cuda_stream
    for call in range(2):          # second call sees the first call's leftovers in the shared array
        gen = torch.Generator().manual_seed(100 * call + dim)
        x = torch.randn(rows, dim, generator=gen).to(dtype).to(dev)
        gate = torch.randn(rows, dim, generator=gen).to(dtype).to(dev)
        dy = torch.randn(rows, dim, generator=gen).to(dtype).to(dev)
        w = (1 + 0.1 * torch.randn(dim, generator=gen)).to(dev)
        y = torch.empty_like(x)
        inv = torch.empty(rows, dtype=torch.float32, device=dev)
        _lib.check(lib.kda_rmsnorm_gate_fwd(rows, dim, io, 1e-6, _ptr(x), _ptr(gate), _ptr(w), _ptr(y), _ptr(inv), stream),
                   "kda_rmsnorm_gate_fwd")
        ref = [torch.empty_like(x), torch.empty_like(x), torch.empty(dim, dtype=torch.float32, device=dev)]
        scr = torch.empty(lib.kda_rmsnorm_gate_bwd_scratch_bytes(rows, dim), dtype=torch.uint8, device=dev)
        _lib.check(lib.kda_rmsnorm_gate_bwd(rows, dim, io, _ptr(x), _ptr(gate), _ptr(w), _ptr(inv), _ptr(dy), _ptr(ref[0]),
                                            _ptr(ref[1]), _ptr(ref[2]), _ptr(scr), scr.numel(), stream), "kda_rmsnorm_gate_bwd")
        got = [torch.empty_like(x), torch.empty_like(x), torch.empty(dim, dtype=torch.float32, device=dev)]
        _lib.check(lib.kda_rmsnorm_gate_bwd_static(rows, dim, io, _ptr(x), _ptr(gate), _ptr(w), _ptr(inv), _ptr(dy),
                                                   _ptr(got[0]), _ptr(got[1]), _ptr(got[2]), stream),
                   "kda_rmsnorm_gate_bwd_static")
        torch.cuda.synchronize(dev)
        for a, b, name in zip(got, ref, ("dx", "dgate", "dweight")):
            assert torch.isfinite(a.float()).all(), name
            # same kernels, same summation order: identical bits
            assert torch.equal(a, b), name


def test_static_scratch_rejects_rows_wider_than_its_array():
    from experiment_swa_kda_b200 import _lib
    lib = _lib.load()
    rc = lib.kda_rmsnorm_gate_bwd_static(4, 512, _lib.DTYPE_F32, *([None] * 8), None)
    assert rc == -2
    assert b"unsupported" in lib.kda_error_string(rc)


def _problem(rows, dim, dtype, seed, shift=0):
    """(a call on a stream, its outputs, what the regular entry point gives, inputs); shift: dx this many elements into its buffer"""
    from experiment_swa_kda_b200 import _lib
    lib, dev, stream = _lib.load(), "cuda:0", torch.cuda.current_stream().cuda_stream
    io = _lib.DTYPE_BF16 if dtype == torch.bfloat16 else _lib.DTYPE_F32
    gen = torch.Generator(device=dev).manual_seed(seed)
    x, gate, dy = (torch.randn(rows, dim, device=dev, generator=gen).to(dtype) for _ in range(3))
    w, y, inv = torch.rand(dim, device=dev, generator=gen), torch.empty_like(x), torch.empty(rows, device=dev)
    _lib.check(lib.kda_rmsnorm_gate_fwd(rows, dim, io, 1e-6, _ptr(x), _ptr(gate), _ptr(w), _ptr(y), _ptr(inv), stream), "forward")
    outs = lambda: [torch.full((rows * dim + shift,), float("nan"), device=dev, dtype=dtype)[shift:].view(rows, dim),
                    torch.full_like(x, float("nan")), torch.full((dim,), float("nan"), device=dev)]
    want, got = outs(), outs()
    scr = torch.empty(lib.kda_rmsnorm_gate_bwd_scratch_bytes(rows, dim), dtype=torch.uint8, device=dev)
    ins = [_ptr(t) for t in (x, gate, w, inv, dy)]
    _lib.check(lib.kda_rmsnorm_gate_bwd(rows, dim, io, *ins, *[_ptr(t) for t in want], _ptr(scr), scr.numel(), stream), "backward")
    torch.cuda.synchronize()
    call = lambda st: _lib.check(lib.kda_rmsnorm_gate_bwd_static(rows, dim, io, *ins, *[_ptr(t) for t in got], st), "static")
    return call, got, want, (x, gate, dy, w, inv)


# one block (up to 8 rows), the fewest rows whose partials lie in dx, and dx at an odd element of its buffer
@pytest.mark.parametrize("rows,dim,dtype,shift", [(1, 128, torch.bfloat16, 0), (8, 64, torch.bfloat16, 1), (9, 128, torch.bfloat16, 1),
                                                  (9, 7, torch.bfloat16, 1), (17, 256, torch.bfloat16, 3), (9, 33, torch.float32, 1)])
def test_partial_sums_fit_in_the_gradient_they_make_way_for(rows, dim, dtype, shift):
    call, got, want, _ = _problem(rows, dim, dtype, rows + dim, shift)
    call(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_calls_on_two_streams_do_not_share_anything():
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    problems = [_problem(24576, 128, torch.bfloat16, 1), _problem(24576, 128, torch.bfloat16, 2)]
    for _ in range(20):
        for st, (call, got, _, _) in zip(streams, problems):
            with torch.cuda.stream(st):
                for t in got:
                    t.fill_(float("nan"))
                call(st.cuda_stream)
    torch.cuda.synchronize()
    for _, got, want, _ in problems:
        assert all(torch.equal(a, b) for a, b in zip(got, want))
