"""The workspace-free compressor entry point, `macko_compress_emit_static`.

Some hosts cannot give the library scratch memory: they run inside an application that has handed all
device memory to its own pool, or they sit on a path where a cudaMalloc is not allowed. The compressor needs
none: both emit entry points write values and packed deltas in one pass, and the workspace of the one that takes
it is left alone. The tests call them through the C ABI with raw device pointers and compare with the oracle, in
a captured graph and from two streams at once too. Collected last so that a failure here cannot hide other
tests behind `-x`.
"""
import numpy as np
import pytest
import torch

import oracle
from macko_spmv_b200 import cabi, workloads

pytestmark = pytest.mark.gpu


def _matrix(rows, cols, density, seed):
    M = workloads.bernoulli_matrix(rows, cols, density, seed=seed, device="cuda")
    M.view(torch.int16)[::7, ::5] = -32768          # some -0.0: pads must keep the sign bit
    return M


def _expected(M):
    return oracle.compress(M.cpu().view(torch.int16).numpy().view(np.uint16))


def _check(got, exp):
    assert np.array_equal(got[0].cpu().view(torch.int16).numpy().view(np.uint16), exp[0]), "values differ"
    assert np.array_equal(got[1].cpu().numpy(), exp[1]), "deltas differ"


def _count(lib, M, stream):
    rows, cols = M.shape
    ri = torch.empty(rows + 1, dtype=torch.int32, device=M.device)
    cabi.check(lib, lib.macko_compress_count(M.data_ptr(), rows, cols, ri.data_ptr(), stream))
    n = int(ri[rows].item())
    return ri, (n + 7) // 8 * 8


def _outputs(P):
    return (torch.full((P,), float("nan"), dtype=torch.float16, device="cuda"),
            torch.full((P // 2,), 0xCD, dtype=torch.uint8, device="cuda"))


def _emit_static(lib, M, ri, P, out, stream):
    rows, cols = M.shape
    cabi.check(lib, lib.macko_compress_emit_static(M.data_ptr(), rows, cols, ri.data_ptr(), P,
                                                   out[0].data_ptr(), out[1].data_ptr(), stream))


def test_both_entry_points_match_the_oracle():
    lib = cabi.load()
    assert lib.macko_compress_static_capacity() == 16 * 1024 * 1024
    stream = torch.cuda.current_stream().cuda_stream
    # first a matrix that comes close to the limit of the static entry point, then a small ragged one
    for (rows, cols, density, seed) in [(4096, 4096, 0.9, 11), (37, 515, 0.3, 12)]:
        M = _matrix(rows, cols, density, seed)
        exp = _expected(M)
        ri, P = _count(lib, M, stream)
        assert 0 < P <= lib.macko_compress_static_capacity() and np.array_equal(ri.cpu().numpy(), exp[2])
        out = _outputs(P)
        _emit_static(lib, M, ri, P, out, stream)
        _check(out, exp)
        out = _outputs(P)
        ws = torch.full((lib.macko_compress_workspace_bytes(P),), 0xAB, dtype=torch.uint8, device="cuda")
        cabi.check(lib, lib.macko_compress_emit(M.data_ptr(), rows, cols, ri.data_ptr(), P, out[0].data_ptr(),
                                                out[1].data_ptr(), ws.data_ptr(), ws.numel(), stream))
        _check(out, exp)
        assert bool((ws == 0xAB).all()), "the workspace was written"


def test_static_entry_point_in_a_captured_graph():
    lib = cabi.load()
    M = _matrix(300, 1027, 0.4, 13)
    ri, P = _count(lib, M, torch.cuda.current_stream().cuda_stream)
    out = _outputs(P)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _emit_static(lib, M, ri, P, out, torch.cuda.current_stream().cuda_stream)
    exp = _expected(M)
    for _ in range(2):
        out[0].fill_(float("nan"))
        out[1].fill_(0xCD)
        graph.replay()
        _check(out, exp)


def test_static_entry_point_from_two_streams_at_once():
    lib = cabi.load()
    mats = [_matrix(2000, 2111, 0.5, 14), _matrix(1999, 2500, 0.3, 15)]
    counted = [_count(lib, M, torch.cuda.current_stream().cuda_stream) for M in mats]
    outs = [[_outputs(P) for _ in range(4)] for _, P in counted]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for k in range(4):
        for M, (ri, P), out, s in zip(mats, counted, outs, streams):
            _emit_static(lib, M, ri, P, out[k], s.cuda_stream)
    torch.cuda.synchronize()
    for M, out in zip(mats, outs):
        exp = _expected(M)
        for o in out:
            _check(o, exp)


def test_static_entry_point_rejects_oversize():
    lib = cabi.load()
    cap = lib.macko_compress_static_capacity()
    a = 0x1000  # never dereferenced: the size check comes first
    st = lib.macko_compress_emit_static(a, 8192, 8192, a, cap + 8, a, a, None)
    assert st == cabi.ERR_WORKSPACE
    assert b"exceeds the built-in scratch" in lib.macko_last_error()
    assert lib.macko_compress_emit_static(a, 4, 4, a, 12, a, a, None) == cabi.ERR_INVALID_ARGUMENT
