"""Stored counts within a few thousand elements of 2^31, the largest that the entry points take: element positions that run
ahead of the last stored element must not wrap. A small matrix sits at the very end of buffers of 2^31 - 8 elements (6 GB
of zeros in front of it, which no row refers to), and has to give what it gives in buffers of its own size."""
import ctypes

import pytest
import torch

import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import cabi, workloads

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
P_MOST = 2**31 - 8


@pytest.fixture(scope="module")
def buffers():
    yield {dt: torch.zeros(P_MOST * 2 if dt == "values" else P_MOST // 2, dtype=torch.uint8, device=DEV) for dt in ("values", "deltas")}
    torch.cuda.empty_cache()


def _at_the_end(comp, buffers):
    """The compressed matrix moved to the last elements of buffers of P_MOST elements: (values, deltas, row_indices)."""
    values, deltas, ri = comp[:3]
    P = values.numel()
    big_v, big_d = buffers["values"].view(torch.float16), buffers["deltas"]
    big_v[P_MOST - P:] = values
    big_d[(P_MOST - P) // 2:] = deltas
    return big_v, big_d, ri + (P_MOST - P)


def _stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("rows,cols", [(5, 4099), (2400, 700), (2, 130003)])   # a CTA per row, a warp per row, rows beyond shared memory
def test_decompress(buffers, rows, cols):
    lib = cabi.load()
    comp = macko_spmv.compress(workloads.bernoulli_matrix(rows, cols, 0.6, seed=rows, device=DEV))
    v, d, ri = _at_the_end(comp, buffers)
    dense = torch.full((rows, cols), 7.0, dtype=torch.float16, device=DEV)
    cabi.check(lib, lib.macko_decompress_fp16(v.data_ptr(), d.data_ptr(), ri.data_ptr(), rows, cols, P_MOST, dense.data_ptr(), _stream()))
    assert torch.equal(dense, macko_spmv.decompress(comp))


def _emit(lib, M, ri, P, v, d, workspace_bytes):
    call = lib.macko_compress_emit_int8 if M.dtype == torch.int8 else lib.macko_compress_emit
    cabi.check(lib, call(M.data_ptr(), *M.shape, ri.data_ptr(), P, v.data_ptr(), d.data_ptr(), v.data_ptr(), workspace_bytes, _stream()))
    count = ctypes.c_uint32()
    cabi.check(lib, lib.macko_compress_overflow(ctypes.byref(count), _stream()))
    return count.value


# few columns: the elements end 1..7 slots in front of the padded count, where the clearing loop's next step lies beyond 2^31
@pytest.mark.parametrize("dtype", [torch.float16, torch.int8])
@pytest.mark.parametrize("rows,cols", [(7, 4099), (3, 9)])
def test_emit(buffers, rows, cols, dtype):
    lib = cabi.load()
    M = workloads.bernoulli_matrix(rows, cols, 0.6, seed=rows, device=DEV)
    M = (M * 30).round().clamp(-100, 100).to(dtype)
    if int(macko_spmv.compress(M)[2][-1]) % 8 == 0:
        M[0, 2] = 1 - (M[0, 2] != 0).to(dtype)        # one element more or less
    values, deltas, ri = macko_spmv.compress(M)[:3]
    P = values.numel()
    assert int(ri[-1]) < P
    v, d = buffers["values"].view(dtype)[-P_MOST:], buffers["deltas"]
    v[-P - 64:] = 3                                   # the slots in front of the matrix keep this
    assert _emit(lib, M, ri + (P_MOST - P), P_MOST, v, d, P_MOST) == 0
    assert torch.equal(v[P_MOST - P:], values) and bool((v[-P - 64: -P] == 3).all())
    assert torch.equal(d[(P_MOST - P) // 2:], deltas) and not d[-P // 2 - 32: -P // 2].any()


def test_emit_refuses_what_lies_beyond(buffers):
    """row_indices of another matrix: a row of 3000 elements that starts 64 slots in front of the end."""
    lib = cabi.load()
    M = torch.ones(2, 3000, dtype=torch.float16, device=DEV)
    v, d = buffers["values"].view(torch.float16), buffers["deltas"]
    v[-128:] = 3
    ri = torch.tensor([P_MOST - 64, P_MOST, P_MOST], dtype=torch.int32, device=DEV)
    assert _emit(lib, M, ri, P_MOST, v, d, P_MOST) == 2
    assert bool((v[-64:] == 1).all()) and bool((v[-128:-64] == 3).all())


@pytest.mark.parametrize("lanes", [4, 8, 16, 32])
@pytest.mark.parametrize("x_in_shared", [0, 1])
def test_product(buffers, lanes, x_in_shared):
    """Rows that end with the buffers, in every launch shape, the same bits as in small buffers."""
    lib = cabi.load()
    rows, cols = 37, 4099
    M = workloads.bernoulli_matrix(rows, cols, 0.6, seed=lanes, device=DEV)
    M[3] = 0
    comp = macko_spmv.compress(M)
    big = _at_the_end(comp, buffers)
    x = torch.randn(cols, device=DEV).half()
    for steps in (2, 4, 6):
        ys = []
        for v, d, ri, P in ((*comp[:3], comp[0].numel()), (*big, P_MOST)):
            y = torch.full((rows,), 7.0, dtype=torch.float16, device=DEV)
            cabi.check(lib, lib.macko_spmv_fp16_tuned(v.data_ptr(), d.data_ptr(), ri.data_ptr(), rows, cols, P, x.data_ptr(), y.data_ptr(),
                                                      1.0, 0.0, _stream(), lanes, steps, x_in_shared, 0))
            ys.append(y)
        assert torch.equal(*ys), steps


@pytest.mark.parametrize("frozen", [False, True])
def test_product_default_and_batched(buffers, frozen):
    rows, cols = 5, 4099      # rows of about 2500 elements take the same launch shape with either count
    comp = macko_spmv.compress(workloads.bernoulli_matrix(rows, cols, 0.6, seed=9, device=DEV))
    big = (*_at_the_end(comp, buffers), rows, cols)
    V = torch.randn(8, cols, device=DEV).half()
    if frozen:
        comp, big = macko_spmv.freeze(comp, plan=False), macko_spmv.freeze(big, plan=False)
    assert torch.equal(macko_spmv.multiply(big, V[0]), macko_spmv.multiply(comp, V[0]))
    for n in (2, 4, 8):
        assert torch.equal(macko_spmv.multiply_batched(big, V[:n]), macko_spmv.multiply_batched(comp, V[:n])), n


def test_planned(buffers):
    """A plan of rows that end with the buffers: the same segments, so the same bits."""
    rows, cols, seg = 3, 60000, 3840
    comp = macko_spmv.compress(workloads.bernoulli_matrix(rows, cols, 0.6, seed=10, device=DEV))
    big = (*_at_the_end(comp, buffers), rows, cols)
    small, large = (macko_spmv.freeze(c, plan=True, segment_elements=seg) for c in (comp, big))
    assert small.plan_meta[:4] == large.plan_meta[:4] and small.plan_meta[3] == rows
    x = torch.randn(cols, device=DEV).half()
    assert torch.equal(macko_spmv.multiply(large, x), macko_spmv.multiply(small, x))
