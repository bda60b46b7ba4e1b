"""Stored counts within a few thousand elements of 2^31, the largest that the entry points take: element positions that run
ahead of the last stored element must not wrap. A small matrix sits at the very end of buffers of 2^31 - 8 elements (6 GB
of zeros in front of it, which no row refers to), and has to give what it gives in buffers of its own size."""
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
