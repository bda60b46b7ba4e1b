"""GPU tests of the compressor at the sizes where its kernels change what they do, bit for bit against the oracle: steps of
256 (count) and 512 (emit) columns, output rings of 512 waiting slots, pad batches of 512 (runs of more than 8192
zeros), rows at every offset from a 16-byte boundary, the row scan's 16384 entries."""
import numpy as np
import pytest
import torch

import oracle
import macko_spmv_b200 as macko_spmv

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _u16(t):
    return t.detach().cpu().contiguous().view(torch.int16).numpy().view(np.uint16)


def _matrix(rows, cols, density, seed):
    g = torch.Generator().manual_seed(seed)
    m = torch.randn(rows, cols, generator=g) * (torch.rand(rows, cols, generator=g) < density)
    m = m.half()
    if cols > 20:
        m[0] = 0                              # nothing stored
        m[1 % rows, : cols - 1] = -0.0        # one element behind as many (negative-zero) pads as the row holds
        m[1 % rows, cols - 1] = 2.0
        m[2 % rows, 1:] = 0                   # zeros to the end of the row
        m[2 % rows, 0] = 3.0
        m[3 % rows] = 1.0                     # every column
        m[4 % rows, cols // 2] = float("nan")
    return m


def _check_compress(m, dev):
    exp = oracle.compress(_u16(m).reshape(m.shape)) if m.dtype != torch.int8 else oracle.compress_int8(m.numpy())
    values, deltas, ri, _, _ = macko_spmv.compress(dev)
    got = values.cpu().numpy() if m.dtype == torch.int8 else _u16(values)
    assert np.array_equal(ri.cpu().numpy(), exp[2]) and np.array_equal(got, exp[0]) and np.array_equal(deltas.cpu().numpy(), exp[1])


SHAPES = [(7, 1), (9, 8), (33, 15), (33, 255), (17, 256), (17, 257), (9, 511), (9, 512), (9, 513), (6, 1025), (6, 4093), (5, 9001), (5, 20011)]


@pytest.mark.parametrize("density", [0.01, 0.5, 0.97])
@pytest.mark.parametrize("rows,cols", SHAPES)
def test_compress_edges(rows, cols, density):
    m = _matrix(rows, cols, density, rows * cols)
    _check_compress(m, m.to(DEV))
    # the matrix two bytes behind a 16-byte boundary: element-wise loads
    shifted = torch.empty(rows * cols + 1, dtype=torch.float16, device=DEV)[1:].view(rows, cols).copy_(m)
    _check_compress(m, shifted)
    m8 = (m.float().nan_to_num().clamp(-3, 3) * 40).round().to(torch.int8)
    _check_compress(m8, m8.to(DEV))


@pytest.mark.parametrize("rows", [16382, 16383, 16384, 40001])
def test_row_scan_of_many_rows(rows):
    m = torch.zeros(rows, 3, dtype=torch.float16)
    m[::3, 1] = 1.0
    m[5::7, 2] = 2.0
    _check_compress(m, m.to(DEV))
