"""GPU tests of the compressor and the decompressor at the sizes where their kernels change what they do, bit for bit
against the oracle: steps of 256 (count) and 512 (emit) columns, output rings of 512 waiting slots, pad batches of 512
(runs of more than 8192 zeros), rows at every offset from a 16-byte boundary, the row scan's 16384 entries; and for the
decompressor windows of 1024 columns, steps that reach over several windows, and both of its kernels."""
import numpy as np
import pytest
import torch

import oracle
import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import cabi

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


# 2400 rows and more, or more columns than shared memory holds: a warp per row; fewer rows: a CTA per row
@pytest.mark.parametrize("density", [0.02, 0.5, 1.0])
@pytest.mark.parametrize("rows,cols", [(2400, 1), (2400, 33), (2401, 1023), (2400, 1024), (2400, 1025), (2401, 2111), (2370, 4096),
                                       (40, 1025), (40, 4099), (4, 130003)])
def test_decompress_edges(rows, cols, density):
    m = _matrix(rows, cols, density, rows + cols)
    comp = macko_spmv.compress(m.to(DEV))
    exp = oracle.decompress((_u16(comp[0]), comp[1].cpu().numpy(), comp[2].cpu().numpy(), rows, cols))
    assert np.array_equal(_u16(macko_spmv.decompress(comp)).reshape(rows, cols), exp)
    # a destination two bytes behind a 16-byte boundary, with guards on both sides
    lib = cabi.load()
    out = torch.full((rows * cols + 64,), 0x5A5A, dtype=torch.int16, device=DEV)
    cabi.check(lib, lib.macko_decompress_fp16(comp[0].data_ptr(), comp[1].data_ptr(), comp[2].data_ptr(), rows, cols, comp[0].numel(),
                                              out.data_ptr() + 2, torch.cuda.current_stream().cuda_stream))
    got = out.cpu().numpy().view(np.uint16)
    assert np.array_equal(got[1 : 1 + rows * cols].reshape(rows, cols), exp)
    assert got[0] == 0x5A5A and (got[1 + rows * cols :] == 0x5A5A).all()
