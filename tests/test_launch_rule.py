"""The default launch of a product: the rule at both sides of every line (pure host arithmetic, 148 SMs), and on the GPU (`-m gpu`) one
product per kernel that it can choose, each checked to be the kernel that the case is there for."""
import ctypes
import random

import pytest
import torch

import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import cabi, workloads

DEV = "cuda:0"
IMMUTABLE, EVEN = cabi.SPMV_MATRIX_IMMUTABLE, cabi.SPMV_ROWS_EVEN


def _launch(rows, cols, padded, flags, sms=148):
    """(lanes per row, threads of a CTA, rows of the tail, rolling loads)"""
    lib = cabi.load()
    out = [ctypes.c_int() for _ in range(4)]
    cabi.check(lib, lib.macko_spmv_default_launch(rows, cols, padded, sms, flags, *[ctypes.byref(v) for v in out]))
    return tuple(v.value for v in out)


@pytest.mark.parametrize("rows,cols,row,want", [
    # lanes: a row, two rows, four rows per warp (4736 warps)
    (4736, 3000, 900, (32, 512, 0, 0)), (4737, 3000, 900, (16, 512, 0, 0)), (9473, 3000, 900, (16, 512, 0, 0)), (9474, 3000, 900, (8, 512, 0, 0)),
    (9474, 37999, 900, (8, 1024, 0, 0)), (9474, 38000, 900, (16, 1024, 0, 0)),
    # threads by columns
    (9474, 9999, 900, (8, 512, 0, 0)), (9474, 10000, 900, (8, 1024, 0, 0)), (4737, 16383, 900, (16, 512, 0, 0)), (4737, 16384, 900, (16, 1024, 0, 0)),
    (4000, 33088, 900, (32, 512, 0, 0)), (4000, 33089, 900, (32, 1024, 0, 0)),
    # six units in flight take more than three sub-steps a row; shorter ones have the shape of macko_spmv_shape
    (9474, 10000, 193, (8, 1024, 0, 0)), (9474, 10000, 192, (16, 512, 0, 0)), (4737, 16384, 385, (16, 1024, 0, 0)), (4737, 16384, 384, (32, 512, 0, 0)),
    (4000, 33089, 769, (32, 1024, 0, 0)), (4000, 33089, 768, (32, 512, 0, 0)),
    # tail: a last round less than half full, rows long enough
    (9473, 3000, 1150, (16, 512, 1, 0)), (9473, 3000, 1149, (16, 512, 0, 0)), (18944, 3000, 575, (8, 512, 0, 0)), (18945, 3000, 575, (8, 512, 1, 0)),
    (18945, 3000, 574, (8, 512, 0, 0)), (18944 + 4736, 3000, 575, (8, 512, 4736, 0)), (18944 + 4737, 3000, 1150, (8, 512, 4737, 0)),
    (18944 + 4737, 3000, 1149, (8, 512, 0, 0)), (28416, 3000, 1200, (8, 512, 9472, 0)), (28417, 3000, 1200, (8, 512, 0, 0)),
    # rolling loads
    (9474, 3000, 1899, (8, 512, 0, 0)), (9474, 3000, 1900, (8, 512, 0, 1)), (18945, 10000, 1900, (8, 1024, 1, 1)), (4737, 3000, 2500, (16, 512, 0, 0)),
])
def test_rule_for_even_rows(rows, cols, row, want):
    assert _launch(rows, cols, rows * row, IMMUTABLE | EVEN) == want
    assert _launch(rows, cols, rows * row, EVEN)[:3] == want[:3]


@pytest.mark.parametrize("rows,cols,row,want", [
    # blocks for 0.55 of the warps
    (5209, 3000, 900, (32, 512, 0, 0)), (5210, 3000, 900, (16, 512, 0, 0)), (10419, 3000, 900, (16, 512, 0, 0)), (10420, 3000, 900, (8, 512, 0, 0)),
    # the chain of the average row: 64 sub-steps, 16 above 16384 columns, 96 where no warp gets a second block of two rows
    (10420, 16384, 4096, (8, 1024, 0, 0)), (10420, 16384, 4097, (16, 1024, 948, 0)), (10420, 16384, 8192, (16, 1024, 948, 0)), (10420, 16384, 8193, (32, 1024, 0, 0)),
    (10420, 16383, 8193, (32, 512, 0, 0)), (10420, 16385, 1024, (8, 1024, 0, 0)), (10420, 16385, 1025, (16, 1024, 0, 0)), (10420, 16385, 2048, (16, 1024, 948, 0)),
    (10420, 16385, 2049, (32, 1024, 0, 0)), (9472, 16384, 9000, (16, 1024, 0, 0)), (9476, 16384, 9000, (32, 1024, 0, 0)),
    # two thirds dense: no row can be much longer
    (11000, 12000, 10000, (16, 512, 1528, 0)), (18943, 12000, 10000, (16, 512, 0, 0)), (18944, 12000, 10000, (8, 1024, 0, 0)), (5209, 12000, 10000, (32, 512, 0, 0)),
    (20000, 38000, 30000, (16, 1024, 1056, 0)), (11000, 30000, 20000, (16, 1024, 1528, 0)), (11000, 30000, 19999, (32, 1024, 0, 0)),
    # threads of a warp per row
    (5209, 33088, 3000, (32, 512, 0, 0)), (5209, 33089, 3000, (32, 1024, 0, 0)), (5210, 16384, 13000, (16, 1024, 0, 0)), (5210, 16385, 3000, (32, 1024, 0, 0)),
    (2368, 20000, 4600, (32, 1024, 0, 1)), (2369, 20000, 4600, (32, 512, 0, 0)), (948, 20000, 4600, (32, 1024, 0, 1)), (947, 20000, 4600, (32, 512, 0, 1)),
    # rolling loads, tail
    (2368, 20000, 3600, (32, 512, 0, 1)), (2368, 20000, 3599, (32, 512, 0, 0)), (10419, 3000, 1150, (16, 512, 947, 0)), (10419, 3000, 1149, (16, 512, 0, 0)),
    (12000, 3000, 2000, (8, 512, 0, 0)),
])
def test_rule_for_rows_that_nobody_has_looked_at(rows, cols, row, want):
    assert _launch(rows, cols, rows * row, 0) == want
    # "immutable" moves loads and changes no bit of the result: lanes and tail do not depend on it
    lanes, threads, tail, rolling = _launch(rows, cols, rows * row, IMMUTABLE)
    assert (lanes, tail, rolling) == (want[0], want[2], 0)
    # CTAs of a warp per row, more than a row per warp: 1024 threads from 16384 columns on if the matrix may change, else from 33089 on
    assert threads == (512 if want[0] == 32 and rows >= 5210 and cols <= 33088 else want[1])


def test_flag_does_not_decide_the_order_of_the_sums():
    rng = random.Random(5)
    for _ in range(3000):   # the number of threads says which warp takes a row, not how the row is added up
        rows, cols = int(2 ** rng.uniform(0, 17)), int(2 ** rng.uniform(3, 18))
        padded = min(int(rows * cols * rng.uniform(0.01, 1.0)), 2 ** 31 - 8)
        for even in (0, EVEN):
            one, two = _launch(rows, cols, padded, even), _launch(rows, cols, padded, even | IMMUTABLE)
            assert (one[0], one[2]) == (two[0], two[2])


def test_refusals():
    lib = cabi.load()
    out = [ctypes.byref(ctypes.c_int()) for _ in range(4)]
    assert lib.macko_spmv_default_launch(4, 4, 8, 148, 2, *out) == cabi.ERR_INVALID_ARGUMENT
    assert lib.macko_spmv_default_launch(4, 4, 8, 148, 8, *out) == cabi.ERR_INVALID_ARGUMENT
    assert lib.macko_spmv_default_launch(-1, 4, 8, 148, 0, *out) == cabi.ERR_INVALID_ARGUMENT
    assert lib.macko_spmv_default_launch(4, 4, 8, 0, 0, *out) == cabi.ERR_INVALID_ARGUMENT
    assert lib.macko_spmv_default_launch(4, 4, 8, 148, 0, None, *out[1:]) == cabi.ERR_INVALID_ARGUMENT
    assert lib.macko_spmv_default_launch(1 << 31, 4, 8, 148, 0, *out) == cabi.ERR_SIZE_OVERFLOW
    assert lib.macko_spmv_default_launch(0, 4, 0, 148, 0, *out) == cabi.OK


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def _matrix(rows, cols, d, dtype):
    """iid, with an empty row, rows that end and start early (the last ones are the tail's): none is longer than the others."""
    M = workloads.bernoulli_matrix(rows, cols, d, seed=rows + cols, device=DEV)
    M[rows // 2] = 0
    M[-1] = 0
    M[-2, cols // 3:] = 0
    M[3, : cols // 2] = 0
    return (M.float() * 30).round().clamp(-127, 127).to(torch.int8) if dtype is torch.int8 else M.to(dtype)


def _reference(M, x):
    ref = torch.cat([part.double() @ x.double() for part in M.split(2048)])
    return ref, torch.cat([part.double().abs() @ x.double().abs() for part in M.split(2048)])


def _vector(cols, dtype):
    x = 0.1 * torch.randn(cols, generator=torch.Generator(device=DEV).manual_seed(cols), device=DEV)
    return x.to(torch.float16 if dtype is torch.int8 else dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("frozen,rows,cols,d,lanes,threads,tail,roll", [
    (True, 4736, 3000, 0.3, 32, 512, 0, 0), (True, 4736, 33100, 0.05, 32, 1024, 0, 0), (True, 4737, 3000, 0.3, 16, 512, 0, 0), (True, 9473, 3000, 0.5, 16, 512, 1, 0),
    (True, 4800, 16384, 0.03, 16, 1024, 0, 0), (True, 9473, 38000, 0.03, 16, 1024, 1, 0), (True, 9474, 2000, 0.3, 8, 512, 0, 0), (True, 19001, 900, 0.7, 8, 512, 57, 0),
    (True, 9501, 4096, 0.5, 8, 512, 0, 1), (True, 19001, 4096, 0.5, 8, 512, 57, 1), (True, 9501, 10001, 0.03, 8, 1024, 0, 0), (True, 19001, 10001, 0.1, 8, 1024, 57, 0),
    (True, 9501, 10001, 0.25, 8, 1024, 0, 1), (True, 19001, 10001, 0.25, 8, 1024, 57, 1),
    (False, 5209, 3000, 0.3, 32, 512, 0, 0), (False, 5210, 3000, 0.3, 16, 512, 0, 0), (False, 10001, 2000, 0.7, 16, 512, 529, 0), (False, 10420, 2000, 0.3, 8, 512, 0, 0),
    (False, 10420, 10000, 0.03, 8, 1024, 0, 0), (False, 5210, 16400, 0.2, 32, 1024, 0, 0), (False, 2368, 6000, 0.85, 32, 1024, 0, 1), (False, 2369, 6000, 0.85, 32, 512, 0, 0),
    (False, 900, 6000, 0.7, 32, 512, 0, 1), (False, 11001, 5000, 0.9, 16, 512, 1529, 0),
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.int8])
def test_product_against_float64(frozen, rows, cols, d, lanes, threads, tail, roll, dtype):
    """Bound: y is rounded once (half a unit in the last place of its type). A lane adds its elements into four fp32 accumulators, at
    most stored / 32 each plus a few of the last iteration, then two additions and five exchanges; every addition is off by at most
    2^-24 of the sum of |value * x|, products are exact."""
    if rows * cols > 64 << 20 and dtype is not torch.float16 and not roll:
        pytest.skip("one type for the large ones")
    M, x = _matrix(rows, cols, d, dtype), _vector(cols, dtype)
    comp = macko_spmv.compress(M)
    matrix = macko_spmv.freeze(comp, windows=False) if frozen else comp
    if _sms() == 148 and dtype is not torch.int8:   # int8 drops the values that round to 0
        assert not frozen or (macko_spmv.rows_are_even(comp) and matrix.plan is None)
        flags = 0 if not frozen else IMMUTABLE | EVEN if matrix.even_rows else IMMUTABLE
        assert _launch(rows, cols, comp[0].numel(), flags) == (lanes, threads, tail, roll)
    ref, l1 = _reference(M, x)
    half_ulp = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
    bound = half_ulp * ref.abs() * (1 + 1e-3) + 2.0 ** -24 * (cols / 32 + 8 + 7) * l1 * 1.01 + 2.0 ** -24
    y = macko_spmv.multiply(matrix, x)
    assert bool(((y.double() - ref).abs() <= bound).all()), float(((y.double() - ref).abs() / bound).max())
    assert torch.equal(y, macko_spmv.multiply(matrix, x))
    assert torch.equal(y, macko_spmv.multiply(matrix, x, out=torch.empty_like(y)))
    if frozen:   # the operator, which a traced program takes
        assert torch.equal(y, torch.ops.macko_spmv.multiply_frozen.default(*comp[:5], x, matrix.even_rows))


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols,d", [(5000, 4096, 0.5), (9473, 4096, 0.5), (10000, 4096, 0.5), (10000, 8192, 0.5), (12000, 20000, 0.1), (11000, 6000, 0.9),
                                         (2000, 6000, 0.8), (7000, 39000, 0.1)])
def test_immutable_flag_changes_no_bit(rows, cols, d):
    M, x = _matrix(rows, cols, d, torch.float16), _vector(cols, torch.float16)
    comp = macko_spmv.compress(M)
    plain = macko_spmv.multiply(comp, x)
    for even in (0, EVEN):
        y = [torch.empty_like(plain), torch.empty_like(plain)]
        for out, flags in zip(y, (even, even | IMMUTABLE)):
            torch.ops.macko_spmv.multiply_ex.default(*comp[:5], x, out, 1.0, 0.0, flags)
        assert torch.equal(y[0], y[1])
        assert even or torch.equal(y[0], plain)
    assert torch.equal(macko_spmv.multiply(macko_spmv.freeze(comp, plan=False), x), plain)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(4800, 3000), (9600, 5000)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.int8])
def test_frozen_uneven_rows_have_the_lanes_of_the_plain_product(rows, cols, dtype):
    """Rows of very uneven length keep the lanes that bound their chains, whatever `freeze` was asked for."""
    M = workloads.skewed_matrix(rows, cols, seed=3, device=DEV, mean_density=0.2)
    M = (M.float() * 30).round().clamp(-127, 127).to(torch.int8) if dtype is torch.int8 else M.to(dtype)
    x = _vector(cols, dtype)
    comp = macko_spmv.compress(M)
    plain = macko_spmv.multiply(comp, x)
    for frozen in (macko_spmv.freeze(comp, plan=False), macko_spmv.freeze(comp)):
        assert not frozen.even_rows and not macko_spmv.rows_are_even(comp)
        assert torch.equal(macko_spmv.multiply(frozen, x, out=torch.empty_like(plain)), plain)
        if frozen.plan is None:
            assert torch.equal(macko_spmv.multiply(frozen, x), plain)


@pytest.mark.gpu
def test_rows_are_even():
    def even(lengths):
        M = torch.zeros(len(lengths), 4096, dtype=torch.float16, device=DEV)
        for r, n in enumerate(lengths):
            M[r, :n] = 1.0
        comp = macko_spmv.compress(M)
        assert all(f.even_rows == macko_spmv.rows_are_even(comp) for f in (macko_spmv.freeze(comp), macko_spmv.freeze(comp, plan=True)))
        assert not macko_spmv.freeze(macko_spmv.compress(M.bfloat16())).even_rows   # so few rows: the launch is the same
        assert not macko_spmv.freeze(comp, plan=False).even_rows   # the sums of the plain product
        return macko_spmv.rows_are_even(comp)

    assert even([800] * 40) and even([0] * 40)
    # 40 rows, mean 800 + 4 = 804: 9/8 of it and 64 are 968.5
    assert even([800] * 39 + [960]) and not even([800] * 39 + [970])
