"""GPU test (`-m gpu`) of the product whose last rows are walked with a warp per row: row counts on both sides of a full round of blocks
and of half a round more (148 SMs, 32 warps each), 8 and 16 lanes per row, every value type, empty and full rows in the tail.

Bound: y is rounded once (half a unit in the last place of its type). In the tail a lane adds its elements into four fp32
accumulators (stored / 128 each), then two additions and five exchanges; with 8 lanes stored / 32, two and three. Every addition is
off by at most 2^-24 of the sum of |value * x| in front of it; products are exact."""
import pytest
import torch

import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import workloads

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
OPS = torch.ops.macko_spmv


# 8 lanes: blocks of four rows, 4736 of them a round, rows of 575 elements for a tail of one row per warp, 1150 for two; 16 lanes: of
# two, 1150 elements a row: from 38000 columns on, and up to 10419 rows where nothing is declared (CTAs of 512 threads)
@pytest.mark.parametrize("rows,cols,d", [(18944, 900, 0.7), (18945, 900, 0.7), (18951, 900, 0.7), (18951, 900, 0.5), (23681, 1700, 0.7), (28416, 1700, 0.7), (28417, 1700, 0.7),
                                         (37889, 900, 0.7),
                                         (18947, 10000, 0.06), (9473, 38000, 0.03), (14208, 38000, 0.03),
                                         (9473, 2000, 0.7), (10001, 2000, 0.7), (10419, 2000, 0.7), (10001, 1600, 0.7)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.int8])
def test_product_against_float64(rows, cols, d, dtype):
    if rows * cols > 100 << 20 and dtype is not torch.float16:
        pytest.skip("one type for the large ones")
    M = workloads.bernoulli_matrix(rows, cols, d, seed=rows + cols, device=DEV)
    M[-1] = 0
    M[-2] = M[-2].abs() + 0.01
    M[-5, : cols // 2] = 0
    M = (M.float() * 30).round().clamp(-127, 127).to(torch.int8) if dtype is torch.int8 else M.to(dtype)
    g = torch.Generator(device=DEV).manual_seed(cols)
    x = (0.1 * torch.randn(cols + 1, generator=g, device=DEV)).to(torch.float16 if dtype is torch.int8 else dtype)[1:]   # not 16-byte aligned
    comp = macko_spmv.compress(M)
    ref = torch.cat([part.double() @ x.double() for part in M.split(4096)])
    l1 = torch.cat([part.double().abs() @ x.double().abs() for part in M.split(4096)])
    half_ulp = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
    bound = half_ulp * ref.abs() * (1 + 1e-3) + 2.0 ** -24 * (cols / 32 + 8 + 7) * l1 * 1.01 + 2.0 ** -24
    for matrix in (comp, macko_spmv.freeze(comp, plan=False)):
        y = macko_spmv.multiply(matrix, x)
        assert bool(((y.double() - ref).abs() <= bound).all()), float(((y.double() - ref).abs() / bound).max())
    y = torch.ones(rows, dtype=x.dtype, device=DEV)
    OPS.multiply_out.default(*comp[:5], x, y, 0.5, -2.0)
    want = 0.5 * ref - 2.0
    assert bool(((y.double() - want).abs() <= half_ulp * want.abs() * (1 + 1e-3) + bound + 2.0 ** -22).all())
