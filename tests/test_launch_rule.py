"""GPU test (`-m gpu`) of the default launch on both sides of every line of its rule (148 SMs): lanes per row by the number of rows, two
CTAs of 512 threads or one of 1024 by the number of columns, and rows that are too short for six units in flight.

Bound as in test_tail_rows: y is rounded once, a lane adds at most stored / 32 / 4 + 8 elements, then at most two additions and five
exchanges, each off by at most 2^-24 of the sum of |value * x|."""
import pytest
import torch

import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import workloads

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("rows,cols,d", [
    (4736, 3000, 0.3), (4737, 3000, 0.3), (9473, 2000, 0.3), (9474, 2000, 0.3),          # a row, two rows, four rows per warp
    (5209, 3000, 0.3), (5210, 3000, 0.3), (10419, 2000, 0.3), (10420, 2000, 0.3),        # the same for a matrix that may change
    (4800, 16383, 0.03), (4800, 16384, 0.03), (9473, 9999, 0.03), (9473, 10000, 0.03),   # 1024 threads with 16 and 8 lanes
    (9473, 37999, 0.02), (2368, 6000, 0.85), (2369, 6000, 0.85), (2368, 6000, 0.7),      # few long rows
    (947, 6000, 0.85), (948, 6000, 0.85), (4736, 1000, 0.75), (4737, 1000, 0.37), (9473, 600, 0.3), (9473, 600, 0.35),         # around three sub-steps a row
])
def test_product_against_float64(rows, cols, d):
    M = workloads.bernoulli_matrix(rows, cols, d, seed=rows + cols, device=DEV)
    M[rows // 2] = 0
    M[-1] = 0.5
    x = torch.randn(cols, generator=torch.Generator(device=DEV).manual_seed(cols), device=DEV).half()
    comp = macko_spmv.compress(M)
    ref = torch.cat([part.double() @ x.double() for part in M.split(2048)])
    l1 = torch.cat([part.double().abs() @ x.double().abs() for part in M.split(2048)])
    bound = 2.0 ** -11 * ref.abs() * (1 + 1e-3) + 2.0 ** -24 * (cols / 32 + 8 + 7) * l1 * 1.01 + 2.0 ** -24
    for matrix in (comp, macko_spmv.freeze(comp, plan=False)):
        y = macko_spmv.multiply(matrix, x)
        assert bool(((y.double() - ref).abs() <= bound).all()), float(((y.double() - ref).abs() / bound).max())
        assert torch.equal(y, macko_spmv.multiply(matrix, x))
