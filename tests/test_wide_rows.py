"""GPU test (`-m gpu`) of the warp-per-row product whose CTAs of 1024 threads share one copy of x: columns around the line where it
starts, around the widest x that shared memory takes, and beyond, for every value type.

Bound: y is rounded once (half a unit in the last place of its type). A lane adds its elements into four fp32 accumulators, stored / 128
each, then two additions and five exchanges; every addition is off by at most 2^-24 of the sum of |value * x| in front of it.
Products are exact (fp16, int8) or rounded once to fp32 (bf16: exact as well, 8 x 8 bits)."""
import pytest
import torch

import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import workloads

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


# x and its frame fill 65 KB at 33088 columns; 116032 is the last width that fits shared memory
@pytest.mark.parametrize("rows,cols,d", [(40, 33088, 0.3), (40, 33089, 0.3), (1, 40001, 1.0), (33, 57409, 0.1), (4737, 33100, 0.03), (9, 116031, 0.2),
                                         (9, 116032, 0.2), (9, 116033, 0.2)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.int8])
def test_product_against_float64(rows, cols, d, dtype):
    M = workloads.bernoulli_matrix(rows, cols, d, seed=rows + cols, device=DEV)
    M = (M.float() * 30).round().clamp(-127, 127).to(torch.int8) if dtype is torch.int8 else M.to(dtype)
    x = (0.05 * torch.randn(cols, generator=torch.Generator(device=DEV).manual_seed(cols), device=DEV)).to(torch.float16 if dtype is torch.int8 else dtype)
    comp = macko_spmv.compress(M)
    ref = torch.mv(M.double(), x.double())
    l1 = torch.mv(M.double().abs(), x.double().abs())
    half_ulp = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
    steps = cols / 128 + 8 + 2 + 5
    bound = half_ulp * ref.abs() * (1 + 1e-3) + 2.0 ** -24 * steps * l1 * 1.01 + 2.0 ** -24   # the last: subnormal fp16
    for matrix in (comp, macko_spmv.freeze(comp, plan=False)):
        y = macko_spmv.multiply(matrix, x)
        assert bool(((y.double() - ref).abs() <= bound).all()), float(((y.double() - ref).abs() / bound).max())
        assert torch.equal(y, macko_spmv.multiply(matrix, x))
