"""`multiply` takes a way around the operator dispatcher when a call only wants the product. These tests check that it
gives the bits of the operator, and that everything else still goes through the operator: gradients, subclasses, modes,
transforms, tracing, profiling, errors."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import workloads

DEV = "cuda:0"


def test_anything_but_a_plain_call_is_declined():
    t = torch.zeros(8)
    for args in ((), (1,), (1, 2), ((), t), ([t] * 5, t), ((t, t, t, 1, 8), t), ((t, t, t, 1.0, 8), t), ((t, t, t, 1), t)):
        assert macko_spmv._direct_multiply(*args) is None
    with pytest.raises(AssertionError):
        macko_spmv.multiply((t.half(), t.byte(), t.int(), 1, 8), t.half())


class _Seen(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.names.append(str(func))
        return func(*args, **(kwargs or {}))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.int8])
def test_same_bits_as_the_operator(dtype):
    M = workloads.bernoulli_matrix(300, 515, 0.4, seed=4, device=DEV)
    M = (M * 30).round().clamp(-100, 100).to(torch.int8) if dtype is torch.int8 else M.to(dtype)
    comp = macko_spmv.compress(M)
    V = torch.randn(515, device=DEV).to(torch.float16 if dtype is torch.int8 else dtype)
    exp = torch.ops.macko_spmv.multiply.default(*comp, V)
    y = macko_spmv._direct_multiply(comp, V)
    assert y is not None and torch.equal(y, exp) and y.dtype == exp.dtype
    frozen = macko_spmv.freeze(comp)
    assert torch.equal(macko_spmv._direct_multiply(frozen, V), exp)
    if dtype is torch.float16:
        planned = macko_spmv.freeze(comp, plan=True)
        got = macko_spmv._direct_multiply(planned, V)
        meta = planned.plan_meta
        assert torch.equal(got, torch.ops.macko_spmv.multiply_planned.default(*comp, planned.plan, meta[0], meta[1], meta[3], V, True))


@pytest.mark.gpu
def test_what_watches_operators_still_sees_them():
    M = workloads.bernoulli_matrix(64, 256, 0.4, seed=4, device=DEV)
    comp = macko_spmv.compress(M)
    V = torch.randn(256, device=DEV).half()
    exp = macko_spmv.multiply(comp, V)
    with _Seen() as seen:
        assert torch.equal(macko_spmv.multiply(comp, V), exp)
    assert any("macko_spmv.multiply" in n for n in seen.names)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as p:
        macko_spmv.multiply(comp, V)
    assert any(e.key == "macko_spmv::multiply" for e in p.key_averages())
    leaf = V.clone().requires_grad_()
    assert macko_spmv._direct_multiply(comp, leaf) is None
    assert macko_spmv._direct_multiply(comp, V.as_subclass(type("Sub", (torch.Tensor,), {}))) is None
    assert torch.equal(torch.vmap(lambda v: macko_spmv.multiply(comp, v))(torch.stack([V, V]))[1], exp)
    assert torch.equal(torch.compile(lambda v: macko_spmv.multiply(comp, v) * 1, fullgraph=True, backend="eager")(V), exp)
    with torch.inference_mode(), torch.no_grad():
        assert torch.equal(macko_spmv.multiply(comp, V), exp)


@pytest.mark.gpu
def test_errors_are_those_of_the_operator():
    M = workloads.bernoulli_matrix(64, 256, 0.4, seed=4, device=DEV)
    comp = macko_spmv.compress(M)
    V = torch.randn(256, device=DEV).half()
    with pytest.raises(RuntimeError, match="torch.half"):
        macko_spmv.multiply(comp, V.float())
    with pytest.raises(RuntimeError, match="M_cols"):
        macko_spmv.multiply(comp, V[:200].contiguous())
    with pytest.raises(RuntimeError, match="M_rows"):
        macko_spmv.multiply((comp[0], comp[1], comp[2], 63, 256), V)
    with pytest.raises(AssertionError):
        macko_spmv.multiply(comp, torch.randn(512, device=DEV).half()[::2])
    with pytest.raises(AssertionError):
        macko_spmv.multiply(comp, V.cpu())
