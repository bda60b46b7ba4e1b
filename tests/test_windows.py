"""GPU tests (`-m gpu`) of the multi-vector product over column windows: the windows against their definition, the product
against float64 at the sizes where it can go wrong, and what a frozen matrix does with them.

Bound of a product: y is the fp16 rounding (2^-11 of |y|) of fp32 sums. A lane adds at most S elements in sequence, S = stored
elements of a row in one window / 8 + 8; the exchanges add three additions, the sum over W windows W more. Each
addition is off by at most 2^-24 of the partial sum, whose size is at most l1 = sum |value * x|; products are exact."""
import copy

import numpy as np
import pytest
import torch

import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import cabi, workloads
from macko_spmv_b200.linear import MackoLinear

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
OPS = torch.ops.macko_spmv


def _layout(rows, cols, padded):
    """The rule of macko_spmv_b200/csrc/windows.cuh: (windows, columns of a window)."""
    least = max(1, -(-cols // 1408))
    blocks, row = (rows + 3) // 4, padded / rows

    def cost(w):
        warps = max(1, 148 // w) * 32
        return 0.5 * (blocks / warps + -(-blocks // warps)) * (row / (64.0 * w) + 1.5) + 0.3 * w

    w = min(range(least, least + 6), key=lambda k: (cost(k), k))
    return w, max(8, (-(-cols // w) + 7) // 8 * 8)


def _check(Y, M, V, what):
    least = max(1, -(-M.shape[1] // 1408))
    ref = V.double() @ M.double().t()
    l1 = V.double().abs() @ M.double().abs().t()
    steps = (1408 + 128) / 8 + 8 + 3 + least + 5   # the widest window, the largest number of windows
    bound = 2.0 ** -11 * ref.abs() + 2.0 ** -24 * steps * l1 * 1.01 + 2.0 ** -25   # the last: spacing of subnormal fp16
    bad = (Y.double() - ref).abs() > bound
    assert not bad.any(), f"{what}: {int(bad.sum())} outside, worst {float(((Y.double() - ref).abs() / bound).max()):.2f} of the bound"


def _multiply(comp, V, frozen=True):
    return OPS.multiply_windowed.default(*comp[:5], OPS.windows_build.default(comp[1], comp[2], comp[3], comp[4]), V, frozen)


@pytest.mark.parametrize("rows,cols,d", [(37, 100, 0.5), (64, 4096, 0.03), (9, 1408, 1.0), (40, 1409, 0.9), (11, 12000, 0.3)])
def test_sections_follow_their_definition(rows, cols, d):
    M = workloads.bernoulli_matrix(rows, cols, d, seed=cols, device=DEV)
    M[1] = 0
    M[2, : cols - 1] = 0
    M[2, cols - 1] = 1.0
    comp = macko_spmv.compress(M)
    W, width = _layout(rows, cols, comp[0].numel())
    got = OPS.windows_build.default(comp[1], comp[2], rows, cols).view(torch.int32).view(W, rows, 2).cpu().numpy().astype(np.int64)
    nibbles = comp[1].cpu().numpy()
    delta = np.stack([nibbles & 15, nibbles >> 4], 1).reshape(-1).astype(np.int64)
    ri = comp[2].cpu().numpy()
    for r in range(rows):
        b, e = int(ri[r]), int(ri[r + 1])
        col = np.cumsum(delta[b:e] + 1) - 1   # column of every stored element
        # a unit belongs to the window of its first element, the row's first unit to window 0
        starts = [b] + [k for k in range((b // 8 + 1) * 8, e, 8)] if e > b else []
        owner = {k: 0 if k == b else min(int(col[k - b]) // width, W - 1) for k in starts}
        for w in range(W):
            mine = [k for k in starts if owner[k] == w]
            later = [k for k in starts if owner[k] > w]
            stop = min(later) if later else e
            n = stop - min(mine) if mine else 0
            assert (got[w, r, 1] & 0xffffffff) >> 8 == n, (r, w)
            if mine:
                first = min(mine)
                front = (int(col[first - b - 1]) + 1 if first > b else 0) - w * width + 16
                assert got[w, r, 0] == first and (got[w, r, 1] & 255) == front, (r, w)


# one column to several windows, rows around the blocks of four, batches around 4 and 8 and over several groups
@pytest.mark.parametrize("rows,cols,d", [(1, 1, 1.0), (3, 7, 0.5), (5, 1407, 0.4), (64, 1408, 0.5), (5000, 1409, 0.3), (40000, 1408, 0.1), (1003, 771, 0.3),
                                         (130, 4096, 0.5), (4097, 3329, 0.9), (257, 11008, 0.2), (31, 30011, 0.05), (12, 140001, 0.01),
                                         (20000, 256, 0.5)])
def test_product_against_float64(rows, cols, d):
    M = workloads.bernoulli_matrix(rows, cols, d, seed=rows + cols, device=DEV)
    comp = macko_spmv.compress(M)
    windows = OPS.windows_build.default(comp[1], comp[2], rows, cols)
    g = torch.Generator(device=DEV).manual_seed(3)
    for batch in (1, 3, 4, 5, 8, 9, 17):
        V = torch.randn(batch, cols, generator=g, device=DEV).half()
        Y = OPS.multiply_windowed.default(*comp[:5], windows, V, True)
        _check(Y, M, V, f"{rows}x{cols} batch {batch}")
        assert torch.equal(Y, OPS.multiply_windowed.default(*comp[:5], windows, V, False))


def test_uneven_rows_and_misaligned_x():
    M = torch.zeros(70, 6000, dtype=torch.float16, device=DEV)
    M[3, ::7] = 1.5
    M[4, 5] = -2.0
    M[9] = 0.25
    M[10, 1650:1700] = 1.0
    M[69, 5999] = 3.0
    comp = macko_spmv.compress(M)
    V = torch.randn(8 * 6000 + 1, generator=torch.Generator(device=DEV).manual_seed(5), device=DEV).half()[1:].view(8, 6000)
    assert V.data_ptr() % 16 != 0
    _check(_multiply(comp, V), M, V, "uneven rows")
    skew = workloads.skewed_matrix(600, 5000, 9, device=DEV, mean_density=0.2)
    V = V.reshape(-1)[: 8 * 5000].view(8, 5000)
    _check(_multiply(macko_spmv.compress(skew), V), skew, V, "skewed")


def test_alpha_beta_and_refusals():
    lib = cabi.load()
    stream = torch.cuda.current_stream().cuda_stream
    for rows, cols in ((70, 3000), (40000, 200)):   # several windows; one
        M = workloads.bernoulli_matrix(rows, cols, 0.4, seed=1, device=DEV)
        comp = macko_spmv.compress(M)
        windows = OPS.windows_build.default(comp[1], comp[2], rows, cols)
        V = torch.randn(5, cols, generator=torch.Generator(device=DEV).manual_seed(2), device=DEV).half()
        Y = torch.ones(5, rows, dtype=torch.float16, device=DEV)
        need = lib.macko_spmm_windowed_workspace_bytes(rows, cols, comp[0].numel(), 5)
        ws = torch.empty(max(need, 1), dtype=torch.uint8, device=DEV)

        def call(batch=5, windows_bytes=windows.numel(), ws_bytes=need, flags=0, win=windows.data_ptr()):
            return lib.macko_spmm_fp16_windowed(comp[0].data_ptr(), comp[1].data_ptr(), comp[2].data_ptr(), rows, cols, comp[0].numel(), win,
                                                windows_bytes, V.data_ptr(), Y.data_ptr(), batch, 2.0, -1.0, ws.data_ptr(), ws_bytes, flags, stream)

        assert call() == cabi.OK
        ref = 2.0 * (V.double() @ M.double().t()) - 1.0
        assert float((Y.double() - ref).norm() / ref.norm()) < 5e-4
        assert call(batch=-1) == cabi.ERR_INVALID_ARGUMENT and call(flags=2) == cabi.ERR_INVALID_ARGUMENT
        assert call(windows_bytes=windows.numel() - 8) == cabi.ERR_WORKSPACE and call(win=None) == cabi.ERR_INVALID_ARGUMENT
        if need:
            assert call(ws_bytes=need - 1) == cabi.ERR_WORKSPACE
        assert call(batch=0) == cabi.OK
    with pytest.raises(RuntimeError):
        OPS.multiply_windowed.default(*comp[:5], windows, V[:, :100].contiguous(), True)
    empty = macko_spmv.compress(torch.zeros(0, 64, dtype=torch.float16, device=DEV))
    assert _multiply(empty, V[:, :64].contiguous()).shape == (5, 0)


def test_graph_and_streams_side_by_side():
    """The partial sums belong to the call: products of one matrix may overlap, in a graph or on two streams."""
    M = workloads.magnitude_pruned_matrix(2000, 5000, 0.4, 3, device=DEV)
    frozen = macko_spmv.freeze(macko_spmv.compress(M))
    g = torch.Generator(device=DEV).manual_seed(8)
    Vs = [torch.randn(8, 5000, generator=g, device=DEV).half() for _ in range(4)]
    want = [macko_spmv.multiply_batched(frozen, V) for V in Vs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [None] * 4
    for i, V in enumerate(Vs):
        with torch.cuda.stream(streams[i % 2]):
            got[i] = macko_spmv.multiply_batched(frozen, V)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [macko_spmv.multiply_batched(frozen, V) for V in Vs]
    for _ in range(2):
        for y in got:
            y.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("frozen", [True, False])
def test_x_written_by_the_kernel_in_front_is_seen(frozen):
    """y of one batched product is x of the next, whose CTAs are already resident while it is written: eager and as one graph.

    Every stage is checked against float64 of what it read, so the bound does not grow along the chain."""
    n = 2000
    M = workloads.bernoulli_matrix(n, n, 0.3, seed=77, device=DEV, scale=0.04)
    comp = macko_spmv.compress(M)
    windows = OPS.windows_build.default(comp[1], comp[2], n, n)
    V = torch.randn(8, n, generator=torch.Generator(device=DEV).manual_seed(4), device=DEV).half()

    def chain():
        out = [V]
        for _ in range(6):
            out.append(OPS.multiply_windowed.default(*comp[:5], windows, out[-1], frozen))
        return out

    eager = chain()
    for a, b in zip(eager, eager[1:]):
        _check(b, M, a, "chain")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain()
    for _ in range(3):
        for y in out[1:]:
            y.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, eager))


def test_route_of_a_frozen_matrix(monkeypatch):
    """Which batches take the windows, and what makes a call take the other routes."""
    M = workloads.magnitude_pruned_matrix(1500, 5000, 0.3, 3, device=DEV)
    comp = macko_spmv.compress(M)
    frozen = macko_spmv.freeze(comp)
    assert frozen.windows is not None and macko_spmv.freeze(comp, plan=False).windows is None
    assert macko_spmv.freeze(macko_spmv.compress(M.bfloat16())).windows is None
    sparse = torch.zeros(2000, 5000, dtype=torch.float16, device=DEV)
    sparse[::7, 3] = 1.0
    assert macko_spmv.freeze(macko_spmv.compress(sparse)).windows is None   # 8 bytes per row and window would outweigh it

    def V(batch, **kw):
        return torch.randn(batch, 5000, generator=torch.Generator(device=DEV).manual_seed(batch), device=DEV).half().requires_grad_(kw.get("grad", False))

    pay = macko_spmv._windows_pay
    assert [pay(frozen, V(b)) for b in (0, 1, 2, 3, 8, 9, 16, 65)] == [False, False, False, True, True, True, True, False]
    assert not pay(frozen, V(9, grad=True)) and pay(frozen, V(8, grad=True))
    with torch.autograd.forward_ad.dual_level():
        assert not pay(frozen, V(9))
    # what the direct calls answer is what the operators give; above the limit the dense copy
    assert frozen.windows_batch >= 16
    for b in (3, 8, 9, 16, 65, 80):
        want = OPS.multiply_windowed.default(*comp[:5], frozen.windows, V(b), True) if b <= frozen.windows_batch else V(b) @ macko_spmv.decompress(comp).t()
        assert torch.equal(macko_spmv.multiply_batched(frozen, V(b)), want)
    with pytest.raises(RuntimeError):
        macko_spmv.multiply_batched(frozen, V(9)[:, :4000].contiguous())
    with pytest.raises(RuntimeError):
        macko_spmv.multiply_batched(frozen, V(9).float())
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(V(70), V(71)[:70])
        tangent = torch.autograd.forward_ad.unpack_dual(macko_spmv.multiply_batched(frozen, dual)).tangent
        assert tangent is not None and float((tangent.float() - V(71)[:70].float() @ M.float().t()).norm()) < 5e-3 * float(tangent.float().norm())
    # gradients and batching rules of the dense copy are still there
    x = V(17, grad=True)
    macko_spmv.multiply_batched(frozen, x).sum().backward()
    assert float((x.grad.float() - M.float().sum(0)).abs().max()) < 0.1
    for batch in (3, 8, 9):
        _check(macko_spmv.multiply_batched(frozen, V(batch)), M, V(batch), f"frozen, batch {batch}")
    # a matrix written after freeze(): another one in the same buffers
    turned = M.roll(1, 0).contiguous()
    for a, b in zip(comp[:3], macko_spmv.compress(turned)[:3]):
        a.copy_(b)
    assert not pay(frozen, V(8))
    _check(macko_spmv.multiply_batched(frozen, V(8)), turned, V(8), "written after freeze()")


@pytest.mark.parametrize("rows,cols,d", [(2048, 2048, 0.7), (2048, 2048, 0.9), (4096, 1024, 0.9)])
def test_sums_of_a_frozen_matrix_stay_in_fp32(rows, cols, d):
    """9..16 vectors of a matrix for which no dense copy pays: compressed passes before `freeze` and after it, never a GEMM whose sums
    may be fp16."""
    M = workloads.magnitude_pruned_matrix(rows, cols, d, 3, device=DEV)
    comp = macko_spmv.compress(M)
    frozen = macko_spmv.freeze(comp)
    assert not macko_spmv._dense_copy_pays(comp, 9) and not macko_spmv._dense_copy_pays(comp, 16)
    for batch in (9, 16):
        V = torch.randn(batch, cols, generator=torch.Generator(device=DEV).manual_seed(batch), device=DEV).half()
        Y = macko_spmv.multiply_batched(frozen, V)
        assert torch.equal(Y, OPS.multiply_windowed.default(*comp[:5], frozen.windows, V, True))
        _check(Y, M, V, f"batch {batch}")


def test_layers_follow_their_buffers():
    """MackoLinear batches over the windows while they are those of its buffers; copies and reloaded layers stay right."""
    W = workloads.magnitude_pruned_matrix(900, 3000, 0.4, 31, device=DEV)
    layer = MackoLinear(macko_spmv.compress(W)).freeze()
    x = torch.randn(7, 3000, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV).half()
    _check(layer(x), W, x, "layer")
    _check(copy.deepcopy(layer)(x), W, x, "copied layer")
    assert layer._frozen_as_is() is layer._frozen
    W2 = W.roll(7, 0).contiguous()   # the same rows in another order: buffers of the same sizes
    two = MackoLinear(macko_spmv.compress(W2))
    assert two.c_0.shape == layer.c_0.shape
    layer.load_state_dict(two.state_dict())   # writes the frozen buffers in place, without another freeze()
    _check(layer(x), W2, x, "reloaded layer")
    layer.c_0, layer.c_1, layer.c_2 = (t.clone() for t in MackoLinear(macko_spmv.compress(W)).compressed[:3])
    assert layer._frozen_as_is() is None
    _check(layer(x), W, x, "replaced buffers")


def test_inference_mode():
    """Nobody counts writes to inference tensors: no windows, so a layer that is reloaded without another freeze() stays right."""
    with torch.inference_mode():
        W = workloads.magnitude_pruned_matrix(640, 2500, 0.5, 7, device=DEV)
        layer = MackoLinear(macko_spmv.compress(W)).freeze()
        x = torch.randn(8, 2500, generator=torch.Generator(device=DEV).manual_seed(2), device=DEV).half()
        assert layer._frozen.windows is None
        _check(layer(x), W, x, "inference tensors")
        _check(layer(x.repeat(2, 1)), W, x.repeat(2, 1), "inference tensors, two groups")
        W2 = W.roll(7, 0).contiguous()   # the same rows in another order: buffers of the same sizes
        layer.load_state_dict(MackoLinear(macko_spmv.compress(W2)).state_dict())
        _check(layer(x), W2, x, "reloaded inference tensors")


def test_windows_argument():
    """False: no windows, the plan as ever; True: also with plan=False, for inference tensors and where they are heavy."""
    M = workloads.magnitude_pruned_matrix(640, 2500, 0.5, 7, device=DEV)
    comp = macko_spmv.compress(M)
    V = torch.randn(8, 2500, generator=torch.Generator(device=DEV).manual_seed(2), device=DEV).half()
    none = macko_spmv.freeze(comp, windows=False)
    assert none.windows is None and none.plan_meta == macko_spmv.freeze(comp).plan_meta
    assert torch.equal(macko_spmv.multiply_batched(none, V), macko_spmv.multiply_batched(comp, V))
    assert MackoLinear(comp).freeze(windows=False)._frozen.windows is None
    want = macko_spmv.multiply_batched(macko_spmv.freeze(comp), V)
    for frozen in (macko_spmv.freeze(comp, windows=True), macko_spmv.freeze(comp, plan=False, windows=True)):
        assert torch.equal(macko_spmv.multiply_batched(frozen, V), want)
    with torch.inference_mode():
        frozen = macko_spmv.freeze(macko_spmv.compress(M), windows=True)
        assert frozen.windows is not None and frozen.windows_of is None
        assert torch.equal(macko_spmv.multiply_batched(frozen, V.clone()), want)
    sparse = torch.zeros(2000, 5000, dtype=torch.float16, device=DEV)
    sparse[::7, 3] = 1.0
    frozen = macko_spmv.freeze(macko_spmv.compress(sparse), windows=True)
    V = V.repeat(1, 2)
    assert frozen.windows is not None
    _check(macko_spmv.multiply_batched(frozen, V), sparse, V, "heavy windows")
    assert macko_spmv.freeze(macko_spmv.compress(M.bfloat16()), windows=True).windows is None


class _WindowedCalls(torch.utils._python_dispatch.TorchDispatchMode):
    """Records the `frozen` argument of every windowed product."""

    def __init__(self):
        super().__init__()
        self.frozen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        if func is OPS.multiply_windowed.default:
            self.frozen.append(args[7])
        return func(*args, **(kwargs or {}))


def test_values_written_after_freeze():
    """The windows do not depend on the values: a write to them alone keeps the windows, but no longer lets a product fetch them ahead
    of stream order."""
    rows, cols = 900, 3000
    W = workloads.magnitude_pruned_matrix(rows, cols, 0.4, 31, device=DEV)
    layer = MackoLinear(macko_spmv.compress(W)).freeze()
    x = torch.randn(8, cols, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV).half()
    assert macko_spmv._direct_batched(layer._frozen, x) is not None
    with _WindowedCalls() as calls:
        layer(x)
    assert calls.frozen == [True]
    layer.c_0.mul_(2.0)
    _check(layer(x), 2 * W, x, "scaled values")
    assert macko_spmv._direct_batched(layer._frozen, x) is None
    with _WindowedCalls() as calls:
        layer(x)
    assert calls.frozen == [False]
    # values that the kernel in front is still writing: y of a product that lets its successor start early
    stored = layer.c_0.numel()
    A = workloads.bernoulli_matrix(stored, 64, 0.5, seed=5, device=DEV)
    v = torch.randn(64, generator=torch.Generator(device=DEV).manual_seed(6), device=DEV).half()
    frozen_A = macko_spmv.freeze(macko_spmv.compress(A), plan=False)
    torch.autograd.graph.increment_version(layer.c_0)   # the operator's `out` argument is not counted
    for _ in range(3):
        layer.c_0.fill_(float("nan"))
        macko_spmv.multiply(frozen_A, v, out=layer.c_0)
        y = layer(x)
        _check(y, macko_spmv.decompress(layer.compressed), x, "values written by the kernel in front")
