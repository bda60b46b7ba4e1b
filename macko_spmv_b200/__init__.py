"""B200-native MACKO SpMV: drop-in for the ``macko_spmv`` Python API.

``compress(M)`` -> ``(values fp16[P], deltas uint8[P/2], row_indices int32[R+1], R, C)``
``multiply(compressed, V)`` -> ``y`` fp16[R]
``move_to_device(compressed, device)``

Same functions, argument meaning and error behaviour as the reference
(src/macko_spmv/__init__.py:110-149); same `macko_spmv::multiply` operator schema
(src/macko_spmv/__init__.py:56-63). The kernels come from a prebuilt sm_100a library
behind a C ABI (``include/macko_b200.h``) instead of an import-time JIT build; there is
no CPU or PyTorch fallback: without the built libraries the import fails, and without a
CUDA device every call raises.

Use ``import macko_spmv_b200 as macko_spmv`` to switch an existing program over.
"""
from __future__ import annotations

import ctypes
import importlib.util
import os
import sysconfig

import torch

LIB_NAME = "macko_spmv"
__version__ = "0.1.0"

_PKG_DIR = os.path.dirname(os.path.abspath(__file__))
_CORE_PATH = os.path.join(_PKG_DIR, "libmacko_b200.so")
_OPS_PATH = os.path.join(_PKG_DIR, "_torch_ops.so")
_DIRECT_PATH = os.path.join(_PKG_DIR, "_torch_direct" + sysconfig.get_config_var("EXT_SUFFIX"))

# The reference reads this variable to choose its JIT cache directory
# (src/macko_spmv/__init__.py:12). Nothing is compiled at import here; it is accepted and ignored.
BUILD_DIRECTORY = os.environ.get("MACKO_SPMV_BUILD_DIRECTORY", "")


def _load_native():
    for path in (_CORE_PATH, _OPS_PATH):
        if not os.path.exists(path):
            raise ImportError(
                f"{path} is missing: build the native libraries first with "
                "`python macko_spmv_b200/build.py` (needs nvcc and g++)."
            )
    core = ctypes.CDLL(_CORE_PATH, mode=ctypes.RTLD_GLOBAL)
    torch.ops.load_library(_OPS_PATH)
    # `multiply` for calls that only want the product; built per Python version, where that has its headers
    direct = None
    if os.path.exists(_DIRECT_PATH):
        spec = importlib.util.spec_from_file_location(__name__ + "._torch_direct", _DIRECT_PATH)
        direct = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(direct)
    return core, direct


_core, _direct = _load_native()
_core.macko_version.restype = ctypes.c_int
_core.macko_last_error.restype = ctypes.c_char_p
_core.macko_status_string.restype = ctypes.c_char_p
_core.macko_status_string.argtypes = [ctypes.c_int]
_core.macko_spmm_windows_bytes.restype = ctypes.c_int64
_core.macko_spmm_windows_bytes.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int64]
_core.macko_spmv_default_launch.restype = ctypes.c_int
_core.macko_spmv_default_launch.argtypes = [ctypes.c_int64] * 3 + [ctypes.c_int, ctypes.c_uint32] + [ctypes.c_void_p] * 4


def native_library_paths() -> tuple[str, str]:
    """Paths of the C-ABI library and of the torch operator library that were loaded."""
    return _CORE_PATH, _OPS_PATH


def native_version() -> int:
    return int(_core.macko_version())


@torch.library.register_fake("macko_spmv::multiply")
def _multiply_fake(M_values, M_deltas, M_row_indices, M_rows, M_cols, V):
    # Same meta kernel as the reference (src/macko_spmv/__init__.py:105-107); int8 values give fp16 like V.
    return torch.empty((M_rows,), device=M_values.device, dtype=V.dtype)


@torch.library.register_fake("macko_spmv::compress_dense")
def _compress_fake(M):
    n = torch.library.get_ctx().new_dynamic_size()
    return (
        M.new_empty((n * 8,)),
        M.new_empty((n * 4,), dtype=torch.uint8),
        M.new_empty((M.shape[0] + 1,), dtype=torch.int32),
    )


@torch.library.register_fake("macko_spmv::multiply_batched")
def _multiply_batched_fake(M_values, M_deltas, M_row_indices, M_rows, M_cols, V):
    return torch.empty((V.shape[0], M_rows), device=M_values.device, dtype=M_values.dtype)


@torch.library.register_fake("macko_spmv::windows_build")
def _windows_build_fake(M_deltas, M_row_indices, M_rows, M_cols):
    n = torch.library.get_ctx().new_dynamic_size()
    return M_deltas.new_empty((n,))


@torch.library.register_fake("macko_spmv::multiply_windowed")
def _multiply_windowed_fake(M_values, M_deltas, M_row_indices, M_rows, M_cols, windows, V, frozen):
    return torch.empty((V.shape[0], M_rows), device=M_values.device, dtype=M_values.dtype)


@torch.library.register_fake("macko_spmv::decompress")
def _decompress_fake(M_values, M_deltas, M_row_indices, M_rows, M_cols):
    return torch.empty((M_rows, M_cols), device=M_values.device, dtype=M_values.dtype)


@torch.library.register_fake("macko_spmv::multiply_frozen")
def _multiply_frozen_fake(M_values, M_deltas, M_row_indices, M_rows, M_cols, V, even_rows=False):
    return torch.empty((M_rows,), device=M_values.device, dtype=V.dtype)


@torch.library.register_fake("macko_spmv::multiply_planned")
def _multiply_planned_fake(M_values, M_deltas, M_row_indices, M_rows, M_cols, plan, virtual_rows, segment_elements, split_rows, V, frozen):
    return torch.empty((M_rows,), device=M_values.device, dtype=M_values.dtype)


@torch.library.register_fake("macko_spmv::add_rmsnorm")
def _add_rmsnorm_fake(x, pending, weight, eps):
    return torch.empty_like(x)


@torch.library.register_fake("macko_spmv::add_rmsnorm_peer")
def _add_rmsnorm_peer_fake(x, pending, weight, eps, flags_address, world, spin_limit):
    return torch.empty_like(x)


@torch.library.register_fake("macko_spmv::rope_attention")
def _rope_attention_fake(qkv, cos_table, sin_table, position, k_cache, v_cache):
    return qkv.new_empty((qkv.numel() // 3,))


@torch.library.register_fake("macko_spmv::silu_mul")
def _silu_mul_fake(gate_up):
    return gate_up.new_empty((gate_up.shape[0] // 2,))


@torch.library.register_fake("macko_spmv::argmax")
def _argmax_fake(values):
    return values.new_empty((1,), dtype=torch.int64)


def move_to_device(compressed, device):
    """Move the three buffers of a compressed matrix (src/macko_spmv/__init__.py:110-117)."""
    return (
        compressed[0].to(device=device),
        compressed[1].to(device=device),
        compressed[2].to(device=device),
        compressed[3],
        compressed[4],
    )


def compress(M):
    """Compress a contiguous fp16 matrix into the MACKO 5-tuple, on the device of ``M``.

    Mirrors src/macko_spmv/__init__.py:120-131, except that the encoder runs on the GPU:
    a CUDA matrix never leaves the device, and a CPU matrix is copied to the current CUDA
    device, compressed there and copied back (there is no host encoder in this package).
    The buffers are bit-identical to the reference's.
    """
    assert M.is_contiguous()
    if M.device.type == "cuda":
        values, deltas, row_indices = torch.ops.macko_spmv.compress_dense.default(M)
        return (values, deltas, row_indices, M.size(0), M.size(1))
    elif M.device.type == "cpu":
        if not torch.cuda.is_available():
            raise RuntimeError("macko_spmv_b200.compress needs a CUDA device: the encoder is a GPU kernel")
        values, deltas, row_indices = torch.ops.macko_spmv.compress_dense.default(M.to("cuda"))
        return move_to_device((values, deltas, row_indices, M.size(0), M.size(1)), "cpu")
    else:
        raise NotImplementedError()


class FrozenMatrix(tuple):
    """The 5-tuple of `compress` for a matrix that will not be written any more (weights), as returned by
    `freeze`. `multiply` recognises it and lets the kernel fetch matrix data while the previous kernel of
    the stream is still finishing; with a plan (see `freeze`) it runs the planned launch. It is still a
    tuple of the same five items, so everything that takes the reference's compressed object takes it."""

    plan = None        # device buffer of the plan, or None
    plan_meta = None   # (virtual_rows, segment_elements, longest_row, split_rows, recommended)
    windows = None      # device buffer of the column windows that `multiply_batched` walks, or None
    windows_of = None   # write counts and addresses of deltas, row_indices and values at `freeze` (see `_written`; None: not counted)
    windows_batch = 0   # the largest batch for which the windows are the faster route
    even_rows = False   # no row is much longer than the mean (see `rows_are_even`), where the launch asks for it

    def __new__(cls, compressed, plan=None, plan_meta=None, windows=None, windows_of=None, windows_batch=0, even_rows=False):
        self = super().__new__(cls, tuple(compressed[:5]))
        self.plan = plan
        self.plan_meta = plan_meta
        self.windows = windows
        self.windows_of = windows_of
        self.windows_batch = windows_batch
        self.even_rows = even_rows
        return self


if _direct is not None:
    _direct.set_frozen_type(FrozenMatrix)
_direct_multiply = _direct.multiply if _direct is not None else lambda compressed_M, V: None
_direct_batched = _direct.multiply_batched if _direct is not None else lambda compressed_M, V: None
_is_compiling = torch.compiler.is_compiling


def freeze(compressed_M, plan="auto", segment_elements=0, windows="auto"):
    """Declare a compressed CUDA matrix immutable and, if it pays, build its launch plan.

    Waits once for the device work that produced the buffers (they must be complete before a kernel may read
    them ahead of stream order). `plan`: "auto" builds the plan and keeps it only if the row statistics
    recommend it (rows far longer than the average, e.g. skewed matrices), True keeps it always, False builds
    none. Unless it is False, products of a matrix of any type whose rows are even (`rows_are_even`) may walk a row with fewer
    lanes; with False `multiply` adds up every row as it does for the plain 5-tuple, bit for bit. The partial sums of cut rows
    live in the plan: products of one planned matrix must not overlap on the GPU (from several streams, order them or freeze
    once per stream).

    `windows`: "auto" gives an fp16 matrix its column windows, which `multiply_batched` walks (8 bytes per row and window of up to
    1408 columns), if they take at most 5 % of the matrix, `plan` is not False, and PyTorch counts writes to the buffers (not for
    inference tensors): windows describe the deltas and row offsets that they were built from, and `multiply_batched` leaves them
    alone once those have been written. Writes that PyTorch does not count (through `.data`, DLPack or a raw pointer) need
    another `freeze`. False builds none, for a matrix that only ever meets single vectors. True builds them for every fp16 matrix
    that they can index, also where writes are not counted (the caller promises that there are none).

    The reference has no counterpart (src/macko_spmv/__init__.py has only compress / multiply)."""
    assert compressed_M[0].is_cuda and compressed_M[1].is_cuda and compressed_M[2].is_cuda
    torch.cuda.synchronize(compressed_M[0].device)
    half = compressed_M[0].dtype == torch.float16
    wanted = half and (windows is True or (windows == "auto" and plan is not False))
    built = _build_windows(compressed_M, windows is True) if wanted else (None, None, 0)   # before the plan, which waits for the device
    if plan is False or not half:
        even = plan is not False and _lanes_depend_on_rows(compressed_M) and rows_are_even(compressed_M)
        return FrozenMatrix(compressed_M, None, None, *built, even)
    buf, meta = torch.ops.macko_spmv.plan_build.default(
        compressed_M[1], compressed_M[2], compressed_M[3], compressed_M[4], compressed_M[0].numel(), int(segment_elements))
    meta = [int(v) for v in meta.tolist()]
    info = (meta[3], meta[4], meta[5], meta[6], meta[7])
    even = _even(info[2], compressed_M[0].numel(), compressed_M[3])
    if plan is True or info[4]:
        return FrozenMatrix(compressed_M, buf, info, *built, even)
    return FrozenMatrix(compressed_M, None, info, *built, even)


def _even(longest_row: int, stored: int, rows: int) -> bool:
    """What MACKO_SPMV_ROWS_EVEN promises: no row above 9/8 of the mean and 64 elements more."""
    return 8 * rows * (longest_row - 64) <= 9 * stored


def _lanes_depend_on_rows(compressed_M) -> bool:
    """Whether the product's launch is another one for rows known to be even (host arithmetic; saves the look at the rows if not)."""
    launches = []
    for flags in (1, 17):   # MACKO_SPMV_MATRIX_IMMUTABLE, the same and MACKO_SPMV_ROWS_EVEN
        out = (ctypes.c_int * 4)()
        at = ctypes.addressof(out)
        status = _core.macko_spmv_default_launch(compressed_M[3], compressed_M[4], compressed_M[0].numel(),
                                                 torch.cuda.get_device_properties(compressed_M[0].device).multi_processor_count,
                                                 flags, at, at + 4, at + 8, at + 12)
        launches.append((status, *out))
    return launches[0] != launches[1]


def rows_are_even(compressed_M) -> bool:
    """Whether no row of a compressed matrix holds many more stored elements than the mean row (reads one number back from the
    device). `freeze` asks this: products of such a matrix may walk a row with fewer lanes, which would make long rows of another
    one take longer. The order of the fp32 sums of a row depends on it."""
    row_indices, rows = compressed_M[2], compressed_M[3]
    return rows > 0 and _even(int((row_indices[1:] - row_indices[:-1]).amax()), compressed_M[0].numel(), rows)


def _written(compressed_M):
    """What tells whether the buffers have been written or moved since: write counts of deltas and row_indices, their addresses, and
    both of values. None where PyTorch does not count writes (inference tensors)."""
    values, deltas, row_indices = compressed_M[:3]
    if deltas.is_inference() or row_indices.is_inference() or values.is_inference():
        return None
    return deltas._version, row_indices._version, deltas.data_ptr(), row_indices.data_ptr(), values._version, values.data_ptr()


def _build_windows(compressed_M, always):
    """(column windows of an fp16 matrix, what they were built from, the largest batch that takes them), or (None, None, 0) where
    they cannot index the matrix. Unless `always`, also where the rows are so short that their 8 bytes per row and window would
    weigh more than 5 % of the matrix, and where nobody would notice a write to it."""
    _, deltas, row_indices, rows, cols = compressed_M[:5]
    stored = 2 * deltas.numel()
    if rows == 0 or rows >= 1 << 30 or cols >= 1 << 24:
        return None, None, 0
    nbytes = _core.macko_spmm_windows_bytes(rows, cols, stored)
    written = _written(compressed_M)
    if not always and (20 * nbytes > 2.5 * stored or written is None):
        return None, None, 0
    windows = torch.ops.macko_spmv.windows_build.default(deltas, row_indices, rows, cols)
    limit = _windows_batch(rows, cols, stored, nbytes // (8 * rows))
    if limit < DENSE_BATCH_THRESHOLD and not _dense_copy_pays(compressed_M, DENSE_BATCH_THRESHOLD):
        # 9..16 vectors that take two passes of the one-kernel product where nothing is frozen: the sums stay in fp32 (the GEMM may
        # add parts in fp16), at about the time of the copy. 16 vectors, windows / copy / passes: 2048x2048 d = 0.7 11.8 / 12.2 / 21.9 us,
        # d = 0.9 12.8 / 12.3 / 26.8, 2000x5000 d = 0.8 18.4 / 20.8 / 47.2, 4096x1024 d = 0.9 11.1 / 9.8 / 28.0
        limit = DENSE_BATCH_THRESHOLD
    return windows, written, limit


# Beyond this many right-hand sides the windowed product has never been ahead of the dense copy.
WINDOWED_BATCH_LIMIT = 64


def _windows_batch(rows, cols, stored, windows) -> int:
    """The largest batch that goes over the column windows of a frozen matrix (`macko_spmm_fp16_windowed`), of 8 or more.

    3..8 vectors always do, where the other choice is one pass of the one-kernel product: 11008x4096 d = 0.5 8 vectors 25.1
    against 41.2 us, 4 vectors 20.5 / 27.9; 8192x8192 d = 0.3 24.1 / 38.7; 512x512 d = 0.5 4.6 / 5.1 and, the only loss, 3 or 4 vectors
    4.1 / 3.7. Two vectors are level or behind (11008x4096 20.3 / 20.0, 4096x4096 d = 0.7 12.6 / 10.9).
    Larger batches take every 8 vectors through the matrix, against one dense copy and a GEMM: the two models below, in us, fit 18
    shapes x 9..48 vectors with a standard deviation of 7 % and 21 %. 16 vectors, windows / copy: 4096x11008 d = 0.5 39.3 / 48.6,
    d = 0.2 24.8 / 42.6, 4096x4096 d = 0.7 23.4 / 21.3, 16384x4096 d = 0.9 92.6 / 77.3; 24 vectors: 4096x11008 d = 0.2 35.9 / 42.9,
    11008x4096 d = 0.5 57.4 / 44.0, 1024x16384 d = 0.3 18.9 / 26.9. The GEMM is slower where rows of the copy do not start on
    16 bytes: 1500x5001 d = 0.15 16 vectors 8.5 / 21.5."""
    blocks = (rows + 3) // 4
    copy_us = (6.9 + 0.63e-6 * rows * cols + 0.52e-6 * stored) * (1.0 if cols % 8 == 0 else 1.7)
    best = 8
    for batch in range(16, WINDOWED_BATCH_LIMIT + 1, 8):
        ctas = windows * batch // 8
        warps = 32 * max(1, 148 // ctas)
        rounds = 0.5 * (blocks / warps - blocks // -warps) * -(ctas // -148)
        if 4.6 + 0.74 * rounds * (stored / (64.0 * rows * windows) + 1.5) + 3.7e-6 * windows * rows * batch >= copy_us:
            break
        best = batch
    return best


def multiply(compressed_M, V, out=None):
    """y = M @ V for a compressed matrix and an fp16 CUDA vector (src/macko_spmv/__init__.py:134-149).

    `out` (not in the reference): a contiguous CUDA vector of M_rows elements that receives y, for callers
    that keep their results in one buffer; without it a new tensor is returned, as in the reference."""
    if out is None and not _is_compiling():
        y = _direct_multiply(compressed_M, V)   # None: not a plain call
        if y is not None:
            return y
    assert compressed_M[0].is_cuda
    assert compressed_M[1].is_cuda
    assert compressed_M[2].is_cuda
    assert V.is_cuda
    assert V.is_contiguous()
    if out is not None:
        flags = 0
        if isinstance(compressed_M, FrozenMatrix):   # MACKO_SPMV_MATRIX_IMMUTABLE, MACKO_SPMV_ROWS_EVEN
            flags = 17 if compressed_M.even_rows else 1
        torch.ops.macko_spmv.multiply_ex.default(
            compressed_M[0], compressed_M[1], compressed_M[2], compressed_M[3], compressed_M[4], V, out, 1.0, 0.0, flags)
        return out
    if isinstance(compressed_M, FrozenMatrix):
        if compressed_M.plan is not None:
            return torch.ops.macko_spmv.multiply_planned.default(
                compressed_M[0], compressed_M[1], compressed_M[2], compressed_M[3], compressed_M[4],
                compressed_M.plan, compressed_M.plan_meta[0], compressed_M.plan_meta[1], compressed_M.plan_meta[3], V, True)
        return torch.ops.macko_spmv.multiply_frozen.default(
            compressed_M[0], compressed_M[1], compressed_M[2], compressed_M[3], compressed_M[4], V, compressed_M.even_rows)
    return torch.ops.macko_spmv.multiply.default(
        compressed_M[0],
        compressed_M[1],
        compressed_M[2],
        compressed_M[3],
        compressed_M[4],
        V,
    )


# Above this many right-hand sides a dense copy of the matrix plus one tensor-core GEMM is always cheaper than
# streaming the compressed matrix once per 8 vectors; from 9 vectors on (two passes) it depends on the density.
DENSE_BATCH_THRESHOLD = 16


def _dense_copy_pays(compressed_M, batch: int) -> bool:
    """9..DENSE_BATCH_THRESHOLD vectors of an fp16 matrix: passes of the multi-vector kernel against one dense copy and a GEMM.

    The line: ceil(batch / 8) passes at 1.3 TB/s of compressed bytes against the copy at 3.0 TB/s of compressed + dense bytes
    plus 19 us. The rates are those of an earlier decompressor; today's takes about 5 TB/s, so the line keeps to the passes where
    the copy is already ahead. Measured (B200, us, passes / copy, * = chosen): 11008x4096 16 vectors d = 0.2 *42.7 / 34.9,
    0.3 *55.6 / 38.0, 0.4 68.8 / *41.6, 0.5 81.2 / *44.6; 9 vectors 0.2 *30.0 / 35.0, 0.4 47.6 / *41.3; 4096x4096 16 vectors
    0.5 *38.3 / 20.2, 0.7 45.2 / *22.7; 8192x8192 9 vectors 0.3 *52.6 / 69.6, 0.5 77.2 / *79.7, 16 vectors 0.3 *75.7 / 69.7."""
    if batch <= 8 or compressed_M[0].dtype != torch.float16:
        return False
    stored_bytes = 2.5 * compressed_M[0].numel()
    passes = (batch + 7) // 8
    multi_vector_us = passes * stored_bytes / 1.3e6
    dense_us = (stored_bytes + 2.0 * compressed_M[3] * compressed_M[4]) / 3.0e6 + 19.0
    return dense_us < multi_vector_us


def decompress(compressed_M):
    """Dense fp16 [rows, cols] of a compressed CUDA matrix (every zero, pads included, comes back as +0)."""
    assert compressed_M[0].is_cuda
    return torch.ops.macko_spmv.decompress.default(*compressed_M[:5])


def _windows_pay(frozen, V) -> bool:
    """Whether a batch goes over the column windows of a frozen matrix."""
    batch = V.shape[0]
    if batch < 3 or batch > frozen.windows_batch:
        return False
    if frozen.windows_of is not None:
        now = _written(frozen)
        if now is None or frozen.windows_of[:4] != now[:4]:
            return False   # written since: the windows may be those of another matrix
    # above 8 vectors the other route is a dense copy and operators that can be differentiated and transformed
    return batch <= 8 or not ((V.requires_grad and torch.is_grad_enabled()) or type(V) is not torch.Tensor
                              or torch._C._functorch.peek_interpreter_stack() is not None or torch.autograd.forward_ad._current_level >= 0)


def _values_as_frozen(frozen) -> bool:
    """Whether the windowed product may fetch the values ahead of stream order: nobody has written them since `freeze`."""
    return frozen.windows_of is None or frozen.windows_of == _written(frozen)


def multiply_batched(compressed_M, V):
    """Y[batch, rows] = V[batch, cols] @ M^T for a compressed matrix and fp16 CUDA vectors.

    The reference runs batched inputs as a loop of `multiply` calls (torch.vmap fallback,
    python_scripts/util_run_pruned_llm.py:112-115). Here up to 8 vectors share one pass over the compressed
    matrix; 9..DENSE_BATCH_THRESHOLD take two passes or, where the matrix is dense enough for that to be cheaper,
    the route of the larger batches: decompress once and run a dense GEMM. A frozen matrix (`freeze`) has column windows, over
    which a pass is up to twice as fast, so more batches stay with the compressed matrix.
    """
    windowed = type(compressed_M) is FrozenMatrix and compressed_M.windows_batch > 0 and not _is_compiling()
    if windowed:
        y = _direct_batched(compressed_M, V)   # None: not a plain call of three vectors or more
        if y is not None:
            return y
    assert compressed_M[0].is_cuda
    assert V.is_cuda
    assert V.is_contiguous()
    if V.dim() != 2:
        raise RuntimeError("V must have shape [batch, cols]")
    batch = V.shape[0]
    if windowed and _windows_pay(compressed_M, V):
        return torch.ops.macko_spmv.multiply_windowed.default(*compressed_M[:5], compressed_M.windows, V, _values_as_frozen(compressed_M))
    if batch > DENSE_BATCH_THRESHOLD or (windowed and batch > compressed_M.windows_batch) or _dense_copy_pays(compressed_M, batch):
        return V @ decompress(compressed_M).t()
    return torch.ops.macko_spmv.multiply_batched.default(*compressed_M[:5], V)


__all__ = ["compress", "multiply", "multiply_batched", "decompress", "move_to_device", "freeze", "rows_are_even", "FrozenMatrix",
           "native_library_paths", "native_version", "LIB_NAME"]
