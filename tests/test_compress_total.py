"""The stored count that the compressor leaves in pinned host memory (`macko_compress_count_total`), against the last row offset: row
counts around the 512 that a warp and the 16384 that the CTA of the prefix sum takes at a time, empty matrices, both value
widths, several threads at once."""
import os
import shutil
import subprocess
import sys
import threading

import pytest
import torch

import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import cabi, workloads


def test_refuses_before_touching_the_device():
    lib = cabi.load()
    a = 0x1000   # never dereferenced
    assert lib.macko_compress_count_total(a, 4, 4, 4, a, a, None) == cabi.ERR_INVALID_ARGUMENT
    assert lib.macko_compress_count_total(a, 4, 4, 2, a, None, None) == cabi.ERR_INVALID_ARGUMENT
    assert lib.macko_compress_count_total(a, 4, 4, 2, a, a + 2, None) == cabi.ERR_MISALIGNED


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(0, 64), (5, 0), (1, 1), (511, 40), (512, 40), (16382, 24), (16383, 24), (16384, 24), (40001, 17)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.int8])
def test_total_is_the_last_row_offset(rows, cols, dtype):
    lib = cabi.load()
    M = (workloads.bernoulli_matrix(rows, cols, 0.4, seed=rows + cols, device="cuda") * 20).to(dtype) if rows and cols else torch.empty(rows, cols, dtype=dtype, device="cuda")
    ri = torch.empty(rows + 1, dtype=torch.int32, device="cuda")
    total = torch.full((1,), -1, dtype=torch.int32).pin_memory()
    cabi.check(lib, lib.macko_compress_count_total(M.data_ptr(), rows, cols, M.element_size(), ri.data_ptr(), total.data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    counts = torch.empty_like(ri)
    count = lib.macko_compress_count_int8 if dtype is torch.int8 else lib.macko_compress_count
    cabi.check(lib, count(M.data_ptr(), rows, cols, counts.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(ri, counts) and int(total[0]) == int(counts[rows])
    values, deltas, row_indices = macko_spmv.compress(M)[:3]
    assert values.numel() == (int(total[0]) + 7) // 8 * 8 == 2 * deltas.numel() and torch.equal(row_indices, ri)


@pytest.mark.gpu
def test_threads_and_streams_at_once():
    mats = [workloads.bernoulli_matrix(700 + 13 * i, 900 + 7 * i, 0.1 + 0.1 * i, seed=i, device="cuda") for i in range(6)]
    want = [macko_spmv.compress(M) for M in mats]
    torch.cuda.synchronize()
    got = [[None] * 8 for _ in mats]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for k in range(8):
                got[i][k] = macko_spmv.compress(mats[i])
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(mats))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w, g in zip(want, got):
        for c in g:
            assert all(torch.equal(a, b) for a, b in zip(w[:3], c[:3]))


# cudaStreamQuery and, on request, cudaStreamSynchronize that answer an error (999) and nothing else, while `fail` says so
_FAKE = """
#define _GNU_SOURCE
#include <dlfcn.h>
int fail_query, fail_synchronize;
typedef int (*call)(void *);
int cudaStreamQuery(void *s) { return fail_query ? 999 : ((call)dlsym(RTLD_NEXT, "cudaStreamQuery"))(s); }
int cudaStreamSynchronize(void *s) { return fail_synchronize ? 999 : ((call)dlsym(RTLD_NEXT, "cudaStreamSynchronize"))(s); }
"""

_CHILD = """
import ctypes, sys
import torch
import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import workloads

fake = ctypes.CDLL(sys.argv[1])
M = workloads.bernoulli_matrix(300, 500, 0.4, seed=1, device="cuda")
want = macko_spmv.compress(M)
torch.cuda.synchronize()
torch.cuda._sleep(400_000_000)   # the count is still to come when the query fails
ctypes.c_int.in_dll(fake, "fail_query").value = 1
ctypes.c_int.in_dll(fake, "fail_synchronize").value = int(sys.argv[2])
try:
    macko_spmv.compress(M)
    raise SystemExit("compress did not notice the failing query")
except RuntimeError as e:
    assert "compress" in str(e), e
ctypes.c_int.in_dll(fake, "fail_query").value = ctypes.c_int.in_dll(fake, "fail_synchronize").value = 0
words = [torch.full((1,), 12345, dtype=torch.int32).pin_memory() for _ in range(4)]
torch.cuda.synchronize()
assert all(int(w) == 12345 for w in words), [int(w) for w in words]
assert all(torch.equal(a, b) for a, b in zip(want[:3], macko_spmv.compress(M)[:3]))
"""


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs a C compiler")
@pytest.mark.parametrize("synchronize_fails", [0, 1])
def test_word_is_not_reused_while_the_count_is_pending(tmp_path, synchronize_fails):
    """A query that fails ends the call with the count still on its way: the pinned word must not go to somebody else."""
    (tmp_path / "fake.c").write_text(_FAKE)
    fake = tmp_path / "fake.so"
    subprocess.run(["gcc", "-shared", "-fPIC", str(tmp_path / "fake.c"), "-o", str(fake), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, LD_PRELOAD=str(fake), PYTHONPATH=root)
    r = subprocess.run([sys.executable, "-c", _CHILD, str(fake), str(synchronize_fails)], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


_BLOCKING = """
import ctypes, time
import torch
cudart = ctypes.CDLL("libcudart.so.12")   # torch's
assert cudart.cudaSetDeviceFlags(4) == 0   # cudaDeviceScheduleBlockingSync
import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import workloads

M = workloads.bernoulli_matrix(300, 500, 0.4, seed=1, device="cuda")
want = macko_spmv.compress(M)
torch.cuda.synchronize()
torch.cuda._sleep(1_000_000_000)   # about half a second
wall, cpu = time.perf_counter(), time.thread_time()
got = macko_spmv.compress(M)
wall, cpu = time.perf_counter() - wall, time.thread_time() - cpu
assert wall > 0.3 and cpu < 0.2 * wall, (wall, cpu)
assert all(torch.equal(a, b) for a, b in zip(want[:3], got[:3]))
"""


@pytest.mark.gpu
def test_blocking_synchronisation_is_respected():
    """A program that asked CUDA to put its threads to sleep while they wait does not find one of them spinning in compress()."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _BLOCKING], env=dict(os.environ, PYTHONPATH=root), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
