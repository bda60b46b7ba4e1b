"""The operator library is for every libtorch program; what needs the Python interpreter lives in a module beside it."""
import shutil
import subprocess

import pytest

import macko_spmv_b200 as macko_spmv


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs a C compiler")
def test_loads_without_an_interpreter(tmp_path):
    src = tmp_path / "load.c"
    src.write_text("#include <dlfcn.h>\n#include <stdio.h>\n"
                   "int main(int n, char **a) { if (dlopen(a[1], RTLD_NOW | RTLD_GLOBAL)) return 0; puts(dlerror()); return 1; }\n")
    exe = tmp_path / "load"
    subprocess.run(["gcc", str(src), "-o", str(exe), "-ldl"], check=True)
    r = subprocess.run([str(exe), macko_spmv.native_library_paths()[1]], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr


def test_the_direct_call_is_built_here():
    assert macko_spmv._direct is not None and macko_spmv._direct.__name__.endswith("._torch_direct")
