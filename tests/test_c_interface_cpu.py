"""The C interface (include/fuselink.h) for programs built against an earlier header."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_product_description_keeps_the_places_of_its_fields(tmp_path):
    """Fields are added at the end: a program built before expect_rows passes its status pointer where the library reads it."""
    cxx = next((c for c in (os.environ.get("CXX"), "g++", "/usr/bin/g++") if c and shutil.which(c)), None)
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "fields.cc", str(tmp_path / "fields")
    src.write_text("""#include "fuselink.h"
#include <stddef.h>
#include <stdio.h>
int main() {
  printf("%zu %zu %zu", offsetof(FlGemmDesc, max_ctas) + sizeof(int), offsetof(FlGemmDesc, status), offsetof(FlGemmDesc, expect_rows));
}
""")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    b = subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "fuselink_b200", "include"), "-I", os.path.join(cuda, "include"), str(src), "-o", exe],
                       capture_output=True, text=True, timeout=300)
    assert b.returncode == 0, b.stderr[-3000:]
    end_of_max_ctas, status, expect_rows = map(int, subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout.split())
    assert status == (end_of_max_ctas + 7) // 8 * 8 and expect_rows == status + 8


@pytest.mark.parametrize("rows,cols", [(0, 4), (1, 0), (1, 2 ** 31 - 127), (1, 2 ** 31 - 1)])
def test_the_relu_gradient_refuses_widths_that_32_bits_do_not_count(rows, cols):
    lib = os.path.join(ROOT, "fuselink_b200", "lib", "libfuselink.so")
    if not os.path.exists(lib):
        pytest.skip("libfuselink.so not built")
    f = ctypes.CDLL(lib).fl_relu_bias_bwd
    f.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p]
    assert f(None, None, None, None, None, rows, cols, None) == -1
