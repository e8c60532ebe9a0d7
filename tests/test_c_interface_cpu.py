"""The C interface (include/fuselink.h) for programs built against an earlier header."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(tmp_path, source, link=False):
    """The output of a C++ program against include/fuselink.h (and lib/libfuselink.so)."""
    cxx = next((c for c in (os.environ.get("CXX"), "g++", "/usr/bin/g++") if c and shutil.which(c)), None)
    lib = os.path.join(ROOT, "fuselink_b200", "lib")
    if cxx is None or (link and not os.path.exists(os.path.join(lib, "libfuselink.so"))):
        pytest.skip("no C++ compiler or library")
    src, exe = tmp_path / "program.cc", str(tmp_path / "program")
    src.write_text('#include "fuselink.h"\n#include <stddef.h>\n#include <stdio.h>\n#include <string.h>\n' + source)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    b = subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "fuselink_b200", "include"), "-I", os.path.join(cuda, "include"), str(src), "-o", exe,
                        *(["-L", lib, "-lfuselink", f"-Wl,-rpath,{lib}"] if link else [])], capture_output=True, text=True, timeout=300)
    assert b.returncode == 0, b.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60, env={k: v for k, v in os.environ.items() if k != "FUSELINK_GEMM_PAIR"})
    assert r.returncode == 0, r.stderr
    return [int(v) for v in r.stdout.split()]


def test_a_product_description_keeps_the_places_of_its_fields(tmp_path):
    """Fields are added at the end: a program built before expect_rows passes its status pointer where the library reads it."""
    end_of_max_ctas, status, expect_rows = _run(tmp_path, """int main() {
  printf("%zu %zu %zu", offsetof(FlGemmDesc, max_ctas) + sizeof(int), offsetof(FlGemmDesc, status), offsetof(FlGemmDesc, expect_rows));
}
""")
    assert status == (end_of_max_ctas + 7) // 8 * 8 and expect_rows == status + 8


# 8 groups of N columns on a GPU that holds 74 pairs: what the faster tiles were (us, pairs of 256 x 256 | of 256 x 512)
@pytest.mark.parametrize("N,K,rows,ctas,variant", [
    (4096, 14336, 250, 0, 1), (4096, 14336, 500, 0, 2), (2048, 5632, 191, 0, 1), (2048, 5632, 700, 0, 1),       # 289|336 398|365 65|99 146|175
    (4096, 14336, 250, 128, 1), (4096, 14336, 500, 128, 1), (2048, 5632, 500, 128, 1), (2048, 5632, 700, 128, 1),   # 283|330 493|526 129|157 131|160
    (4096, 14336, 250, 96, 2), (4096, 14336, 191, 96, 1), (2048, 5632, 700, 96, 2),                            # 343|311 289|337 176|169
    (2048, 5632, 250, 64, 1), (4096, 14336, 700, 64, 2), (4096, 14336, 250, 32, 2), (2048, 5632, 700, 32, 2),  # 115|139 936|834 774|686 383|357
    (4096, 14336, 0, 32, 2), (4096, 14336, 1024, 32, 2), (256, 14336, 250, 0, 1), (4096, 14336, 250, 1, 2), (4096, 14336, 250, 1000, 1),
])
def test_tiles_by_expected_rows_on_the_pairs_that_a_launch_may_use(N, K, rows, ctas, variant, tmp_path):
    got, = _run(tmp_path, f"""int main() {{
  FlGemmDesc d;
  memset(&d, 0, sizeof d);
  d.num_groups = 8; d.N = {N}; d.K = {K}; d.epilogue = FL_EPI_SCATTER; d.max_ctas = {ctas}; d.expect_rows = {rows};
  printf("%d", fl_gemm_choose(&d, 74));
}}
""", link=True)
    assert got == variant


@pytest.mark.parametrize("push_world,rows,variant", [(0, 191, 1), (0, 1024, 1), (2, 191, 0), (8, 447, 0), (2, 448, 1), (2, 1024, 1), (2, 0, 1)])
def test_tiles_of_weight_gradients_that_other_ranks_receive(push_world, rows, variant, tmp_path):
    """Pairs store a gradient of few rows faster only where it leaves through shared memory, which it does if it stays on this GPU."""
    got, = _run(tmp_path, f"""int main() {{
  FlGemmDesc d;
  memset(&d, 0, sizeof d);
  d.group_mode = 1; d.num_groups = 8; d.M = 28672; d.N = 4096; d.epilogue = FL_EPI_WGRAD; d.push_world = {push_world}; d.expect_rows = {rows};
  printf("%d", fl_gemm_choose(&d, 74));
}}
""", link=True)
    assert got == variant


@pytest.mark.parametrize("rows,cols", [(0, 4), (1, 0), (1, 2 ** 31 - 127), (1, 2 ** 31 - 1)])
def test_the_relu_gradient_refuses_widths_that_32_bits_do_not_count(rows, cols):
    lib = os.path.join(ROOT, "fuselink_b200", "lib", "libfuselink.so")
    if not os.path.exists(lib):
        pytest.skip("libfuselink.so not built")
    f = ctypes.CDLL(lib).fl_relu_bias_bwd
    f.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p]
    assert f(None, None, None, None, None, rows, cols, None) == -1


@pytest.mark.parametrize("ctas", [1, 2, 7, 296])
def test_a_hand_off_with_a_cta_that_gave_up_is_not_published(ctas, tmp_path):
    """fl_kv_ticket and fl_kv_end over a launch's CTAs, where nobody gives up, then where the first, the last or all of them do: one CTA is the
    last, and it publishes only what is whole."""
    published = _run(tmp_path, f"""int main() {{
  const unsigned n = {ctas};
  for (unsigned who = 0; who < 4; ++who) {{
    unsigned counter = 0, lasts = 0, published = 0;
    for (unsigned c = 0; c < n; ++c) {{
      const bool ok = who == 0 || !(who == 3 || (who == 1 && c == 0) || (who == 2 && c == n - 1));
      const unsigned before = counter;
      counter += fl_kv_ticket(ok);
      const FlKvEnd e = fl_kv_end(before, ok, n);
      lasts += e.last; published += e.publish;
      if (e.last && c != n - 1) return 1;
    }}
    if (lasts != 1) return 1;
    printf("%u ", published);
  }}
}}
""")
    assert published == [1, 0, 0, 0]
    text = open(os.path.join(ROOT, "fuselink_b200", "csrc", "kernels", "kv_pack.cu")).read()
    body = text[text.index("kv_pack_bulk_kernel("):]
    behind = body[body.index("if (!ok) let_copies_land"):body.index("st_release_sys(a.done_flag")]
    assert "fl_kv_ticket(ok)" in behind and "if (end.publish && a.hdr_bytes" in behind and behind.endswith("if (end.publish && a.done_flag) ")
