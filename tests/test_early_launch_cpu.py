"""Rules of the kernels that are launched to start while the one before them in the stream still runs, read off their source."""
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fuselink_b200", "csrc", "kernels")
EARLY = ["decoder.cu", "thin_gemm.cu", "comm_kernels.cu"]


def _functions(name):
    """{function: body} of the __global__ and __device__ functions of a file, comments removed."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(KERNELS, name)).read())
    found = {}
    for m in re.finditer(r"\b__(global|device)__\b", text):
        start, semicolon = text.find("{", m.end()), text.find(";", m.end())
        if start < 0 or 0 <= semicolon < start:
            continue
        head = re.sub(r"__launch_bounds__\s*\([^)]*\)", "", text[m.end():start])
        depth, at = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        found[re.search(r"(\w+)\s*\(", head).group(1)] = found.get(re.search(r"(\w+)\s*\(", head).group(1), "") + text[start:at]
    return found


def _reached(functions, kernel):
    """The kernel's body and those of the functions of its file that it calls, through any number of calls."""
    names, todo = set(), [kernel]
    while todo:
        n = todo.pop()
        if n not in names:
            names.add(n)
            todo += [f for f in functions if re.search(rf"\b{f}\b", functions[n])]
    return {n: functions[n] for n in names}


@pytest.mark.parametrize("name", EARLY)
def test_what_another_kernel_writes_is_not_read_as_read_only(name):
    """ld.global.nc is defined only for memory that nobody writes while the kernel runs; the kernel before an early one does."""
    functions = _functions(name)
    early = [k for k, body in functions.items() if "grid_dep_wait()" in body]
    assert early
    for k in early:
        for n, body in _reached(functions, k).items():
            assert not re.search(r"ld_nc|\.nc\b|__ldg|__restrict__", body), f"{name}: {n}, reached from {k}"


def test_a_product_that_gave_up_waits_for_its_copies():
    """Whichever role gives up (the products while the loader has no more blocks to wait for, say), a warp waits behind the CTA's
    barrier before it frees TMEM and the CTA may end: copies into its shared memory may be on the way."""
    body = _functions("thin_gemm.cu")["thin_gemm_kernel"]
    behind = body[body.rindex("mbar_wait"):]                     # nobody gives up later than that
    barrier, look, free = (re.search(r, behind) for r in (r"else __syncthreads\(\);", r"if \([^{;]*abort_flag\)+ let_copies_land\(\);", r"tmem_dealloc"))
    assert barrier and look and free and barrier.end() < look.start() < look.end() < free.start()


def test_the_limit_of_a_wait_counts_from_the_end_of_the_kernel_before():
    """Every bounded wait of an early kernel stands behind a grid_dep_wait of its role: the kernel before may poll a flag for longer."""
    for name in ("decoder.cu", "thin_gemm.cu"):
        for n, body in _functions(name).items():
            roles = re.split(r"\belse if \(warp == 1", body)
            for role in roles if "mbar_wait" in body else []:
                assert re.search(r"grid_dep_wait\(\)", role[:role.index("mbar_wait")]), f"{name}: {n}"


@pytest.mark.parametrize("kernel", ["thin_gemm_kernel", "dec_attention_ring_kernel"])
def test_a_warp_goes_on_together_behind_a_wait(kernel):
    """mbar_wait answers thread by thread; outside of the roles of a single lane it is mbar_wait_warp, since shuffles, cluster barriers
    and .aligned instructions follow, also where the wait ran out."""
    body = next(f[kernel] for f in map(_functions, EARLY) if kernel in f)
    while m := re.search(r"if \([^{}]*lane == 0[^{}]*\) \{", body):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(body[at], 0)
            at += 1
        body = body[:m.start()] + body[at:]
    assert "mbar_wait_warp(" in body and "mbar_wait(" not in body


def test_a_kernel_that_polls_flags_lets_nobody_start_before_it_has_seen_them():
    """The next kernel's CTAs would hold their SMs while flags are polled, and what a peer waits for before it sets them may need those SMs."""
    functions = _functions("comm_kernels.cu")
    polling = [k for k, body in functions.items() if "grid_dep_wait()" in body and any("wait_flag_ge" in b for b in _reached(functions, k).values())]
    assert sorted(polling) == ["barrier_kernel", "put_chunks_kernel", "wait_flags_kernel"]
    for k in polling:
        body = functions[k].replace("if (a.nwait == 0) grid_dep_launch();", "nobody_polls_from_here();")
        assert "grid_dep_launch()" not in body, k
        if "nobody_polls_from_here" in body:                     # what is polled behind it is a loop over a.nwait flags
            behind = body[body.index("nobody_polls_from_here"):]
            assert all("a.nwait" in line for line in re.findall(r"if \([^;]*wait_flag_ge", behind)) and behind.count("wait_flag_ge") == 1


@pytest.mark.parametrize("name,kernel", [("fp8_gemm.cu", "fp8_grouped_gemm_kernel"), ("grouped_gemm.cu", "grouped_gemm_kernel"),
                                         ("grouped_gemm.cu", "grouped_gemm_pair_kernel"), ("grouped_gemm.cu", "grouped_gemm_wide_kernel")])
def test_a_grouped_product_that_gave_up_waits_for_its_copies(name, kernel):
    """As above: behind the CTA's barrier, before TMEM is freed, whichever role gave up and although the loader may have ended before that."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(KERNELS, name)).read())
    start = re.search(rf"\n{kernel}\(const __grid_constant__", text).start()
    body = text[start:text.index("\n}\n", start)]
    behind = body[body.rindex("mbar_wait"):]
    barrier, look, free = (re.search(r, behind) for r in (r"\n  __syncthreads\(\);", r"if \([^{;]*\*abort_flag\) let_copies_land\(\);", r"tmem_dealloc"))
    assert barrier and look and free and barrier.end() < look.start() < look.end() < free.start()
    if kernel.startswith("fp8"):                                 # sums are asked for ahead of their use: none is on its way at the end
        assert re.search(r"if \(!ok\) tmem_ld_wait\(\);", behind[:barrier.start()])


@pytest.mark.parametrize("kernel", ["grouped_gemm_kernel", "grouped_gemm_pair_kernel", "grouped_gemm_wide_kernel"])
def test_an_epilogue_warp_goes_on_together_behind_a_wait(kernel):
    """Loads from TMEM and the stores through shared memory want the whole warp, also where a wait ran out; single lanes wait by themselves."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(KERNELS, "grouped_gemm.cu")).read())
    start = re.search(rf"\n{kernel}\(const __grid_constant__", text).start()
    body = text[start:text.index("\n}\n", start)]
    epilogue = body[body.index("half = (warp - 2) >> 2"):]
    assert "mbar_wait_warp(" in epilogue and "mbar_wait(" not in epilogue
