"""How a put is split over its CTAs (csrc/kernels/comm_kernels.cu, by the functions that the kernel and its launch go by): every slot has one
owner, a segment's arrivals add up to its chunks, and they do so only once all of its owners are done."""
import ctypes as ct
import os
import random

import pytest

SLOT = 16 * 1024
MAX_SEGS, FLAG_COUNT, FLAG_SEQ_PER_CHUNK = 8, 2, 1
LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fuselink_b200", "lib", "libfuselink.so")


class Seg(ct.Structure):                  # FlSeg
    _fields_ = [("src", ct.c_void_p), ("dst", ct.c_void_p), ("bytes", ct.c_ulonglong), ("flags", ct.c_void_p), ("flag_mode", ct.c_int),
                ("wait_flags", ct.c_void_p), ("bytes_done", ct.c_void_p)]


class Put(ct.Structure):                  # FlPutArgs
    _fields_ = [("seg", Seg * MAX_SEGS), ("nseg", ct.c_int), ("chunk_bytes", ct.c_uint), ("seq", ct.c_uint), ("use_bulk", ct.c_int),
                ("status", ct.c_void_p), ("wait_flag", ct.c_void_p * 8), ("wait_want", ct.c_uint * 8), ("nwait", ct.c_int),
                ("done_scratch", ct.c_void_p)]


class Split(ct.Structure):                # FlPutSplit
    _fields_ = [("slots", ct.c_uint), ("slot_end", ct.c_uint * MAX_SEGS), ("first_cta", ct.c_uint * MAX_SEGS), ("first_adds", ct.c_uint * MAX_SEGS)]


class Shifted(ct.Structure):              # FlPutShifted
    _fields_ = [("head", ct.c_ulonglong), ("vectors", ct.c_ulonglong), ("shift", ct.c_uint)]


@pytest.fixture(scope="module")
def lib():
    if not os.path.exists(LIB):
        pytest.skip("libfuselink.so not built")
    lib = ct.CDLL(LIB)
    lib.fl_put_split.argtypes = [ct.POINTER(Put), ct.c_uint, ct.POINTER(Split)]
    lib.fl_put_shifted.argtypes = [ct.c_ulonglong] * 3 + [ct.POINTER(Shifted)]
    return lib


def split(lib, sizes, chunk, G, mode=FLAG_COUNT, wait=None):
    out, put = Split(), Put(nseg=len(sizes), chunk_bytes=chunk, use_bulk=1)
    for s, b in zip(put.seg, sizes):
        s.bytes, s.flag_mode, s.wait_flags = b, mode, wait
    assert lib.fl_put_split(ct.byref(put), G, ct.byref(out)) == 0
    return out


@pytest.mark.parametrize("seed", range(40))
def test_arrivals_of_an_even_split(lib, seed):
    rng = random.Random(seed)
    U = 0
    while U == 0:                         # launches whose CTAs take chunks in turn are drawn again
        chunk = 16 * rng.choice([1, 100, 1024, 4096, 32768])
        most = rng.choice([1 << 16, 1 << 20, 1 << 26])
        sizes = [rng.randint(0, most) if rng.random() < 0.8 else 16 * rng.randint(0, 100) for _ in range(rng.randint(1, 8))]
        chunks = [-(-b // chunk) for b in sizes]
        G = min(max(sum(chunks), 1), 296)
        sp = split(lib, sizes, chunk, G)
        U = sp.slots
    assert U == sum(-(-b // SLOT) for b in sizes) >= G
    u0 = 0
    for i, (b, n_chunks) in enumerate(zip(sizes, chunks)):
        n = -(-b // SLOT)
        assert sp.slot_end[i] == u0 + n
        if n == 0:
            continue
        took = []                         # (CTA, first slot, last slot)
        for c in range(G):
            lo, hi = max(U * c // G, u0), min(U * (c + 1) // G, u0 + n)
            if lo < hi:
                took.append((c, lo, hi))
        assert [t[1] for t in took[1:]] == [t[2] for t in took[:-1]] and took[0][1] == u0 and took[-1][2] == u0 + n
        assert [t[0] for t in took] == list(range(took[0][0], took[-1][0] + 1)) and took[0][0] == sp.first_cta[i]
        adds = [sp.first_adds[i] if c == sp.first_cta[i] else 1 for c, _, _ in took]
        assert sum(adds) == n_chunks and min(adds) >= 1         # none finishes without adding: n_chunks is reached by the last
        u0 += n


def test_common_launches_are_split_evenly(lib):
    from fuselink_b200.ops.comm import chunking
    for sizes in ([64 << 10], [16 << 20], [1 << 30], [2621440] * 8, [8 << 20] * 4):
        chunk, n = chunking(sizes[0])
        G = min(n * len(sizes), 296)
        assert split(lib, sizes, chunk, G).slots > 0
        assert split(lib, sizes, chunk, G, FLAG_SEQ_PER_CHUNK).slots == 0 and split(lib, sizes, chunk, G, wait=16).slots == 0


def test_what_the_kernel_multiplies_fits_32_bits(lib):
    for G in (1, 37, 296):
        most = (2 ** 32 - 1) // G
        assert split(lib, [most * SLOT], 1 << 30, G).slots == (most if most * SLOT >> 30 >= G - 1 else 0)
        assert split(lib, [most * SLOT + 1], 1 << 30, G).slots == 0


@pytest.mark.parametrize("sh", range(1, 16))
def test_shifted_copy_stays_inside_the_source(lib, sh):
    """copy_shifted: vectors read lie inside the source, begin at multiples of 16, as do those written, which cover the destination once."""
    for to in range(16):
        src, dst, p = 4096 + (to + sh) % 16, 8192 + to, Shifted()
        for nbytes in list(range(0, 120)) + [1000, 65536, 65537]:
            assert lib.fl_put_shifted(src, dst, nbytes, ct.byref(p)) == 0
            head, n, shift = p.head, p.vectors, p.shift
            if n == 0:
                assert nbytes < 64                                                       # nothing longer goes byte by byte
                continue
            assert (src + head - shift) % 16 == 0 and (dst + head) % 16 == 0
            assert 0 < shift < 16 and head - shift >= 0 and head - shift + 16 * (n - 1) + 32 <= nbytes        # first and last byte read
            assert head + 16 * n <= nbytes and nbytes - head - 16 * n < 48
