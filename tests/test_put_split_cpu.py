"""How a put is split over its CTAs (csrc/kernels/comm_kernels.cu), in arithmetic: every slot has one owner, a segment's arrivals add up to
its chunks, and they do so only once all of its owners are done."""
import random

import pytest

SLOT = 16 * 1024


def owner(u, U, G):                       # put_owner
    return ((u + 1) * G - 1) // U


def even_split(sizes, chunk, G):
    units = [-(-b // SLOT) for b in sizes]
    U, u0 = sum(units), 0
    if U < G:
        return 0
    for b, n in zip(sizes, units):
        if n and owner(u0 + n - 1, U, G) - owner(u0, U, G) + 1 > -(-b // chunk):
            return 0
        u0 += n
    return U


@pytest.mark.parametrize("seed", range(40))
def test_arrivals_of_an_even_split(seed):
    rng = random.Random(seed)
    chunk = 16 * rng.choice([1, 100, 1024, 4096, 32768])
    most = rng.choice([1 << 16, 1 << 20, 1 << 26])
    sizes = [rng.randint(0, most) if rng.random() < 0.8 else 16 * rng.randint(0, 100) for _ in range(rng.randint(1, 8))]
    chunks = [-(-b // chunk) for b in sizes]
    G = min(max(sum(chunks), 1), 296)
    U = even_split(sizes, chunk, G)
    if U == 0:
        return
    u0 = 0
    for b, n_chunks in zip(sizes, chunks):
        n = -(-b // SLOT)
        if n == 0:
            continue
        took = []                         # (CTA, first unit, last unit)
        for c in range(G):
            lo, hi = max(U * c // G, u0), min(U * (c + 1) // G, u0 + n)
            if lo < hi:
                took.append((c, lo, hi))
        assert [t[1] for t in took[1:]] == [t[2] for t in took[:-1]] and took[0][1] == u0 and took[-1][2] == u0 + n
        first, last = owner(u0, U, G), owner(u0 + n - 1, U, G)
        assert [t[0] for t in took] == list(range(first, last + 1))
        adds = [n_chunks - (last - first) if c == first else 1 for c, _, _ in took]
        assert sum(adds) == n_chunks and min(adds) >= 1         # none finishes without adding: n_chunks is reached by the last
        u0 += n


def test_common_launches_are_split_evenly():
    from fuselink_b200.ops.comm import chunking
    for sizes in ([64 << 10], [16 << 20], [1 << 30], [2621440] * 8, [8 << 20] * 4):
        chunk, n = chunking(sizes[0])
        assert even_split(sizes, chunk, min(n * len(sizes), 296)) > 0


@pytest.mark.parametrize("sh", range(1, 16))
def test_shifted_copy_stays_inside_the_source(sh):
    """copy_shifted: vectors read lie inside the source and the bytes written cover the destination once."""
    for to16 in range(16):
        for nbytes in list(range(0, 120)) + [1000, 65536, 65537]:
            head = to16 + 16
            body = nbytes - head - 16 + sh
            if body < 16:
                continue
            n = body >> 4
            assert head - sh >= 0 and head - sh + 16 * (n - 1) + 32 <= nbytes        # first and last byte read
            assert head + 16 * n <= nbytes and nbytes - head - 16 * n < 48
