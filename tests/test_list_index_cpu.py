"""Entry numbers of voxel lists near the limit of 2^31 - 1 voxels (prologue.cu
terma_body and blocked_adjoint_kernel, list_chunks), in 32-bit arithmetic
(CPU): every entry is taken once, none beyond the list.
"""
import numpy as np
import pytest

U = np.uint32


def _taken(count, stride, live):
    """First and last entry and number of entries that a launch of `stride` threads takes."""
    rounds = int((U(count) + U(stride - 1)) // U(stride))
    lo, hi, n = None, None, 0
    thread = np.arange(stride, dtype=U)
    for it in {0, 1, rounds - 2, rounds - 1} & set(range(rounds)):   # the others lie between
        with np.errstate(over="ignore"):
            e = U(it) * U(stride) + thread
        e = e[live(e, count)]
        n += e.size
        if e.size:
            lo = int(e.min()) if lo is None else min(lo, int(e.min()))
            hi = int(e.max()) if hi is None else max(hi, int(e.max()))
    return rounds, lo, hi, n


# 2047 x 2049 x 512 and 2317 x 1661 x 558 pass the check on the grid's size
@pytest.mark.parametrize("count", [1, 31, 32, 33, 70000, 1 << 30, 2047 * 2049 * 512, 2317 * 1661 * 558])
@pytest.mark.parametrize("ctas", [1, 3, 152 * 3, 152 * 8])
def test_strided_entries(count, ctas):
    stride = ctas * 256
    rounds, lo, hi, n = _taken(count, stride, lambda e, c: e < U(c))
    assert rounds == -(-count // stride)
    assert (lo, hi) == (0, count - 1)
    seen = {0, 1, rounds - 2, rounds - 1} & set(range(rounds))
    assert n == sum(min(stride, count - it * stride) for it in seen)


def test_signed_entries_would_pass_the_end():
    """What the unsigned comparison is for: read as int, the last round's tail is below 0."""
    count, stride = 2047 * 2049 * 512, 152 * 8 * 256
    rounds = -(-count // stride)
    e = U(rounds - 1) * U(stride) + np.arange(stride, dtype=U)
    assert (e.view(np.int32) < 0).any() and (e.view(np.int32) < np.int32(count)).sum() > (e < U(count)).sum()


@pytest.mark.parametrize("count", [0, 1, 32, 33, 2 ** 31 - 33, 2 ** 31 - 32, 2 ** 31 - 2, 2 ** 31 - 1])
def test_chunks(count):
    chunks = int((U(count) + U(31)) >> U(5))
    assert chunks == -(-count // 32)
    assert chunks == 0 or ((chunks - 1) << 5) + 31 < 2 ** 31
