"""Segments that do not tile the input: the call reports them, leaves them alone and
partitions the others, and writes nothing outside the output, whatever the malformed
ones' lengths."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx
import oracle

pytestmark = pytest.mark.gpu

M = 5


def run(torch, x, call, rec):
    """The output between two guards and the latched status."""
    n = x.size
    kind, dtype = (np.int64, torch.int64) if rec else (np.int32, torch.int32)
    out = torch.full((n + (1 << 17),), -1, dtype=dtype, device="cuda")
    lo = 1 << 16
    call(torch.from_numpy(x.view(kind)).cuda(), out[lo:lo + n])
    status = mdx.workspace(0).error()
    got = out.cpu().numpy()
    assert (got[:lo] == -1).all() and (got[lo + n:] == -1).all()
    return got[lo:lo + n], status


def values(n, rec):
    x = oracle.fill_uniform_u32(n, n)
    return x.astype(np.uint64) | (np.arange(n, dtype=np.uint64) << np.uint64(32)) if rec else x


def check(got, x, offs, good):
    for s in range(len(offs) - 1):
        a, b = int(offs[s]), int(offs[s + 1])
        if s in good:
            assert np.array_equal(got[a:b].view(x.dtype), oracle.partition(x[a:b], M)[0]), s
        else:
            assert (got[a:b] == -1).all(), s


@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("run_tiles", [1, 2, 8])
def test_first_segment_off_the_start(cuda_ready, run_tiles, rec):
    """Its runs have no room among the entries; the next segment is shorter by half a
    run, so that one entry of the first in its place would pass the output's end."""
    torch = cuda_ready
    P = 2048 if rec else 4096
    for first, second in ((9 * run_tiles * P, 7 * run_tiles * P + 10), (3 * P, 2 * P + 1), (100, 5 * P), (5 * P, 7)):
        offs = np.array([P, P + first, P + first + second], dtype=np.int64)
        x = values(int(offs[-1]), rec)
        do = torch.from_numpy(offs).cuda()
        elem = mdx.ELEM_REC8 if rec else mdx.ELEM_U32
        try:
            mdx.set_tuning(elem, M, 0, 33, plain_two_kernel=1, run_tiles=run_tiles)
            got, status = run(torch, x, lambda d, o: mdx.partition_segmented(d, do, ("mod", M), out=o), rec)
        finally:
            mdx.load_tuning(mdx.TUNING_PATH, missing_ok=True)
        assert status == mdx.MDX_ERR_SEGMENTS
        check(got, x, offs, {1})
        assert (got[:P] == -1).all()


@pytest.mark.parametrize("rec", [False, True])
def test_last_segment_short_of_the_end(cuda_ready, rec):
    torch = cuda_ready
    P = 2048 if rec else 4096
    for lengths in ((7 * P + 10, 30 * P), (P, 30), (9 * P, 30)):
        offs = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
        x = values(int(offs[-1]) + 100, rec)
        do = torch.from_numpy(offs).cuda()
        got, status = run(torch, x, lambda d, o: mdx.partition_segmented(d, do, ("mod", M), out=o), rec)
        assert status == mdx.MDX_ERR_SEGMENTS
        check(got, x, offs, {0})
        assert (got[int(offs[-1]):] == -1).all()


def test_head_flags_without_a_first_one(cuda_ready):
    torch = cuda_ready
    P = 4096
    offs = np.array([P, P + 72 * P, P + 72 * P + 56 * P + 10], dtype=np.int64)
    x = values(int(offs[-1]), False)
    flags = np.zeros(x.size, dtype=np.int32)
    flags[offs[:-1]] = np.diff(offs)
    df = torch.from_numpy(flags).cuda()
    got, status = run(torch, x, lambda d, o: mdx.mdiscr_segm(d, df, ("mod", M), d_out=o), False)
    assert status == mdx.MDX_ERR_SEGMENTS
    check(got, x, offs, {1})


def test_more_runs_than_32_bits_count(cuda_ready):
    """Segments that all cover the whole input, 2^20 + 1 of 2^12 runs each: their sum,
    taken modulo 2^32, would fit the run table."""
    torch = cuda_ready
    n = 1 << 24
    offs = torch.zeros(2 * ((1 << 20) + 1), dtype=torch.int64, device="cuda")
    offs[1::2] = n
    x = values(n, False)
    try:
        mdx.set_tuning(mdx.ELEM_U32, M, 0, 33, plain_two_kernel=1, run_tiles=1)
        got, status = run(torch, x, lambda d, o: mdx.partition_segmented(d, offs, ("mod", M), out=o), False)
    finally:
        mdx.load_tuning(mdx.TUNING_PATH, missing_ok=True)
    assert status == mdx.MDX_ERR_SEGMENTS
    assert (got == -1).all()
