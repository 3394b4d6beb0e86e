"""The small-segment groups of the segmented path at their edges, bit-exact against
the oracle: segments that begin and end inside a thread's 16-byte words, several in
one word, empty ones at a group's ends, groups of one segment and of 128, lengths at
the window, buffers off their alignment, every class bound, and a class count per
segment."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx
import oracle

pytestmark = pytest.mark.gpu


def lengths_of(form, P, rng):
    if form == "tiny":  # many heads in every word
        return rng.integers(0, 5, 9000)
    if form == "empty":  # runs of empty segments before, between and after full ones
        x = np.zeros(3000, dtype=np.int64)
        x[rng.choice(3000, 120, replace=False)] = rng.integers(1, P + 1, 120)
        return x
    if form == "window":  # at the small-segment bound and the window
        return rng.choice([1, 2, 3, P - 5, P - 4, P - 3, P - 1, P], 60)
    if form == "words":  # around a thread's words at every number of them
        return rng.choice([3, 4, 5, 12, 19, 20, 21, 28, 36, 37, 1019, 1020, 1025], 900)
    return np.concatenate([[P, 0, 1], rng.integers(1, 400, 200), [P - 1], np.zeros(130, np.int64), [7]])


@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("form", ["tiny", "empty", "window", "words", "mixed"])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 7, 8, 13, 16])
def test_groups(cuda_ready, m, form, rec):
    torch = cuda_ready
    rng = np.random.default_rng(m * 7 + len(form))
    P = 2048 if rec else 4096
    offs = np.concatenate([[0], np.cumsum(lengths_of(form, P, rng))]).astype(np.uint64)
    n = int(offs[-1])
    x = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    if rec:
        x = x.astype(np.uint64) | (np.arange(n, dtype=np.uint64) << np.uint64(32))
    eo, es, ef = oracle.partition_segmented(x, offs, m, headflags=True)
    kind = np.int64 if rec else np.int32
    do = torch.from_numpy(offs.view(np.int64)).cuda()
    for off_in, off_out in ((0, 0), (1, 0), (0, 1)):
        base = torch.zeros(n + 4, dtype=torch.int64 if rec else torch.int32, device="cuda")
        base[off_in:off_in + n] = torch.from_numpy(x.view(kind)).cuda()
        out = torch.zeros_like(base)
        o, sizes, hf = mdx.partition_segmented(base[off_in:off_in + n], do, ("mod", m),
                                               out=out[off_out:off_out + n], headflags=True)
        torch.cuda.synchronize()
        assert mdx.workspace(0).error() == mdx.MDX_OK
        assert np.array_equal(sizes.cpu().numpy(), es)
        assert np.array_equal(o.cpu().numpy().view(x.dtype), eo), (off_in, off_out)
        assert np.array_equal(hf.cpu().numpy(), ef)


def test_class_count_per_segment(cuda_ready):
    torch = cuda_ready
    rng = np.random.default_rng(2)
    lengths = np.concatenate([rng.integers(0, 40, 2000), rng.integers(1, 4097, 60), [9000, 5, 70_000]])
    seg_m = rng.integers(1, 17, lengths.size).astype(np.int32)
    offs = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    x = rng.integers(0, 1 << 32, int(offs[-1]), dtype=np.uint64).astype(np.uint32)
    out, sizes = mdx.partition_segmented_multi(
        torch.from_numpy(x.view(np.int32)).cuda(), torch.from_numpy(offs.view(np.int64)).cuda(),
        torch.from_numpy(seg_m).cuda(), 16)
    torch.cuda.synchronize()
    assert mdx.workspace(0).error() == mdx.MDX_OK
    got, gs = out.cpu().numpy().view(np.uint32), sizes.cpu().numpy()
    for s in range(lengths.size):
        a, b = int(offs[s]), int(offs[s + 1])
        cls = x[a:b] % seg_m[s]
        assert np.array_equal(got[a:b], x[a:b][np.argsort(cls, kind="stable")]), s
        assert np.array_equal(gs[s], np.bincount(cls, minlength=16)), s


@pytest.mark.parametrize("batch", [1, 3, 32])
@pytest.mark.parametrize("groups", [1, 2, 443, 2300])
def test_groups_a_cta(cuda_ready, batch, groups):
    """From one group in all to several tickets a CTA, with batches that end before
    and at the last group."""
    torch = cuda_ready
    rng = np.random.default_rng(groups + batch)
    offs = np.concatenate([[0], np.cumsum(rng.integers(1500, 4097, 2 * groups))]).astype(np.uint64)
    n = int(offs[-1])
    x = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    eo, es, ef = oracle.partition_segmented(x, offs, 5, headflags=True)
    try:
        mdx.set_tuning(mdx.ELEM_U32, 8, 0, 33, run_tiles=4, group_batch=batch)
        o, sizes, hf = mdx.partition_segmented(torch.from_numpy(x.view(np.int32)).cuda(),
                                               torch.from_numpy(offs.view(np.int64)).cuda(), ("mod", 5),
                                               headflags=True)
        torch.cuda.synchronize()
    finally:
        mdx.load_tuning(mdx.TUNING_PATH, missing_ok=True)
    assert mdx.workspace(0).error() == mdx.MDX_OK
    assert np.array_equal(sizes.cpu().numpy(), es)
    assert np.array_equal(o.cpu().numpy().view(np.uint32), eo)
    assert np.array_equal(hf.cpu().numpy(), ef)


@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("m", [8, 9, 16])
def test_groups_longer_than_the_buffers(cuda_ready, m, rec):
    """Above 8 classes a group of more than 7/4 windows gives up its last segment: ranges
    around that, the last segment as long as it can be, heads around it, a class count
    per segment."""
    torch = cuda_ready
    rng = np.random.default_rng(m)
    P = 2048 if rec else 4096
    most = P // 4 * 7
    lengths = []
    for total in (most - 1, most, most + 1, most + 9, 2 * P - 1):
        for parts in ([total - P, P], [3, 0, total - P - 3, P], [0, 1, total - P - 1, P, 0],
                      [5] * 40 + [total - P - 200, P], [P - 1, total - P + 1]):
            lengths += parts + [-sum(parts) % P]  # the next group starts a window
    lengths = np.array(lengths * 3)
    offs = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    n = int(offs[-1])
    x = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    seg_m = rng.integers(1, m + 1, lengths.size).astype(np.int32)
    cls = x % np.repeat(seg_m, lengths).astype(np.uint32)
    if rec:
        x = x.astype(np.uint64) | (np.arange(n, dtype=np.uint64) << np.uint64(32))
    eo, es, ef = oracle.partition_segmented(x, offs, m, headflags=True)
    d = torch.from_numpy(x.view(np.int64 if rec else np.int32)).cuda()
    do = torch.from_numpy(offs.view(np.int64)).cuda()
    o, sizes, hf = mdx.partition_segmented(d, do, ("mod", m), headflags=True)
    torch.cuda.synchronize()
    assert mdx.workspace(0).error() == mdx.MDX_OK
    assert np.array_equal(sizes.cpu().numpy(), es)
    assert np.array_equal(o.cpu().numpy().view(x.dtype), eo)
    assert np.array_equal(hf.cpu().numpy(), ef)
    o, sizes = mdx.partition_segmented_multi(d, do, torch.from_numpy(seg_m).cuda(), m)
    torch.cuda.synchronize()
    assert mdx.workspace(0).error() == mdx.MDX_OK
    seg = np.repeat(np.arange(lengths.size), lengths)
    assert np.array_equal(o.cpu().numpy().view(x.dtype), x[np.lexsort((cls, seg))])
    counts = np.bincount(seg * m + cls, minlength=lengths.size * m).reshape(-1, m)
    assert np.array_equal(sizes.cpu().numpy(), counts)
