"""Records above 16 classes whose neighbours share a class: threads of one class beside
threads of several, in every launch form, bit-exact against the oracle."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx
import oracle

pytestmark = pytest.mark.gpu


def classes(n, m, form, per, rng):
    if form == "threads":  # each thread's records are of one class
        return np.repeat(rng.integers(0, m, n // per + 1), per)[:n]
    if form == "some":  # of one class, or of any, in turn and at random
        c = np.repeat(rng.integers(0, m, n // per + 1), per)[:n]
        mixed = np.repeat(rng.random(n // per + 1) < 0.4, per)[:n]
        return np.where(mixed, rng.integers(0, m, n), c)
    if form == "lane":  # all but one thread of a warp
        c = rng.integers(0, m, n)
        t = np.arange(n) // per
        return np.where(t % 32 == (t // 32) % 32, c, (t // 7) % m)
    lengths = rng.integers(1, 41, n)  # runs that begin anywhere in a thread's records
    return np.repeat(rng.integers(0, m, n), lengths)[:n]


def records(n, m, form, per, seed):
    rng = np.random.default_rng(seed)
    key = rng.integers(0, 1 << 24, n) * m + classes(n, m, form, per, rng)
    return key.astype(np.uint64) | (np.arange(n, dtype=np.uint64) << np.uint64(32))


FORMS = ["threads", "some", "lane", "runs"]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("m", [17, 32, 64])
def test_records_of_8_bytes(cuda_ready, m, form):
    torch = cuda_ready
    for knobs in (dict(plain_two_kernel=1), dict(plain_two_kernel=1, tile_threads=512),
                  dict(plain_two_kernel=1, tile_bytes=32), dict(plain_two_kernel=0)):
        x = records(150_001, m, form, 4 if knobs.get("tile_bytes") else 8, m)
        eo, es = oracle.partition(x, m)
        d = torch.from_numpy(x.view(np.int64)).cuda()
        for n in (9_000, 150_001):  # one launch of a few tiles, and more
            eo, es = oracle.partition(x[:n], m)
            try:
                mdx.set_tuning(mdx.ELEM_REC8, m, 0, 33, **knobs)
                out, sizes = mdx.partition(d[:n], ("mod", m))
                torch.cuda.synchronize()
            finally:
                mdx.set_tuning(mdx.ELEM_REC8, m, 0, 33)
                mdx.load_tuning(mdx.TUNING_PATH, missing_ok=True)
            assert mdx.workspace(0).error() == mdx.MDX_OK
            assert np.array_equal(sizes.cpu().numpy(), es), knobs
            assert np.array_equal(out.cpu().numpy().view(np.uint64), eo), knobs


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("m", [32, 64])
def test_sharded_output(cuda_ready, m, form):
    torch = cuda_ready
    n = 150_001
    x = records(n, m, form, 8, m + 1)
    eo, es = oracle.partition(x, m)
    d = torch.from_numpy(x.view(np.int64)).cuda()
    ws = mdx.new_workspace(mdx.workspace_size(n, mdx.ELEM_REC8, m))
    counts = mdx.dist_count(d, ("mod", m), ws)
    out = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    mdx.dist_scatter(d, ("mod", m), counts.reshape(1, m), 0, [out.data_ptr()], n + 1, n, ws)
    torch.cuda.synchronize()
    assert ws.error() == mdx.MDX_OK
    assert np.array_equal(out[:n].cpu().numpy().view(np.uint64), eo)
    assert np.array_equal(counts.cpu().numpy(), es)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("m", [32, 64])
def test_records_of_16_bytes(cuda_ready, m, form):
    torch = cuda_ready
    for n in (5_000, 150_001):
        x = records(n, m, form, 4, m + 2)
        rows = np.empty((n, 4), dtype=np.uint32)
        rows[:, 0], rows[:, 1] = x & np.uint64(0xffffffff), x >> np.uint64(32)
        rows[:, 2:] = rows[:, :2] ^ 0x5bd1e995
        out, sizes = mdx.partition_records(torch.from_numpy(rows.view(np.int32)).cuda(), 16, ("mod", m))
        torch.cuda.synchronize()
        cls = rows[:, 0] % m
        assert np.array_equal(sizes.cpu().numpy(), np.bincount(cls, minlength=m))
        assert np.array_equal(out.cpu().numpy().view(np.uint32), rows[np.argsort(cls, kind="stable")])
