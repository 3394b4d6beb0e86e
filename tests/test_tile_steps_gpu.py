"""The plain path's tile steps where they can go wrong, bit-exact against the
oracle: remainders over the whole range of 32-bit keys, sorted and clustered
inputs (warps of one class next to mixed ones), and every tile geometry at the
edges of its tiles."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx
import oracle

pytestmark = pytest.mark.gpu


def partition(torch, x, m, kind="mod"):
    d = torch.from_numpy(x.view(np.int64 if x.dtype == np.uint64 else np.int32)).cuda()
    out, sizes, hf = mdx.partition(d, (kind, m), headflags=True)
    torch.cuda.synchronize()
    assert mdx.workspace(0).error() == mdx.MDX_OK
    return out.cpu().numpy().view(x.dtype), sizes.cpu().numpy(), hf.cpu().numpy().view(np.uint32)


def check(torch, x, m, kind="mod"):
    eo, es, ef = oracle.partition(x, m, kind=oracle.DISCR_MASK if kind == "mask" else oracle.DISCR_MOD,
                                  headflags=True)
    go, gs, gf = partition(torch, x, m, kind)
    assert np.array_equal(gs, es)
    assert np.array_equal(go, eo)
    assert np.array_equal(gf, ef)


def test_remainders_of_every_class_count(cuda_ready):
    """Keys at and around multiples of m up to 2^32 - 1: the reciprocal's
    quotient is off by one there first."""
    rng = np.random.default_rng(1)
    for m in range(1, 65):
        q = np.concatenate([np.arange(0, 40), rng.integers(0, (1 << 32) // m, 1500),
                            np.arange((1 << 32) // m - 40, (1 << 32) // m + 1)]).astype(np.uint64) * m
        k = np.concatenate([q - 1, q, q + 1, rng.integers(0, 1 << 32, 1000).astype(np.uint64)])
        x = k[k < (1 << 32)].astype(np.uint32)
        x[-1] = 0xffffffff
        check(cuda_ready, x, m)


def clustered(n, m, form, seed):
    rng = np.random.default_rng(seed)
    if form == "sorted":
        cls = np.sort(rng.integers(0, m, n))
    elif form == "one":
        cls = np.full(n, m - 1)
    elif form == "runs":  # lengths around a warp's and a thread's elements
        lengths = rng.choice([1, 15, 16, 17, 127, 128, 255, 256, 511, 512, 513, 2000, 9000], n)
        cls = np.repeat(rng.integers(0, m, n), lengths)[:n]
    else:  # two classes hold nearly all
        cls = np.where(rng.random(n) < 0.02, rng.integers(0, m, n), (np.arange(n) // 3000) % 2)
    return (rng.integers(0, 1 << 24, n) * m + cls).astype(np.uint32)


@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("m", [2, 3, 8, 13, 32, 64])
def test_clustered_inputs(cuda_ready, m, threads, rec):
    elem = mdx.ELEM_REC8 if rec else mdx.ELEM_U32
    tile = threads * (8 if rec else 16)
    try:
        mdx.set_tuning(elem, m, 0, 33, plain_two_kernel=1, tile_bytes=64, tile_threads=threads)
        for form in ("sorted", "one", "runs", "two"):
            for n in (tile - 1, tile, 3 * tile + 1, 700_001):
                x = clustered(n, m, form, m + n)
                if rec:
                    x = x.astype(np.uint64) | (np.arange(n, dtype=np.uint64) << np.uint64(32))
                check(cuda_ready, x, m)
    finally:
        mdx.set_tuning(elem, m, 0, 33)
        mdx.load_tuning(mdx.TUNING_PATH, missing_ok=True)


@pytest.mark.parametrize("m", [5, 16, 32, 64])
def test_records_of_16_bytes(cuda_ready, m):
    """Four records a thread: the count columns and byte groups at their smallest."""
    torch = cuda_ready
    for n in (1023, 1024, 4097, 300_001):
        for form in ("sorted", "runs"):
            keys = clustered(n, m, form, n)
            rows = np.empty((n, 4), dtype=np.uint32)
            rows[:, 0] = keys
            rows[:, 1:] = np.random.default_rng(n).integers(0, 1 << 32, (n, 3))
            order = np.argsort(keys % m, kind="stable")
            d = torch.from_numpy(rows.view(np.int32)).cuda()
            out, sizes = mdx.partition_records(d, 16, ("mod", m))
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy().view(np.uint32), rows[order])
            assert np.array_equal(sizes.cpu().numpy(), np.bincount(keys % m, minlength=m))


@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("m", [1, 2, 3, 8, 13, 32, 64])
def test_a_few_tiles_in_one_launch(cuda_ready, m, rec):
    """Up to eight tiles of 16 KB go through one cluster launch: its tile edges, the
    largest size it takes and the first it does not, buffers off their alignment."""
    torch = cuda_ready
    tile = 2048 if rec else 4096
    kind = np.int64 if rec else np.int32
    for n in (1, 15, tile - 1, tile, tile + 1, 5 * tile + 77, 8 * tile - 1, 8 * tile, 8 * tile + 1):
        for form in ("runs", "sorted"):
            x = clustered(n, m, form, m + n)
            if rec:
                x = x.astype(np.uint64) | (np.arange(n, dtype=np.uint64) << np.uint64(32))
            eo, es, ef = oracle.partition(x, m, headflags=True)
            for off_in, off_out in ((0, 0), (1, 0), (0, 1)):
                base = torch.zeros(n + 2, dtype=torch.int64 if rec else torch.int32, device="cuda")
                base[off_in:off_in + n] = torch.from_numpy(x.view(kind)).cuda()
                out = torch.zeros_like(base)
                o, sizes, hf = mdx.partition(base[off_in:off_in + n], ("mod", m),
                                             out=out[off_out:off_out + n], headflags=True)
                torch.cuda.synchronize()
                assert np.array_equal(sizes.cpu().numpy(), es), (n, form)
                assert np.array_equal(o.cpu().numpy().view(x.dtype), eo), (n, form, off_in, off_out)
                assert np.array_equal(hf.cpu().numpy().view(np.uint32), ef), (n, form)
                assert not out[:off_out].any() and not out[off_out + n:].any()
        host, host_sizes = mdx.mdiscr(base[:n].clone(), ("mod", m))
        assert sum(host_sizes) == n


@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("m", [2, 7, 16, 40])
def test_inputs_off_a_16_byte_address(cuda_ready, m, rec):
    """An input that begins inside a 16-byte word is read from that word's address:
    every position in it, at and around whole tiles counted from there."""
    torch = cuda_ready
    tile = 2048 if rec else 4096
    kind = np.int64 if rec else np.int32
    for off in (1,) if rec else (1, 2, 3):
        for n in (8 * tile + 1, 9 * tile - off, 9 * tile - off + 1, 9 * tile, 20 * tile - 1, 700_001):
            x = clustered(n, m, "two" if off == 2 else "runs", m + n)
            if rec:
                x = x.astype(np.uint64) | (np.arange(n, dtype=np.uint64) << np.uint64(32))
            eo, es, ef = oracle.partition(x, m, headflags=True)
            base = torch.full((n + 8,), -1, dtype=torch.int64 if rec else torch.int32, device="cuda")
            base[off:off + n] = torch.from_numpy(x.view(kind)).cuda()
            out, sizes, hf = mdx.partition(base[off:off + n], ("mod", m), headflags=True)
            torch.cuda.synchronize()
            assert mdx.workspace(0).error() == mdx.MDX_OK
            assert np.array_equal(sizes.cpu().numpy(), es), (n, off)
            assert np.array_equal(out.cpu().numpy().view(x.dtype), eo), (n, off)
            assert np.array_equal(hf.cpu().numpy().view(np.uint32), ef), (n, off)
