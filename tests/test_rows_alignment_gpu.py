"""Rows whose memory begins inside a 16-byte word: a tile comes by copies of whole
words, the last one of a column only if it ends inside it.  Every position in a word,
numbers of rows at whole tiles, four and eight rows a thread."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx
import oracle

pytestmark = pytest.mark.gpu


def order_of(keys, m):
    rec = keys.astype(np.uint64) | (np.arange(len(keys), dtype=np.uint64) << np.uint64(32))
    out, sizes = oracle.partition(rec, m)
    return (out >> np.uint64(32)).astype(np.int64), sizes


def tile_rows(row_bytes, leads, m):
    """Rows of a tile when there are many: see run_rows."""
    threads = 512 if m > 16 else 256
    buf = (26624 if row_bytes <= 6 else 73728) if m > 32 else 36864 if m > 16 else 20480
    fit = (buf - 16 * leads) // row_bytes
    return min(fit & ~15, threads * (8 if fit >= 6 * threads else 4))


@pytest.mark.parametrize("m", [2, 7, 16, 20, 64])
@pytest.mark.parametrize("words", [3, 5, 8, 33])
def test_records(cuda_ready, words, m):
    torch = cuda_ready
    tile = tile_rows(4 * words, 1, m)
    for n in (tile, 300 * tile, 300 * tile + 1):
        rng = np.random.default_rng(n + m)
        rows = rng.integers(0, 1 << 32, (n, words), dtype=np.uint64).astype(np.uint32)
        perm, es = order_of(rows[:, 0], m)
        expect = rows[perm].reshape(-1)
        for off in (1, 2, 3):
            base = torch.zeros(n * words + off, dtype=torch.int32, device="cuda")
            base[off:] = torch.from_numpy(rows.view(np.int32).reshape(-1)).cuda()
            out, sizes = mdx.partition_records(base[off:], 4 * words, ("mod", m))
            torch.cuda.synchronize()
            assert mdx.workspace(0).error() == mdx.MDX_OK
            assert np.array_equal(out.cpu().numpy().view(np.uint32), expect), (n, off)
            assert np.array_equal(sizes.cpu().numpy(), es)


@pytest.mark.parametrize("m", [2, 7, 16, 20, 64])
@pytest.mark.parametrize("widths", [[], [1], [8, 2, 4], [8] * 7])
def test_columns(cuda_ready, widths, m):
    torch = cuda_ready
    types = {1: np.uint8, 2: np.int16, 4: np.int32, 8: np.int64}
    tile = tile_rows(4 + sum(widths), 1 + len(widths), m)
    for n in (300 * tile, 300 * tile + 17):
        rng = np.random.default_rng(n + m)
        keys = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
        perm, es = order_of(keys, m)
        host = [keys.view(np.int32)] + [
            rng.integers(0, 256, n * w, dtype=np.uint8).view(types[w]) for w in widths]
        expect = [h[perm] for h in host]
        for off in (1, 2, 3):  # the key's words; the others at offsets of their own
            cols = []
            for i, h in enumerate(host):
                at = off if i == 0 else (off + 2 * i) % 16
                base = torch.zeros(n + at, dtype=torch.from_numpy(h[:0]).dtype, device="cuda")
                base[at:] = torch.from_numpy(h).cuda()
                cols.append(base[at:])
            got, sizes = mdx.partition_columns(cols, ("mod", m))
            torch.cuda.synchronize()
            assert mdx.workspace(0).error() == mdx.MDX_OK
            for e, g in zip(expect, got):
                assert np.array_equal(g.cpu().numpy(), e), (n, off, e.dtype)
            assert np.array_equal(sizes.cpu().numpy(), es)


@pytest.mark.parametrize("m", [2, 16, 64])
def test_numbers_of_rows_after_the_last_whole_tile(cuda_ready, m):
    """Fewer rows of a one-byte column than a 16-byte word holds, and more."""
    torch = cuda_ready
    tile = tile_rows(5, 2, m)
    for n in (5, 15, 16, 17, 300 * tile + 1, 300 * tile + 15, 300 * tile + 16, 300 * tile + 17):
        rng = np.random.default_rng(n + m)
        keys = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
        perm, es = order_of(keys, m)
        other = rng.integers(0, 256, n, dtype=np.uint8)
        for at in (1, 15):
            base = torch.zeros(n + 3, dtype=torch.int32, device="cuda")[3:]
            base.copy_(torch.from_numpy(keys.view(np.int32)))
            col = torch.zeros(n + at, dtype=torch.uint8, device="cuda")[at:]
            col.copy_(torch.from_numpy(other))
            got, sizes = mdx.partition_columns([base, col], ("mod", m))
            torch.cuda.synchronize()
            assert mdx.workspace(0).error() == mdx.MDX_OK
            assert np.array_equal(got[0].cpu().numpy().view(np.uint32), keys[perm]), (n, at)
            assert np.array_equal(got[1].cpu().numpy(), other[perm]), (n, at)
            assert np.array_equal(sizes.cpu().numpy(), es)
