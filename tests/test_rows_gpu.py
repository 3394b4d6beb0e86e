"""The row kernels (mdx_partition_records, mdx_partition_columns) at the edges of
their tiles and units: every unit a record is moved in, the widest record they
take and the first they do not, inputs and outputs off their alignment, partial
tiles, one to eight columns, and every class bound."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx
import oracle

pytestmark = pytest.mark.gpu


def order_of(keys, m):
    rec = keys.astype(np.uint64) | (np.arange(len(keys), dtype=np.uint64) << np.uint64(32))
    out, sizes, flags = oracle.partition(rec, m, headflags=True)
    return (out >> np.uint64(32)).astype(np.int64), sizes, flags


@pytest.mark.parametrize("size", [12, 24, 48, 124, 1020, 1024, 1028])
@pytest.mark.parametrize("m", [1, 2, 7, 16, 33])
def test_record_units(cuda_ready, size, m):
    torch = cuda_ready
    words = size // 4
    for n in (1, 15, 16, 17, 1023, 20_000 // words + 1, 40_000):
        rng = np.random.default_rng(n * m + size)
        rows = rng.integers(0, 1 << 32, (n, words), dtype=np.uint64).astype(np.uint32)
        perm, es, ef = order_of(rows[:, 0], m)
        for off_in, off_out in ((0, 0), (1, 0), (0, 2), (3, 3)):  # words off a 16-byte address
            base = torch.zeros(n * words + 4, dtype=torch.int32, device="cuda")
            d = base[off_in:off_in + n * words]
            d.copy_(torch.from_numpy(rows.view(np.int32).reshape(-1)))
            out = torch.zeros(n * words + 4, dtype=torch.int32, device="cuda")
            o, sizes, hf = mdx.partition_records(d, size, ("mod", m), out=out[off_out:off_out + n * words],
                                                 headflags=True)
            torch.cuda.synchronize()
            assert mdx.workspace(0).error() == mdx.MDX_OK
            assert np.array_equal(o.cpu().numpy().view(np.uint32).reshape(n, words), rows[perm]), (n, off_in)
            assert np.array_equal(sizes.cpu().numpy(), es)
            assert np.array_equal(hf.cpu().numpy(), ef)
            assert not out[:off_out].any() and not out[off_out + n * words:].any()


@pytest.mark.parametrize("widths", [[], [1], [2, 1], [8, 4, 2, 1], [8] * 7, [1] * 7, [4, 8, 4, 1, 8, 2, 2]])
@pytest.mark.parametrize("m", [1, 2, 6, 16, 64])
def test_column_widths(cuda_ready, widths, m):
    torch = cuda_ready
    types = {1: np.uint8, 2: np.int16, 4: np.int32, 8: np.int64}
    for n in (1, 17, 1024, 2049, 60_001):
        rng = np.random.default_rng(n * m + len(widths))
        keys = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
        perm, es, ef = order_of(keys, m)
        host = [keys.view(np.int32)] + [
            rng.integers(0, 256, n * w, dtype=np.uint8).view(types[w]) for w in widths]
        for off in (0, 1):  # elements off a 16-byte address, inputs and outputs
            cols, outs = [], []
            for h in host:
                base = torch.from_numpy(np.concatenate([h[:1], h])).cuda()
                cols.append(base[1:] if off else base[1:].clone())
                outs.append(torch.zeros(n + 1, dtype=base.dtype, device="cuda")[off:off + n])
            got, sizes, hf = mdx.partition_columns(cols, ("mod", m), outs=outs, headflags=True)
            torch.cuda.synchronize()
            assert mdx.workspace(0).error() == mdx.MDX_OK
            for h, g in zip(host, got):
                assert np.array_equal(g.cpu().numpy(), h[perm]), (n, off, h.dtype)
            assert np.array_equal(sizes.cpu().numpy(), es)
            assert np.array_equal(hf.cpu().numpy(), ef)
