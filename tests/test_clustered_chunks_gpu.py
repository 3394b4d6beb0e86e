"""The scatter's loop for chunks that two classes fill, at 3 to 16 classes: it is taken
by chunks of several tiles, so the grid is kept small, with numbers of tiles that give
chunks of unequal length, and inputs off a 16-byte address, whose first tile begins
inside a word."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx
import oracle

pytestmark = pytest.mark.gpu


def classes(n, m, form, rng):
    if form == "sorted":
        return np.sort(rng.integers(0, m, n))
    if form == "one":
        return np.full(n, m - 1)
    if form == "two":  # two at a time, a warp of one class here and there
        pair = np.arange(n) * 4 // n % (m - 1)
        return pair + np.repeat(rng.integers(0, 2, n // 500 + 1), 500)[:n]
    few = np.arange(n) * 3 // n % m  # one class, and others within an eighth of a chunk
    return np.where(rng.random(n) < 0.1, rng.integers(0, m, n), few)


@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("m", [3, 4, 8, 13, 16])
def test_chunks_of_two_classes(cuda_ready, m, threads, rec):
    torch = cuda_ready
    elem = mdx.ELEM_REC8 if rec else mdx.ELEM_U32
    kind, dtype = (np.int64, torch.int64) if rec else (np.int32, torch.int32)
    tile = threads * (8 if rec else 16)
    ctas = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(m)
    try:
        mdx.set_tuning(elem, m, 0, 33, plain_two_kernel=1, plain_ctas_per_sm=1, tile_threads=threads)
        for form in ("sorted", "one", "two", "few"):
            # at least four tiles a CTA: exactly, one element more, and five here and there
            for n in (4 * ctas * tile, 4 * ctas * tile + 1, 9 * ctas * tile // 2 - 3):
                x = (rng.integers(0, 1 << 24, n) * m + classes(n, m, form, rng)).astype(np.uint32)
                if rec:
                    x = x.astype(np.uint64) | (np.arange(n, dtype=np.uint64) << np.uint64(32))
                eo, es = oracle.partition(x, m)
                for off in (0, 1) if rec or form != "two" else (0, 3):
                    base = torch.full((n + 4,), -1, dtype=dtype, device="cuda")
                    base[off:off + n] = torch.from_numpy(x.view(kind)).cuda()
                    out, sizes = mdx.partition(base[off:off + n], ("mod", m))
                    torch.cuda.synchronize()
                    assert mdx.workspace(0).error() == mdx.MDX_OK
                    assert np.array_equal(sizes.cpu().numpy(), es), (form, n, off)
                    assert np.array_equal(out.cpu().numpy().view(x.dtype), eo), (form, n, off)
    finally:
        mdx.set_tuning(elem, m, 0, 33)
        mdx.load_tuning(mdx.TUNING_PATH, missing_ok=True)


@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("geometry", [dict(tile_bytes=64), dict(tile_bytes=32), dict(tile_threads=512)])
@pytest.mark.parametrize("m", [2, 5, 16, 40])
def test_tile_edges_of_every_geometry(cuda_ready, m, geometry, rec):
    """More than the eight tiles that go in one launch whatever the geometry."""
    torch = cuda_ready
    elem = mdx.ELEM_REC8 if rec else mdx.ELEM_U32
    tile = geometry.get("tile_threads", 256) * geometry.get("tile_bytes", 64) // (8 if rec else 4)
    base = 8 * (2048 if rec else 4096)
    first = base // tile + 1
    x = oracle.fill_uniform_u32((first + 1) * tile + 1, m)
    if rec:
        x = x.astype(np.uint64) | (np.arange(x.size, dtype=np.uint64) << np.uint64(32))
    d = torch.from_numpy(x.view(np.int64 if rec else np.int32)).cuda()
    try:
        mdx.set_tuning(elem, m, 0, 33, plain_two_kernel=1, **geometry)
        for n in (base + 1, first * tile - 1, first * tile, first * tile + 1, (first + 1) * tile):
            eo, es = oracle.partition(x[:n], m)
            out, sizes = mdx.partition(d[:n], ("mod", m))
            torch.cuda.synchronize()
            assert mdx.workspace(0).error() == mdx.MDX_OK
            assert np.array_equal(sizes.cpu().numpy(), es), n
            assert np.array_equal(out.cpu().numpy().view(x.dtype), eo), n
    finally:
        mdx.set_tuning(elem, m, 0, 33)
        mdx.load_tuning(mdx.TUNING_PATH, missing_ok=True)
