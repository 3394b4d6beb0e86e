"""16-byte records at the edges of their tiles: up to eight tiles in one launch, above
16 classes tiles of 512 threads whatever the knobs, below those of 256."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two_kernel", [0, 1])
@pytest.mark.parametrize("m", [2, 16, 17, 32, 40, 64])
def test_tile_edges(cuda_ready, m, two_kernel):
    torch = cuda_ready
    rng = np.random.default_rng(m)
    rows = rng.integers(0, 1 << 32, (610_000, 4), dtype=np.uint64).astype(np.uint32)
    rows[300_000:, 0] = np.sort(rows[300_000:, 0] % m)  # and in class order
    d = torch.from_numpy(rows.view(np.int32)).cuda()
    try:
        mdx.set_tuning(mdx.ELEM_U32, m, 0, 33, plain_two_kernel=two_kernel)
        for n in (8 * 1024, 8 * 1024 + 1, 5 * 2048 - 1, 5 * 2048, 5 * 2048 + 1, 296 * 2048, 296 * 2048 + 1):
            cls = rows[:n, 0] % m
            out, sizes, hf = mdx.partition_records(d[:n].contiguous(), 16, ("mod", m), headflags=True)
            torch.cuda.synchronize()
            assert mdx.workspace(0).error() == mdx.MDX_OK
            counts = np.bincount(cls, minlength=m)
            assert np.array_equal(sizes.cpu().numpy(), counts), n
            assert np.array_equal(out.cpu().numpy().view(np.uint32), rows[:n][np.argsort(cls, kind="stable")]), n
            flags = np.zeros(n, dtype=np.uint32)
            flags[(np.cumsum(counts) - counts)[counts > 0]] = counts[counts > 0]
            assert np.array_equal(hf.cpu().numpy().view(np.uint32), flags), n
    finally:
        mdx.set_tuning(mdx.ELEM_U32, m, 0, 33)
        mdx.load_tuning(mdx.TUNING_PATH, missing_ok=True)
