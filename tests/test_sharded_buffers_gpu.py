"""The two steps of a sharded partition on two buffers: the scatter's input holds the
elements that were counted, at another alignment within a 16-byte word.  The steps
share their chunks of tiles, so these must not depend on where the elements lie."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("m", [2, 7, 16, 40])
def test_scatter_from_a_copy_at_another_alignment(cuda_ready, m, rec):
    torch = cuda_ready
    tile = 2048 if rec else 4096
    kind, dtype = (np.int64, torch.int64) if rec else (np.int32, torch.int32)
    per_word = 2 if rec else 4
    for n in (5, tile - 1, tile, 9 * tile - 1, 9 * tile + 1, 700_001):
        x = oracle.fill_uniform_u32(n, n + m)
        if rec:
            x = x.astype(np.uint64) | (np.arange(n, dtype=np.uint64) << np.uint64(32))
        eo, es = oracle.partition(x, m)
        at = []
        for off in range(per_word):
            base = torch.full((n + 8,), -1, dtype=dtype, device="cuda")
            base[off:off + n] = torch.from_numpy(x.view(kind)).cuda()
            at.append(base[off:off + n])
        ws = mdx.new_workspace(mdx.workspace_size(n, mdx.ELEM_REC8 if rec else mdx.ELEM_U32, m))
        room = (n + per_word - 1) // per_word * per_word
        for counted, scattered in [(0, q) for q in range(per_word)] + [(1, 0)]:
            counts = mdx.dist_count(at[counted], ("mod", m), ws)
            out = torch.full((room + 16,), -1, dtype=dtype, device="cuda")
            sizes = mdx.dist_scatter(at[scattered], ("mod", m), counts.reshape(1, m), 0,
                                     [out[8:].data_ptr()], room, n, ws)
            torch.cuda.synchronize()
            assert ws.error() == mdx.MDX_OK
            assert np.array_equal(sizes.cpu().numpy(), es)
            got = out.cpu().numpy()
            assert np.array_equal(got[8:8 + n].view(x.dtype), eo), (n, counted, scattered)
            assert (got[:8] == -1).all() and (got[8 + n:] == -1).all()
