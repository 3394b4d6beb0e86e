"""Segments of many runs, whose counts a warp scans: numbers of runs around the lanes
and around the rows that a lane has in flight, bit-exact against the oracle."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [2, 3, 8, 13])
def test_numbers_of_runs(cuda_ready, m):
    torch = cuda_ready
    P = 4096
    for runs in (5, 31, 32, 33, 127, 128, 129, 255, 256, 257, 515):
        lengths = [runs * P, 7, (runs - 1) * P + 1]  # in the second one runs begin inside a row
        offs = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
        x = oracle.fill_uniform_u32(int(offs[-1]), runs)
        eo, es, ef = oracle.partition_segmented(x, offs, m, headflags=True)
        try:
            mdx.set_tuning(mdx.ELEM_U32, m, 0, 33, plain_two_kernel=1, run_tiles=1)
            o, sizes, hf = mdx.partition_segmented(torch.from_numpy(x.view(np.int32)).cuda(),
                                                   torch.from_numpy(offs.view(np.int64)).cuda(),
                                                   ("mod", m), headflags=True)
            torch.cuda.synchronize()
        finally:
            mdx.load_tuning(mdx.TUNING_PATH, missing_ok=True)
        assert mdx.workspace(0).error() == mdx.MDX_OK
        assert np.array_equal(sizes.cpu().numpy(), es), runs
        assert np.array_equal(o.cpu().numpy().view(np.uint32), eo), runs
        assert np.array_equal(hf.cpu().numpy(), ef), runs
