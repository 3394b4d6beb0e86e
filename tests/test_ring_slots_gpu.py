"""The plain scatter's ring at the numbers of tiles where it has one slot, two, and one
again: around whole rounds of the CTAs of either form, bit-exact against the oracle."""
import numpy as np
import pytest

import mdiscriminator_b200 as mdx
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("m", [2, 8, 16, 32])
def test_tiles_around_rounds_of_ctas(cuda_ready, m, rec):
    torch = cuda_ready
    tile = 2048 if rec else 4096
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x = oracle.fill_uniform_u32(10 * sms * tile, m)
    if rec:
        x = x.astype(np.uint64) | (np.arange(x.size, dtype=np.uint64) << np.uint64(32))
    d = torch.from_numpy(x.view(np.int64 if rec else np.int32)).cuda()
    for tiles in (3 * sms, 4 * sms, 5 * sms, 6 * sms, 8 * sms):
        for n in (tiles * tile, tiles * tile + 1):
            eo, es = oracle.partition(x[:n], m)
            out, sizes = mdx.partition(d[:n], ("mod", m))
            torch.cuda.synchronize()
            assert mdx.workspace(0).error() == mdx.MDX_OK
            assert np.array_equal(sizes.cpu().numpy(), es), n
            assert np.array_equal(out.cpu().numpy().view(x.dtype), eo), n
