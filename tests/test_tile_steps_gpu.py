"""The plain path's tile steps where they can go wrong, bit-exact against the
oracle: remainders over the whole range of 32-bit keys."""
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
