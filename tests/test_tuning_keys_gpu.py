"""Which entry of the tuning table a call takes."""
import pytest

import mdiscriminator_b200 as mdx

pytestmark = pytest.mark.gpu


def test_records_of_16_bytes_take_the_entry_of_as_many_bytes(cuda_ready):
    m = 6
    try:
        mdx.set_tuning(mdx.ELEM_U32, m, 0, 33, plain_two_kernel=1, plain_ctas_per_sm=1)
        mdx.set_tuning(mdx.ELEM_U32, m, 20, 21, plain_two_kernel=1, plain_ctas_per_sm=3)
        ctas = lambda n: mdx.get_tuning(mdx.ELEM_REC16, m, n)["plain_ctas_per_sm"]  # noqa: E731
        assert [ctas(n) for n in (1 << 17, 1 << 18, (1 << 18) + 1, 1 << 19, (1 << 19) + 1)] == [1, 3, 3, 3, 1]
        assert ctas(0xffffffff) == 1
        mdx.set_tuning(mdx.ELEM_REC16, m, 19, 33, plain_two_kernel=1, plain_ctas_per_sm=2)
        assert [ctas(n) for n in (1 << 18, 1 << 19, 1 << 20, 0xffffffff)] == [3, 2, 2, 2]
        assert mdx.get_tuning(mdx.ELEM_U32, m, 1 << 21)["plain_ctas_per_sm"] == 2
        assert mdx.get_tuning(mdx.ELEM_U32, m, 1 << 20)["plain_ctas_per_sm"] == 3
    finally:
        mdx.set_tuning(mdx.ELEM_U32, m, 0, 33)
        mdx.load_tuning(mdx.TUNING_PATH, missing_ok=True)
