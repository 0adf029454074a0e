"""The cutoff scan over order ranges that end within, at and beyond the 256
orders a warp looks at together: the cutoffs and the outputs of one range per
frequency.  Ranges only cut the same sequence of orders, so both are equal
(outputs: the sums' order depends on the cutoff alone)."""
import numpy as np
import pytest

import dsmsgt
from cases import psv_small, sh_small


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["psv", "sh"])
@pytest.mark.parametrize("chunk", [32, 224, 256, 288, 512, 4096])
def test_order_ranges_give_the_same_cutoffs(built, mode, chunk):
    s = dsmsgt.Setup(psv_small() if mode == "psv" else sh_small(imax=64), mode)
    freqs = [1, 12, 64]
    ref = dsmsgt.Context(s)
    want = ref.run(freqs)
    ref.close()
    ctx = dsmsgt.Context(s, l_chunk=chunk)
    got = ctx.run(freqs)
    ctx.close()
    assert list(got[-1]) == list(want[-1])
    for a, b in zip(got[:-1], want[:-1]):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)
