"""Groups of sources whose segments are factored side by side: as many as a
group holds, one more, and two groups, deep sources beside shallow ones, at
the same depth, below every separator of the shallowest, and with a small
order range.  Bit for bit the outputs of a context of each source alone (the
same operations run on the same numbers)."""
import numpy as np
import pytest

import dsmsgt
from cases import psv_small

GROUPS = [
    (6361.0, 6071.0),
    (6071.0, 6361.0, 6071.0, 5471.0),
    (6366.0, 6361.0, 6271.0, 5071.0, 4071.0),
    (3900.0, 6361.0, 6350.0, 6271.0, 6171.0, 6071.0, 5971.0, 5771.0, 900.0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [dsmsgt.DSM_PREC_FP64, dsmsgt.DSM_PREC_MIXED])
@pytest.mark.parametrize("radii", GROUPS)
@pytest.mark.parametrize("chunk", [0, 64])
def test_source_groups_equal_single_source_contexts(built, radii, prec, chunk):
    setups = [dsmsgt.Setup(psv_small(r0=r0, rdelta=700.0), "psv") for r0 in radii]
    freqs = [3, 29]
    kw = dict(precision=prec, l_chunk=chunk) if chunk else dict(precision=prec)
    mc = dsmsgt.MultiSourceContext(setups, **kw)
    mc.set_depth_cutoff(0.0)
    got = mc.run(freqs)
    mc.close()
    for s, g in zip(setups, got):
        c = dsmsgt.Context(s, **kw)
        c.set_depth_cutoff(0.0)
        want = c.run(freqs)
        c.close()
        assert list(g[3]) == list(want[3])
        for a, b in zip(g[:3], want[:3]):
            assert np.array_equal(a, b)
