"""Groups of sources with the depth cut (the mixed path's default): a system's
bottom segment then lies in a shared segment for one source and in the
source's own for another, on a stream of its own.  Against a context of each
source alone without the cut (with it, a source's own cut lies higher than that
of a group with a deeper one): equal cutoffs, outputs to 1e-12 (FP64, the cut's
bound squared and rounding) or 1e-6 (mixed) relative L2."""
import numpy as np
import pytest

import dsmsgt
from cases import psv_small
from conftest import rel_l2

GROUPS = [(6366.0, 6361.0, 6271.0, 5071.0, 4071.0), (6361.0, 6071.0, 5971.0, 3900.0)]


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(dsmsgt.DSM_PREC_FP64, 1e-12), (dsmsgt.DSM_PREC_MIXED, 1e-6)])
@pytest.mark.parametrize("radii", GROUPS)
def test_source_groups_with_the_cut(built, radii, prec, tol):
    setups = [dsmsgt.Setup(psv_small(r0=r0, rdelta=350.0), "psv") for r0 in radii]
    freqs = [64, 3, 29]
    mc = dsmsgt.MultiSourceContext(setups, precision=prec)
    mc.set_depth_cutoff(1e-20)
    for _ in range(2):
        got = mc.run(freqs)
    mc.close()
    for s, g in zip(setups, got):
        c = dsmsgt.Context(s, precision=prec)
        c.set_depth_cutoff(0.0)
        want = c.run(freqs)
        c.close()
        assert list(g[3]) == list(want[3])
        for a, b in zip(g[:3], want[:3]):
            assert np.all(np.isfinite(a))
            for i in range(len(freqs)):
                assert rel_l2(a[i], b[i]) <= tol
