"""dsm_stats.solve_bytes: the bytes a run's band solves move.  Without the depth
cut every system of a model moves the same; with it the rows below a system's
first one do not count; a second source adds its own walk."""
import pytest

import dsmsgt
from cases import psv_small, sh_small


def _per_system(ctx, freqs):
    ctx.run(freqs)
    st = ctx.stats()
    assert st.systems > 0
    return st.solve_bytes / st.systems


@pytest.mark.gpu
@pytest.mark.parametrize("mode,prec", [("sh", dsmsgt.DSM_PREC_FP64), ("psv", dsmsgt.DSM_PREC_FP64),
                                       ("psv", dsmsgt.DSM_PREC_MIXED)])
def test_solve_bytes_of_a_system(built, mode, prec):
    s = dsmsgt.Setup(sh_small() if mode == "sh" else psv_small(), mode)
    ctx = dsmsgt.Context(s, precision=prec)
    if mode == "psv":
        ctx.set_depth_cutoff(0.0)
    one = _per_system(ctx, [3])
    # the solutions at a receiver's three nodes at least, for every right-hand side
    assert one >= 3 * (3 if mode == "sh" else 6) * 16
    assert _per_system(ctx, [7, 20, 31]) == one   # a run's count starts at zero
    if mode == "psv":
        ctx.set_depth_cutoff(1e-20)
        assert 0 < _per_system(ctx, [3, 40]) < one
    ctx.close()


@pytest.mark.gpu
def test_solve_bytes_of_two_sources(built):
    setups = [dsmsgt.Setup(psv_small(r0=r0), "psv") for r0 in (6071.0, 6071.0)]
    single = dsmsgt.Context(setups[0])
    one = _per_system(single, [3, 40])
    single.close()
    both = dsmsgt.MultiSourceContext(setups)
    both.run([3, 40])
    two = both.stats().solve_bytes / both.stats().systems
    both.close()
    assert one < two < 2 * one  # the segments below the sources are factored once
