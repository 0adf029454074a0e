"""The P-SV band solve in row segments (csrc/psv_seg.cu) where its segments
are at their edges, against the oracle's sequential band solve (dcsymbdl0 /
dcsbdlv0, src/SGTpsv/dcsymbdl.f90:2-166).

Another elimination order of the same FP64 equations: results differ by
rounding, which the small model amplifies to about 1e-13; bar 1e-10 relative
L2 per array, the repository's bar of FP64 parity, and identical cutoffs."""
import numpy as np
import pytest

import dsmsgt
from cases import psv_small
from conftest import rel_l2

TOL = 1e-10

# source radii: in the topmost element (the source rows are the surface
# rows), in the element below it (no row between the source and the surface
# rows), mid-crust, mantle, near a separator of the inner core, and in the
# second element from the centre (no row below the source)
RADII = [6370.0, 6360.0, 6350.0, 6071.0, 3700.0, 900.0, "second"]


def _r0(job, where):
    if where != "second":
        return where
    s = dsmsgt.Setup(job, "psv")
    z0 = s.s.vrmax[0] / s.s.nlayer[0]  # first element of the innermost zone
    return 1.5 * z0


@pytest.mark.gpu
@pytest.mark.parametrize("where", RADII)
@pytest.mark.parametrize("imax", [64, 9])
def test_source_at_segment_edges_matches_oracle(built, where, imax):
    from oracle import driver_setup, oracle as orc
    r0 = _r0(psv_small(imax=imax, rdelta=700.0), where)
    job = psv_small(imax=imax, rdelta=700.0, r0=r0)
    freqs = [5, imax]
    ctx = dsmsgt.Context(dsmsgt.Setup(job, "psv"))
    t, r, y, llog = ctx.run(freqs)
    ctx.close()
    ot, orr, oy, ollog = orc.run(driver_setup.psv_setup(job), freqs, threads=8)
    assert list(llog) == list(ollog)
    for a, b in ((t, ot), (r, orr), (y, oy)):
        assert np.all(np.isfinite(a))
        assert rel_l2(a, b) <= TOL


@pytest.mark.gpu
def test_orders_and_frequencies_sharing_a_warp(built):
    """Order ranges of 32 with more frequencies than fit one warp's stage:
    the same outputs as one frequency at a time."""
    s = dsmsgt.Setup(psv_small(), "psv")
    freqs = [3, 11, 12, 40, 64]
    one = dsmsgt.Context(s, freq_batch=1, l_chunk=32)
    want = [one.run([f]) for f in freqs]
    one.close()
    many = dsmsgt.Context(s, freq_batch=5, l_chunk=32)
    got = many.run(freqs)
    many.close()
    for k, w in enumerate(want):
        assert got[3][k] == w[3][0]
        for a, b in zip(got[:3], w[:3]):
            assert np.array_equal(a[k], b[0])


# source radii of the SH model (3480 to 6371 km): in the first and the last
# element, next to them, mid-mantle
@pytest.mark.gpu
@pytest.mark.parametrize("r0", [3480.5, 3500.0, 5000.0, 6300.0, 6360.0, 6370.9])
@pytest.mark.parametrize("imax", [48, 5])
def test_sh_source_at_segment_edges_matches_oracle(built, r0, imax):
    from cases import sh_small
    from oracle import driver_setup, oracle as orc
    job = sh_small(imax=imax)
    job.param_text = job.param_text.replace("# 6. source radius (km)\n6271.0", f"# 6. source radius (km)\n{r0!r}")
    assert f"\n{r0!r}\n" in job.param_text
    freqs = [2, imax]
    ctx = dsmsgt.Context(dsmsgt.Setup(job, "sh"))
    t, r, y, llog = ctx.run(freqs)
    ctx.close()
    ot, orr, oy, ollog = orc.run(driver_setup.sh_setup(job), freqs, threads=8)
    assert list(llog) == list(ollog)
    for a, b in ((t, ot), (r, orr), (y, oy)):
        assert np.all(np.isfinite(a))
        assert rel_l2(a, b) <= TOL
