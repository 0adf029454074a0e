"""The sums beyond 90 degrees on a distance grid that is symmetric about 90
degrees, against the same distances of a grid that is not (the whole
contraction, order by order).  The norms are taken over the far half alone:
near the source radius its values are far below the near half's.

FP64: the repository's bar of FP64 parity, 1e-10 relative L2 (the grids' angles
differ by the rounding of their radians, and the sums start from different
tables).  Mixed: the same products in the same order, so the same bits."""
import numpy as np
import pytest

import dsmsgt
from conftest import rel_l2
from dsmsgt import synth


def _run(mode, precision, freqs, rmin, rmax, rdelta, r0, thmax):
    model = synth.sh_mantle_model(0) if mode == "sh" else synth.psv_earth_model(0)
    job = dsmsgt.Job(
        synth.param_file(tlen=1638.4, rmin=rmin, rmax=rmax, rdelta=rdelta, r0=r0, thmin=0.0, thmax=thmax, thdelta=1.0,
                         imin=0, imax=64), synth.dsm_config(), model)
    ctx = dsmsgt.Context(dsmsgt.Setup(job, mode), precision=precision, freq_batch=len(freqs))
    out = ctx.run(freqs)
    ctx.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["psv", "sh"])
@pytest.mark.parametrize("freqs", [[1], [3]])
def test_fp64_far_half_next_to_the_source(built, mode, freqs):
    geo = (6046.0, 6067.0, 10.0, 6061.0)  # receivers 15, 5 and 5 km from the source radius
    got = _run(mode, dsmsgt.DSM_PREC_FP64, freqs, *geo, 180.0)
    want = _run(mode, dsmsgt.DSM_PREC_FP64, freqs, *geo, 178.0)
    assert list(got[-1]) == list(want[-1])
    for a, b in zip(got[:-1], want[:-1]):
        assert np.all(np.isfinite(a))
        assert rel_l2(a[:, 91:179], b[:, 91:]) <= 1e-10
        assert rel_l2(a[:, :91], b[:, :91]) <= 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["psv", "sh"])
@pytest.mark.parametrize("r0", [6061.0, 5871.0])
def test_mixed_distances_do_not_depend_on_the_grid(built, mode, r0):
    geo = (3571.0, 6330.0, 250.0, r0)
    got = _run(mode, dsmsgt.DSM_PREC_MIXED, [1, 33, 64], *geo, 180.0)
    want = _run(mode, dsmsgt.DSM_PREC_MIXED, [1, 33, 64], *geo, 178.0)
    assert list(got[-1]) == list(want[-1])
    for a, b in zip(got[:-1], want[:-1]):
        assert np.array_equal(a[:, :179], b)
