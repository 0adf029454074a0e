"""The P-SV depth cut above the topmost receiver, whose two rows are the
cutoff probe (receivers in the lower mantle, a shallow source): the probe of a
system that starts above them is zero, whatever an earlier launch or batch
left behind.  Against the uncut FP64 path: the same cutoffs, and outputs to
1e-12 (FP64: the cut's own bound, 1e-20 squared, and rounding) or 1e-6 (the
mixed path's bar)."""
import numpy as np
import pytest

import dsmsgt
from conftest import rel_l2
from dsmsgt import synth

FREQS = [64, 3, 50, 64, 7, 33, 64]


def _setup(r0=6071.0):
    return dsmsgt.Setup(dsmsgt.Job(
        synth.param_file(tlen=1638.4, rmin=3600.0, rmax=4000.0, rdelta=100.0, r0=r0, thmin=0.0, thmax=180.0,
                         thdelta=15.0, imin=0, imax=64), synth.dsm_config(maxlmax=4000),
        synth.psv_earth_model(0)), "psv")


def _check(got, want, tol):
    assert list(got[3]) == list(want[3])
    for x, y in zip(got[:3], want[:3]):
        assert np.all(np.isfinite(x))
        for i in range(len(FREQS)):
            assert rel_l2(x[i], y[i]) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(dsmsgt.DSM_PREC_FP64, 1e-12), (dsmsgt.DSM_PREC_MIXED, 1e-6)])
@pytest.mark.parametrize("kw", [dict(freq_batch=1), dict(freq_batch=2, l_chunk=96), dict(freq_batch=7)])
def test_probe_rows_below_the_cut_are_zero(built, prec, tol, kw):
    s = _setup()
    a = dsmsgt.Context(s, freq_batch=7)
    want = a.run(FREQS)
    a.close()
    b = dsmsgt.Context(s, precision=prec, **kw)
    b.set_depth_cutoff(1e-20)
    for _ in range(2):  # the second run finds the first one's values in the scratch
        _check(b.run(FREQS), want, tol)
    b.close()


@pytest.mark.gpu
def test_probe_rows_below_the_cut_are_zero_for_several_sources(built):
    setups = [_setup(r0) for r0 in (6071.0, 6361.0, 5771.0)]
    m = dsmsgt.MultiSourceContext(setups, freq_batch=2)
    m.set_depth_cutoff(1e-20)
    got = m.run(FREQS)
    m.close()
    for s, g in zip(setups, got):
        c = dsmsgt.Context(s, freq_batch=7)
        want = c.run(FREQS)
        c.close()
        _check(g, want, 1e-12)
