"""An interpolated value is divided by the sum of its weights, rounded as a
division: with windows of one distance and a record whose value is a power of
two, the weight times the value is exact and the quotient is the value."""
import numpy as np
import pytest

import dsmsgt
import test_gpu_catalogue as cat


@pytest.mark.gpu
def test_single_weight_divides_out(built):
    value = 2.0 ** -70
    scale = value / 1e-21          # the library multiplies records by 1e-21
    assert scale * 1e-21 == value
    p = cat._params(num=4, fmin=0, fmax=40, ipdistance=0.1, c_red_reci=0.0)
    rec = np.full_like(cat._records(p, 4, 1), 1 + 1j)
    dist = np.random.default_rng(3).uniform(p["theta_min"], p["theta_min"] + 25.0, 997)
    c = dsmsgt.Catalogue(p)
    c.add(rec, scale=np.full(4, scale))
    got = c.spectra(dist)
    c.close()
    assert np.all(got[:, :, 0] == 0.0)   # frequency 0 has no record
    assert np.all(got[:, :, 1:].real == value) and np.all(got[:, :, 1:].imag == value)


@pytest.mark.gpu
def test_call_after_a_refused_one(built):
    """The staging memory of a refused call is written by the next one."""
    p = cat._params(num=4, fmax=40)
    rng = np.random.default_rng(5)
    rec, dist, coef = cat._records(p, 4, 1), rng.uniform(0.0, 30.0, 3000), rng.standard_normal((3000, 6, 4))
    bad = coef.copy()
    bad[-1, -1, -1] = np.nan
    c = dsmsgt.Catalogue(p)
    c.add(rec)
    want = c.series(dist[::-1], coef)
    for _ in range(5):
        with pytest.raises(dsmsgt.DsmError):
            c.series(dist, bad)
        assert np.array_equal(c.series(dist[::-1], coef), want)
    c.close()
