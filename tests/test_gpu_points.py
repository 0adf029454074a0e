"""Edges of the point interpolation (chunks of distances, columns of
components, blocks of frequencies, rows of outputs) and of the filter stage
(segments, lanes of an item, windows kept in shared memory or not) against
the oracle, with the bar of the whole catalogue path: 1e-10 relative L2 (FP64
throughout)."""
import numpy as np
import pytest

import test_gpu_catalogue as cat
import test_gpu_kernels as ker
from conftest import rel_l2


@pytest.mark.gpu
@pytest.mark.parametrize("num,nout", [(1, 1), (3, 64), (4, 5), (7, 2), (32, 64), (32, None)])
@pytest.mark.parametrize("fmin,fmax,width", [(0, 64, 0.5), (3, 6, 3.0), (6, 50, 8.0), (0, 0, 15.5)])
def test_points_match_oracle(built, num, nout, fmin, fmax, width):
    p = cat._params(num=num, fmin=fmin, fmax=fmax, ipdistance=width, c_red_reci=4.0)
    rng = np.random.default_rng(num + fmax)
    dist = np.sort(rng.uniform(0.0, 30.0, 71))       # a full tile of 32, another, and the rest
    rec = cat._records(p, num, 9)
    coef = None if nout is None else rng.standard_normal((dist.size, nout, num))
    got = cat._run(p, [(rec, None, None)], dist, coef)
    want = cat._oracle(p, [(rec, np.arange(num), np.ones(num))], dist, coef)
    assert got.shape == want.shape
    assert np.sqrt(np.sum((got - want) ** 2)) <= cat.TOL * max(np.sqrt(np.sum(want ** 2)), 1e-300)


# samples of the window: fewer than a segment, one segment and the start of
# the next, 16 segments, just within and beyond the shared memory of a block
@pytest.mark.gpu
@pytest.mark.parametrize("npoles", [1, 7, 8])
@pytest.mark.parametrize("nwin", [12, 33, 513, 2700, 6000])
def test_filters_match_oracle(built, npoles, nwin):
    rng = np.random.default_rng(nwin + npoles)
    p = cat._params(np1=4096, tlen=4096.0, omegai=np.log(100.0) / 4096.0, fmax=60, iwin_start=7, iwin_end=6 + nwin)
    kp = ker._kparams(p, 2, 1, 3, rng, npoles)
    kp["nt1"] = [p["iwin_start"], p["iwin_start"] + nwin // 3]
    kp["nt2"] = [p["iwin_end"], p["iwin_start"] + nwin // 2]
    ir = np.array([0, 1, 1])
    h3, h4 = ker._spectra(rng, ir.size, 61)
    want = ker._oracle(p, kp, ir, h3, h4)
    got = ker._device(p, kp, ir, h3, h4)
    assert rel_l2(got[1], want[1]) <= ker.TOL
    assert rel_l2(got[0], want[0]) <= ker.TOL
