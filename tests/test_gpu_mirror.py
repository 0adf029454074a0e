"""Distances symmetric about 90 degrees, where even and odd orders are
contracted with half the distances (Engine::set_distances), against the
general contraction of the same distances: the grid without its last ones is
not symmetric.

FP64: the two differ by the order of the sums and by one unit in the last
place of 180 degrees; bar 1e-10 relative L2 per array, the repository's bar of
FP64 parity.  Mixed: contraction outputs are rounded to FP32 (6e-8 of each,
tens of them in a record, with cancellation); bar 2e-6."""
import numpy as np
import pytest

import dsmsgt
from conftest import rel_l2
from dsmsgt import synth

# first distance, step, number of distances: both poles and 90 degrees; even
# counts (no distance is its own mirror image); halves that need 0 to 3
# columns of padding; the smallest count; column tiles of 128 that end inside
# a basis function
GRIDS = [(0.0, 1.5, 121), (0.5, 1.0, 180), (0.0, 1.0, 181), (42.5, 1.0, 96), (41.0, 1.0, 99), (0.0, 0.5, 361)]


def _job(mode, thmin, thmax, thdelta):
    sh = mode == "sh"
    model = synth.sh_mantle_model(0) if sh else synth.psv_earth_model(0)
    return dsmsgt.Job(
        synth.param_file(tlen=1638.4, rmin=3500.0 if sh else 1000.0, rmax=6300.0, rdelta=700.0, r0=6071.0,
                         thmin=thmin, thmax=thmax, thdelta=thdelta, imin=0, imax=64), synth.dsm_config(), model)


def _run(job, mode, precision, freqs, **kw):
    ctx = dsmsgt.Context(dsmsgt.Setup(job, mode), precision=precision, **kw)
    out = ctx.run(freqs)
    st = ctx.stats()
    ctx.close()
    return out, st


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [dsmsgt.DSM_PREC_FP64, dsmsgt.DSM_PREC_MIXED])
@pytest.mark.parametrize("mode", ["psv", "sh"])
@pytest.mark.parametrize("grid", GRIDS)
def test_symmetric_distances_match_general_contraction(built, grid, mode, precision):
    t0, dt, n = grid
    freqs = [3, 33, 64]
    # 32 orders at first: field rows and tables grow
    job = _job(mode, t0, t0 + (n - 1) * dt, dt)
    got, gst = _run(job, mode, precision, freqs, l_chunk=32)
    assert dsmsgt.Setup(job, mode).theta_n == n
    want, wst = _run(_job(mode, t0, t0 + (n - 3) * dt, dt), mode, precision, freqs, l_chunk=32)
    assert list(got[-1]) == list(want[-1])
    assert gst.lsum_flops < 0.6 * wst.lsum_flops
    tol = 1e-10 if precision == dsmsgt.DSM_PREC_FP64 else 2e-6
    for a, b in zip(got[:-1], want[:-1]):
        if b.size == 0:
            continue
        ax = [i for i in range(b.ndim) if a.shape[i] != b.shape[i]]
        assert len(ax) == 1 and b.shape[ax[0]] == n - 2
        a = np.take(a, range(n - 2), axis=ax[0])
        assert np.all(np.isfinite(a))
        assert rel_l2(a, b) <= tol
