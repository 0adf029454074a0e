"""The FP64 contraction at the edges of its tiles: column counts around 32 and
64 against the oracle (1e-10 relative L2, the repository's bar of FP64
parity), and its two tile shapes against each other: a grid whose tiles fill
the SMs against a coarser grid of the same distances (1e-11 of each array's
largest value: the same products in another order of some thousand terms)."""
import numpy as np
import pytest

import dsmsgt
from cases import sh_small
from conftest import rel_l2
from dsmsgt import synth


@pytest.mark.gpu
@pytest.mark.parametrize("thdelta", [180.0, 22.5, 12.0, 11.25, 5.8, 5.625, 1.0])   # 2, 9, 16, 17, 32, 33, 181 distances
def test_column_counts_match_oracle(built, thdelta):
    from oracle import driver_setup, oracle as orc
    job = sh_small(imax=16, thdelta=thdelta, rdelta=900.0)
    freqs = [4, 15]
    ctx = dsmsgt.Context(dsmsgt.Setup(job, "sh"))
    got = ctx.run(freqs)
    ctx.close()
    want = orc.run(driver_setup.sh_setup(job), freqs, threads=8)
    assert list(got[-1]) == list(want[-1])
    for a, b in zip(got[:-1], want[:-1]):
        assert np.all(np.isfinite(a)) and rel_l2(a, b) <= 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["psv", "sh"])
@pytest.mark.parametrize("step", [1.0, 0.7])         # mirrored at 90 degrees, and not
def test_tile_shapes_agree(built, mode, step):
    sh = mode == "sh"

    def run(thdelta):
        job = dsmsgt.Job(
            synth.param_file(tlen=1638.4, rmin=3500.0, rmax=6300.0, rdelta=45.0, r0=6071.0, thmin=0.0, thmax=180.0,
                             thdelta=thdelta, imin=0, imax=64), synth.dsm_config(),
            (synth.sh_mantle_model if sh else synth.psv_earth_model)(0))
        ctx = dsmsgt.Context(dsmsgt.Setup(job, mode))
        out = ctx.run([21, 64])
        ctx.close()
        return out
    fine, coarse = run(step), run(60 * step)
    assert list(fine[-1]) == list(coarse[-1])
    for a, b in zip(fine[:-1], coarse[:-1]):
        ax = next(i for i in range(b.ndim) if a.shape[i] != b.shape[i])
        a = np.take(a, range(0, 60 * b.shape[ax], 60), axis=ax)
        assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(b))
