"""SH receiver fields and slot weights where the receivers do not fill the
warps of a block (1 to 6 with the surface) and the orders do not fill a warp,
against the oracle: 1e-10 relative L2 per array, the repository's bar of FP64
parity."""
import numpy as np
import pytest

import dsmsgt
from conftest import rel_l2
from dsmsgt import synth


@pytest.mark.gpu
@pytest.mark.parametrize("rmin,rdelta", [(6300.0, 50.0), (6200.0, 100.0), (6000.0, 100.0), (5900.0, 100.0)])
@pytest.mark.parametrize("freqs", [[1], [2, 63, 64]])
def test_sh_fields_match_oracle(built, rmin, rdelta, freqs):
    from oracle import driver_setup, oracle as orc
    job = dsmsgt.Job(
        synth.param_file(tlen=1638.4, rmin=rmin, rmax=6300.0, rdelta=rdelta, r0=6271.0, thmin=0.0, thmax=180.0,
                         thdelta=20.0, imin=0, imax=64), synth.dsm_config(), synth.sh_mantle_model(0))
    ctx = dsmsgt.Context(dsmsgt.Setup(job, "sh"))
    got = ctx.run(freqs)
    ctx.close()
    want = orc.run(driver_setup.sh_setup(job), freqs, threads=8)
    assert list(got[-1]) == list(want[-1])
    for a, b in zip(got[:-1], want[:-1]):
        assert np.all(np.isfinite(a)) and rel_l2(a, b) <= 1e-10
