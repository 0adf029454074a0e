"""Split of field rows for the tensor-core sums at the edges of its vectors
(four orders), the groups of 128 orders a warp keeps in registers and its
re-reading beyond them: order ranges from a few to more than 2048, FP32 rows
(P-SV) and FP64 rows (SH), one parity and two.  Against the FP64 sums of the
same fields; bar 5e-6 relative L2 per array: contraction outputs rounded to
FP32 (6e-8 each, tens in a record with cancellation), fields rounded to FP32
(P-SV) and pieces of 22 bits."""
import numpy as np
import pytest

import dsmsgt
from conftest import rel_l2
from dsmsgt import synth


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["psv", "sh"])
@pytest.mark.parametrize("thdelta", [1.0, 1.7])     # mirrored at 90 degrees, and not
@pytest.mark.parametrize("freq,r0", [(1, 5700.0), (40, 6071.0), (129, 6071.0), (60, 6361.0)])
def test_split_rows_of_all_lengths(built, mode, thdelta, freq, r0):
    sh = mode == "sh"
    job = dsmsgt.Job(
        synth.param_file(tlen=1638.4, rmin=3500.0, rmax=6300.0, rdelta=700.0, r0=r0, thmin=0.0, thmax=180.0,
                         thdelta=thdelta, imin=0, imax=130), synth.dsm_config(),
        synth.sh_mantle_model(0) if sh else synth.psv_earth_model(0))
    s = dsmsgt.Setup(job, mode)
    outs = []
    for precision in (dsmsgt.DSM_PREC_FP64, dsmsgt.DSM_PREC_MIXED):
        ctx = dsmsgt.Context(s, precision=precision)
        outs.append(ctx.run([freq, freq + 1]))
        ctx.close()
    want, got = outs
    assert list(got[-1]) == list(want[-1])
    for a, b in zip(got[:-1], want[:-1]):
        assert np.all(np.isfinite(a)) and rel_l2(a, b) <= 5e-6
