"""complex64 records where nothing else is asked for (written by the
epilogues) against those formed from the complex128 outputs of the same call
(the packing kernel), bit for bit: both round each value once."""
import ctypes as C

import numpy as np
import pytest

import dsmsgt
from cases import psv_small, sh_small


def _records_only(ctx, setup, freqs, which):
    nt, nr, ns = setup.num
    n = len(freqs)
    shapes = dict(tsgt32=(n, setup.r_n, setup.theta_n, nt), rsgt32=(n, setup.r_n, setup.theta_n, nr),
                  synn32=(n, setup.theta_n, ns))
    rec = {k: np.zeros(shapes[k], np.complex64) for k in which}
    out = dsmsgt.Out()
    for k, a in rec.items():
        setattr(out, k, a.ctypes.data_as(C.POINTER(C.c_float)))
    fl = np.asarray(freqs, np.int32)
    rc = dsmsgt.lib().dsm_run_freqs(ctx.h, fl.ctypes.data_as(C.POINTER(C.c_int)), n, C.byref(out))
    assert rc == 0
    return rec


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [dsmsgt.DSM_PREC_FP64, dsmsgt.DSM_PREC_MIXED])
@pytest.mark.parametrize("mode", ["psv", "sh"])
@pytest.mark.parametrize("which", [("tsgt32", "rsgt32", "synn32"), ("synn32",), ("rsgt32",)])
@pytest.mark.parametrize("thdelta", [15.0, 1.0])
def test_records_alone_equal_packed_records(built, mode, precision, which, thdelta):
    s = dsmsgt.Setup(psv_small(thdelta=thdelta) if mode == "psv" else sh_small(imax=64, thdelta=thdelta), mode)
    freqs = [64, 3, 17, 40, 9]                       # batches of 3 and 2, not in the order of their cutoffs
    ctx = dsmsgt.Context(s, precision=precision, freq_batch=3)
    want = dict(zip(("tsgt32", "rsgt32", "synn32"), ctx.run(freqs, want32=True)[4]))
    got = _records_only(ctx, s, freqs, which)
    ctx.close()
    for k in which:
        assert np.array_equal(got[k], want[k]) and np.any(got[k] != 0)
