"""Models whose densities, and so all stiffnesses, are scaled by a power of
ten: the band's pivots then exceed 1e154 or fall below 1e-154, where |D|^2 leaves
FP64's range but 1/D does not.  Against the oracle, which divides by Smith's
rule; bar 1e-10 relative L2 per array, the repository's bar of FP64 parity."""
import re

import numpy as np
import pytest

import dsmsgt
from cases import psv_small, sh_small
from conftest import rel_l2


def _scaled(job, k):
    def line(text):
        if not re.match(r"\s*\d+\.\d{3}\s+\d+\.\d{3}$", text[:20]) or len(text) < 90:
            return text
        rho = [re.sub(r"e([+-]\d+)", lambda m: f"e{int(m.group(1)) + k:+04d}", text[20 + 19 * i:39 + 19 * i])
               for i in range(4)]
        return text[:20] + "".join(f" {c.strip()}" for c in rho)
    return dsmsgt.Job(job.param_text, job.conf_text, "\n".join(line(t) for t in job.model_text.split("\n")))


@pytest.mark.gpu
@pytest.mark.parametrize("mode,k", [("sh", 158), ("sh", -166), ("psv", 146), ("psv", 150)])
def test_scaled_model_matches_oracle(built, mode, k):
    from oracle import driver_setup, oracle as orc
    job = _scaled(sh_small() if mode == "sh" else psv_small(rdelta=900.0), k)
    freqs = [3, 11]
    ctx = dsmsgt.Context(dsmsgt.Setup(job, mode))
    got = ctx.run(freqs)
    ctx.close()
    want = orc.run(driver_setup.setup(job, mode), freqs, threads=8)
    assert list(got[3]) == list(want[3])
    for a, b in zip(got[:3], want[:3]):
        top = np.max(np.abs(b))
        assert np.all(np.isfinite(a)) and top > 0.0
        assert rel_l2(a / top, b / top) <= 1e-10
