"""Writes far_half.npz: outputs beyond 90 degrees of small seeded models in
80-bit arithmetic (rounded to FP64), and how far the FP64 oracle is from them.

The 80-bit values come from the oracle's own sources with ``double`` replaced
by ``long double`` (set-up arrays and outputs stay FP64), compiled here into a
scratch folder.  Run from the repository root: python tests/golden/make_far_half.py
"""
import ctypes as C
import os
import re
import subprocess
import sys
import tempfile

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
for p in (ROOT, os.path.dirname(HERE), os.path.join(ROOT, "dsm-kernel_b200")):
    sys.path.insert(0, p)

import dsmsgt  # noqa: E402
from dsmsgt import synth  # noqa: E402
from oracle import driver_setup, oracle as orc  # noqa: E402


def _widen(text):
    head, brace, api = text.partition('extern "C"')
    head = re.sub(r"(?<!const )\bdouble\b", "real", head)          # internal values and work arrays
    head = re.sub(r"\bconst double\b(?!\*)", "const real", head)
    api = api.replace("double tt", "oracle::real tt").replace("&lg, probe, n)", "&lg)")
    text = head + brace + api
    text = re.sub(r"(?<![\w.])(\d+\.\d*(?:e[-+]?\d+)?)(?![\w.])", r"\1L", text)
    text = re.sub(r"std::memcpy\((\w+) \+ 2 \* (\w+) \* k, (\w+)\.data\(\), sizeof\(cplx\) \* \2\);",
                  r"for (long q = 0; q < \2; ++q) { \1[2 * (\2 * k + q)] = (double)\3[q].re; "
                  r"\1[2 * (\2 * k + q) + 1] = (double)\3[q].im; }", text)
    return text


def _library(tmp):
    src = os.path.join(ROOT, "oracle")
    for name in ("oracle_common.hpp", "oracle_sh.cpp", "oracle_psv.cpp"):
        text = _widen(open(os.path.join(src, name)).read())
        if name.endswith(".hpp"):
            text = text.replace("namespace oracle {", "namespace oracle {\ntypedef long double real;", 1)
        open(os.path.join(tmp, name), "w").write(text)
    out = os.path.join(tmp, "liboracle80.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-fPIC", "-std=c++17", "-I" + os.path.join(ROOT, "include"),
                    "-shared", "-o", out, os.path.join(tmp, "oracle_sh.cpp"), os.path.join(tmp, "oracle_psv.cpp")],
                   check=True)
    return C.CDLL(out)


def cases(mode):
    """(name, job, frequencies) of seeded models: sources 20 to 670 km deep,
    receivers from the inner core (every other P-SV model) or the lower mantle up."""
    rng = np.random.default_rng(11)
    for k in range(24):
        r0, rd = round(float(rng.uniform(5700.0, 6350.0)), 1), round(float(rng.uniform(500.0, 900.0)), 1)
        deep, shallow = float(rng.uniform(900.0, 3400.0)), float(rng.uniform(3600.0, 4200.0))
        freq = int(rng.integers(1, 65))
        model = (synth.psv_earth_model if mode == "psv" else synth.sh_mantle_model)(100 + k)
        rmin = round(deep if mode == "psv" and k % 2 == 0 else shallow, 1)
        text = synth.param_file(tlen=1638.4, rmin=rmin, rmax=6340.0, rdelta=rd, r0=r0, thmin=95.0, thmax=179.0,
                                thdelta=28.0, imin=0, imax=64)
        yield f"{mode}{k}", dsmsgt.Job(text, synth.dsm_config(), model), [freq]


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def main():
    out = {}
    with tempfile.TemporaryDirectory() as tmp:
        lib = _library(tmp)
        for mode in ("psv", "sh"):
            for name, job, freqs in cases(mode):
                s = driver_setup.setup(job, mode)
                fl = np.array(freqs, np.int32)
                exact = dsmsgt.alloc_outputs(s, len(freqs))
                getattr(lib, f"oracle_{mode}_run")(
                    C.cast(s.ptr, C.c_void_p), fl.ctypes.data_as(C.POINTER(C.c_int)), len(freqs),
                    *(C.c_void_p(x.ctypes.data) for x in exact[:3]), exact[3].ctypes.data_as(C.POINTER(C.c_int)))
                fp64 = orc.run(s, freqs)
                assert list(fp64[3]) == list(exact[3])
                for k, a in zip("try", exact):
                    out[f"{name}_{k}"] = a
                out[f"{name}_err"] = np.array([rel(b, a) for a, b in zip(exact[:3], fp64[:3])])
                print(name, freqs, list(exact[3]), out[f"{name}_err"], flush=True)
    np.savez_compressed(os.path.join(HERE, "far_half.npz"), **out)


if __name__ == "__main__":
    main()
