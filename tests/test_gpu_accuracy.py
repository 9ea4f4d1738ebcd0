"""Rounding error of the FP64 step.  The oracle's source compiled a second time
with long double in place of double (64-bit mantissas, its literals and the
inputs in double) gives a step without rounding error to speak of; against it
the GPU step may be no further off than the same formulas in double."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

import gks_ic
from conftest import ORACLE

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def exact(tmp_path_factory):
    """exact(W, params, dt): one step of the long double build, interior cells."""
    tmp = tmp_path_factory.mktemp("exact")
    src, lib = str(tmp / "wide.c"), str(tmp / "libwide.so")
    with open(src, "w") as f:
        f.write("#include <tgmath.h>\n#include <stdlib.h>\n#include <string.h>\n#define double long double\n")
        f.write('#include "%s"\n' % os.path.join(ORACLE, "gks_oracle.c"))
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-std=gnu11", "-o", lib, src, "-lm"], check=True)
    step = ctypes.CDLL(lib).orc_step

    def run(W, prm, dt):
        fields = [(n, ctypes.c_int if t is ctypes.c_int else ctypes.c_longdouble) for n, t in prm._fields_]
        wide = type("WideParams", (ctypes.Structure,), {"_fields_": fields})()
        for n, _ in fields:
            setattr(wide, n, getattr(prm, n))
        X = W.astype(np.longdouble)
        F = np.zeros((15,) + W.shape[1:], np.longdouble)
        step(ctypes.c_void_p(X.ctypes.data), ctypes.byref(wide), ctypes.c_longdouble(dt), ctypes.c_void_p(F.ctypes.data))
        return X[:, 3:-3, 3:-3, 3:-3]

    return run


@pytest.mark.parametrize("nc,mach,flags,power", [(16, 0.45, 0, False), (24, 0.2, 0, True), (31, 0.3, 0, False),
                                                 (32, 0.2, 3, False), (33, 0.55, 2, True)])
def test_fp64_step_rounds_no_worse_than_the_formulas_in_double(gks, oracle, exact, nc, mach, flags, power):
    case = gks_ic.make_dhit(nc, k0=3.0, Mt=mach, seed=nc)
    W = gks_ic.to_conservative_padded(case)
    pr = gks.PR_FACTOR_GPU if flags & gks.DIRECT_ENERGY else gks.PR_FACTOR_CPU
    law = gks.VISC_POWER if power else gks.VISC_SUTHERLAND
    with gks.Solver(gks.phys_from_case(case, visc_law=law, pr_factor=pr), gks.FP64, flags) as s:
        s.upload(W)
        dt = s.timestep(0.5)
        s.step(1)
        s.sync()
        got = s.download()[:, 3:-3, 3:-3, 3:-3]
    prm = oracle.params(nc, case.gam, case.mu0, case.p0, 1.0, case.Mt, case.t0, visc_law=law, pr_factor=pr, flags=flags)
    want = exact(W, prm, dt)
    plain = oracle.step(W.copy(), prm, dt, 1)[:, 3:-3, 3:-3, 3:-3]

    def rms(A):
        return np.sqrt(((A - want).astype(np.float64).reshape(5, -1) ** 2).mean(1))

    assert np.all(rms(got) <= rms(plain)), rms(got) / rms(plain)
