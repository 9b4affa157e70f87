"""Refinement ratios other than 2 (they are even): the general forms of the restriction, the
interpolation and the moments' sub-columns against the oracle port, from the port's own
initial hierarchy, bit for bit but for what the logarithm moves; the FP32 form against the
FP64 one within its bar.  J, whose contributions carry a logarithm that CUDA and the host library each give
to one ulp, and what it moves in a step: 2^-48."""
import dataclasses

import numpy as np
import pytest

import vxstate
from helpers import gpu_vs_port

CASES = {"r4": dict(r=4, nx=64, np=32, Lfinest=2), "r4_3": dict(r=4, nx=64, np=32, Lfinest=3),
         "r6": dict(r=6, nx=60, np=36, Lfinest=2), "r8": dict(r=8, nx=64, np=32, Lfinest=2)}


@pytest.fixture(scope="module")
def ctx():
    from veritas_gb300 import Context

    c = Context(0)
    yield c
    c.set_pipelined(True)
    c.close()


def _problem(name, **kw):
    from veritas_gb300 import Problem

    return Problem(L=8.0, pmax=2.0, Te=50.0, x1=1.5, x2=2.0, x3=6.0, x4=6.5, pert_amp=0.2, pert_k=2.0, a0=2.0, fwhm=2.0,
                   delay=1.0, **CASES[name], **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("pipelined", [True, False])
@pytest.mark.parametrize("name", list(CASES))
def test_fp64_steps_match_port(ctx, tmp_path, name, pipelined):
    ctx.set_pipelined(pipelined)
    err = gpu_vs_port(ctx, _problem(name), 2, tmp_path)
    assert all(v <= 2.0**-48 for v in err.values()), err


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["r4", "r8"])  # the FP32 form takes up to 8 finest cells per coarse one
def test_fp32_steps_match_fp64(ctx, tmp_path, name):
    from veritas_gb300 import SolverManager

    p = _problem(name)
    a = SolverManager(ctx, p)
    a.save_state(tmp_path / "in.bin")
    b = SolverManager(ctx, dataclasses.replace(p, precision=32))
    b.load_state(tmp_path / "in.bin")
    for _ in range(3):
        dt = a.CalculateDt()
        a.Advance(dt)
        b.Advance(dt)
    out = []
    for k, s in enumerate((a, b)):
        s.save_state(tmp_path / f"{k}.bin")
        out.append(vxstate.read_state(tmp_path / f"{k}.bin"))
        s.close()
    worst = peak = 0.0
    for la, lb in zip(out[0]["species"][0], out[1]["species"][0]):
        for ra, rb in zip(la, lb):
            worst = max(worst, float(np.max(np.abs(ra["f"][..., :2] - rb["f"][..., :2]))))
            peak = max(peak, float(np.max(np.abs(ra["f"][..., 0]))))
    assert worst <= 1e-5 * peak
