"""a^2 on the faces from A (EMSolver.cpp:555-619) after field-only steps, bit for bit
against the same expression in numpy: over the range where its quotients take the short
form with the rounding of `/`, and beyond it (A of 1e45 and more, infinities).
"""
import numpy as np
import pytest

import vxstate
from helpers import golden, problem_for


@pytest.fixture(scope="module")
def ctx():
    from veritas_gb300 import Context

    c = Context(0)
    yield c
    c.close()


def _face(f1, f2, f3, f4):
    c6, c43, mm = 1.0 / 6, 4.0 / 3, 1.0e-10
    fL = c6 * (-f1 + 5 * f2 + 2 * f3)
    fR = c6 * (2 * f2 + 5 * f3 - f4)
    AL, BL = f1 - 2 * f2 + f3, f3 - f1
    AR, BR = f2 - 2 * f3 + f4, f4 - f2
    bL = c43 * (AL * AL) + 0.5 * AL * BL + 0.25 * (BL * BL)
    bR = c43 * (AR * AR) - 0.5 * AR * BR + 0.25 * (BR * BR)
    oL, oR = 0.5 / ((mm + bL) * (mm + bL)), 0.5 / ((mm + bR) * (mm + bR))
    return (oL / (oL + oR)) * fL + (oR / (oL + oR)) * fR


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0.0, 1e-30, 1.0, 1e20, 1e44, 1e46, 1e77, 1e160])
def test_face_a_squared_matches_expression(ctx, tmp_path, scale):
    from veritas_gb300 import SolverManager

    st = golden("slab64", 0)
    rng = np.random.default_rng(5)
    for k in ("Ay", "Az"):
        st[k] = np.array(st[k])
        st[k][:] = scale * rng.standard_normal(st[k].shape)
    vxstate.write_state(st, tmp_path / "in.bin")
    s = SolverManager(ctx, problem_for("slab64"))
    s.load_state(tmp_path / "in.bin")
    s.AdvanceFields(1e-18)
    s.save_state(tmp_path / "out.bin")
    s.close()
    got = vxstate.read_state(tmp_path / "out.bin")
    n, pre = got["n"], got["pre"]
    with np.errstate(all="ignore"):
        a = [_face(*(np.asarray(got[k])[pre + np.arange(n) + d] for d in (-2, -1, 0, 1))) for k in ("Ay", "Az")]
        want = a[0] * a[0] + a[1] * a[1]
    np.testing.assert_array_equal(np.asarray(got["a_squared"])[:n], want)
