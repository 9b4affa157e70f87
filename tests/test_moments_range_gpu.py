"""Column sums where g + c1 p cancels: from about gamma = 1e8 on it is 0 at negative momenta,
its logarithm infinite and J, 0 x infinity in empty cells, not a number.  The windows that
hold those cells must not be left out for being empty.  Below, J is finite.  Against the
sums in numpy (separate and pipelined launch)."""
import numpy as np
import pytest

import vxstate

ME, QE, C, C_INV = 9.10938291e-31, 1.60217657e-19, 299792458.0, 3.33564095e-9
NX, NP = 40, 120


@pytest.fixture(scope="module")
def ctx():
    from veritas_gb300 import Context

    c = Context(0)
    yield c
    c.set_pipelined(True)
    c.close()


def _current(f, pmax):
    """J of the interior columns of f (NX + 4, NP + 4) without fields."""
    dp, c1 = 2 * pmax * ME * C / NP, C_INV / ME
    p = -pmax * ME * C + dp * np.arange(-1, NP + 2)
    G = np.sqrt(1 + p * p * c1 * c1) + c1 * p
    with np.errstate(divide="ignore", invalid="ignore"):
        L = np.log(G[1:] / G[:-1]) / c1  # cells -1 .. NP
        v = f[2:-2, 1:-1]
        cj = v[:, 1:-1] * L[1:-1] + (L[2:] - L[:-2]) * (v[:, 2:] - v[:, :-2]) / 48
        return cj.sum(axis=1) * (-QE * QE / ME)


@pytest.mark.gpu
@pytest.mark.parametrize("pmax", [2.0, 1e4, 1e6, 3e8])
def test_current_over_the_momentum_range(ctx, tmp_path, pmax):
    from veritas_gb300 import Problem, SolverManager

    s = SolverManager(ctx, Problem(L=5.0, nx=NX, np=NP, pmax=pmax))
    s.save_state(tmp_path / "in.bin")
    st = vxstate.read_state(tmp_path / "in.bin")
    f = np.zeros((NX + 4, NP + 4))
    f[2:-2, 2 + 80:2 + 84] = 1e46 * (1 + np.random.default_rng(1).random((NX, 4)))  # in one window of 29 cells
    st["species"][0][0][0]["f"] = np.repeat(f[..., None], 3, axis=2)
    vxstate.write_state(st, tmp_path / "in.bin")
    s.load_state(tmp_path / "in.bin")
    s.moments()
    s.save_state(tmp_path / "out.bin")
    J = np.array(vxstate.read_state(tmp_path / "out.bin")["J"][:NX])
    want = _current(f, pmax)
    assert np.isnan(want).all() == (pmax > 1e8)
    np.testing.assert_array_equal(np.isfinite(J), np.isfinite(want))
    if pmax < 1e8:
        # dp in units of p differs from the framework's by the roundings of its constants
        assert np.max(np.abs(J - want)) <= 1e-9 * np.max(np.abs(want))
        s.close()
        return
    # the pipelined launch forms them too: the step's J makes the fields not a number
    s.Advance(1e-18)
    s.save_state(tmp_path / "out.bin")
    assert np.isnan(vxstate.read_state(tmp_path / "out.bin")["J"][:NX]).all()
    s.close()
