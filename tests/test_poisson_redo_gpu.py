"""The exact solve's backward sweep checks each chunk of rows against IEEE division while
the next one is swept, and redoes chunks that fail.  The quotients' short form holds down
to solutions of 1e-21, so a right-hand side scaled by 2^-100 has every chunk redone; the
system is linear and a power of two exact, so the solution has to be 2^-100 times the one
of the unscaled right-hand side, bit for bit.  Sizes: one chunk of 256 rows before the last
eight, exactly one, two rows more, several.
"""
import numpy as np
import pytest

import vxstate


@pytest.fixture(scope="module")
def ctx():
    from veritas_gb300 import Context

    c = Context(0)
    yield c
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [40, 264, 266, 600, 1100])
def test_redone_chunks_give_the_same_solution(ctx, tmp_path, nx):
    from veritas_gb300 import Problem, SolverManager

    s = SolverManager(ctx, Problem(L=min(100.0, nx / 8.0), nx=nx, np=32))
    s.save_state(tmp_path / "in.bin")
    st = vxstate.read_state(tmp_path / "in.bin")
    n = st["n"]
    rng = np.random.default_rng(nx)
    rhs = np.sin(np.arange(n) * 0.1) + 0.1 * rng.standard_normal(n)
    rhs -= rhs.mean()
    phi = []
    for scale in (1.0, 2.0**-100):
        for k, v in (("charge", 0.0 * rhs), ("neut", scale * rhs)):
            st[k] = np.array(st[k])
            st[k][:n] = v
        vxstate.write_state(st, tmp_path / "in.bin")
        s.load_state(tmp_path / "in.bin")
        s.poisson()
        s.save_state(tmp_path / "out.bin")
        phi.append(np.array(vxstate.read_state(tmp_path / "out.bin")["phi"][:n]))
    s.close()
    assert np.max(np.abs(phi[0])) > 0
    assert np.max(np.abs(phi[1])) < 1e-21
    np.testing.assert_array_equal(phi[1] * 2.0**100, phi[0])
