"""The FP32 step forms the limiter's coefficients where it uses them and hands the limiter
exchange the ones it needs; the per-class calls form whole planes of them first.  The two
must agree also where a refined patch reaches the lowest momentum (a hierarchy that a state
file brings): the bottom row's faces move nothing themselves, but the coefficient of a
coarse one starts the exchange over r fine faces that do.  f is drawn at random, cell by
cell, so that the limiter acts everywhere.

Both ways round each update to FP32 (eight roundings of sums no larger than the largest f,
6e-8 each, in six stages): 3e-6 of the largest f; a coefficient of the wrong branch moves
cells by 1e-3 of it and more."""
import numpy as np
import pytest

import vxstate

TOL = 3e-6
NX, NP = 64, 32
# boxes (x0, p0, x1, p1) in base cells, finest level first
BOXES = {2: [(20, 0, 44, 12)], 3: [(28, 0, 36, 8), (20, 0, 44, 16)]}


@pytest.fixture(scope="module")
def ctx():
    from veritas_gb300 import Context

    c = Context(0)
    yield c
    c.set_persistent(False)
    c.close()


def _edge_state(st, levels):
    """The state's base level with refined patches that touch p = -pmax."""
    rng = np.random.default_rng(5)
    base = st["species"][0][-1][0]
    assert (base["n_x"], base["n_p"]) == (NX, NP)
    peak = float(base["f"].max())
    coarse = np.zeros((NX + 4, NP + 4))
    coarse[2:-2, 2:-2] = peak * (0.2 + 0.8 * rng.random((NX, NP)))
    base["f"][..., 0] = base["f"][..., 1] = coarse
    new = []
    for depth, (x0, p0, x1, p1) in enumerate(BOXES[levels]):
        k = 2 ** (levels - 1 - depth)
        xs, ps = np.arange(x0 * k - 2, x1 * k + 2), np.arange(p0 * k - 2, p1 * k + 2)
        f = coarse[np.ix_(xs // k + 2, ps // k + 2)] * (0.5 + 0.5 * rng.random((xs.size, ps.size)))
        f[:, ps < 0] = 0.0
        new.append([dict(x_pos=x0 * k, p_pos=p0 * k, n_x=(x1 - x0) * k, n_p=(p1 - p0) * k, depth=depth, up=0, down=1,
                         left=0, right=0, f=np.repeat(f[..., None], 3, axis=2))])
    st["species"][0] = new + [[base]]
    return peak


@pytest.mark.gpu
@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("levels", [2, 3])
def test_step_equals_per_class_calls_at_the_momentum_edge(ctx, tmp_path, levels, persistent):
    from veritas_gb300 import Problem, SolverManager

    p = Problem(L=8.0, nx=NX, np=NP, Lfinest=levels, pmax=1.0, Te=200.0, x1=0.0, x2=1.0, x3=7.0, x4=8.0, a0=1.0, fwhm=2.0,
                delay=1.0, precision=32)
    runs = [SolverManager(ctx, p) for _ in range(2)]
    runs[0].save_state(tmp_path / "in.bin")
    st = vxstate.read_state(tmp_path / "in.bin")
    peak = _edge_state(st, levels)
    vxstate.write_state(st, tmp_path / "in.bin")
    for s in runs:
        s.load_state(tmp_path / "in.bin")
    a, b = runs
    dt = a.CalculateDt()
    ctx.set_persistent(persistent)
    a.Advance(dt)
    ctx.sync()
    ctx.set_persistent(False)
    for stage in range(6):
        b.moments()
        b.poisson()
        b.vlasov_stage(stage, dt)
        b.update_time(stage, dt)
        b.maxwell_stage(stage, dt)
    out = []
    for k, s in enumerate(runs):
        s.save_state(tmp_path / f"{k}.bin")
        out.append(vxstate.read_state(tmp_path / f"{k}.bin"))
        s.close()
    worst = 0.0
    for la, lb in zip(out[0]["species"][0], out[1]["species"][0]):
        for ra, rb in zip(la, lb):
            worst = max(worst, float(np.max(np.abs(ra["f"][..., :2] - rb["f"][..., :2]))))
    assert worst <= TOL * peak, worst / peak
