"""The scan solve of sets whose runs differ in size: the scan's threads follow the largest run,
so that most blocks of a small run's cluster hold no cells; and the sizes about which the
assembly moves into the solve.  phi, E_x and Ex0 against the same run alone (other carries)
and against the exact solve, within 4 n^2 2^-52 of their scale: the discrete system's
conditioning is about n^2, and either side errs by two units of it."""
import numpy as np
import pytest

FIELDS = ("phi", "Ex", "charge")


@pytest.fixture(scope="module")
def ctx():
    from veritas_gb300 import Context

    c = Context(0)
    yield c
    c.close()


def _problem(nx, poisson=1, levels=1):
    from veritas_gb300 import Problem

    L = min(100.0, nx / 8.0)
    return Problem(L=L, nx=nx, np=40, Lfinest=levels, poisson=poisson, x1=0.15 * L, x2=0.20 * L, x3=0.80 * L, x4=0.85 * L,
                   Te=40.0, p0=0.1, pert_amp=0.2, pert_k=2.0)


def _compare(a, b, n):
    for name in FIELDS:
        x, y = a[name], b[name]
        assert np.isfinite(x).all()
        assert np.max(np.abs(x - y)) <= 4 * n * n * 2.0**-52 * np.max(np.abs(y)), (name, n)


@pytest.mark.gpu
def test_sets_of_mixed_sizes(ctx):
    from veritas_gb300 import SolverManager, advance_many

    probs = [_problem(nx, levels=lv) for nx, lv in ((32, 1), (34, 2), (76, 1), (322, 1), (1026, 2), (4096, 1), (4098, 1))]
    for last in (6, 7):  # largest run 4096, then 4098
        alone, together = [], []
        for p in probs[:last]:
            s = SolverManager(ctx, p)
            s.Advance(1e-17)
            alone.append({k: s.field(k) for k in FIELDS})
            s.close()
        sms = [SolverManager(ctx, p) for p in probs[:last]]
        advance_many(sms, [1e-17] * last)
        together = [{k: s.field(k) for k in FIELDS} for s in sms]
        for s in sms:
            s.close()
        for p, a, b in zip(probs, together, alone):
            _compare(a, b, p.nx * 2 ** (p.Lfinest - 1))


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [2048, 4096, 4098])
def test_scan_fields_match_exact_solve(ctx, nx):
    from veritas_gb300 import SolverManager

    out = []
    for poisson in (1, 0):
        s = SolverManager(ctx, _problem(nx, poisson))
        s.Advance(1e-17)
        out.append({k: s.field(k) for k in FIELDS})
        s.close()
    _compare(*out, nx)
