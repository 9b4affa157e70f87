"""Contexts on threads of their own launch the same kernels at different sizes at once: what one
sets up for its launch must not undo what another has set up for a larger one."""
import threading

import numpy as np
import pytest

# (Problem of the larger run, of the smaller, the call, the array it fills)
CASES = {
    "exact": (dict(nx=8192, np=32), dict(nx=256, np=32), "poisson", "phi"),
    "scan": (dict(nx=16384, np=32, poisson=1), dict(nx=256, np=32, poisson=1), "poisson", "phi"),
    "screen": (dict(nx=32, np=60000), dict(nx=32, np=20000), "moments", "charge"),
}


@pytest.mark.gpu
@pytest.mark.parametrize("case", list(CASES))
def test_two_contexts_on_two_threads(case):
    from veritas_gb300 import Context, Problem, SolverManager

    big, small, call, name = CASES[case]
    runs, before = [], []
    for kw in (big, small):
        ctx = Context(0)
        s = SolverManager(ctx, Problem(L=100.0, **kw))
        for c in ("moments", call):
            getattr(s, c)()
        ctx.sync()
        runs.append((ctx, s))
        before.append(np.array(s.field(name)))
    errors = []
    start = threading.Barrier(2)

    def work(ctx, s):
        try:
            start.wait()
            for _ in range(40):
                for _ in range(25):
                    getattr(s, call)()
                ctx.sync()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=r) for r in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for (ctx, s), b in zip(runs, before):
        np.testing.assert_array_equal(s.field(name), b)
        s.close()
        ctx.close()
