"""The tile autotuner times the kernels of the step's first FCT stage, the fused limiter and
update among them, and leaves the run's state as it is, also where f's slots differ."""
import dataclasses

import pytest

import vxstate
from helpers import golden, problem_for

# kernels of a stage's FCT part: FP64 gamma, two face and two flux passes, f2, limiter R, C and
# update; FP32 x and p fluxes, flux combination, f2, limiter R, C and update
KERNELS = {64: 8, 32: 6}
SHAPES = {64: 7, 32: 5}


@pytest.fixture(scope="module")
def ctx():
    from veritas_gb300 import Context

    c = Context(0)
    yield c
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision,fast,poisson", [(64, 0, 0), (64, 0, 1), (64, 1, 0), (64, 1, 1), (32, 0, 0)])
def test_autotune_times_the_step_and_changes_nothing(ctx, tmp_path, precision, fast, poisson):
    from veritas_gb300 import SolverManager, autotune_many

    st = golden("beam2", 1)
    for levels in st["species"]:
        for rects in levels:
            for r in rects:
                r["f"][..., 1] *= 0.5
    vxstate.write_state(st, tmp_path / "in.bin")
    s = SolverManager(ctx, dataclasses.replace(problem_for("beam2"), precision=precision, fast=fast, poisson=poisson))
    s.load_state(tmp_path / "in.bin")
    s.save_state(tmp_path / "a.bin")
    before = ctx.kernel_launches()
    autotune_many([s])
    launches = ctx.kernel_launches() - before
    s.save_state(tmp_path / "b.bin")
    s.close()
    a, b = vxstate.read_state(tmp_path / "a.bin"), vxstate.read_state(tmp_path / "b.bin")
    for la, lb in zip(a["species"][0], b["species"][0]):
        for ra, rb in zip(la, lb):
            assert (ra["f"][..., :2] == rb["f"][..., :2]).all()
    assert launches == 6 * SHAPES[precision] * KERNELS[precision]  # a warm-up and five timed


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
def test_profile_times_the_update_of_the_step(ctx, precision):
    """The step forms the limiter's C in the update's pass: that pass is timed, and no other."""
    from veritas_gb300 import SolverManager

    s = SolverManager(ctx, dataclasses.replace(problem_for("beam2"), precision=precision))
    s.Advance(s.CalculateDt())
    prof = s.profile_kernels(reps=1)
    s.close()
    assert prof["limC"] == 0.0 and prof["update"] > 0.0
