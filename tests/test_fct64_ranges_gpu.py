"""The FP64 kernels' short paths against the oracle port, bit for bit, on states whose f
crosses the lines between them: zeros, values about the 1e-14 below which the face weights
are not formed, negative values and -0 (the limiter's general extrema), and values so large
that the quotients take IEEE division."""
import numpy as np
import pytest

import vxstate
from helpers import golden, gpu_vs_port, problem_for


@pytest.fixture(scope="module")
def ctx():
    from veritas_gb300 import Context

    c = Context(0)
    yield c
    c.close()


def _edit(f, how):
    """f: (n_x + 4, n_p + 4, 3) block; edits the interior of slots 0 and 1 alike."""
    g = f[2:-2, 2:-2, 0].copy()
    rng = np.random.default_rng(11)
    if how == "tiny":       # the profile's tail on both sides of 1e-14, zeros in between
        g *= 1e-14 / np.median(g[g > 0])
        g[rng.random(g.shape) < 0.2] = 0.0
    elif how == "signs":    # negative values, -0 and zeros among ordinary ones
        u = rng.random(g.shape)
        g[u < 0.05] *= -1e-3
        g[(u >= 0.05) & (u < 0.1)] = -0.0
        g[(u >= 0.1) & (u < 0.2)] = 0.0
    elif how == "wide":     # neighbours up to 1e70 apart (weights below 1e-250)
        g *= 10.0 ** rng.integers(-70, 1, g.shape)
    elif how == "huge":     # smoothness indicators above 1e95
        g *= 1e4
    f[2:-2, 2:-2, 0] = g
    f[2:-2, 2:-2, 1] = g


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["tiny", "signs", "wide", "huge"])
@pytest.mark.parametrize("name", ["slab64", "ragged2"])
def test_short_paths_match_port(ctx, tmp_path, name, how):
    st = golden(name, 1)
    for levels in st["species"]:
        for rects in levels:
            for r in rects:
                _edit(r["f"], how)
    path = tmp_path / "in.bin"
    vxstate.write_state(st, path)
    err = gpu_vs_port(ctx, problem_for(name), 1, tmp_path, init_state=path)
    assert all(v == 0.0 for v in err.values()), err
