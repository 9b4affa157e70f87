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


def _edit_windows(f, how):
    """f's interior from its own values and a far smaller tail, window by window (29 cells)."""
    g = np.abs(f[2:-2, 2:-2, 0])
    tail, bulk = 1e-45 * g.max(), g.max() * (0.5 + 0.5 * np.random.default_rng(3).random(g.shape))
    n_p = g.shape[1]
    j = np.arange(n_p)[None, :]
    h = np.full(g.shape, tail)
    if how == "gap":         # a window of tail between two bulks
        h = np.where((j < 20) | (j >= n_p - 4), bulk, tail)
    elif how == "cancel":    # the bulk's charge cancels: what lies below and above it decides
        h = np.where(j == n_p // 2, bulk[:, :1], np.where(j == n_p // 2 + 1, -bulk[:, :1], tail))
    elif how == "void":      # nothing at all in half of the columns
        h = np.where(j < n_p // 3, bulk, tail)
        h[::2] = 0.0
    f[2:-2, 2:-2, 0] = h
    f[2:-2, 2:-2, 1] = h


@pytest.mark.gpu
@pytest.mark.parametrize("pipelined", [True, False])
@pytest.mark.parametrize("how", ["tail", "gap", "cancel", "void"])
@pytest.mark.parametrize("name", ["drift128", "ragged2"])
def test_skipped_moment_windows_match_port(ctx, tmp_path, name, how, pipelined):
    """Moment windows that are not formed leave the column sums as they are (and are formed
    after all where they do not): every array against the port, bit for bit; J, whose
    contributions carry a logarithm that CUDA and the host library each give to one ulp, to
    2^-51 (the separate and the fully formed sums differ from the port alike)."""
    st = golden(name, 1)
    for levels in st["species"]:
        for rects in levels:
            for r in rects:
                _edit_windows(r["f"], how)
    path = tmp_path / "in.bin"
    vxstate.write_state(st, path)
    ctx.set_pipelined(pipelined)
    try:
        err = gpu_vs_port(ctx, problem_for(name), 1, tmp_path, init_state=path)
    finally:
        ctx.set_pipelined(True)
    assert err.pop("J") <= 2.0 ** -51
    assert all(v == 0.0 for v in err.values()), err
