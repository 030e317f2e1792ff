"""Crowded blocks as several P2G items: block counts around the lines of small
(1280 and 640) and large scenes (2560 and 1280) and scenes on both sides of
65,536 particles, against the FP64 oracle, and the same bits in a batch as
alone."""
import numpy as np
import pytest

from conftest import relerr
from mpm_b200 import _abi, scenes
from mpm_b200.batch import Batch
from mpm_b200.scenes import Scene
from mpm_b200.solver import Material, Particles
from oracle import oracle as O

pytestmark = pytest.mark.gpu

RES = 24
# Terms of one sign: 192 / 2 of a segment in turn, its groups (8), an item's
# segments (2560 / 192 + 16), a block's items (65,537 / 1280) and the tiles (8).
MASS_TOL = (96 + 8 + 30 + 52 + 8) * 2.0 ** -24


def _scene(n, extent, transfer, seed=0):
    rng = np.random.default_rng(seed or n)
    x = ((8.05 + extent * rng.random((n, 3))) / RES).astype(np.float32)
    p = Particles(x, rng.normal(size=(n, 3)).astype(np.float32), 0.01, [Material(**scenes.SNOW)])
    return Scene("split", p, (0.0, 0.0, 0.0), (RES,) * 3, 1.0 / RES, 1e-5, transfer, _abi.INTERP_QUADRATIC)


@pytest.mark.parametrize("n", [640, 1280, 1281, 2560, 2561, 65_536, 65_537])
@pytest.mark.parametrize("transfer", [0, 1])
def test_grid_matches_oracle(gpu, transfer, n):
    sc = _scene(n, 3.9, transfer)
    g, o = sc.solver(), O.OracleSolver(sc.desc(), sc.particles, bits=64)
    g.resetGrid()
    g.particlesToGrid()
    o.reset_grid()
    o.particles_to_grid()
    assert relerr(g.download_grid(_abi.GRID_MASS), o.grid(_abi.GRID_MASS)) < MASS_TOL
    # momentum terms of both signs, as in test_gpu_p2g_rows.py
    assert relerr(g.download_grid(_abi.GRID_VELOCITY), o.grid(_abi.GRID_VELOCITY)) < 4.0 * MASS_TOL * np.sqrt(n)


def test_batch_equals_solo_on_both_sides_of_the_line(gpu):
    scs = [_scene(n, e, k % 2, seed=k + 1) for k, (n, e) in enumerate([(65_536, 7.0), (65_537, 7.0), (9_000, 1.5), (70_000, 3.0)])]
    with Batch() as b:
        ids = [b.add(s) for s in scs]
        b.step(8)
        got = [[b.download(i, f) for f in (_abi.FIELD_POSITION, _abi.FIELD_VELOCITY)] for i in ids]
    for s, want in zip(scs, got):
        g = s.solver()
        g.step(8)
        for f, w in zip((_abi.FIELD_POSITION, _abi.FIELD_VELOCITY), want):
            assert np.array_equal(g.download(f), w)
        g.close()
