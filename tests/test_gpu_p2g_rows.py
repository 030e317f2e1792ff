"""P2G by rows at the sizes where it can go wrong: counts around the staging
pass (32) and the row segment (192), more segments than a round holds (16),
one cell, one row and a full block, against the FP64 oracle, and bitwise the
same by single warps and by whole CTAs."""
import numpy as np
import pytest

from conftest import relerr
from mpm_b200 import _abi, scenes
from mpm_b200.solver import APICMPMSolver3D, Material, MPMSolver3D, Particles
from oracle import oracle as O

pytestmark = pytest.mark.gpu

COMBOS = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2)]  # (transfer, interpolation)
RES = 24
# extent of the particles in cells along x, y, z
SHAPES = {"cell": (0.9, 0.9, 0.9), "row": (3.9, 0.9, 0.9), "blocks": (6.0, 6.0, 6.0)}
# A node's mass is a sum of terms of one sign: at most 192 / 2 of a segment in
# turn, the groups (8), the segments of an item (38) and the tiles (8), each
# rounding within 2^-24 of the running sum.
MASS_TOL = (96 + 8 + 38 + 8) * 2.0 ** -24


def _particles(n, shape, seed):
    rng = np.random.default_rng(seed)
    h = 1.0 / RES
    lo = np.array([8.05, 8.05, 8.05]) * h
    x = (lo + np.asarray(SHAPES[shape]) * h * rng.random((n, 3))).astype(np.float32)
    v = rng.normal(size=(n, 3)).astype(np.float32)
    Fe = (np.eye(3)[None] + 0.01 * rng.normal(size=(n, 3, 3))).astype(np.float32).reshape(n, 9)
    B = (5.0 * h * h * rng.normal(size=(n, 3, 3))).astype(np.float32).reshape(n, 9)
    return Particles(x, v, 0.01, [Material(**scenes.SNOW)]), Fe, B


def _solver(p, transfer, interp):
    args = (p, (0, 0, 0), (RES,) * 3, 1.0 / RES, 0.9)
    return (APICMPMSolver3D(*args, interp, 1e-4) if transfer else MPMSolver3D(*args, 0.95, interp, 1e-4))


@pytest.mark.parametrize("n,shape", [(1, "cell"), (31, "cell"), (33, "row"), (192, "cell"), (193, "row"),
                                     (4095, "row"), (4097, "cell"), (9000, "row"), (5000, "blocks")])
@pytest.mark.parametrize("transfer,interp", COMBOS)
def test_grid_matches_oracle(gpu, transfer, interp, n, shape):
    p, Fe, B = _particles(n, shape, n)
    g = _solver(p, transfer, interp)
    o = O.OracleSolver(g._desc, p, bits=64)
    for field, val in [(_abi.FIELD_FE, Fe)] + ([(_abi.FIELD_B, B)] if transfer else []):
        g.upload(field, val)
        o.set(field, val.astype(np.float64))
    g.resetGrid()
    g.particlesToGrid()
    o.reset_grid()
    o.particles_to_grid()
    assert relerr(g.download_grid(_abi.GRID_MASS), o.grid(_abi.GRID_MASS)) < MASS_TOL
    # momentum terms of both signs: the bound of their absolute sum, |v| up to ~4 of an rms sum sqrt(n) smaller
    tol = 4.0 * MASS_TOL * max(1.0, np.sqrt(n))
    assert relerr(g.download_grid(_abi.GRID_VELOCITY), o.grid(_abi.GRID_VELOCITY)) < tol
    # the FP32 stress, see test_gpu_parity.py, in sums of both signs
    assert relerr(g.download_grid(_abi.GRID_FORCE), o.grid(_abi.GRID_FORCE)) < 1e-4 + tol


@pytest.mark.parametrize("n,shape", [(1, "cell"), (33, "row"), (193, "row"), (4095, "row"), (5000, "blocks")])
@pytest.mark.parametrize("transfer,interp", COMBOS)
def test_warps_stages_and_ctas_agree_bitwise(gpu, transfer, interp, n, shape):
    p, Fe, B = _particles(n, shape, n)
    first = None
    for stage, warps in ((32, 0), (32, 4096), (16, 0), (24, 100)):
        g = _solver(p, transfer, interp)
        g.set_tuning(1024, stage, warps)
        g.upload(_abi.FIELD_FE, Fe)
        if transfer:
            g.upload(_abi.FIELD_B, B)
        g.step(3)
        got = [g.download(f) for f in (_abi.FIELD_POSITION, _abi.FIELD_VELOCITY, _abi.FIELD_FE)]
        first = first or got
        for a, b in zip(got, first):
            assert np.array_equal(a, b), (stage, warps)
