"""The scatter of the semi-implicit solve (P2G by rows on the stress
differential) and its gather at the sizes where they can go wrong: counts
around the staging pass (32) and the row segment (192), blocks of two and more
work items (chunk 2560): the FP64 oracle's residual of the solution."""
import numpy as np
import pytest

from mpm_b200 import _abi, scenes
from mpm_b200.solver import APICMPMSolver3D, Material, MPMSolver3D, Particles
from oracle import oracle as O

pytestmark = pytest.mark.gpu

RES = 24
SHAPES = {"cell": (0.9, 0.9, 0.9), "row": (3.9, 0.9, 0.9), "blocks": (6.0, 6.0, 6.0)}
# As in test_gpu_p2g_rows.py: sums of an item's segments, groups and tiles.
SUM_TOL = (96 + 8 + 38 + 8) * 2.0 ** -24


@pytest.mark.parametrize("n,shape", [(1, "cell"), (33, "row"), (193, "cell"), (2561, "cell"), (5200, "row"),
                                     (6000, "blocks")])
@pytest.mark.parametrize("transfer,interp", [(0, 0), (0, 1), (1, 1), (1, 2)])
def test_solve_matches_oracle(gpu, transfer, interp, n, shape):
    rng = np.random.default_rng(n)
    h = 1.0 / RES
    x = (8.05 * h + np.asarray(SHAPES[shape]) * h * rng.random((n, 3))).astype(np.float32)
    v = rng.normal(size=(n, 3)).astype(np.float32)
    mass = float(400.0 * np.prod(SHAPES[shape]) * h ** 3 / n)  # 400 kg/m^3 however crowded
    p = Particles(x, v, mass, [Material(**scenes.SNOW)])
    args = (p, (0, 0, 0), (RES,) * 3, h, 0.9)
    g = APICMPMSolver3D(*args, interp, 1e-4) if transfer else MPMSolver3D(*args, 0.95, interp, 1e-4)
    o = O.OracleSolver(g._desc, p, bits=64)
    Fe = (np.eye(3)[None] + 0.01 * rng.normal(size=(n, 3, 3))).astype(np.float32).reshape(n, 9)
    g.upload(_abi.FIELD_FE, Fe)
    o.set(_abi.FIELD_FE, Fe.astype(np.float64))
    dt, tol = 1e-3, 1e-6
    g.set_implicit(1.0, max_iter=200, tol=tol)
    g.resetGrid()
    g.particlesToGrid()
    g.updateGridVelocities(dt)
    g.gridCollision(dt)
    vs = g.download_grid(_abi.GRID_VELOCITY_STAR).reshape(-1, 3).astype(np.float64)
    m = g.download_grid(_abi.GRID_MASS).reshape(-1, 1).astype(np.float64)
    g.solveLinearSystem(dt)
    it, res = g.solve_info()
    assert it < 200 and res <= tol, (it, res)
    act = m > np.finfo(np.float32).eps  # the unknowns
    x = np.where(act, g.download_grid(_abi.GRID_VELOCITY_STAR).reshape(-1, 3), 0.0)
    o.reset_grid()
    o.particles_to_grid()
    hx = np.where(act, dt * dt * o.hessian_action(x), 0.0)
    b = np.where(act, m * vs, 0.0)
    # FP64 residual of the GPU's x for its own v*: the stop tolerance, plus the
    # FP32 stress differential (1e-5) and sums in terms of both signs of c H x.
    bound = tol + (1e-5 + 4.0 * SUM_TOL * max(1.0, np.sqrt(n))) * np.linalg.norm(hx) / np.linalg.norm(b)
    assert np.linalg.norm(np.where(act, m * x, 0.0) + hx - b) / np.linalg.norm(b) < bound
