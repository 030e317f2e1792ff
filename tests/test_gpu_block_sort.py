"""The block sort (blocks put together from the particles that stayed in them
and the arrivals from their neighbours) gives exactly the stable sort of all
keys, so a run with it is bitwise the run that sorts all keys every step
(MPM_FULL_SORT=1): slow and fast particles (no, few and many movers past the
neighbouring blocks), crowded blocks, more arrivals than shared memory holds,
particles that leave the grid, and several scenes."""
import os

import numpy as np
import pytest

from mpm_b200 import _abi
from mpm_b200.batch import Batch
from mpm_b200.scenes import Scene
from mpm_b200.solver import Material, Particles

pytestmark = pytest.mark.gpu

FIELDS = (_abi.FIELD_POSITION, _abi.FIELD_VELOCITY, _abi.FIELD_FE)
RES, DT = 32, 1e-3
CELL = 1.0 / (RES * DT)  # a cell per step


def _scene(n, extent, cells_per_step, spread=0.0, seed=1, at=(12.1, 12.1, 12.1)):
    """n stress-free particles in `extent` cells from cell `at`, all moving by
    cells_per_step along x + y (and by up to `spread` cells more each)."""
    rng = np.random.default_rng(seed)
    x = ((np.asarray(at) + extent * rng.random((n, 3))) / RES).astype(np.float32)
    v = np.array([1.0, 0.7, 0.1]) * cells_per_step * CELL + spread * CELL * rng.uniform(-1, 1, (n, 3))
    p = Particles(x, v.astype(np.float32), 0.01, [Material(youngs_modulus=0.0)])
    return Scene("moving", p, (0.0, 0.0, 0.0), (RES,) * 3, 1.0 / RES, DT, _abi.TRANSFER_PIC_FLIP,
                 _abi.INTERP_LINEAR, blend=1.0, gravity=0.0, sticky_cells=0)


def _states(make, steps, full_sort):
    if full_sort:
        os.environ["MPM_FULL_SORT"] = "1"
    try:
        eng = make()  # the engine reads the switch when it is created
    finally:
        os.environ.pop("MPM_FULL_SORT", None)
    out = []
    for _ in range(steps):
        eng.step(1)
        out.append([eng.download(f) for f in FIELDS])
    eng.close()
    return out


@pytest.mark.parametrize("n,extent,cells,spread", [
    (1, 1.0, 0.3, 0.0), (500, 6.0, 0.05, 0.02), (20_000, 7.0, 0.1, 0.05),  # steady movement
    (3_000, 6.0, 1.5, 1.0), (20_000, 6.0, 3.0, 2.0),                        # most particles change block
    (2_000, 3.0, 9.0, 0.0), (20_000, 6.0, 9.0, 3.0),                        # past the neighbours, and out of the grid
    (12_000, 0.8, 0.35, 0.0), (30_000, 2.5, 0.2, 0.1),                      # crowded blocks that cross together
])
def test_block_sort_equals_full_sort(gpu, n, extent, cells, spread):
    make = _scene(n, extent, cells, spread).solver
    a, b = _states(make, 12, False), _states(make, 12, True)
    for k, (sa, sb) in enumerate(zip(a, b)):
        for x, y in zip(sa, sb):
            assert np.array_equal(x, y), k


def test_block_sort_equals_full_sort_in_a_batch(gpu):
    scs = [_scene(5_000, 6.0, 0.4, 0.3, seed=2), _scene(9_000, 1.5, 0.5, 0.0, seed=3), _scene(700, 4.0, 6.0, 2.0, seed=4)]

    def run(full_sort):
        if full_sort:
            os.environ["MPM_FULL_SORT"] = "1"
        try:
            bt = Batch()
        finally:
            os.environ.pop("MPM_FULL_SORT", None)
        ids = [bt.add(s) for s in scs]
        bt.step(10)
        out = [bt.download(i, f) for i in ids for f in FIELDS]
        bt.close()
        return out

    for x, y in zip(run(False), run(True)):
        assert np.array_equal(x, y)
