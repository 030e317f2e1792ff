"""The step's sort goes block by block or, where many particles leave their
blocks, by radix passes in the same launch.  Either way it is the stable sort of
all keys (bitwise the run with MPM_FULL_SORT=1), and no movement makes it much
slower than that sort."""
import os
import time

import numpy as np
import pytest

from mpm_b200 import _abi
from mpm_b200.batch import Batch
from mpm_b200.scenes import Scene
from mpm_b200.solver import Material, Particles

pytestmark = pytest.mark.gpu

FIELDS = (_abi.FIELD_POSITION, _abi.FIELD_VELOCITY)
DT = 1e-3


def _scene(n, extent, cells_per_step, res=64, at=12.1, seed=1):
    """n stress-free particles in a cube of `extent` cells from cell `at`, all
    moving by cells_per_step along x and less along y and z."""
    rng = np.random.default_rng(seed)
    x = ((at + extent * rng.random((n, 3))) / res).astype(np.float32)
    v = np.tile(np.array([1.0, 0.7, 0.3]) * cells_per_step / (res * DT), (n, 1)).astype(np.float32)
    p = Particles(x, v, 0.01, [Material(youngs_modulus=0.0)])
    return Scene("moving", p, (0.0, 0.0, 0.0), (res,) * 3, 1.0 / res, DT, _abi.TRANSFER_PIC_FLIP,
                 _abi.INTERP_LINEAR, blend=1.0, gravity=0.0, sticky_cells=0)


def _engine(make, full_sort):
    if full_sort:
        os.environ["MPM_FULL_SORT"] = "1"
    try:
        return make()  # the engine reads the switch when it is created
    finally:
        os.environ.pop("MPM_FULL_SORT", None)


# Sizes around one radix tile (8192) and the smallest scene that has radix
# passes (4096); grids of 16, 20 and 26 key bits (3, 3 and 5 passes).  0.02
# cells a step: block by block; 0.35: about one particle in six changes block;
# 6: past the neighbours, and out of the grid in the end.
@pytest.mark.parametrize("n,res", [(4095, 32), (4096, 32), (8191, 64), (8192, 64), (8193, 64), (16_385, 32),
                                   (100_003, 96), (50_000, 320)])
@pytest.mark.parametrize("cells", [0.02, 0.35, 6.0])
def test_either_route_equals_full_sort(gpu, n, res, cells):
    make = _scene(n, min(18.0, res / 2.5), cells, res=res).solver
    a, b = _engine(make, False), _engine(make, True)
    for k in range(8):
        a.step(1)
        b.step(1)
        for f in FIELDS:
            assert np.array_equal(a.download(f), b.download(f)), (k, f)
    a.close()
    b.close()


def test_route_follows_the_movement_of_every_step(gpu):
    """Graph-replayed steps whose route changes on the way: a sheet of 30,000
    particles crosses the border of the grid in some of the steps."""
    sc = _scene(40_000, 20.0, 0.02)
    sc.particles.positions[:30_000, 0] = (64 - 7.5 + 0.2 * np.random.default_rng(5).random(30_000)) / 64
    sc.particles.velocities = sc.particles.velocities.copy()
    sc.particles.velocities[:30_000, 0] = 0.5 / (64 * DT)
    a, b = _engine(sc.solver, False), _engine(sc.solver, True)
    a.step(24)
    b.step(24)
    for f in FIELDS:
        assert np.array_equal(a.download(f), b.download(f)), f
    a.close()
    b.close()


def test_far_movers_of_one_scene_in_a_batch(gpu):
    scs = [_scene(30_000, 16.0, 0.05, seed=2), _scene(20_000, 12.0, 6.0, seed=3), _scene(700, 8.0, 0.2, seed=4)]
    with Batch() as b:
        ids = [b.add(s) for s in scs]
        b.step(10)
        got = [[b.download(i, f) for f in FIELDS] for i in ids]
    for s, want in zip(scs, got):
        g = _engine(s.solver, True)
        g.step(10)
        for f, w in zip(FIELDS, want):
            assert np.array_equal(g.download(f), w)
        g.close()


def _ms_per_step(make, full_sort):
    best = 1e9
    for _ in range(3):
        eng = _engine(make, full_sort)
        eng.step(4)
        eng.synchronize()
        t = time.perf_counter()
        eng.step(8)
        eng.synchronize()
        best = min(best, (time.perf_counter() - t) / 8 * 1e3)
        eng.close()
    return best


# All particles past the neighbouring blocks; a third of the particles of eight
# crowded blocks into the next.
@pytest.mark.parametrize("n,extent,cells,res,at", [(400_000, 37.0, 6.0, 128, 24.1), (1_000_000, 8.0, 0.3, 64, 12.0)])
def test_much_movement_is_no_slower_than_a_full_sort(gpu, n, extent, cells, res, at):
    make = _scene(n, extent, cells, res=res, at=at).solver
    assert _ms_per_step(make, False) < 1.5 * _ms_per_step(make, True)
