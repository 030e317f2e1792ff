"""Where a scene has more small blocks than the block sort's CTAs take, single
warps put them together: the result is the stable sort of all keys (bitwise the
run with MPM_FULL_SORT=1), with few and many arrivals in a block, from lower and
higher blocks, and with particles past the neighbouring blocks."""
import os

import numpy as np
import pytest
import torch

from mpm_b200 import _abi
from mpm_b200.batch import Batch
from mpm_b200.scenes import Scene
from mpm_b200.solver import Material, Particles

pytestmark = pytest.mark.gpu

FIELDS = (_abi.FIELD_POSITION, _abi.FIELD_VELOCITY, _abi.FIELD_FE)
RES, DT = 96, 1e-3


def _scene(n, cells_per_step, spread=0.0, groups=(), far=0, seed=1):
    """n stress-free particles over nearly all of the grid, moving by
    cells_per_step along x + y (and by up to `spread` more each).  `groups` of
    particles lie close together at the border of a block, half of them on
    either side, and change sides between the first and the sixth step; `far`
    particles move by six cells a step."""
    rng = np.random.default_rng(seed)
    x = 6.0 + (RES - 12) * rng.random((n, 3))
    v = np.array([1.0, 0.7, 0.1]) * cells_per_step + spread * rng.uniform(-1, 1, (n, 3))
    at = 0
    for k, size in enumerate(groups):
        # the border of two blocks along one axis, anywhere in the others
        axis, half = k % 3, size // 2
        c = 4.0 * rng.integers(3, RES // 4 - 3, 3) + rng.uniform(0.5, 3.5, 3)
        c[axis] = 4.0 * np.floor(c[axis] / 4.0)
        g = slice(at, at + size)
        x[g] = c + rng.uniform(-0.4, 0.4, (size, 3))
        x[g][:half, axis] = c[axis] - 0.05 - 0.5 * rng.random(half)
        x[g][half:, axis] = c[axis] + 0.05 + 0.5 * rng.random(size - half)
        v[g] = 0.0
        v[g][:half, axis] = 0.12
        v[g][half:, axis] = -0.12
        if k % 2:  # all together, from one side, within one step
            x[g][:, axis] = c[axis] - 0.05 - 0.1 * rng.random(size)
            v[g][:, axis] = 0.2
        at += size
    v[at:at + far] = 6.0 * np.sign(rng.uniform(-1, 1, (far, 3)))
    p = Particles((x / RES).astype(np.float32), (v / (RES * DT)).astype(np.float32), 0.01,
                  [Material(youngs_modulus=0.0, hardening=0.0)])
    return Scene("sparse", p, (0.0, 0.0, 0.0), (RES,) * 3, 1.0 / RES, DT, _abi.TRANSFER_PIC_FLIP,
                 _abi.INTERP_LINEAR, blend=1.0, gravity=0.0, sticky_cells=0)


def _engine(make, full_sort):
    if full_sort:
        os.environ["MPM_FULL_SORT"] = "1"
    try:
        return make()  # the engine reads the switch when it is created
    finally:
        os.environ.pop("MPM_FULL_SORT", None)


# A warp sorts up to 192 arrivals in shared memory, more in global memory; the
# blocks stay below the 768 particles from which CTAs take them.
@pytest.mark.parametrize("n,cells,spread,groups,far", [
    (200_000, 0.03, 0.02, (), 0), (200_000, 0.3, 0.2, (), 0), (60_000, 0.05, 0.0, (), 1_500),
    (200_000, 0.02, 0.0, (191, 192, 193, 194, 380, 384, 388, 600, 700, 730) * 3, 0),
    (200_000, 0.25, 0.1, (400, 700, 64, 65, 33, 192, 193) * 4, 4_000)])
def test_warps_put_blocks_together_as_the_full_sort(gpu, n, cells, spread, groups, far):
    make = _scene(n, cells, spread, groups, far).solver
    a, b = _engine(make, False), _engine(make, True)
    ctas = 5 * torch.cuda.get_device_properties(0).multi_processor_count
    for k in range(6):
        a.step(1)
        b.step(1)
        assert a.stats()["active_blocks"] > 2 * ctas + 100  # (a few blocks may be large)
        for f in FIELDS:
            assert np.array_equal(a.download(f), b.download(f)), (k, f)
    a.close()
    b.close()


def test_warps_in_a_batch(gpu):
    scs = [_scene(80_000, 0.2, 0.2, (193, 500, 191), 300, seed=2), _scene(30_000, 0.4, 0.1, (), 0, seed=3),
           _scene(120_000, 0.01, 0.0, (700, 730, 300), 900, seed=4)]

    def run(full_sort):
        bt = _engine(Batch, full_sort)
        ids = [bt.add(s) for s in scs]
        bt.step(6)
        out = [bt.download(i, f) for i in ids for f in FIELDS]
        bt.close()
        return out

    for x, y in zip(run(False), run(True)):
        assert np.array_equal(x, y)
