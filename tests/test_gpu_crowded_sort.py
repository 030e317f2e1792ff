"""Crowded blocks: where one block holds many of a batch's particles, the steps
sort all keys, by the full sort where the first step finds it so, by radix
passes in the block sort's launch where the block fills later.  Any route is the
stable sort of all keys (bitwise the run with MPM_FULL_SORT=1), and none is
much slower than it."""
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
RES, DT = 32, 1e-3


def _scene(n, blocks, part=1.0, converge=0, seed=1, res=RES):
    """n stress-free particles; `part` of them in blocks^3 whole blocks, the rest
    spread out.  They drift by 0.005 cells a step, or (converge) meet at the
    middle of a block after that many steps."""
    rng = np.random.default_rng(seed)
    x = 12.05 + (4 * blocks - 0.1) * rng.random((n, 3))
    k = n - int(n * part)
    x[:k] = 3.0 + (res - 8) * rng.random((k, 3))
    v = 0.005 * rng.uniform(-1, 1, (n, 3))
    if converge:
        v = (14.0 - x) / converge
    p = Particles((x / res).astype(np.float32), (v / (res * DT)).astype(np.float32), 0.01,
                  [Material(youngs_modulus=0.0)])
    return Scene("crowded", p, (0.0, 0.0, 0.0), (res,) * 3, 1.0 / res, DT, _abi.TRANSFER_PIC_FLIP,
                 _abi.INTERP_LINEAR, blend=1.0, gravity=0.0, sticky_cells=0)


def _engine(make, full_sort):
    if full_sort:
        os.environ["MPM_FULL_SORT"] = "1"
    try:
        return make()  # the engine reads the switch when it is created
    finally:
        os.environ.pop("MPM_FULL_SORT", None)


# On both sides of the lines of the first step (in the fullest block 4096 + n / 64
# on the 32^3 grid, 4096 + n / 16 on 64^3, 16384 + n / 16 on 320^3) and at the
# smallest dense block (4096).
@pytest.mark.parametrize("n,blocks,part,res", [
    (4095, 1, 1.0, 32), (4096, 1, 1.0, 32), (4161, 1, 1.0, 32), (4162, 1, 1.0, 32), (40_000, 1, 1.0, 32),
    (40_000, 2, 1.0, 32), (60_000, 1, 0.08, 32), (60_000, 1, 0.2, 32), (4369, 1, 1.0, 64), (4370, 1, 1.0, 64),
    (60_000, 1, 0.1, 64), (60_000, 1, 0.2, 64), (17_000, 1, 1.0, 320), (18_000, 1, 1.0, 320)])
def test_crowded_scene_equals_full_sort(gpu, n, blocks, part, res):
    make = _scene(n, blocks, part, res=res).solver
    a, b = _engine(make, False), _engine(make, True)
    for k in range(6):
        for e in (a, b):
            e.step(3)
            e.synchronize()  # (the read-back of the first step has landed)
        for f in FIELDS:
            assert np.array_equal(a.download(f), b.download(f)), (k, f)
    a.close()
    b.close()


def test_block_that_fills_later_equals_full_sort(gpu):
    """150,000 particles of 27 blocks meet in one: past 65,536 + n / 13 = 77,074
    in a block the radix passes take over."""
    make = _scene(150_000, 3, converge=30).solver
    a, b = _engine(make, False), _engine(make, True)
    for k in range(9):
        a.step(3)
        b.step(3)
        for f in FIELDS:
            assert np.array_equal(a.download(f), b.download(f)), (k, f)
    a.close()
    b.close()


def test_crowded_scene_joins_and_leaves_a_batch(gpu):
    scs = [_scene(5_000, 3, seed=2), _scene(30_000, 1, seed=3), _scene(700, 1, seed=4)]

    def run(full_sort):
        bt = _engine(Batch, full_sort)
        ids = [bt.add(scs[0])]
        bt.step(4)
        ids.append(bt.add(scs[1]))
        bt.step(5)
        ids.append(bt.add(scs[2]))
        bt.step(4)
        out = [bt.download(i, f) for i in ids for f in FIELDS]
        bt.remove(ids[1])
        bt.step(6)
        out += [bt.download(i, f) for i in (ids[0], ids[2]) for f in FIELDS]
        bt.close()
        return out

    for x, y in zip(run(False), run(True)):
        assert np.array_equal(x, y)


def _ms_per_step(make, full_sort):
    best = 1e9
    for _ in range(8):
        eng = _engine(make, full_sort)
        eng.step(4)
        eng.synchronize()
        t = time.perf_counter()
        eng.step(12)
        eng.synchronize()
        best = min(best, (time.perf_counter() - t) / 12 * 1e3)
        eng.close()
    return best


@pytest.mark.parametrize("n,blocks", [(250_000, 1), (1_000_000, 1), (1_000_000, 2)])
def test_crowded_scene_is_no_slower_than_a_full_sort(gpu, n, blocks):
    make = _scene(n, blocks).solver
    assert _ms_per_step(make, False) < 1.15 * _ms_per_step(make, True)
