"""Step statistics: blocks that hold particles and scenes with particles outside
their grid, however P2G splits a block's particles into work items."""
import numpy as np
import pytest

from mpm_b200 import _abi
from mpm_b200.batch import Batch
from mpm_b200.scenes import Scene
from mpm_b200.solver import Material, Particles

pytestmark = pytest.mark.gpu

RES = 64


def _scene(n, crowded, outside, seed):
    """n particles at rest over the grid, `crowded` of them in one block and
    `outside` of them off the grid; with the number of blocks they occupy."""
    rng = np.random.default_rng(seed)
    cell = rng.integers(1, RES - 2, (n, 3))
    cell[:crowded] = 20 + rng.integers(0, 4, (crowded, 3))
    x = (cell + rng.uniform(0.3, 0.6, (n, 3))) / RES  # (well inside a cell: its base is the cell)
    inside = np.ones(n, bool)
    if outside:
        x[-outside:, 0] = -2.0
        inside[-outside:] = False
    blocks = len(np.unique((cell[inside] + 4) // 4, axis=0))
    p = Particles(x.astype(np.float32), np.zeros((n, 3), np.float32), 0.01, [Material(youngs_modulus=0.0)])
    return Scene("stats", p, (0.0, 0.0, 0.0), (RES,) * 3, 1.0 / RES, 1e-4, _abi.TRANSFER_PIC_FLIP,
                 _abi.INTERP_LINEAR, gravity=0.0, sticky_cells=0), blocks


# Scenes on both sides of 65,536 particles, whose blocks are split differently (the
# grid of 4,914 blocks is compacted by one cluster, the batch below is not).
@pytest.mark.parametrize("n,crowded,outside", [(1, 0, 0), (1, 0, 1), (3_000, 1_500, 700), (60_000, 9_000, 5_000),
                                               (200_000, 30_000, 0), (200_000, 2_600, 9_000)])
def test_blocks_are_counted_once(gpu, n, crowded, outside):
    sc, blocks = _scene(n, crowded, outside, seed=n)
    s = sc.solver()
    for _ in range(3):
        s.step(2)
        st = s.stats()
        assert (st["active_blocks"], st["outside_blocks"]) == (blocks, int(outside > 0))
    s.close()


def test_blocks_of_a_batch(gpu):
    scs = [_scene(60_000, 9_000, 5_000, seed=1), _scene(200_000, 30_000, 12_000, seed=2), _scene(50, 0, 0, seed=3)]
    with Batch() as b:
        for sc, _ in scs:
            b.add(sc)
        b.step(4)
        st = b.stats()
    assert (st["active_blocks"], st["outside_blocks"]) == (sum(blocks for _, blocks in scs), 2)
