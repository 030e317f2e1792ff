"""Scenes of a batch are copied while the ones before them are still sorted and
written: the caller's arrays, page-locked or not, may be overwritten as soon as
add() returns, and every scene holds its own particles, at sizes around the
cell-sorted upload (65,536) and in an order that makes a staging buffer grow,
be reused while the other is busy, and shrink."""
import numpy as np
import pytest
import torch

from mpm_b200 import _abi
from mpm_b200.batch import Batch
from mpm_b200.scenes import Scene
from mpm_b200.solver import Material, Particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("sizes", [(1, 65_535, 65_536, 200_000, 7, 300_000, 65_537, 3), (2_500_000, 10, 2_500_001, 40_000)])
def test_arrays_may_be_reused_after_add(gpu, sizes, pinned):
    top = max(sizes)
    if pinned:
        bufs = [torch.empty(top, c, pin_memory=True).numpy() for c in (3, 3, 1)]
    else:
        bufs = [np.empty((top, c), np.float32) for c in (3, 3, 1)]
    want, ids = [], []
    with Batch() as b:
        for k, n in enumerate(sizes):
            rng = np.random.default_rng(k)
            x, v, m = bufs[0][:n], bufs[1][:n], bufs[2][:n, 0]
            x[:] = 0.2 + 0.6 * rng.random((n, 3), dtype=np.float32)
            v[:] = rng.random((n, 3), dtype=np.float32)
            m[:] = 0.01
            want.append((x.copy(), v.copy()))
            p = Particles(x, v, m, [Material()])
            assert p.positions.ctypes.data == x.ctypes.data
            ids.append(b.add(Scene("upload", p, (0.0, 0.0, 0.0), (32, 32, 32), 1.0 / 32, 1e-4, k % 2,
                                   _abi.INTERP_QUADRATIC)))
            for a in bufs:
                a[:] = np.nan
        for sid, (x, v) in zip(ids, want):
            assert np.array_equal(b.download(sid, _abi.FIELD_POSITION), x)
            assert np.array_equal(b.download(sid, _abi.FIELD_VELOCITY), v)
