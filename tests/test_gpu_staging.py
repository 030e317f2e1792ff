"""The buffers that stage particles on their way in stage the blocking field
transfers as well, are not overwritten while still read, and are given back
where memory runs out."""
import numpy as np
import pytest
import torch

from mpm_b200 import _abi
from mpm_b200.batch import Batch
from mpm_b200.scenes import Scene, tiny_scene
from mpm_b200.solver import Material, Particles

pytestmark = pytest.mark.gpu


def _scene(n, seed, res=32):
    rng = np.random.default_rng(seed)
    x = 0.2 + 0.6 * rng.random((n, 3), dtype=np.float32)
    v = rng.random((n, 3), dtype=np.float32)
    return Scene("staging", Particles(x, v, 0.01, [Material()]), (0.0, 0.0, 0.0), (res,) * 3, 1.0 / res, 1e-4,
                 _abi.TRANSFER_APIC, _abi.INTERP_QUADRATIC)


def _held():
    """Device memory in use, without what the scene pool only keeps."""
    torch.cuda.synchronize()
    _abi.load().mpm_release_cached_memory(0)
    free, total = torch.cuda.mem_get_info(0)
    return total - free


def test_field_transfers_share_the_upload_buffer(gpu):
    """4M particles are staged in 112 MB, their Fe in 144 MB: held are the 144,
    not both (the rest of the bound is the allocator's granularity)."""
    s = _scene(4_000_000, 1, res=64).solver()
    s.step(1)
    s.synchronize()
    before = _held()
    fe = s.download(_abi.FIELD_FE)
    assert _held() - before < 80e6
    s.upload(_abi.FIELD_FE, fe)
    assert np.array_equal(s.download(_abi.FIELD_FE), fe)
    s.close()


def test_transfers_between_adds(gpu):
    """Field downloads and density grids of every size between adds."""
    sizes = (300, 70_000, 1_000, 200_000, 50_000)
    with Batch() as b:
        scs, ids = [_scene(n, k) for k, n in enumerate(sizes)], []
        for sc in scs:
            ids.append(b.add(sc))
            for sid, s in zip(ids, scs):
                assert np.array_equal(b.download(sid, _abi.FIELD_POSITION), s.particles.positions)
            rho = b.density(ids[0])
            assert np.isclose(rho.sum(dtype=np.float64) / 32 ** 3, 300 * 0.01, rtol=1e-4)
        for sid, s in zip(ids, scs):
            assert np.array_equal(b.download(sid, _abi.FIELD_VELOCITY), s.particles.velocities)


def test_scene_that_does_not_fit(gpu):
    """A grid of 1.1 TB is refused; the scenes before and after it are as if it
    had not been tried."""
    huge = tiny_scene(n=100_000)
    huge.resolution = (4096,) * 3
    fits = [_scene(70_000, 2), _scene(90_000, 3)]

    def run(with_huge):
        with Batch() as b:
            ids = [b.add(fits[0])]
            if with_huge:
                with pytest.raises(Exception, match="(?i)memory|alloc"):
                    b.add(huge)
            ids.append(b.add(fits[1]))
            if with_huge:
                with pytest.raises(Exception, match="(?i)memory|alloc"):
                    b.add(huge)
            b.step(3)
            return [b.download(i, f) for i in ids for f in (_abi.FIELD_POSITION, _abi.FIELD_FE)]

    for x, y in zip(run(True), run(False)):
        assert np.array_equal(x, y)
