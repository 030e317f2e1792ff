"""Admission counts what a scene holds on the device."""
import numpy as np
import pytest
import torch

from mpm_b200 import _abi
from mpm_b200.batch import Batch
from mpm_b200.scenes import Scene
from mpm_b200.serving import scene_device_bytes
from mpm_b200.solver import Material, Particles

pytestmark = pytest.mark.gpu


def _held():
    """Device memory in use, without what the scene pool only keeps."""
    torch.cuda.synchronize()
    _abi.load().mpm_release_cached_memory(0)
    free, total = torch.cuda.mem_get_info(0)
    return total - free


# Crowded blocks (tiles of split items), a sparse scene on a large grid (block
# tables), and one of a few particles on it.
@pytest.mark.parametrize("n,res,extent,transfer", [(6_000_000, 128, 0.3, _abi.TRANSFER_APIC),
                                                   (3_000_000, 400, 0.9, _abi.TRANSFER_PIC_FLIP),
                                                   (1_000, 400, 0.9, _abi.TRANSFER_APIC)])
def test_estimate_covers_what_a_scene_holds(gpu, n, res, extent, transfer):
    rng = np.random.default_rng(0)
    x = 0.05 + extent * rng.random((n, 3), dtype=np.float32)
    p = Particles(x, (0.0, -1.0, 0.0), 0.01, [Material()], volume=np.full(n, 1e-6, np.float32))
    sc = Scene("memory", p, (0.0, 0.0, 0.0), (res,) * 3, 1.0 / res, 1e-5, transfer, _abi.INTERP_CUBIC)
    with Batch() as b:
        # kernels and page tables of a first run are no part of a scene
        sid = b.add(Scene("warm", Particles(x[:1000], (0.0, 0.0, 0.0), 0.01, [Material()]), (0.0, 0.0, 0.0), (32,) * 3,
                          1.0 / 32, 1e-5, transfer, _abi.INTERP_CUBIC))
        b.step(8)
        b.remove(sid)
        b.synchronize()
        before = _held()
        b.add(sc)
        b.step(8)
        b.synchronize()
        held = _held() - before
    want = scene_device_bytes(sc)
    # the allocator hands out memory in pieces of up to 32 MB
    assert held <= want + 64e6
    assert want <= 1.5 * held + 64e6
