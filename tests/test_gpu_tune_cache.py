"""Entries of the tuning file hold for the kernels they were measured on: lines
without a version, or of another one, are not used, and their keys are tuned
again."""
import os
import subprocess
import sys

import pytest
import torch

from mpm_b200 import _abi

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (a process of its own: the file is read once in a process)
PROGRAM = """
from mpm_b200 import _abi, scenes
s = scenes.tiny_scene(n=4000, transfer=_abi.TRANSFER_APIC, interpolation=_abi.INTERP_CUBIC).solver()
print(sorted(s.autotune(steps_per_candidate=1).items()))
"""


@pytest.mark.parametrize("prefix,used", [("", False), ("v1 ", False), ("v2 ", True), ("v3 ", False)])
def test_entries_of_other_kernels_are_tuned_again(gpu, tmp_path, prefix, used):
    path = tmp_path / "tuning.txt"
    dev = torch.cuda.get_device_name(0).replace(" ", "_")
    path.write_text("".join(f"{prefix}{dev} 4 {_abi.TRANSFER_APIC} {b} 2048 16 7\n" for b in range(4)))
    out = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, env=dict(os.environ, MPM_TUNE_CACHE=str(path)),
                         capture_output=True, text=True, check=True).stdout
    got = dict(eval(out))
    stale = dict(g2p_chunk=2048, p2g_stage=16, p2g_warp_max=7)
    assert all(got[k] == v for k, v in stale.items()) == used
    assert (got["steps"] == 1) == used
    # what was tuned is found again, behind the lines that were there
    again = dict(eval(subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT,
                                     env=dict(os.environ, MPM_TUNE_CACHE=str(path)), capture_output=True, text=True,
                                     check=True).stdout))
    assert again == dict(got, steps=1)
