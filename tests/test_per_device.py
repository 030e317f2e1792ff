"""A kernel's shared-memory limit belongs to a device: the set-up step that
raises it runs once for each device, again after a failure, and with several
threads no caller goes on before it has run."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "per_device.hpp"
#include <thread>
#include <vector>
int main() {
    mpm::OncePerDevice once;
    int runs[80] = {};
    for (int round = 0; round < 3; ++round)
        for (int d = 0; d < 64; ++d)
            if (once(d, [&] { ++runs[d]; return 0; }) != 0) return 1;
    for (int d = 0; d < 64; ++d)
        if (runs[d] != 1) return 2;
    for (int round = 0; round < 3; ++round) once(70, [&] { ++runs[70]; return 0; });
    if (runs[70] != 3) return 3;

    mpm::OncePerDevice failing;
    int tries = 0;
    if (failing(1, [&] { return ++tries < 3 ? 2 : 0; }) != 2) return 4;
    if (failing(1, [&] { return ++tries < 3 ? 2 : 0; }) != 2) return 5;
    if (failing(1, [&] { return ++tries < 3 ? 2 : 0; }) != 0 || tries != 3) return 6;
    failing(1, [&] { return ++tries, 0; });
    if (tries != 3) return 7;

    mpm::OncePerDevice shared;
    std::atomic<int> ready[4] = {}, early{0};
    std::vector<std::thread> ts;
    for (int t = 0; t < 16; ++t)
        ts.emplace_back([&, t] {
            shared(t % 4, [&] { ready[t % 4] = 1; return 0; });
            if (!ready[t % 4]) ++early;
        });
    for (auto& t : ts) t.join();
    return early ? 8 : 0;
}
"""


def test_setup_runs_once_for_each_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run([os.environ.get("MPM_HOSTCXX", "/usr/bin/g++"), "-std=c++17", "-pthread", "-I",
                    os.path.join(ROOT, "mpm_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_shared_memory_limits_are_raised_per_device():
    """Every limit is raised through the per-device step or at each launch."""
    src = open(os.path.join(ROOT, "mpm_b200", "csrc", "kernels.cu")).read()
    calls = src.split("cudaFuncSetAttribute")[:-1]
    assert calls and all("once(device" in c.splitlines()[-1] for c in calls)
