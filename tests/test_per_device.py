"""A kernel's shared memory limit belongs to the device that was current when it was raised: a process that uses
a second device has to raise it there as well.  rg_perdevice.cuh is run on the host with several threads and
devices; the sources must not set attributes once per process."""
import glob
import re
import shutil
import subprocess

import pytest

from conftest import PKG_DIR

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "rg_perdevice.cuh"
int main()
{
    rg::PerDevice once;
    std::atomic<int> calls[rg::kMaxDevices + 2] = {};
    auto use = [&](int dev, int result) { return once.run(dev, 0, [&] { ++calls[dev]; return result; }); };
    if (use(0, 7) != 7 || use(0, 0) != 0 || calls[0] != 2) return 1;   // a failure is tried again
    std::vector<std::thread> t;
    for (int k = 0; k < 8; ++k)
        t.emplace_back([&] { for (int i = 0; i < 1000; ++i) for (int d = 0; d < 4; ++d) use(d, 0); });
    for (auto& x : t) x.join();
    if (calls[0] != 2 || calls[1] != 1 || calls[2] != 1 || calls[3] != 1) return 2;
    use(rg::kMaxDevices, 0);
    use(rg::kMaxDevices, 0);
    return calls[rg::kMaxDevices] == 2 ? 0 : 3;                        // no room to remember: every time
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_set_up_runs_once_on_every_device(tmp_path):
    (tmp_path / "p.cpp").write_text(PROGRAM)
    exe = tmp_path / "p"
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", PKG_DIR + "/csrc", "-o", str(exe), str(tmp_path / "p.cpp")], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_attribute_is_set_once_per_process():
    for name in glob.glob(PKG_DIR + "/csrc/*.cu"):
        src = open(name).read()
        assert "call_once" not in src, name
        assert not re.search(r"static bool (attr|done) = false", src), name
