"""Kernel attributes are set once per device, not once per process (tm_per_device.h), and
every kernel that needs more shared memory than the default asks for it that way.  Host
only: a counter takes the place of the CUDA call."""
import os
import re
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "trophic_maelstorm_gb300", "csrc")

MAIN = r"""
#include "%s"
#include <cstdio>
#include <thread>
#include <vector>
int main()
{
    static tmg::PerDevice once;
    int calls[2] = {0, 0}, fail = 3;
    auto on = [&](int d) { return once.run(d, [&] { ++calls[d]; return 0; }); };
    // a device whose setup fails is asked again, and reports the error each time
    if (once.run(1, [&] { return fail; }) != 3 || once.run(1, [&] { return fail; }) != 3) return 1;
    for (int i = 0; i < 3; ++i)
        if (on(0) != 0) return 2;
    if (calls[0] != 1 || calls[1] != 0) return 3;
    if (on(1) != 0 || on(1) != 0 || calls[1] != 1) return 4;        // the second device has its own
    int far = 0;                                                     // ordinals beyond the mask: every time
    for (int d : {-1, 64, 1000})
        if (once.run(d, [&] { ++far; return 0; }) != 0) return 5;
    if (far != 3) return 6;
    // threads that come first together: each returns after a setup of its device
    static tmg::PerDevice shared;
    std::atomic<int> set[8]{}, bad{0};
    std::vector<std::thread> ts;
    for (int t = 0; t < 16; ++t)
        ts.emplace_back([&, t] {
            for (int i = 0; i < 20000; ++i) {
                const int d = (t + i) %% 8;
                shared.run(d, [&] { set[d].store(1); return 0; });
                if (set[d].load() != 1) ++bad;
            }
        });
    for (auto& t : ts) t.join();
    return bad.load() ? 7 : 0;
}
"""


def test_setup_runs_on_every_device(tmp_path):
    (tmp_path / "m.cpp").write_text(MAIN % os.path.join(CSRC, "tm_per_device.h"))
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-o", str(tmp_path / "m"), str(tmp_path / "m.cpp")], check=True)
    assert subprocess.run([str(tmp_path / "m")]).returncode == 0


def test_no_process_wide_attribute_flag():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
            assert not re.search(r"\bstatic\s+bool\b", src), f
            # set through allow_smem, or unconditionally when the object is created (the network)
            if f not in ("tm_kernels.cuh", "tm_mlp.cu"):
                assert "cudaFuncSetAttribute" not in src, f
