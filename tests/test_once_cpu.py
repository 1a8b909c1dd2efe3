"""CPU: deo_once.h, what a kernel's launcher knows per device: found once for each device
(its function attributes hold on that device alone), complete before any thread sees it,
and not kept after an error."""
import os
import subprocess

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "diffeqoperators.jl_gb300", "csrc", "deo_once.h")
PROGRAM = r"""
#include "%s"
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
int main() {
    deo::PerDevice<long> known;
    std::atomic<int> steps[2] = {{0}, {0}}, bad{0};
    long v = 0;
    if (known.get(0, v, [](long&) { return 7; }) != 7) return 1;  // an error, not kept
    std::vector<std::thread> t;
    for (int i = 0; i < 8; ++i)
        t.emplace_back([&, dev = i %% 2] {
            long g = 0;
            const int e = known.get(dev, g, [&](long& out) {
                for (int k = 0; k < 2; ++k) {  // two instantiations, one after the other
                    out = 100 + dev;
                    ++steps[dev];
                    std::this_thread::sleep_for(std::chrono::milliseconds(20));
                }
                return 0;
            });
            if (e || g != 100 + dev || steps[dev] != 2) ++bad;
        });
    for (auto& x : t) x.join();
    return bad || steps[0] != 2 || steps[1] != 2 ? 2 : 0;
}
"""


def test_found_once_per_device_and_whole(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM % HEADER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
