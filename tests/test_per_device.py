"""Values kept per device (pmsim_b200/csrc/pms_per_device.h): host logic, compiled here without CUDA."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pmsim_b200", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "pms_per_device.h"
#define CHECK(c) if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; }
int main() {
    pms::PerDevice<int, 4> t;
    int v = -1, made = 0;
    auto make = [&](int dev) { return [&made, dev](int& x) { made++; x = 10 + dev; return true; }; };
    CHECK(t.get(0, v, make(0)) && v == 10 && made == 1);
    CHECK(t.get(1, v, make(1)) && v == 11 && made == 2);  // another device makes its own
    CHECK(t.get(0, v, make(0)) && v == 10 && made == 2);  // kept
    CHECK(t.get(1, v, make(1)) && v == 11 && made == 2);
    // a failure is not kept and leaves the caller's value alone
    v = 5;
    CHECK(!t.get(2, v, [](int& x) { x = 99; return false; }) && v == 5);
    CHECK(t.get(2, v, make(2)) && v == 12 && made == 3);
    // no such device number
    CHECK(!t.get(4, v, make(4)) && !t.get(-1, v, make(-1)) && made == 3);
    // threads on one new device make one value
    std::atomic<int> n{0}, bad{0};
    std::vector<std::thread> th;
    for (int k = 0; k < 8; k++)
        th.emplace_back([&] {
            int w = 0;
            if (!t.get(3, w, [&](int& x) { x = 40 + n++; return true; }) || w != 40) bad++;
        });
    for (auto& x : th) x.join();
    CHECK(n == 1 && bad == 0);
    return 0;
}
"""


def test_each_device_has_its_own_value(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_no_kernel_attribute_is_kept_for_the_whole_process():
    """Kernel attributes and occupancy figures hold for the device that was current: the solver keeps them
    through PerDevice, not in a static of its own."""
    text = open(os.path.join(CSRC, "pms_solver.cu")).read()
    for name in ("int team_setup(", "void count_team_slots("):
        a = text.index(name)
        body = text[a:text.index("\n}\n", a)]
        assert "PerDevice<" in body and "cudaGetDevice" in body
        assert "static int" not in body and "static bool" not in body
