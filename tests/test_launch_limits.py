"""SmemLimits (csrc/launch_limits.cuh), what each device's launches may ask of shared memory, against a fake of the call
that sets it: no GPU is needed."""
import os
import subprocess

from kipp_b200.csrc import build

PROGRAM = r"""
#include "launch_limits.cuh"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    const int a = 0, b = 0;                                  // two kernels
    {
        SmemLimits limits;
        int calls = 0;
        size_t set_to = 0;
        auto set = [&](size_t n) { ++calls; set_to = n; return 0; };
        CHECK(limits.raise(0, &a, 48 * 1024, set) == 0 && calls == 0);                   // what every launch may ask
        CHECK(limits.raise(0, &a, 100000, set) == 0 && calls == 1 && set_to == 100000);
        CHECK(limits.raise(0, &a, 100000, set) == 0 && calls == 1);
        CHECK(limits.raise(0, &a, 60000, set) == 0 && calls == 1);                       // a smaller form lowers nothing
        CHECK(limits.raise(1, &a, 60000, set) == 0 && calls == 2 && set_to == 60000);    // another device
        CHECK(limits.raise(0, &b, 60000, set) == 0 && calls == 3);                       // another kernel
        CHECK(limits.raise(0, &a, 120000, set) == 0 && calls == 4 && set_to == 120000);
        CHECK(limits.raise(0, &a, 100000, set) == 0 && calls == 4);
        auto refuse = [&](size_t) { ++calls; return 7; };
        CHECK(limits.raise(0, &a, 300000, refuse) == 7 && calls == 5);
        CHECK(limits.raise(0, &a, 120000, refuse) == 0 && calls == 5);                   // what was allowed still is
        CHECK(limits.raise(0, &a, 300000, refuse) == 7 && calls == 6);                   // and a refusal is asked again
    }
    {
        // many threads, each about to launch with a size of its own: the device allows it when raise() returns
        SmemLimits limits;
        std::atomic<size_t> device{0};
        std::atomic<int> bad{0};
        std::vector<std::thread> threads;
        for (int t = 0; t < 8; ++t)
            threads.emplace_back([&, t] {
                unsigned x = 17 * t + 1;
                for (int i = 0; i < 20000; ++i) {
                    x = x * 1664525u + 1013904223u;
                    const size_t want = 50000 + (x >> 8) % (1000 + 10 * (size_t)i);
                    if (limits.raise(0, &a, want, [&](size_t n) { std::this_thread::yield(); device = n; return 0; }) != 0 || device < want) ++bad;
                }
            });
        for (auto& t : threads) t.join();
        CHECK(bad == 0);
    }
    puts("ok");
    return 0;
}
"""


def test_the_limit_is_kept_per_device_and_kernel_and_never_lowered(tmp_path):
    source, program = tmp_path / "limits.cpp", tmp_path / "limits"
    source.write_text(PROGRAM)
    folder = os.path.dirname(build.__file__)
    subprocess.run([build._cxx(), "-std=c++17", "-O2", "-pthread", "-I", folder, str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)], capture_output=True, text=True, check=False).stdout == "ok\n"


def test_no_kernel_file_sets_the_limit_by_itself():
    folder = os.path.dirname(build.__file__)
    for name in os.listdir(folder):
        if name.endswith(".cu"):
            with open(os.path.join(folder, name), encoding="utf-8") as f:
                assert "cudaFuncSetAttribute" not in f.read(), name
