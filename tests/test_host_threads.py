"""Host work on threads: an exception in a part, or a thread that cannot be started, reaches
the caller as an exception or as work done by the caller, and never ends the process."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAIN = """
#include <sys/resource.h>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include "host_threads.hpp"
int main(int argc, char** argv) {
    std::atomic<int> done{0};
    const bool starved = !std::strcmp(argv[1], "starved");
    if (starved) {  // no room for a thread's stack
        long pages = 0;
        if (FILE* f = std::fopen("/proc/self/statm", "r")) {
            if (std::fscanf(f, "%ld", &pages) != 1) return 2;
            std::fclose(f);
        }
        rlimit r;
        r.rlim_cur = r.rlim_max = rlim_t(pages) * 4096 + (4u << 20);
        if (setrlimit(RLIMIT_AS, &r)) return 2;
    }
    try {
        gaia::run_parts(8, [&](int k) {
            if (!starved && (k == 0 || k == 5)) throw std::bad_alloc();
            ++done;
        });
        std::printf("returned %d\\n", done.load());
    } catch (const std::bad_alloc&) {
        std::printf("bad_alloc %d\\n", done.load());
    }
}
"""


@pytest.mark.parametrize("case,out", [("throws", "bad_alloc 6"), ("starved", "returned 8")])
def test_parts_end_and_errors_reach_the_caller(tmp_path, case, out):
    (tmp_path / "t.cpp").write_text(MAIN)
    exe = str(tmp_path / "t")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-pthread", "-I",
                    os.path.join(ROOT, "gaia_gb300", "csrc"), str(tmp_path / "t.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, case], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == out, (r.returncode, r.stdout, r.stderr)


def test_engine_records_are_built_through_it():
    with open(os.path.join(ROOT, "gaia_gb300", "csrc", "vbd_engine.cuh")) as f:
        src = f.read()
    assert "run_parts(nt, work)" in src and "std::thread>" not in src
