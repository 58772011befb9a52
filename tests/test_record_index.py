"""Scenes of up to 2^31 - 1 incidences are accepted, and their records are found: rows are
counted in 32 bits, records in 64."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAIN = """
#include <cstdio>
#include "record_index.hpp"
using namespace gaia;
int main() {
    const int32_t last = std::numeric_limits<int32_t>::max();
    std::printf("%d\\n", checked_count(last) == last);
    try {
        checked_count(int64_t(last) + 1);
        std::printf("0\\n");
    } catch (const std::runtime_error&) {
        std::printf("1\\n");
    }
    std::printf("%d\\n", dev::record_index(last, 7) == (size_t(last) << 3) + 7);
    int ok = 1;
    for (int n = 0; n <= dev::kSegNbrs; ++n)
        for (int p = 0; p < dev::kSlice; ++p) {
            const int32_t z = dev::pack_nbrs(n, p);
            ok &= dev::nbrs_of(z) == n && dev::place_of(z) == p;
        }
    std::printf("%d\\n", ok);
}
"""


def test_counts_and_places(tmp_path):
    (tmp_path / "t.cpp").write_text(MAIN)
    exe = str(tmp_path / "t")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-I", os.path.join(ROOT, "gaia_gb300", "csrc"),
                    str(tmp_path / "t.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split() == ["1"] * 4
