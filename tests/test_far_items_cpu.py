"""Cost of a far-field item for the largest leaves (the device header's function on the host).

A leaf of 16,843,009 bodies with 255 far nodes has 2^32 - 1 pairs; its item must keep a cost, since
items without one are left out.
"""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "galaxy-collision-simulation_b200" / "csrc"
SOURCE = """
#include "fmm.cuh"
#include <cstdio>
int main() {
    int t, n;
    while (std::scanf("%d %d", &t, &n) == 2) std::printf("%u\\n", gx::far_item_cost(t, n));
}
"""


def test_cost_never_wraps(tmp_path):
    src = tmp_path / "cost.cu"
    src.write_text(SOURCE)
    exe = tmp_path / "cost"
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC), str(src), "-o",
                    str(exe)], check=True)
    cases = [(1, 1), (5, 512), (64, 300), (4194303, 512), (4194304, 512), (16843009, 255), (8421505, 510), (2**31 - 1, 512)]
    out = subprocess.run([str(exe)], input="\n".join(f"{t} {n}" for t, n in cases), capture_output=True, text=True,
                         check=True).stdout.split()
    assert [int(v) for v in out] == [min(t * n + 1, 2**31 - 1) for t, n in cases]
