"""The in-place line kernels do not depend on the order in which a block's threads run
between two barriers: their source, compiled for the CPU, leaves the same bits with the
threads taken in ascending and in descending order (`line_emu/order.cpp`).  Lengths
whose butterfly counts are, and are not, multiples of the block size, with every radix,
two to four passes, and compile-time plans (33, 64)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "ads4-holographic-quantum-turbulence_b200" / "csrc"
LENGTHS = [4, 6, 12, 26, 33, 48, 64, 96, 100, 121, 150, 180, 200, 250, 384, 500, 600, 750, 768,
           1000, 1001, 1024, 1300, 2048]


@pytest.fixture(scope="module")
def order(tmp_path_factory):
    exe = tmp_path_factory.mktemp("order") / "order"
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", "/usr/local/cuda/include",
                    "-I", str(ROOT / "include"), "-I", str(CSRC),
                    str(ROOT / "tests" / "line_emu" / "order.cpp"),
                    str(CSRC / "hqt_ops_host.cpp"), "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("axis", ["x", "y"])
def test_thread_order_does_not_matter(order, axis):
    out = subprocess.run([str(order), axis, *map(str, LENGTHS)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout
