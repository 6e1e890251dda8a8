"""The runtime-length block FFT's planner (kfr_gb300/csrc/rp.cpp) on the CPU: its descriptors are walked pass by
pass, every shared-memory address checked against the buffer and the result against the direct DFT."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "kfr_gb300", "csrc")

# every radix alone, in each place of two and three passes, odd and even group sizes, four and more passes, the
# longest lengths of the one-CTA plans
LENGTHS = [2, 3, 5, 7, 11, 13, 16, 18, 22, 26, 49, 121, 143, 169, 200, 256, 360, 539, 600, 847, 1001, 1024, 1080, 1331,
           1536, 1920, 2187, 2197, 2401, 3125, 3600, 4095, 4096,
           # primes of 17 to 127 as passes of their own
           17, 34, 127, 17 * 19, 289, 2 * 37 * 5, 23 * 12 * 11, 17 * 19 * 11]


@pytest.fixture(scope="module")
def walker(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("rp") / "test_rp")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, os.path.join(ROOT, "tests", "cpp", "test_rp.cpp"),
                    os.path.join(CSRC, "rp.cpp"), "-o", exe], check=True)
    return exe


# layout (0 signals, 1 columns, 2 rows), signals per tile, bytes of a complex value, both ends in shared memory,
# values a thread holds
@pytest.mark.parametrize("layout,s,elem,io,hold", [
    (0, 1, 8, 0, 16), (0, 1, 16, 0, 16), (0, 1, 8, 1, 16), (0, 1, 8, 0, 32), (0, 1, 16, 1, 32), (1, 16, 8, 0, 16),
    (1, 4, 8, 0, 16), (1, 8, 16, 0, 32), (1, 1, 8, 0, 16), (2, 16, 8, 0, 16), (2, 8, 16, 0, 16), (2, 2, 8, 0, 32)])
def test_descriptors(walker, layout, s, elem, io, hold):
    lengths = LENGTHS if s <= 4 else [n for n in LENGTHS if n <= 1080]
    r = subprocess.run([walker, str(layout), str(s), str(elem), str(io), str(hold)] + [str(n) for n in lengths], capture_output=True,
                       text=True)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout


def test_lengths_without_a_plan(walker):
    for n in (131, 2 * 137, 2 * 65537):
        assert subprocess.run([walker, "0", "1", "8", "0", "16", str(n)], capture_output=True).returncode == 1
