"""Plans built on the CPU against stubs of the CUDA calls (tests/cpp/cuda_stub.cpp): which lengths and sizes they take."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "kfr_gb300", "csrc")
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def compile_test(tmp, name, *sources):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp / name)
    cpp = os.path.join(ROOT, "tests", "cpp")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CUDA, "-I", CSRC, "-Wl,--unresolved-symbols=ignore-all",
                    os.path.join(cpp, name + ".cpp"), os.path.join(cpp, "cuda_stub.cpp")] +
                   [os.path.join(CSRC, s) for s in sources] + ["-o", exe], check=True)
    return exe


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    return compile_test(tmp_path_factory.mktemp("plans"), "test_plan_lengths", "plan.cpp", "rp.cpp")


# every short length, and the longest ones that one CTA transforms
@pytest.mark.parametrize("precision,lo,hi", [("f", 1, 2000), ("f", 11000, 17000), ("f", 20000, 20600), ("d", 1, 2000),
                                             ("d", 5500, 8500), ("d", 10000, 10300)])
def test_every_length_plans(plans, precision, lo, hi):
    r = subprocess.run([plans, precision, str(lo), str(hi)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:]


# dot products where a convolution would round more, one CTA where the plain radices fit in place, the four-step or
# Bluestein's multi-kernel transform beyond
@pytest.mark.parametrize("precision,strategy,lengths", [
    ("sf", "direct", [13, 19, 23, 31, 58, 62, 124, 946, 1955, 8177, 12000, 12312, 14880, 16384]),
    ("sf", "bluestein", [142, 149, 8178]), ("sf", "fourstep", [11297, 11550, 11880, 13851, 14400, 16383, 16385]),
    ("sf", "rader", [137, 7561, 8641]), ("sf", "multi", [12433, 13933, 14401, 15319]),
    ("sd", "direct", [19, 23, 31, 56, 946, 2140, 3268, 6144, 6384, 8192]), ("sd", "bluestein", [149]),
    ("sd", "fourstep", [5676, 7056, 7200, 8099]), ("sd", "multi", [6217, 7039, 7057])])
def test_strategy(plans, precision, strategy, lengths):
    r = subprocess.run([plans, precision] + [str(n) for n in lengths], capture_output=True, text=True, check=True)
    assert dict(zip(lengths, r.stdout.split())) == {n: strategy for n in lengths}


# launches of a forward transform, what the plan says of itself, its half length's four-step split
@pytest.mark.parametrize("precision,n,launches,says", [
    ("rf", 7200, 1, "fused split/merge"), ("rf", 88200, 2, "split fused into the four-step row pass, merge fused"),
    ("rf", 1 << 20, 3, "separate split, merge fused into the column pass"), ("rf", 2 * 8209, 2, "separate split, separate merge"),
    ("rd", 88200, 2, "split fused into the four-step row pass, merge fused"),
    # enough tiles for either pass of lengths with large primes
    ("rd", 16206, 2, "n=8103 = 73 x 111"), ("rd", 31450, 2, "n=15725 = 85 x 185"), ("rf", 31750, 2, "n=15875 = 125 x 127")])
def test_real_plans(plans, precision, n, launches, says):
    r = subprocess.run([plans, precision, str(n)], capture_output=True, text=True, check=True)
    count, text = r.stdout.split(" ", 1)
    assert int(count) == launches and says in text, r.stdout


def test_plan_cache_per_device(tmp_path):
    exe = compile_test(tmp_path, "test_plan_cache", "plan_cache.cpp", "plan.cpp", "rp.cpp")
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
