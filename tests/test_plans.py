"""Plans of the register passes, made on the host (csrc/reg_tiles.cu), by a
C++ program that links against the library."""
import shutil
import subprocess
from pathlib import Path

import pytest

from yao_rs import _abi as A

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    nvcc = shutil.which("nvcc")
    if shutil.which("g++") is None or nvcc is None:
        pytest.skip("no C++ compiler or CUDA headers")
    exe, lib = tmp_path_factory.mktemp("plans") / "plans", A.LIB_PATH.parent
    cmd = ["g++", "-std=c++17", "-O2", str(ROOT / "tests/c/plans.cpp"), "-I", str(ROOT / "yao-rs_b200/csrc"),
           "-I", str(Path(nvcc).resolve().parent.parent / "include"), "-L", str(lib), "-lyao_gpu", f"-Wl,-rpath,{lib}",
           "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

    def run(*args):
        return subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, check=True, timeout=300).stdout
    return run


# Every matrix is rounded (1e-16 an entry, up and down alike) and the state's
# scale holds what that changes; the scale itself is rounded once, 2e-16, and
# the sum of the logarithms adds 1e-19 a gate.  A bias of an ulp a CNOT would
# be 6e-14 for 18 qubits and 40 layers.
@pytest.mark.parametrize("n,layers", [(4, 400), (18, 40), (30, 160)])
def test_split_program_keeps_the_norm(plans, n, layers):
    count, off = plans("norm", n, layers).split()
    assert int(count) > n * layers
    assert abs(float(off)) < 1e-15


def test_gates_without_targets_or_with_a_qubit_twice_are_not_planned(plans):
    """They are left to the passes of one gate."""
    assert plans("supported").split() == ["1", "0", "0", "0"]


# four times the gates: four times the time, twice that allowed (16 times and
# more where every scan runs to the program's end)
@pytest.mark.parametrize("n,nbits,what", [(13, 13, "exact"), (13, 14, "exact"), (13, 14, "last"), (13, 14, "fused"),
                                          (8, 9, "exact"), (24, 30, "fused"), (13, 14, "sweep"), (8, 9, "sweep")])
def test_planning_time_is_linear(plans, n, nbits, what):
    few, many = (float(plans("time", n, nbits, what, gates)) for gates in (20000, 80000))
    assert many < 8.0 * few, (few, many)


def test_descriptions_fit(plans):
    """8 KiB a pass (three CTAs an SM), with 16 bytes for one more segment."""
    sizes = [int(x) for x in plans("sizes").split()]
    assert len(sizes) == 2 and max(sizes) <= 8192 + 16
