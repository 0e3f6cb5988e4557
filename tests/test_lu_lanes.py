"""The warp's LU of the affine Gauss-Newton solve on the CPU: its lanes run one
after the other between the warp-synchronous calls, in several orders, so that
a value one lane reads after another has overwritten it shows (with the lanes
in step on a GPU it need not).  Matrices of two to six parameters, with zero
pivots, ties, infinities and NaN, bit for bit against the same steps done by
one thread."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_lu_does_not_depend_on_the_order_of_lanes(tmp_path):
    exe = str(tmp_path / "lu_lanes")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wno-unknown-pragmas", "-o", exe,
                           os.path.join(ROOT, "tests", "cpp", "lu_lanes.cpp")])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and "LU PASSED" in out.stdout, out.stdout + out.stderr
