"""The slices of the one-shot runs' pending edges fit the lists they are written to."""
import subprocess

from efficientstructuralgraphclusteringongpus_gb300 import build as pkg_build

HERE = pkg_build.ROOT / "tests"


def test_slices_of_any_plan_fit_their_lists(tmp_path):
    exe = tmp_path / "pending_slices_check"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{pkg_build.CSRC}", str(HERE / "pending_slices_check.cpp"), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    state, plans, full = out.stdout.split()
    assert state == "ok" and int(plans) == 4000 and int(full) > 0
