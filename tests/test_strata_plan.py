"""The dense-phase solve plan on the host (csrc/arap_strata.h): groups, tiles,
update lists and inversion items against the solution of the factorised
system, with the kernels' index arithmetic."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "mesh-deform_gb300" / "csrc"


def test_plan_solves_the_system(tmp_path):
    exe = tmp_path / "strata_plan"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-Wall", f"-I{CSRC}",
                    str(ROOT / "tests" / "cpp" / "strata_plan.cpp"), str(CSRC / "arap_strata.cpp"),
                    str(CSRC / "arap_symbolic.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.endswith("ok\n")
