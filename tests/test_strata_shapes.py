"""Launch shapes of the dense-phase plan on the host against the instances the
kernels have."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "mesh-deform_gb300" / "csrc"


def test_shapes_have_kernels(tmp_path):
    exe = tmp_path / "strata_shapes"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-Wall", f"-I{CSRC}",
                    str(ROOT / "tests" / "cpp" / "strata_shapes.cpp"), str(CSRC / "arap_strata.cpp"),
                    str(CSRC / "arap_symbolic.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.endswith("ok\n")
