"""The local step's rotation fits (csrc/arap_device.cuh) compiled for the host,
over conditionings down to 1e-7 and both signs of the determinant."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "mesh-deform_gb300" / "csrc"


def test_fits_against_the_covariances_rotation(tmp_path):
    import build_lib

    exe = tmp_path / "rotation_fit"
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Wno-unknown-pragmas", f"-I{CSRC}",
                    f"-I{build_lib.cuda_include()}", str(ROOT / "tests" / "cpp" / "rotation_fit.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.endswith("ok\n")
