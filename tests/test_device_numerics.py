"""The device code's arithmetic on FP32 and FP64 bit patterns
(csrc/arap_device.cuh) compiled for the host."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "mesh-deform_gb300" / "csrc"


@pytest.mark.parametrize("name", ["conversions", "split_difference"])
def test_on_the_host(tmp_path, name):
    import build_lib

    exe = tmp_path / name
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Wno-unknown-pragmas", f"-I{CSRC}",
                    f"-I{build_lib.cuda_include()}", str(ROOT / "tests" / "cpp" / f"{name}.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.endswith("ok\n")
