"""CPU test of the tensor-core M2L's shared operator rows (csrc/i8_ops.h)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "simplefmm_b200" / "csrc"


def test_i8_shared_rows(tmp_path):
    exe = tmp_path / "i8_shared_test"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{CSRC}", f"-I{ROOT / 'include'}",
                    str(ROOT / "tests/native/i8_shared_test.cpp"), str(CSRC / "tables.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "i8 shared ok" in r.stdout, r.stdout
