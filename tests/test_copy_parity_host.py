"""CPU test of the phases a giving-up kernel waits for (csrc/copy_parity.h):
barriers whose copies have landed cost one poll, the others are waited for, and
the waits' parities at any point of a pass give the issues'."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_copy_parity(tmp_path):
    exe = tmp_path / "copy_parity_test"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{ROOT / 'simplefmm_b200/csrc'}",
                    str(ROOT / "tests/native/copy_parity_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "copy parity ok" in r.stdout, (r.returncode, r.stdout)
