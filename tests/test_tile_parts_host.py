"""CPU test of the part sums' sizes (csrc/tile_parts.h): what the server sets
aside covers the node counts of measured trees."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_tile_part_sizes(tmp_path):
    exe = tmp_path / "tile_parts_test"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'simplefmm_b200/csrc'}",
                    str(ROOT / "tests/native/tile_parts_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "tile parts ok" in r.stdout, r.stdout
