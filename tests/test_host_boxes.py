"""The rules of the mixed form's shared-memory boxes, checked by a host program
over every extent they meet (tests/box_check.cpp)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_box_rules(tmp_path):
    exe = tmp_path / "box_check"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{ROOT / 'interparts_mpich_gb300' / 'csrc'}",
                    str(ROOT / "tests" / "box_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "boxes ok" in r.stdout, r.stdout
