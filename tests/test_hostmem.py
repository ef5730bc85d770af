"""pages_present and pages_allow, which decide whether ordinary host rows are
read and written in place (untouched pages come in one GPU fault at a time, and
a store to a page that the program may not write would end the context)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "dynearthsol-old_gb300" / "csrc"
BUILD = ROOT / "dynearthsol-old_gb300" / "_build"


def test_pages_present():
    BUILD.mkdir(exist_ok=True)
    exe = BUILD / "hostmem_check"
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{CSRC}", str(ROOT / "tests" / "hostmem_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "0 mismatches\n", r.stdout
