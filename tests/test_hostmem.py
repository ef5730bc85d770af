"""pages_ready, which brings ordinary host rows into memory before kernels read
or write them in place and keeps kernels from those the program itself may not
access (csrc/des_hostmem.h)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "dynearthsol-old_gb300" / "csrc"
BUILD = ROOT / "dynearthsol-old_gb300" / "_build"


def test_pages_ready():
    BUILD.mkdir(exist_ok=True)
    exe = BUILD / "hostmem_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", f"-I{CSRC}", str(ROOT / "tests" / "hostmem_check.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "0 mismatches\n", r.stdout
