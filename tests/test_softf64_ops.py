"""The grouped integer-pipe product and the quotient of the FP64 element and
node passes (csrc/des_softf64.cuh), bit for bit against the host's IEEE
arithmetic at the edges of their range; the GPU's own FP64 unit is compared in
test_softf64.py through des_gpu_softf64_check."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "dynearthsol-old_gb300" / "csrc"
BUILD = ROOT / "dynearthsol-old_gb300" / "_build"


def test_host_bit_identical_to_ieee():
    BUILD.mkdir(exist_ok=True)
    exe = BUILD / "softf64_ops_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{CSRC}",
                    str(ROOT / "tests" / "softf64_ops_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), "300000"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.count(" 0 mismatches") == r.stdout.count("\n"), r.stdout
