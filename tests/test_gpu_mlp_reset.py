"""The closure's calls across a device reset, as a program of its own
(mlp_reset_check.cu): blocks allocated after the reset are never written or
freed by a later call or by the end of a thread that called before it.  And
more calls at a time than there are kept blocks."""
import subprocess
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from des_gb300 import closure
from des_gb300.build import ARCH, BUILD, INCLUDE, ROOT, _nvcc


@pytest.mark.gpu
def test_blocks_after_a_reset_are_the_programs(gpu):
    exe = BUILD / "mlp_reset_check"
    subprocess.run([_nvcc(), "-O1", "-std=c++17", ARCH, f"-I{INCLUDE}", str(ROOT / "tests" / "mlp_reset_check.cu"),
                    str(BUILD / "des_mlp.cu.o"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


@pytest.mark.gpu
def test_more_calls_at_a_time_than_kept_blocks(gpu):
    cases = []
    for k in range(24):
        rng = np.random.default_rng(k)
        x = np.zeros((2000 + k, 16), np.float32)
        x[:, :14] = rng.normal(0, 1, (len(x), 14))
        cases.append((closure.new_net(k), x))
    want = [closure.forward(net, x) for net, x in cases]
    with ThreadPoolExecutor(24) as ex:
        for _ in range(3):
            got = list(ex.map(lambda c: closure.forward(*c), cases))
            assert all(np.array_equal(a, b) for a, b in zip(got, want))
