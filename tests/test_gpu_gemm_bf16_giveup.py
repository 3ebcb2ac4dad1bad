"""What the bf16 tile kernels do when a wait runs out: the CTA, or both of a pair, stop, the copies and MMAs in flight end before the
memory goes to the next launch, and the status word says so.  The waits run out by a host program's choice (the kernel's source,
compiled with a condition in front of them); nothing faults or hangs."""
import os
import subprocess
import tempfile

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_every_role_may_give_up_anywhere():
    exe = os.path.join(tempfile.mkdtemp(), "gemm_bf16_giveup")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-o", exe,
                    os.path.join(HERE, "gemm_bf16_giveup_harness.cu")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    tried, complaints = (int(v) for v in out.stdout.split()[-2:])
    assert out.returncode == 0 and tried > 100 and complaints == 0, out.stdout
