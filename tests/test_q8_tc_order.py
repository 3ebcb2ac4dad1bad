"""The waits of the Q8_0 / Q4_0 prompt kernel's MMA warps (emel.cpp_b200/csrc/q8_tc_order.h, the source the kernel compiles):
over every interleaving of producers, MMA warps and epilogue, an MMA reads the operands of its own pair, and the roles come to
their end.  The other order of the same waits, which a timing hid on the device, is seen to fail here."""
import os
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def walk():
    exe = os.path.join(tempfile.mkdtemp(), "q8_tc_order")
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", exe, os.path.join(HERE, "q8_tc_order_harness.cc")], check=True)

    def run(*args):
        out = subprocess.run([exe, *args], check=True, capture_output=True, text=True)
        return [int(v) for v in out.stdout.split()]
    return run


def test_every_mma_reads_its_own_operands(walk):
    states, wrong, ends, stuck = walk()
    assert states > 1000 and wrong == 0 and ends == 1 and stuck == 0


def test_operands_first_is_seen_to_fail(walk):
    assert walk("ad")[1] > 0
    assert walk("da")[1:] == [0, 1, 0]
