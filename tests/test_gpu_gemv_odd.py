"""Mat-vec products whose K is no multiple of 2048 (csrc/gemv2.cu, gemv_odd_kernel): bits equal to the oracle's, over one
block, the 32 blocks of a turn and its edges, odd rows, several columns, rows at every even address, a residual-free sum."""
import numpy as np
import pytest

import emel_cpp_b200 as eb
from oracle import bindings as ob
from tests import synth

pytestmark = pytest.mark.gpu
TYPES = [eb.Q4_K, eb.Q6_K, eb.Q8_0, eb.Q4_0]


@pytest.fixture(scope="module")
def be():
    b = eb.Backend(0)
    yield b
    b.close()


def operands(port, t, k, m, n):
    w = synth.random_blocks(t, 7 * k + m, m, k)
    x = synth.activations_f32(k + n, k, n).reshape(k, n)
    want = np.zeros((m, n), np.float32)
    assert port.mul_mat(ob.mul_mat_op(w, t, k, m, x, n, want), route="blocks")
    return w, x, want


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("blocks,m,n", [
    (1, 1, 1), (3, 5, 1), (31, 9, 2), (32, 16, 3), (33, 8, 4), (43, 2500, 1), (65, 7, 4), (127, 3, 1),
])
def test_blocks_of_a_row(be, port, t, blocks, m, n):
    k = blocks * eb.BLOCK_ELEMS[t]
    w, x, want = operands(port, t, k, m, n)
    got = np.full((m, n), np.nan, np.float32)
    assert be.mul_mat(eb.mul_mat_op(w, t, k, m, x, n, got)), be.last_error
    assert be.sync()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("t", [eb.Q8_0, eb.Q4_0])
@pytest.mark.parametrize("blocks,m,n", [(33, 130, 8), (35, 70, 9), (129, 33, 70), (1023, 5, 17)])
def test_many_columns_of_odd_rows(be, port, t, blocks, m, n):
    test_blocks_of_a_row(be, port, t, blocks, m, n)


@pytest.mark.parametrize("t", [eb.Q6_K, eb.Q8_0, eb.Q4_0])
@pytest.mark.parametrize("offset", [2, 8, 14])
def test_rows_at_even_addresses(be, port, t, offset):
    torch = pytest.importorskip("torch")
    k, m, n = 43 * eb.BLOCK_ELEMS[t], 21, 1
    w, x, want = operands(port, t, k, m, n)
    room = torch.zeros(w.size + 64, dtype=torch.uint8, device="cuda")
    dev_w = room[offset:offset + w.size]
    dev_w.copy_(torch.from_numpy(w.reshape(-1)))
    dev_x, dev_y = torch.from_numpy(x).cuda(), torch.zeros((m, n), device="cuda")
    torch.cuda.synchronize()
    assert be.mul_mat(eb.mul_mat_op(dev_w, t, k, m, dev_x, n, dev_y)), be.last_error
    assert be.sync()
    assert np.array_equal(dev_y.cpu().numpy().view(np.uint32), want.view(np.uint32))
