"""The tcgen05 kernels of K-quant products (csrc/gemm_tc.cu, gemm_q6k_tc.cu) and the lines between them and their neighbours:
bits equal to the oracle's, which adds block values in the reference's x86 order.  Q6_K sums exact integers in f32, so
the cases that could break it are the largest sums, every row alignment of 210-byte blocks, and partial tiles.  Which
kernel a call takes shows in the number of launches: every route has the same bits."""
import numpy as np
import pytest

import emel_cpp_b200 as eb
from oracle import bindings as ob
from tests import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    b = eb.Backend(0)
    yield b
    b.close()


def check(be, port, t, w, k, m, x, n):
    got, want = np.full((m, n), np.nan, np.float32), np.zeros((m, n), np.float32)
    assert be.mul_mat(eb.mul_mat_op(w, t, k, m, x, n, got)), be.last_error
    assert be.sync()
    assert port.mul_mat(ob.mul_mat_op(w, t, k, m, x, n, want), route="blocks")
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), float(np.abs(got - want).max())


def extreme_blocks(t, m, k):
    """Rows of the largest and smallest codes in turn: quants all low, all high, alternating; scales at both ends."""
    n = m * k // 256
    b = np.zeros((n, eb.BLOCK_BYTES[t]), np.uint8)
    i = np.arange(n)
    quant = np.array([0x00, 0xff, 0x0f, 0xf0], np.uint8)[i % 4]
    if t == eb.Q4_K:
        b[:, 1], b[:, 3] = 0x20, 0x21                                     # d, dmin
        b[:, 4:16] = np.where(i % 3 == 2, 0x3f, 0xff).astype(np.uint8)[:, None]
        b[:, 16:] = quant[:, None]
    else:
        b[:, :192] = quant[:, None]
        b[:, 192:208] = np.array([0x80, 0x7f, 0xf8, 0x07], np.uint8)[(i // 4) % 4][:, None]
        b[:, 209] = 0x20
    return b.reshape(-1)


@pytest.mark.parametrize("t,m", [(eb.Q4_K, 136), (eb.Q6_K, 136), (eb.Q6_K, 1000)])
def test_largest_sums(be, port, t, m):
    k, n = 768, 40
    x = np.ones((k, n), np.float32)
    x[:, 1::4] = -1.0
    x[::2, 2::4] = -1.0
    x[:, 3::4] = np.where(np.arange(k) % 64 < 32, 1.0, -1.0)[:, None]
    x *= np.linspace(0.5, 2.0, n, dtype=np.float32)
    check(be, port, t, extreme_blocks(t, m, k), k, m, x, n)


@pytest.mark.parametrize("t", [eb.Q4_K, eb.Q6_K])
@pytest.mark.parametrize("k,m,n", [
    (256, 1, 32), (256, 129, 5), (1280, 127, 33), (1792, 260, 64), (3328, 128, 65), (2816, 300, 96), (768, 384, 129),
    (256, 3000, 300), (1280, 1300, 517), (1280, 300, 8), (1280, 4630, 5), (1792, 1100, 33), (2816, 400, 96),
])
def test_partial_tiles(be, port, t, k, m, n):
    check(be, port, t, synth.random_blocks(t, 3 * k + n, m, k), k, m, synth.activations_f32(k + n, k, n).reshape(k, n), n)


def one_sided(k, n):
    """Activations whose means, and sums on either side of them, are the largest that 8 bits allow: all one value, halves and
    quarters at opposite ends in several orders, one value far from the others, ramps."""
    x = np.ones((k, n), np.float32)
    i = np.arange(k)
    for j in range(n):
        x[:, j] = [np.ones(k), -np.ones(k), np.where(i % 2, 1, -1), np.where(i % 256 < 128, 1, -1), np.where(i % 256 < 192, 1, -1),
                   np.where(i % 256 < 64, 1, -1), np.where(i % 256 == 7, 1, -0.99), (i % 256) / 255.0 * 2 - 1, np.where(i % 4, 0, 1)][j % 9]
    return x * np.linspace(0.5, 2.0, n, dtype=np.float32)


@pytest.mark.parametrize("m,n", [(136, 32), (300, 33), (2400, 128), (14300, 130), (12700, 131), (2500, 1154)])
@pytest.mark.parametrize("extreme", [False, True])
def test_q4_k_tiles_of_every_width(be, port, m, n, extreme):
    """Tiles of 32 and, the last three, 128 columns, whole and ragged, with and without 16-byte rows of results.  (64: see
    test_q4_k_short_sums; 128 with a table of the rows: test_q4_k_columns_in_turns and the benchmarked shapes.)"""
    k = 512
    w = extreme_blocks(eb.Q4_K, m, k) if extreme else synth.random_blocks(eb.Q4_K, m + n, m, k)
    x = one_sided(k, n) if extreme else synth.activations_f32(m * n, k, n).reshape(k, n)
    check(be, port, eb.Q4_K, w, k, m, x, n)


@pytest.mark.parametrize("offset", [2, 6, 10, 14])
@pytest.mark.parametrize("m", [140, 525])
def test_q6_k_rows_at_even_addresses(be, port, offset, m):
    torch = pytest.importorskip("torch")
    k, n = 1280, 70
    w = synth.random_blocks(eb.Q6_K, 5, m, k)
    x = synth.activations_f32(6, k, n).reshape(k, n)
    want = np.zeros((m, n), np.float32)
    assert port.mul_mat(ob.mul_mat_op(w, eb.Q6_K, k, m, x, n, want), route="blocks")
    room = torch.zeros(w.size + 64, dtype=torch.uint8, device="cuda")
    dev_w = room[offset:offset + w.size]
    dev_w.copy_(torch.from_numpy(w.reshape(-1)))
    dev_x, dev_y = torch.from_numpy(x).cuda(), torch.zeros((m, n), device="cuda")
    torch.cuda.synchronize()
    assert be.mul_mat(eb.mul_mat_op(dev_w, eb.Q6_K, k, m, dev_x, n, dev_y)), be.last_error
    assert be.sync()
    assert np.array_equal(dev_y.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("k,m,n", [(2048, 4737, 130), (2048, 10000, 96), (10240, 130, 97), (256, 6500, 201), (1280, 9472, 192), (10496, 128, 192)])
@pytest.mark.parametrize("extreme", [False, True])
def test_q6_k_prompts(be, port, k, m, n, extreme):
    """The prompt kernel's sizes: streamed rows and others, whole and ragged tiles, rows of 8 bytes and not."""
    w = extreme_blocks(eb.Q6_K, m, k) if extreme else synth.random_blocks(eb.Q6_K, m + n, m, k)
    x = one_sided(k, n) if extreme else synth.activations_f32(m * n, k, n).reshape(k, n)
    count = launches_of(be, lambda: check(be, port, eb.Q6_K, w, k, m, x, n))
    assert count == 4      # quantizer, operand layout, slabs, product


@pytest.mark.parametrize("offset", [2, 8, 14])
def test_q6_k_prompts_at_even_addresses(be, port, offset):
    torch = pytest.importorskip("torch")
    k, m, n = 768, 6500, 194
    w = synth.random_blocks(eb.Q6_K, 5, m, k)
    x = synth.activations_f32(6, k, n).reshape(k, n)
    want = np.zeros((m, n), np.float32)
    assert port.mul_mat(ob.mul_mat_op(w, eb.Q6_K, k, m, x, n, want), route="blocks")
    room = torch.zeros(w.size + 64, dtype=torch.uint8, device="cuda")
    dev_w = room[offset:offset + w.size]
    dev_w.copy_(torch.from_numpy(w.reshape(-1)))
    dev_x, dev_y = torch.from_numpy(x).cuda(), torch.zeros((m, n), device="cuda")
    torch.cuda.synchronize()
    assert be.mul_mat(eb.mul_mat_op(dev_w, eb.Q6_K, k, m, dev_x, n, dev_y)), be.last_error
    assert be.sync()
    assert np.array_equal(dev_y.cpu().numpy().view(np.uint32), want.view(np.uint32))


def test_q6_k_prompt_rows_in_turns(monkeypatch):
    """More rows than the workspace holds unpacked: slabs and product once per turn.  Four columns equal those of the mat-vec kernels."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("EMELB_ACT_MELEMS", "1")
    b = eb.Backend(0)
    try:
        k, m, n = 256, 220000, 192
        w = torch.from_numpy(synth.random_blocks(eb.Q6_K, 9, 1000, k).reshape(1000, -1)).cuda()
        w = w[torch.arange(m, device="cuda") * 7 % 997].contiguous()
        x = torch.from_numpy(synth.activations_f32(10, k, n).reshape(k, n)).cuda()
        y, few = torch.zeros((m, n), device="cuda"), torch.zeros((m, 4), device="cuda")
        x4 = x[:, :4].contiguous()
        torch.cuda.synchronize()

        def call():
            assert b.mul_mat(eb.mul_mat_op(w, eb.Q6_K, k, m, x, n, y)), b.last_error
        assert launches_of(b, call) == 6      # quantizer, operand layout, and two turns
        assert b.mul_mat(eb.mul_mat_op(w, eb.Q6_K, k, m, x4, 4, few)), b.last_error
        assert b.sync()
        assert torch.equal(y[:, :4].contiguous().view(torch.int32), few.view(torch.int32))
    finally:
        b.close()


def launches_of(be, call):
    before = be.diagnostics()["kernel_launches"]
    call()
    return be.diagnostics()["kernel_launches"] - before


@pytest.mark.parametrize("k,m", [(2048, 70), (4096, 150), (8192, 33), (8192, 8200), (14336, 65)])
@pytest.mark.parametrize("n", [4, 5, 6, 7, 8, 9])
def test_q6_k_few_columns_of_long_aligned_rows(be, port, k, m, n):
    """K a multiple of 2048 never takes the tcgen05 kernel (quantizer, operand layout, product: three launches): behind the
    quantizer one mma.sync launch, or mat-vec launches of eight, four, two and one columns."""
    w = synth.random_blocks(eb.Q6_K, 3 * k + n, m, k)
    x = synth.activations_f32(k + n, k, n).reshape(k, n)
    count = launches_of(be, lambda: check(be, port, eb.Q6_K, w, k, m, x, n))
    few_long_rows = k >= 8192 and m < k   # the activations of eight columns do not fit beside the mat-vec kernel's rings
    assert count == 1 + {4: 1, 5: 2, 6: 2, 7: 3 if few_long_rows else 1, 8: 2 if few_long_rows else 1, 9: 1}[n]


@pytest.mark.parametrize("m,n,tc", [
    (4608, 8, True), (4600, 8, False), (4601, 5, True), (1024, 33, True), (1024, 32, False), (9300, 4, False), (8, 4609, True), (8, 4604, False),
    (1, 4609, True),
])
@pytest.mark.parametrize("k", [256, 2304])
def test_q6_k_line_to_the_mat_vec_kernel(be, port, m, n, tc, k):
    """Rows that no streaming kernel takes: the tcgen05 kernel (operand layout, product) from 9216 passes of four columns times
    rows on, one mat-vec launch below."""
    w = synth.random_blocks(eb.Q6_K, 5 * m + n, m, k)
    x = synth.activations_f32(m + n, k, n).reshape(k, n)
    assert launches_of(be, lambda: check(be, port, eb.Q6_K, w, k, m, x, n)) == (3 if tc else 2)


def device_bytes_of_a_context(monkeypatch, melems):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("EMELB_ACT_MELEMS", str(melems))
    free = torch.cuda.mem_get_info()[0]
    b = eb.Backend(0)
    held = free - torch.cuda.mem_get_info()[0]
    b.close()
    return held


def test_a_context_holds_one_copy_of_the_activations_in_operand_order(be, monkeypatch):
    """1.25 bytes an element for the quantized planes and 1.08 for the Q4_K operand; the f16 operand of Q6_K shares it."""
    grown = device_bytes_of_a_context(monkeypatch, 320) - device_bytes_of_a_context(monkeypatch, 64)
    assert grown < 2.4 * (256 << 20)


def test_q6_k_columns_in_turns(port, monkeypatch):
    """More columns than the workspace holds in f16: the operand is laid out, and the product made, once per turn."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("EMELB_ACT_MELEMS", "72")
    b = eb.Backend(0)
    try:
        k, m = 256, 3
        n = (72 << 20) // k - 5
        w = synth.random_blocks(eb.Q6_K, 9, m, k)
        x = synth.activations_f32(10, k, n).reshape(k, n)
        want = np.zeros((m, n), np.float32)
        assert port.mul_mat(ob.mul_mat_op(w, eb.Q6_K, k, m, x, n, want), route="blocks")
        dev_w, dev_x, dev_y = torch.from_numpy(w.reshape(-1)).cuda(), torch.from_numpy(x).cuda(), torch.zeros((m, n), device="cuda")
        torch.cuda.synchronize()

        def call():
            assert b.mul_mat(eb.mul_mat_op(dev_w, eb.Q6_K, k, m, dev_x, n, dev_y)), b.last_error
        assert launches_of(b, call) == 5      # quantizer, and two turns
        assert b.sync()
        assert np.array_equal(dev_y.cpu().numpy().view(np.uint32), want.view(np.uint32))
    finally:
        b.close()


def test_q4_k_columns_in_turns(port, monkeypatch):
    """More columns than the workspace holds in f16: layout, table and product once per turn."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("EMELB_ACT_MELEMS", "72")
    b = eb.Backend(0)
    try:
        k, m = 256, 3
        n = (72 << 20) // k - 5
        w = synth.random_blocks(eb.Q4_K, 9, m, k)
        x = synth.activations_f32(10, k, n).reshape(k, n)
        want = np.zeros((m, n), np.float32)
        assert port.mul_mat(ob.mul_mat_op(w, eb.Q4_K, k, m, x, n, want), route="blocks")
        dev_w, dev_x, dev_y = torch.from_numpy(w.reshape(-1)).cuda(), torch.from_numpy(x).cuda(), torch.zeros((m, n), device="cuda")
        torch.cuda.synchronize()

        def call():
            assert b.mul_mat(eb.mul_mat_op(dev_w, eb.Q4_K, k, m, dev_x, n, dev_y)), b.last_error
        assert launches_of(b, call) == 7      # quantizer, and two turns
        assert b.sync()
        assert np.array_equal(dev_y.cpu().numpy().view(np.uint32), want.view(np.uint32))
    finally:
        b.close()


@pytest.mark.parametrize("t", [eb.Q8_0, eb.Q4_0])
@pytest.mark.parametrize("k,m,n,launches", [
    (5376, 4801, 33, 3), (5120, 130, 1601, 3), (5120, 1300, 333, 3),      # one turn of tiles, ragged rows and columns
    (2304, 2500, 900, 3),                                                  # several tiles a CTA, odd turns of K
    (4096, 1300, 192, 2), (2304, 2500, 800, 2), (3840, 1300, 333, 2),      # on the other side of each line: mma.sync
    (4096, 1300, 333, {eb.Q8_0: 3, eb.Q4_0: 2}),                           # tiles for two thirds of the SMs
])
def test_q8_0_and_q4_0_prompts(be, port, t, k, m, n, launches):
    w = synth.random_blocks(t, m + n, m, k)
    x = synth.activations_f32(m * n, k, n).reshape(k, n)
    assert launches_of(be, lambda: check(be, port, t, w, k, m, x, n)) == (launches if isinstance(launches, int) else launches[t])      # quantizer, (operand layout,) product


@pytest.mark.parametrize("t", [eb.Q8_0, eb.Q4_0])
def test_q8_0_and_q4_0_prompts_largest_sums(be, port, t):
    """Quants and activations at the ends of their range; scales from subnormal to large, of either sign."""
    k, m, n = 5120, 1300, 260
    b = np.zeros((m * k // 32, eb.BLOCK_BYTES[t]), np.uint8)
    i = np.arange(len(b))
    d = np.array([2.0 ** -24, -2.0 ** -14, 0.5, -8.0, 0.0], np.float16)[i % 5]
    b[:, :2] = d.view(np.uint8).reshape(-1, 2)
    b[:, 2:] = np.array([0x80, 0x7f, 0xff, 0x00, 0x88], np.uint8)[i // 5 % 5][:, None]
    check(be, port, t, b.reshape(-1), k, m, one_sided(k, n), n)


@pytest.mark.parametrize("k,m,n", [(256, 3100, 513), (512, 4100, 515), (768, 6500, 162), (1024, 4096, 333), (1024, 14300, 97), (2048, 5700, 130), (512, 2500, 250), (768, 14300, 63)])
@pytest.mark.parametrize("extreme", [False, True])
def test_q4_k_short_sums(be, port, k, m, n, extreme):
    """Tiles of 128 and, the last three, 64 columns without a table of the rows: two launches behind the quantizer.  Odd and even
    strides."""
    w = extreme_blocks(eb.Q4_K, m, k) if extreme else synth.random_blocks(eb.Q4_K, m + n, m, k)
    x = one_sided(k, n) if extreme else synth.activations_f32(m * n, k, n).reshape(k, n)
    assert launches_of(be, lambda: check(be, port, eb.Q4_K, w, k, m, x, n)) == 3


def tiled_rows(torch, t, seed, m, k):
    """Rows 7 i % 997 of 997 random ones, on the device."""
    few = torch.from_numpy(synth.random_blocks(t, seed, 997, k).reshape(997, -1)).cuda()
    return few, few[torch.arange(m, device="cuda") * 7 % 997].contiguous()


def test_q4_k_table_larger_than_the_workspace(monkeypatch):
    """Rows whose table does not fit beside the activations: all columns in one turn, without it."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("EMELB_ACT_MELEMS", "8")
    b = eb.Backend(0)
    try:
        k, m, n = 4096, 83001, 2047
        few, w = tiled_rows(torch, eb.Q4_K, 9, m, k)
        x = torch.from_numpy(synth.activations_f32(10, k, n).reshape(k, n)).cuda()
        y, want = torch.zeros((m, n), device="cuda"), torch.zeros((997, n), device="cuda")
        torch.cuda.synchronize()

        def call():
            assert b.mul_mat(eb.mul_mat_op(w, eb.Q4_K, k, m, x, n, y)), b.last_error
        assert launches_of(b, call) == 3      # quantizer, operand layout, product
        assert b.mul_mat(eb.mul_mat_op(few, eb.Q4_K, k, 997, x, n, want)), b.last_error
        assert b.sync()
        assert torch.equal(y.view(torch.int32), want[torch.arange(m, device="cuda") * 7 % 997].view(torch.int32))
    finally:
        b.close()


@pytest.mark.parametrize("k,m,n,launches", [
    (2048, 1030, 768, 2), (2048, 2048, 512, 2), (2048, 2048, 645, 4), (2048, 2600, 250, 4),    # aligned rows: mma.sync, or the prompt kernel
    (768, 6500, 320, 3), (768, 6500, 777, 4), (1280, 2500, 700, 4), (512, 14300, 200, 3),      # others: 128 x 64 tiles, or the prompt kernel
])
def test_q6_k_line_to_the_prompt_kernel(be, port, k, m, n, launches):
    w = synth.random_blocks(eb.Q6_K, m + n, m, k)
    x = synth.activations_f32(m * n, k, n).reshape(k, n)
    assert launches_of(be, lambda: check(be, port, eb.Q6_K, w, k, m, x, n)) == launches


@pytest.mark.parametrize("offset", [2, 8, 14])
def test_q6_k_prompt_kernel_at_even_addresses(be, port, offset):
    torch = pytest.importorskip("torch")
    k, m, n = 1280, 2500, 702
    w = synth.random_blocks(eb.Q6_K, 5, m, k)
    x = synth.activations_f32(6, k, n).reshape(k, n)
    want = np.zeros((m, n), np.float32)
    assert port.mul_mat(ob.mul_mat_op(w, eb.Q6_K, k, m, x, n, want), route="blocks")
    room = torch.zeros(w.size + 64, dtype=torch.uint8, device="cuda")
    dev_w = room[offset:offset + w.size]
    dev_w.copy_(torch.from_numpy(w.reshape(-1)))
    dev_x, dev_y = torch.from_numpy(x).cuda(), torch.zeros((m, n), device="cuda")
    torch.cuda.synchronize()

    def call():
        assert be.mul_mat(eb.mul_mat_op(dev_w, eb.Q6_K, k, m, dev_x, n, dev_y)), be.last_error
    assert launches_of(be, call) == 4
    assert be.sync()
    assert np.array_equal(dev_y.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("t", [eb.Q8_0, eb.Q4_0])
def test_q8_0_and_q4_0_prompt_columns_in_turns(monkeypatch, t):
    """More columns than the workspace holds (9088): layout and product once per turn.  Columns at the turns' and tiles' ends and
    between them equal those of the mma.sync kernel."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("EMELB_ACT_MELEMS", "40")
    b = eb.Backend(0)
    try:
        k, m, n = 4096, 130, 10001
        w = torch.from_numpy(synth.random_blocks(t, 9, m, k)).cuda()
        x = torch.randn((k, n), device="cuda", generator=torch.Generator("cuda").manual_seed(3))
        at = torch.tensor([0, 1, 63, 64, 4000, 4001, 9023, 9086, 9087, 9088, 9089, 9151, 9152, 9900, 9983, 9984, 9999, 10000], device="cuda")
        some = x[:, at].contiguous()
        y, want = torch.zeros((m, n), device="cuda"), torch.zeros((m, len(at)), device="cuda")
        torch.cuda.synchronize()

        def call():
            assert b.mul_mat(eb.mul_mat_op(w, t, k, m, x, n, y)), b.last_error
        assert launches_of(b, call) == 5      # quantizer, and two turns
        assert launches_of(b, lambda: b.mul_mat(eb.mul_mat_op(w, t, k, m, some, len(at), want))) == 2
        assert b.sync()
        assert torch.equal(y[:, at].contiguous().view(torch.int32), want.view(torch.int32)) and bool(want.any())
    finally:
        b.close()


def test_q6_k_prompt_columns_and_rows_in_turns(monkeypatch):
    """Columns that fill the workspace but for one tile row of unpacked weights: three turns of rows, then the other columns with
    all rows at once.  Columns at the turns' and tiles' ends equal those of the kernels for few columns."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("EMELB_ACT_MELEMS", "72")
    b = eb.Backend(0)
    try:
        k, m = 256, 300
        n = (72 << 20) // k - 5               # 268928 columns and 25979
        w = torch.from_numpy(synth.random_blocks(eb.Q6_K, 9, m, k)).cuda()
        x = torch.randn((k, n), device="cuda", generator=torch.Generator("cuda").manual_seed(4))
        at = torch.tensor([0, 63, 64, 127, 128, 100000, 268863, 268927, 268928, 268929, 269055, 269056, n - 2, n - 1], device="cuda")
        some = x[:, at].contiguous()
        y, want = torch.zeros((m, n), device="cuda"), torch.zeros((m, len(at)), device="cuda")
        torch.cuda.synchronize()

        def call():
            assert b.mul_mat(eb.mul_mat_op(w, eb.Q6_K, k, m, x, n, y)), b.last_error
        assert launches_of(b, call) == 1 + (1 + 2 * 3) + (1 + 2)      # quantizer; layout, and slabs and product of each turn of rows
        assert b.mul_mat(eb.mul_mat_op(w, eb.Q6_K, k, m, some, len(at), want)), b.last_error
        assert b.sync()
        assert torch.equal(y[:, at].contiguous().view(torch.int32), want.view(torch.int32)) and bool(want.any())
    finally:
        b.close()


@pytest.mark.parametrize("t,k,n,launches", [(eb.Q8_0, 2304, 901, 3), (eb.Q4_0, 2304, 901, 2), (eb.Q4_0, 2304, 902, 2), (eb.Q4_0, 2304, 904, 3),
                                            (eb.Q4_0, 3072, 901, 3)])
def test_q8_0_and_q4_0_prompts_of_other_strides(be, port, t, k, n, launches):
    """Rows of results that are no multiple of 16 bytes: short Q4_0 sums stay on mma.sync."""
    m = 2500
    w = synth.random_blocks(t, m + n, m, k)
    x = synth.activations_f32(m * n, k, n).reshape(k, n)
    assert launches_of(be, lambda: check(be, port, t, w, k, m, x, n)) == launches
