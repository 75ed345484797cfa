"""mm8_seq on tcgen05 kind::i8 (csrc/mm8_seq_i8.cu): the edges of its tiles, K blocks, splits and forms."""
import ctypes

import pytest
import torch

from oracle import rwkv_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from chatrwkv_b200 import ops as o
    return o


def _error_word(ops):
    from chatrwkv_b200 import _lib
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), 1024, "mm8_seq")
    e = ctypes.c_int(-1)
    assert _lib.lib().rwkv_mm8_seq_tc_take_error(ws.data_ptr(), None, ctypes.byref(e)) == 0
    return e.value


# rows around the tile sizes (16 / 32 up to 128) and the one-CTA / CTA-pair boundary, in-features around the K block of 128
# and past the one-chunk-per-thread preparation, out-features that are no multiple of 8 or 128, and more tiles than CTAs
@pytest.mark.parametrize("T,N,M", [(2, 16, 8), (15, 127, 277), (16, 128, 128), (17, 129, 129), (32, 640, 4096), (33, 4096, 1000),
                                   (64, 2048, 256), (65, 300, 50277), (96, 256, 2304), (127, 1024, 640), (129, 512, 384),
                                   (300, 384, 9000), (3, 16400, 200), (40, 20480, 136)])
def test_edges_against_oracle_and_one_cta_form(ops, T, N, M):
    from chatrwkv_b200 import _lib
    from tests.util import packed_case
    cpu, dev = packed_case(N, M, seed=T + N + M)
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, N, generator=g).half()
    y = torch.full((T, M), float("nan"), dtype=torch.float16, device="cuda")
    torch.ops.rwkv.mm8_seq(T, N, M, x.cuda(), *dev, y)
    _lib.lib().rwkv_mm8_seq_set_path(8)
    try:
        y1 = torch.full((T, M), float("nan"), dtype=torch.float16, device="cuda")
        torch.ops.rwkv.mm8_seq(T, N, M, x.cuda(), *dev, y1)
    finally:
        _lib.lib().rwkv_mm8_seq_set_path(0)
    torch.cuda.synchronize()
    assert _error_word(ops) == 0
    assert torch.equal(y, y1)                       # exact integer sums: no dependence on the form or the K split
    ref = orc.mm8_kernel(x, *cpu)
    # one rounding to fp16 (2^-11 relative), and fp32 terms of a few times the result's size
    assert ((y.float().cpu() - ref).abs() <= ref.abs() * 2 ** -10 + 1e-4).all()


def test_non_finite_rows_stay_in_their_row(ops):
    from tests.util import packed_case
    T, N, M = 40, 512, 300
    cpu, dev = packed_case(N, M, seed=2)
    x = torch.randn(T, N, generator=torch.Generator().manual_seed(3)).half()
    ref = orc.mm8_kernel(x, *cpu)
    bad = x.clone()
    bad[5, 17], bad[33, 500] = float("nan"), float("-inf")
    bad[7] = 0
    y = torch.empty((T, M), dtype=torch.float16, device="cuda")
    torch.ops.rwkv.mm8_seq(T, N, M, bad.cuda(), *dev, y)
    y = y.float().cpu()
    assert not torch.isfinite(y[[5, 33]]).any()
    assert (y[7] == 0).all()
    rest = [t for t in range(T) if t not in (5, 7, 33)]
    assert ((y[rest] - ref[rest]).abs() <= ref[rest].abs() * 2 ** -10 + 1e-4).all()


@pytest.mark.parametrize("magnitude", [6e-8, 1e-3, 3e4])
def test_range_of_the_fixed_point_scale(ops, magnitude):
    """The power-of-two scale follows the row: subnormal and huge activations keep their relative accuracy."""
    from tests.util import packed_case
    T, N, M = 16, 256, 128
    cpu, dev = packed_case(N, M, seed=4)
    x = (torch.randn(T, N, generator=torch.Generator().manual_seed(5)).clamp(-2, 2) * magnitude).half()
    ref = orc.mm8_kernel(x, *cpu)
    y = torch.empty((T, M), dtype=torch.float16, device="cuda")
    torch.ops.rwkv.mm8_seq(T, N, M, x.cuda(), *dev, y)
    scale = ref.abs().max().item()
    ok = (y.float().cpu() - ref.half().float()).abs() <= ref.abs() * 2 ** -10 + max(scale * 1e-5, 6e-8)
    assert ok[ref.abs() < 6e4].all()


# forms: few rows with a K split, pairs of 64 / 96 / 128 tokens with several tiles a CTA, rows read twice (N past one chunk per thread)
@pytest.mark.parametrize("T,N,M", [(2, 640, 264), (16, 4096, 512), (16, 1024, 40000), (32, 4096, 1000), (40, 4096, 1000), (130, 4096, 640),
                                   (256, 4096, 9728), (500, 2048, 300), (5, 20480, 136)])
def test_wide_rows_keep_what_an_outlier_dwarfs(ops, T, N, M):
    """A row with one huge element: the rest keeps its bits (a fourth digit), which shows in columns whose weight there is zero.
    W = (q - 128) / 4096 exactly; the other elements are multiples of 2^-8, so that all fp32 row sums are exact."""
    from chatrwkv_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(T + N + M)
    q = torch.zeros((N, ops.padded_stride(M)), dtype=torch.uint8, device="cuda")[:, :M]
    q.copy_(torch.randint(0, 256, (N, M), generator=g, device="cuda"))
    q[7] = 128
    c = lambda n, v: torch.full((n,), v, dtype=torch.float16, device="cuda")
    pack = (q, c(M, -128.5 / 4096), c(M, 2.0 ** -10), c(N, 0.0), c(N, 0.25))
    x = (torch.randn(T, N, generator=g, device="cuda") * 256).round().div(256).clamp(-4, 4).half()
    plain, wide = x.clone(), sorted({1, T // 2, T - 1})
    x[wide, 7] = 60000.0

    def run(a):
        y = torch.full((T, M), float("nan"), dtype=torch.float16, device="cuda")
        torch.ops.rwkv.mm8_seq(T, N, M, a, *pack, y)
        return y
    y = run(x)
    ref = (x.double() @ (q.double() - 128)) / 4096
    # the store's rounding, and one fp32 rounding of mx * SX = 1882 (half a step: 2^-14); three digits alone miss by 1e-2
    assert ((y.double() - ref).abs() <= ref.abs() * 2 ** -11 * 1.001 + 2 ** -13)[wide].all()
    others = [t for t in range(T) if t not in wide]
    assert torch.equal(y[others], run(plain)[others])           # a wide row changes no other row
    _lib.lib().rwkv_mm8_seq_set_path(8)
    try:
        assert torch.equal(y, run(x))                           # one CTA per tile: the same bits
    finally:
        _lib.lib().rwkv_mm8_seq_set_path(0)
    assert _error_word(ops) == 0
