"""The CTA-pair GEMM (csrc/gemm_tc.cu) at the edges of its tiles: rows around the 128 of a CTA and the 256 of a pair, columns
that end inside a tile, inside a half and inside a 64-column block, one k-block and more than the ring holds, several tiles
per pair, every width that real layers get; both orders of the weight, bf16 and INT8.  The oracle is a float64 product of the
operands as the path rounds them."""
import numpy as np
import pytest

import cases

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def sgq():
    from __graft_entry__ import load_package
    return load_package()


SHAPES = [(1, 64, 32), (64, 64, 96), (127, 128, 160), (128, 192, 416), (129, 512, 288), (255, 576, 1056), (256, 1024, 4064),
          (257, 64, 22016), (300, 448, 2080), (600, 640, 9632), (2500, 256, 2592)]
# one shape per width from 96 to 256 whose last tile is partial, then 256 columns with several row tiles and several rounds
WIDE = {(200, 128, 4768): 96, (129, 128, 14240): 128, (255, 128, 21344): 160, (250, 576, 11872): 192, (100, 576, 14240): 224,
        (256, 576, 16608): 256, (513, 640, 11040): 256, (700, 1024, 17312): 256}
WIDE_I8 = {(65, 240, 4763): 96, (129, 144, 14235): 128, (255, 256, 21333): 160, (100, 592, 23701): 192, (257, 208, 23705): 224,
           (257, 592, 17787): 256}


def pair_columns(M, N, kblocks, pairs):
    """The launch's rule for the width, restated: rounds of the persistent grid times the cycles of a k-block, and the last
    tile's epilogue."""
    cost = {bn: -(-(-(-M // 256) * -(-N // bn)) // pairs) * max(2 * bn, 256 + bn) * kblocks + 16 * bn for bn in range(256, 63, -32)}
    return min(cost, key=cost.get)           # of equal ones the widest: the first in this order


def test_widths_that_the_shapes_below_take():
    """On the 148 SMs of a B200, k-blocks of 64 (bf16) and 128 (INT8)."""
    assert {s: pair_columns(s[0], s[2], -(-s[1] // 64), 74) for s in WIDE} == WIDE
    assert {s: pair_columns(s[0], s[2], -(-s[1] // 128), 74) for s in WIDE_I8} == WIDE_I8


def check(y, x, w, K):
    want = x.double() @ w.double()
    mag = x.double().abs() @ w.double().abs()
    # exact products, fp32 sums of K of them (one rounding of at most 2^-23 of the running magnitude each) and the epilogue's two
    assert bool(((y.double() - want).abs() <= mag * (K + 4) * 2.0 ** -23 + 1e-12).all())


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,N", SHAPES + list(WIDE))
def test_pair_gemm_edges(sgq, M, K, N):
    gen = torch.Generator(device="cuda").manual_seed(M * 7 + K * 3 + N)
    x = torch.randn(M, K, device="cuda", generator=gen)
    b = torch.randn(N, device="cuda", generator=gen)
    xb = x.bfloat16()
    ws = sgq.Workspace(torch.device("cuda"))
    for layout in (cases.LAYOUT_NK, cases.LAYOUT_KN):
        n = N - 3 if layout == cases.LAYOUT_NK else N               # rows of 4n bytes: also the epilogue without 128-bit stores
        w = torch.randn((n, K) if layout == cases.LAYOUT_NK else (K, n), device="cuda", generator=gen) * 0.05
        for q, deq in ((sgq.quantize_int4(w, 32), sgq.dequantize_int4),
                       (sgq.quantize_int8(w, cases.PER_ROW), sgq.dequantize_int8),
                       (sgq.quantize_int8(w, cases.PER_TENSOR), sgq.dequantize_int8)):
            real = deq(q)
            # the scales of INT8 codes stored [N,K] multiply the sums in fp32; else code * scale is rounded to bf16
            wf = real if q.qdata.dtype == torch.int8 and layout == cases.LAYOUT_NK else real.bfloat16().float()
            wf = wf.t() if layout == cases.LAYOUT_NK else wf
            for bias in (None, b[:n]):
                y = sgq.quantized_matmul(x, q, bias, layout=layout, path=sgq.PATH_TC_BF16, workspace=ws)
                assert sgq.device_status() == 0
                check(y if bias is None else y.double() - bias.double(), xb, wf, K + (0 if bias is None else 4096))


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,N", list(WIDE_I8))
def test_pair_gemm_i8_widths(sgq, M, K, N):
    """kind::i8 at the widths of real layers: the int32 sums are exact, the epilogue's two products and one sum round once each."""
    gen = torch.Generator(device="cuda").manual_seed(M + K + N)
    x = torch.randn(M, K, device="cuda", generator=gen)
    bias = torch.randn(N, device="cuda", generator=gen)
    w = torch.randn(N, K, device="cuda", generator=gen) * 0.05
    for scheme in (cases.PER_ROW, cases.PER_TENSOR):
        q = sgq.quantize_int8(w, scheme)
        for b in (bias, None):
            y, xq, sx, acc = sgq.linear_w8a8(x, q, b, want_parts=True)
            assert sgq.device_status() == 0
            assert torch.equal(acc.double(), xq.double() @ q.qdata.double().t())
            want = acc.float() * sx[:, None] * q.scales.view(1, -1)
            assert torch.equal(y, want if b is None else want + b)
            assert torch.equal(sgq.linear_w8a8(x, q, b), y)             # codes and scales of x in the call's own scratch


@pytest.mark.gpu
def test_expansion_of_2_31_steps(sgq):
    """A [K,N] weight of 2^34 codes: 2^31 steps of eight, one more than 32-bit indices hold.  x in {-1, 0, 1} and scales that are
    powers of two from 1/2 to 4: every product is a multiple of 1/2 and the sums stay below 2^23, so fp32 holds them exactly."""
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB of device memory")
    K = N = 1 << 17
    M, group = 64, 128
    gen = torch.Generator(device="cuda").manual_seed(1)
    codes = torch.randint(0, 256, (K * N // 2,), dtype=torch.uint8, device="cuda", generator=gen)
    scales = torch.exp2(torch.randint(-1, 3, (K * N // group,), device="cuda", generator=gen, dtype=torch.int32).float())
    q = sgq.QuantizedTensor(codes, scales, sgq.PER_TENSOR, (K, N), group, 4)
    x = torch.randint(-1, 2, (M, K), device="cuda", generator=gen, dtype=torch.int32).float()
    y = sgq.quantized_matmul(x, q, path=sgq.PATH_TC_BF16)
    assert sgq.device_status() == 0
    for n in (0, 1, 127, 128, 65535, 65536, 100001, N - 130, N - 1):
        nibble = (codes.view(K, N // 2)[:, n // 2] >> (4 * (n % 2))) & 0xF
        column = ((nibble.int() ^ 8) - 8).double() * scales.view(K, N // group)[:, n // group].double()
        assert torch.equal(y[:, n].double(), x.double() @ column), n
