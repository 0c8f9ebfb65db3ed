"""The tensor-core decode kernel for weights stored [K,N] (csrc/linear_kn.cu) against a float64 product: every padded
batch size, both feature widths of a CTA, ragged K and N, one and several slices of K, groups wider than 32."""
import numpy as np
import pytest

import cases
from util import TOL_FP32, heavy_tailed_rows, rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sgq():
    from __graft_entry__ import load_package
    return load_package()


SHAPES = [(1, 64, 32, 32), (1, 1024, 1024, 32), (2, 4096, 11008, 32), (2, 68, 96, 96), (3, 1000, 416, 32), (4, 8192, 1024, 128),
          (4, 60, 256, 64), (5, 2048, 4160, 32), (8, 4096, 288, 32), (9, 516, 12800, 64), (13, 2052, 160, 32), (16, 4096, 4096, 128)]


@pytest.mark.parametrize("M,K,N,group", SHAPES)
def test_kn_tensor_core_decode(sgq, port, M, K, N, group):
    rng = np.random.default_rng(M * 131 + K + N)
    x = heavy_tailed_rows(M + N, M, K, 300.0, 2) * rng.uniform(0.01, 50.0, (M, 1)).astype(np.float32)
    w = cases.weight_with_outliers(K + N, (K, N))
    b = (rng.standard_normal(N) * 0.1).astype(np.float32)
    xd, wd, bd = (torch.from_numpy(a).cuda() for a in (x, w, b))
    ws = sgq.Workspace(torch.device("cuda"))
    runs = [(sgq.quantize_int4(wd, group), port.dequantize_int4(*port.quantize_int4(w, group), (K, N), group))]
    for scheme in (cases.PER_TENSOR, cases.PER_ROW):
        runs.append((sgq.quantize_int8(wd, scheme), port.dequantize_int8(*port.quantize_int8(w, scheme), scheme).reshape(K, N)))
    for q, deq in runs:
        for bias in (bd, None):
            y = sgq.quantized_matmul(xd, q, bias, layout=cases.LAYOUT_KN, workspace=ws).cpu().numpy()
            assert sgq.device_status() == 0
            # fp32: factors x * s rounded once, products with the codes exact, K / 16 accumulations of at most 2^-23 of the sums
            # of absolute products each
            xf = x.astype(np.float64)
            want = xf @ deq.astype(np.float64) + (b[None, :] if bias is not None else 0.0)
            mag = np.abs(xf) @ np.abs(deq.astype(np.float64))
            assert np.all(np.abs(y - want) <= mag * (K / 16 + 8) * 2.0 ** -23 + 1e-6), (M, K, N, np.max(np.abs(y - want) / mag))
            assert rel_err(y, want) <= TOL_FP32
        again = sgq.quantized_matmul(xd, q, None, layout=cases.LAYOUT_KN, workspace=ws).cpu().numpy()
        assert np.array_equal(again, y)                     # slices of K are added in a fixed order
    xd[M - 1, K // 2] = float("nan")
    y = sgq.quantized_matmul(xd, runs[0][0], None, layout=cases.LAYOUT_KN, workspace=ws)
    assert torch.isnan(y[M - 1]).all() and torch.isfinite(y[: M - 1]).all()


EXTREMES = ["inf", "-inf", "both", "nan", "huge", "tiny"]


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("kind", EXTREMES)
def test_kn_decode_non_finite_and_extreme_activations(sgq, M, kind):
    """Factors x * s that the three bf16 parts do not hold: Inf, NaN, a finite one above bf16's largest value, and a row of
    factors whose parts lie below bf16's smallest.  Codes with zeros among them, every scale exactly 1; +-Inf and NaN per
    output as in the reference's fp32 chain, the other rows the same bits as without that row."""
    K, N = 520, 288
    gen = torch.Generator(device="cuda").manual_seed(M)
    w = torch.randint(-7, 8, (K, N), device="cuda", generator=gen).float()
    w[:, ::32] = 7.0                                        # every scale is exactly 1
    w8 = torch.randint(-127, 128, (K, N), device="cuda", generator=gen).float() * (torch.rand(K, N, device="cuda", generator=gen) < 0.9)
    w8[:, 0] = 127.0
    x = torch.randn(M, K, device="cuda", generator=gen)
    clean, m = x.clone(), M - 1
    if kind == "huge":
        x[m] = 0.0
        x[m, 77] = 3.4e38                                   # above the largest bf16 value
    elif kind == "tiny":
        x[m] *= 1e-37
    elif kind == "both":
        x[m, 3], x[m, 400] = float("inf"), float("-inf")
    else:
        x[m, 77] = float(kind)
    ws = sgq.Workspace(x.device)
    runs = [(sgq.quantize_int4(w, 32), w), (sgq.quantize_int8(w8, sgq.PER_ROW), w8), (sgq.quantize_int8(w8, sgq.PER_TENSOR), w8)]
    bias = torch.randn(N, device="cuda", generator=gen)
    for q, deq in runs:
        for b in (None, bias):
            y = sgq.quantized_matmul(x, q, b, layout=sgq.LAYOUT_KN, path=sgq.PATH_GEMV, workspace=ws)
            y_clean = sgq.quantized_matmul(clean, q, b, layout=sgq.LAYOUT_KN, path=sgq.PATH_GEMV, workspace=ws)
            assert sgq.device_status() == 0
            assert torch.equal(y[:m], y_clean[:m])          # rows do not mix
            terms = x[m].double()[:, None] * deq.double()
            want = terms.sum(0) + (0.0 if b is None else b.double())
            got, want32 = y[m], want.float()
            assert torch.equal(torch.isnan(got), torch.isnan(want32)), kind
            assert torch.equal(torch.isinf(got), torch.isinf(want32)) and torch.equal(got[got.isinf()], want32[want32.isinf()])
            fin = torch.isfinite(want32)
            mag = terms.abs().sum(0) + (0.0 if b is None else b.abs().double())
            err = (got.double() - want).abs()               # one rounding of the running sum per term, or of the smallest subnormal
            assert bool((err <= mag * (K + 8) * 2.0 ** -23 + K * 2.0 ** -149)[fin].all()), (kind, float((err / mag)[fin].max()))


@pytest.mark.parametrize("M", [1, 3, 16, 40, 128])
def test_kn_forward_in_place(sgq, M):
    """The output may be the activations' own buffer (K == N): every launch that stores it starts behind the ones that read x.
    Up to 63 rows the bits are those of the any-shape form, which is what an overlapping output takes; a view that starts four
    bytes off a row is one that the tensor-core form does not take either."""
    K = N = 512
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, device="cuda", generator=gen)
    w = torch.randn(K, N, device="cuda", generator=gen) * 0.05
    ws = sgq.Workspace(x.device)
    for q in (sgq.quantize_int4(w, 32), sgq.quantize_int8(w, sgq.PER_ROW)):
        apart = sgq.quantized_matmul(x, q, workspace=ws)
        shifted = torch.empty(M * K + 1, device="cuda")[1:].view(M, K)
        shifted.copy_(x)
        other = sgq.quantized_matmul(shifted, q, workspace=ws) if M < 64 else apart
        for _ in range(20):
            buf = x.clone()
            got = sgq.quantized_matmul(buf, q, out=buf, workspace=ws)
            assert got is buf and torch.equal(got, other)
        assert rel_err(got.cpu().numpy(), apart.cpu().numpy()) <= 1e-5
    assert sgq.device_status() == 0
