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
