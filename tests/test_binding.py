"""The native calls of the Python package (csrc/torch_binding.cpp): what they refuse, and what they read of the objects they
are given.  Shapes are checked before the device, so the refusals need no GPU."""
import pytest

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def sgq():
    from __graft_entry__ import load_package
    return load_package()


def int8_weight(sgq, shape):
    n = 1
    for d in shape:
        n *= d
    return sgq.QuantizedTensor(torch.zeros(shape, dtype=torch.int8), torch.ones(shape[0]), sgq.PER_ROW, shape, n, 8)


def test_w8a8_refuses_weights_that_are_not_int8_matrices(sgq):
    """A weight of three dimensions must not be read as the matrix of its first two."""
    for shape in ((2, 16, 4), (32,), (2, 16, 1, 1)):
        with pytest.raises(RuntimeError, match="2D"):
            sgq.linear_w8a8(torch.zeros(3, 16), int8_weight(sgq, shape))
    packed = sgq.QuantizedTensor(torch.zeros(2 * 16 // 2, dtype=torch.uint8), torch.ones(1), sgq.PER_TENSOR, (2, 16), 32, 4)
    with pytest.raises(RuntimeError, match="INT8"):
        sgq.linear_w8a8(torch.zeros(3, 16), packed)


def test_w8a8_refuses_operands_that_do_not_fit_the_weight(sgq):
    """Narrower activations or a short bias would be read past their end."""
    q = int8_weight(sgq, (8, 32))
    for x in (torch.zeros(32), torch.zeros(1, 3, 32)):
        with pytest.raises(RuntimeError, match="2D"):
            sgq.linear_w8a8(x, q)
    for k in (16, 48):
        with pytest.raises(RuntimeError, match="inner dimensions"):
            sgq.linear_w8a8(torch.zeros(3, k), q)
    for n in (1, 7, 9):
        with pytest.raises(RuntimeError, match="broadcasting"):
            sgq.linear_w8a8(torch.zeros(3, 32), q, torch.zeros(n))
    with pytest.raises(ValueError, match="CUDA"):                     # everything fits: the device is what is left to refuse
        sgq.linear_w8a8(torch.zeros(3, 32), q, torch.zeros(8))


@pytest.mark.gpu
def test_scratch_comes_from_the_workspace_objects_own_get(sgq):
    """A caller's workspace is asked through get(), whether it derives from Workspace and overrides it or only has it; one that
    has nothing to give leaves the call without scratch."""
    x, w = torch.randn(2, 256, device="cuda"), torch.randn(256, 96, device="cuda")
    q = sgq.quantize_int4(w, 32)
    want = sgq.quantized_matmul(x, q)
    asked = []

    class Derived(sgq.Workspace):
        def get(self, nbytes):
            asked.append(nbytes)
            return super().get(nbytes)

    class Duck:
        def get(self, nbytes):
            asked.append(nbytes)
            return torch.empty(nbytes + 64, dtype=torch.uint8, device="cuda")

    for ws in (Derived(x.device), Duck()):
        asked.clear()
        for _ in range(3):
            assert torch.equal(sgq.quantized_matmul(x, q, workspace=ws), want)
        assert asked == [sgq.linear_workspace_bytes(4, 2, 256, 96, sgq.LAYOUT_KN)] * 3

    class Nothing:
        def get(self, nbytes):
            return None

    serial = sgq.quantized_matmul(x, q, path=sgq.PATH_SIMT)
    assert torch.equal(sgq.quantized_matmul(x, q, workspace=Nothing()), serial)
    assert torch.equal(sgq.quantized_matmul_backward_x(want, q, workspace=Nothing()), sgq.quantized_matmul_backward_x(want, q, path=sgq.PATH_SIMT))


@pytest.mark.gpu
def test_fields_that_a_bit_width_does_not_use_are_not_read(sgq):
    """INT4 has no scheme and INT8 no group: what a checkpoint loader left there does not matter."""
    x, w = torch.randn(2, 256, device="cuda"), torch.randn(256, 96, device="cuda")
    q4, q8 = sgq.quantize_int4(w, 32), sgq.quantize_int8(w)
    bare4 = sgq.QuantizedTensor(q4.qdata, q4.scales, None, (256, 96), 32, 4)
    bare8 = sgq.QuantizedTensor(q8.qdata, q8.scales, sgq.PER_ROW, (256, 96), None, 8)
    for q, bare, deq in ((q4, bare4, sgq.dequantize_int4), (q8, bare8, sgq.dequantize_int8)):
        assert torch.equal(sgq.quantized_matmul(x, bare), sgq.quantized_matmul(x, q))
        assert torch.equal(deq(bare), deq(q))
    assert torch.equal(sgq.linear_w8a8(x[:, :96].contiguous(), bare8), sgq.linear_w8a8(x[:, :96].contiguous(), q8))
