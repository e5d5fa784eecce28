"""Host side of the product of unaligned rows, with the library replaced by a recorder (no GPU)."""
import pytest
import torch

from basedxl_b200 import _lib, ops
from basedxl_b200.cascaded_lowp_matmul import cascaded_lowp_matmul


class _Recorder:
    """Stands for the loaded library: remembers the arguments of the launch."""

    def __init__(self):
        self.calls = []

    def bxl_gemm_ragged_workspace_bytes(self, M, N, K):
        return 2 * (M * ((K + 7) // 8 * 8) + K * ((N + 7) // 8 * 8))

    def bxl_gemm_ragged_f16(self, *args):
        self.calls.append(args)
        return 0


@pytest.fixture
def recorder(monkeypatch):
    rec = _Recorder()
    monkeypatch.setattr(_lib, "lib", lambda: rec)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "_f16_cuda", lambda t, name: ops._req(t.dtype == torch.float16, f"{name}: expected fp16"))
    return rec


def _h(*shape):
    return torch.zeros(*shape, dtype=torch.float16)


@pytest.mark.parametrize(
    "what,kw",
    [
        ("sliced b", {"b": _h(7, 20)[:, :9]}),
        ("transposed b", {"b": _h(9, 7).t()}),
        ("expanded b", {"b": _h(1, 9).expand(7, 9)}),
        ("one-dimensional b", {"b": _h(7)}),
        ("transposed a", {"a": _h(7, 5).t()}),
        ("every second column of a", {"a": _h(5, 14)[:, ::2]}),
        ("three-dimensional a", {"a": _h(1, 5, 7)}),
        ("residual of another shape", {"residual": _h(5, 8)}),
        ("transposed residual", {"residual": _h(9, 5).t()}),
        ("fp32 residual", {"residual": _h(5, 9).float()}),
        ("bias of another length", {"bias": _h(8)}),
        ("bias of another rank", {"bias": _h(1, 9)}),
        ("every second value of bias", {"bias": _h(18)[::2]}),
        ("fp32 bias", {"bias": _h(9).float()}),
        ("bias on another device", {"bias": torch.zeros(9, dtype=torch.float16, device="meta")}),
        ("residual on another device", {"residual": torch.zeros(5, 9, dtype=torch.float16, device="meta")}),
        ("b on another device", {"b": torch.zeros(7, 9, dtype=torch.float16, device="meta")}),
    ],
)
def test_operands_that_the_kernel_would_misread_are_refused(recorder, what, kw):
    with pytest.raises(ValueError):
        ops.gemm_ragged(**{"a": _h(5, 7), "b": _h(7, 9), **kw})
    assert not recorder.calls, what


@pytest.mark.parametrize(
    "kw,lda,ldr",
    [
        ({}, 7, 0),
        ({"a": _h(1, 7).expand(5, 7)}, 0, 0),
        ({"a": _h(5, 12)[:, 3:10]}, 12, 0),
        ({"residual": _h(1, 9).expand(5, 9), "bias": _h(11)[1:10]}, 7, 0),
        ({"residual": _h(5, 17)[:, 2:11]}, 7, 17),
        ({"a": _h(1, 5).t(), "b": _h(1, 9)}, 1, 0),       # one column: its stride means nothing
    ],
)
def test_operands_that_the_kernel_reads_are_passed_on(recorder, kw, lda, ldr):
    args = {"a": _h(5, 7), "b": _h(7, 9), **kw}
    assert ops.gemm_ragged(**args).shape == (5, 9)
    (call,) = recorder.calls
    assert (call[1], call[3], call[6]) == (lda, 9, ldr) and call[9:12] == (5, 9, args["a"].shape[1])


@pytest.mark.parametrize(
    "a,b,launches",
    [
        (_h(5, 8), _h(8, 16), 1),
        (_h(5, 16)[:, :7], _h(7, 16), 1),            # padded rows of seven
        (_h(5, 7), _h(7, 16), 2),
        (_h(5, 8), _h(8, 9), 2),
        (_h(41)[1:].view(5, 8), _h(8, 16), 2),       # odd address
        (_h(1, 8).expand(5, 8), _h(8, 16), 2),       # rows on top of one another
    ],
)
def test_only_launches_that_run_are_counted(recorder, a, b, launches):
    before = _lib.launches
    ops.gemm_ragged(a, b)
    assert _lib.launches - before == launches


@pytest.fixture
def product(monkeypatch):
    """The kernel replaced by PyTorch, with the operands it takes."""

    def gemm_ragged(a, b, bias=None, residual=None):
        for t in (bias, residual):
            ops._req(t is None or t.dtype == torch.float16, "gemm_ragged: expected fp16")
        y = a.float() @ b.float()
        y = y if bias is None else y + bias.detach().float()
        return (y if residual is None else y + residual.float()).half()

    monkeypatch.setattr(ops, "gemm_ragged", gemm_ragged)


@pytest.mark.parametrize("bias_type", [None, torch.float16, torch.float32])
@pytest.mark.parametrize("residual", ["fp16", "fp32", "one row", "one value", "transposed"])
def test_any_residual_is_added(product, residual, bias_type):
    """Whatever its type and broadcast, and whatever the bias is."""
    g = torch.Generator().manual_seed(1)
    a, b = torch.randn(2, 5, 7, generator=g).half(), torch.randn(7, 9, generator=g).half()
    full = torch.randn(2, 5, 9, generator=g).half()
    r = {"fp16": full, "fp32": full.float(), "one row": full[0, 0], "one value": full[0, 0, :1], "transposed": full.transpose(1, 2).contiguous().transpose(1, 2)}[residual]
    bias = None if bias_type is None else torch.randn(9, generator=g).to(bias_type)
    y = cascaded_lowp_matmul(a, b, bias=bias, residual=r)
    ref = a.float() @ b.float() + r.float() + (0 if bias is None else bias.float())
    assert y.shape == (2, 5, 9) and y.dtype == (torch.float32 if bias_type == torch.float32 else torch.float16)
    assert float((y.float() - ref).abs().max()) <= 3 * 2.0**-11 * float(ref.abs().max() + 4)


def test_gradient_of_a_bias(product):
    """A bias that asks for a gradient gets it from unaligned extents, as the sum outside the kernel gives it."""
    bias = torch.zeros(9, dtype=torch.float16, requires_grad=True)
    cascaded_lowp_matmul(_h(5, 7), _h(7, 9), bias=bias).float().sum().backward()
    assert torch.equal(bias.grad, torch.full((9,), 5.0, dtype=torch.float16))
    with torch.no_grad():
        assert not cascaded_lowp_matmul(_h(5, 7), _h(7, 9), bias=bias).requires_grad
