"""The native host side of a product call, without a GPU: what it leaves to the Python path, and how it is built."""
import pytest

torch = pytest.importorskip("torch")

from mojolearn_b200 import _native, torch_ops  # noqa: E402


def test_a_missing_library_does_not_come_before_the_operands_refusals(monkeypatch):
    def missing():
        raise _native.NativeError("missing")

    monkeypatch.setattr(torch_ops, "_plain_product", torch_ops._bind_plain_product)
    monkeypatch.setattr(_native, "lib", missing)
    with pytest.raises(TypeError, match="a must be a CUDA tensor"):
        torch_ops.product(torch.zeros(2, 16), torch.zeros(3, 16), op=torch_ops.OP_NT)
