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


def test_the_cuda_library_is_built_without_torch(monkeypatch, capsys):
    from mojolearn_b200.csrc import build as cuda_build
    done = []

    def no_torch(force=False):
        assert done == ["cuda"]
        raise ImportError("No module named 'torch'")

    monkeypatch.setattr(cuda_build, "build", lambda **kw: done.append("cuda") or "libb200i.so")
    monkeypatch.setattr(cuda_build, "build_host", no_torch)
    cuda_build.main([])
    assert done == ["cuda"] and "No module named 'torch'" in capsys.readouterr().err


def test_a_host_extension_of_another_torch_is_stale_and_not_used(monkeypatch, tmp_path):
    import types
    from mojolearn_b200.csrc import build as cuda_build
    lib = tmp_path / "_host_call.so"
    assert cuda_build.host_stale(str(lib))
    lib.write_bytes(b"\0" + cuda_build.host_tag().encode() + b"\0")
    assert not cuda_build.host_stale(str(lib))
    lib.write_bytes(b"\0torch 2.0.0, python 3.12\0")
    assert cuda_build.host_stale(str(lib))
    import mojolearn_b200
    monkeypatch.setattr(mojolearn_b200, "_host_call", types.SimpleNamespace(BUILT_FOR="torch 2.0.0, python 3.12"), raising=False)
    with pytest.warns(RuntimeWarning, match="built for torch 2.0.0"):
        assert torch_ops._load_host_call() is None
