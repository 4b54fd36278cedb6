"""The native host side of a product call: the plain case gives the Python path's words, everything else keeps its refusals."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from mojolearn_b200 import _native, linalg, torch_ops  # noqa: E402


def _operands(m, n, k, kind, op=linalg.OP_NT, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn((k, m) if op == linalg.OP_TN else (m, k), generator=g, device="cuda")
    b = torch.randn((n, k) if op == linalg.OP_NT else (k, n), generator=g, device="cuda")
    if kind == linalg.W_F32:
        return a, b, None
    if kind == linalg.W_BF16:
        return a, b.to(torch.bfloat16).view(torch.uint16), None
    codes = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8)
    e = torch.randint(-9, -5, (n,), generator=g, device="cuda", dtype=torch.int32)
    return a, codes, e if kind == linalg.W_INT8_EXP else torch.exp2(e.float())


def _python(monkeypatch, *args, **kw):
    with monkeypatch.context() as mp:
        mp.setattr(torch_ops, "_plain_product", None)
        return torch_ops.product(*args, **kw)


@pytest.mark.parametrize("kind", [linalg.W_F32, linalg.W_BF16, linalg.W_INT8_EXP, linalg.W_INT8_SCALE])
def test_the_plain_case_is_taken_and_gives_the_same_words(kind, monkeypatch):
    assert torch_ops._host_call is not None, "mojolearn_b200/_host_call.so is not built"
    for m, n, k in ((1, 40, 256), (5, 305, 784), (33, 130, 300), (130, 260, 144)):
        for op in (linalg.OP_NT,) if kind in (linalg.W_INT8_EXP, linalg.W_INT8_SCALE) else (linalg.OP_NN, linalg.OP_NT, linalg.OP_TN):
            a, b, s = _operands(m, n, k, kind, op)
            want = _python(monkeypatch, a, b, s, kind, op)
            got = torch_ops._plain_product(a, b, s, kind, op, torch_ops.PLAN_AUTO, 0)
            assert got is not None and got.shape == want.shape and got.dtype == want.dtype and got.device == want.device and not got.requires_grad
            assert torch.equal(got.view(torch.int32), want.view(torch.int32))


def test_other_streams_and_threads():
    import threading
    a, b, _ = _operands(8, 640, 512, linalg.W_F32)
    want = torch_ops.product(a, b, None, linalg.W_F32, linalg.OP_NT)
    torch.cuda.synchronize()
    wrong = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                got = torch_ops.product(a, b, None, linalg.W_F32, linalg.OP_NT)
                torch.cuda.current_stream().synchronize()
                if not torch.equal(got, want):
                    wrong.append(1)

    threads = [threading.Thread(target=work) for _ in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong


def test_refusals_are_the_python_paths(monkeypatch):
    a, b, _ = _operands(4, 64, 128, linalg.W_F32)
    _, codes, e = _operands(4, 64, 128, linalg.W_INT8_EXP)
    F, B, I8, NT = linalg.W_F32, linalg.W_BF16, linalg.W_INT8_EXP, linalg.OP_NT
    for args, kw in (((a.double(), b, None, F, NT), {}), ((a, b.half(), None, F, NT), {}), ((a[:, ::2], b[:, ::2], None, F, NT), {}), ((a, b.T, None, F, linalg.OP_NN), {}),
                     ((a, b[:, :64].contiguous(), None, F, NT), {}), ((a[0], b, None, F, NT), {}), ((a.cpu(), b, None, F, NT), {}), ((a, b, None, F, 7), {}),
                     ((a, b, None, B, NT), {}), ((a, codes, None, I8, NT), {}), ((a, codes, e[:3], I8, NT), {}), ((a, codes, e.float(), I8, NT), {}),
                     ((a, codes.T.contiguous(), e, I8, linalg.OP_NN), {}), ((a[:0], b, None, F, NT), {}), ((a, b, None, F, NT), {"plan": 99}),
                     ((a, b, None, F, NT), {"plan": torch_ops.PLAN_DECODE, "group_leaves": 3}), ((a.tolist(), b, None, F, NT), {})):
        outcomes = []
        for run in (lambda: _python(monkeypatch, *args, **kw), lambda: torch_ops.product(*args, **kw)):
            try:
                outcomes.append(run().cpu().numpy().view(np.int32).tobytes())
            except Exception as x:  # noqa: BLE001
                outcomes.append((type(x), str(x)))
        assert outcomes[0] == outcomes[1], outcomes


def test_wrapped_tensors_are_left_to_the_python_path():
    class Sub(torch.Tensor):
        pass

    a, b, _ = _operands(4, 64, 128, linalg.W_F32)
    run = lambda x, y: torch_ops._plain_product(x, y, None, linalg.W_F32, linalg.OP_NT, torch_ops.PLAN_AUTO, 0)  # noqa: E731
    assert run(a.as_subclass(Sub), b) is None and run(torch._neg_view(a), b) is None and run(a.cpu(), b) is None
    seen = []
    torch.func.vmap(lambda x: (seen.append(run(x, b)), x)[1])(a[None])
    assert seen == [None]
    assert run(torch.nn.Parameter(a), b) is not None
    with pytest.raises(_native.NativeError):
        torch_ops.product(a, b, None, linalg.W_F32, linalg.OP_NT, plan=99)
