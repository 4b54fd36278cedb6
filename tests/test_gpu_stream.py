"""The streaming kernel for 5 to 16 rows over a large float32 or bf16 weight (`plan=PLAN_STREAM`, and what the automatic choice
takes from nine million words up), bit for bit against the CPU oracle."""
import os
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import oracle  # noqa: E402
from mojolearn_b200 import _native, linalg, torch_ops  # noqa: E402


def _bits(t):
    return t.cpu().numpy().view(np.int32) if isinstance(t, torch.Tensor) else t.view(np.int32)


def _run(a, w, kind, **kw):
    stored = oracle.to_bf16(w) if kind == linalg.W_BF16 else w
    return torch_ops.product(torch.from_numpy(a).cuda(), torch.from_numpy(stored).cuda(), None, kind, linalg.OP_NT, **kw)


def _bf16_exact(rng, *shape):
    return (rng.integers(-127, 128, shape).astype(np.float32)) / 64


@pytest.mark.parametrize("kind", [linalg.W_F32, linalg.W_BF16])
@pytest.mark.parametrize("m", [1, 5, 8, 9, 13, 16])
def test_stream_plan(m, kind):
    """Ragged column units, depths of one leaf, of a part of one (sixteen steps) and of several groups, a CTA that meets two
    leaf groups; a subnormal activation and weight, an infinity, zeros in both operands."""
    for n, k in ((1, 16), (24, 128), (64, 144), (770, 784), (1001, 400), (300, 5136), (12007, 272)):
        rng = np.random.default_rng(m * 31 + n + k + kind)
        a, w = rng.standard_normal((m, k)).astype(np.float32), _bf16_exact(rng, n, k)
        a[m // 2, k // 3], w[n - 1, k - 1], w[n // 2, 3], w[n // 3, 5] = 1e-41, np.inf, 2.0**-130, 0.0
        want = oracle.nan_canon(oracle.gemm_rows(a, w, oracle.OP_NT))
        for gl in (1, 2, 4):
            if -(-oracle.leaf_count(k) // gl) <= 64 and gl <= oracle.leaf_count(k):
                assert np.array_equal(_bits(_run(a, w, kind, plan=torch_ops.PLAN_STREAM, group_leaves=gl)), want.view(np.int32)), (n, k, gl)


@pytest.mark.parametrize("act", [torch_ops.ACT_GELU_ERF, torch_ops.ACT_SILU, torch_ops.ACT_PAIR_SWIGLU, torch_ops.ACT_PAIR_GEGLU_TANH])
@pytest.mark.parametrize("m,n,k,gl", [(7, 1000, 400, 4), (16, 1000, 400, 4), (7, 132, 1040, 1)])
def test_stream_plan_store_epilogues(m, n, k, gl, act):
    """In the kernel's own store (one leaf group) and in the group fold."""
    rng = np.random.default_rng(n + act)
    a, w = (torch.from_numpy(rng.standard_normal(s).astype(np.float32)).cuda() for s in ((m, k), (n, k)))
    bias = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    want = torch_ops.product(a, w, None, linalg.W_F32, linalg.OP_NT, plan=torch_ops.PLAN_SKINNY, bias=bias, act=act)
    got = torch_ops.product(a, w, None, linalg.W_F32, linalg.OP_NT, plan=torch_ops.PLAN_STREAM, group_leaves=gl, bias=bias, act=act)
    assert np.array_equal(_bits(got), _bits(want))


@pytest.mark.parametrize("m,n,k,kind", [(5, 4801, 2000, linalg.W_F32), (16, 8467, 2048, linalg.W_F32), (9, 60001, 784, linalg.W_F32), (8, 11008, 4096, linalg.W_BF16),
                                        (12, 11008, 4096, linalg.W_BF16)])
def test_automatic_choice_at_the_sizes_that_stream(m, n, k, kind):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert _native.lib().b200i_auto_plan(m, n, k, linalg.OP_NT, kind, sms, -1, None) == torch_ops.PLAN_STREAM
    rng = np.random.default_rng(n)
    a, w = rng.standard_normal((m, k)).astype(np.float32), (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
    got = _run(a, w, kind)
    assert np.array_equal(_bits(got), _bits(_run(a, w, kind, plan=torch_ops.PLAN_SKINNY)))
    assert np.array_equal(_bits(got), _bits(_run(a, w, kind, plan=torch_ops.PLAN_STREAM, group_leaves=2)))


def forcing_cases():
    """One cell whose chain needs the flushed step, the rest admitted: the smallness in the weight, the activations or both."""
    for kind in (linalg.W_F32, linalg.W_BF16):
        for m, n, k, gl in ((8, 305, 784, 2), (16, 70, 528, 4)):
            for where, (small, large) in (("w", (2.0**-120, 2.0**-7)), ("a", (2.0**-120, 2.0**-7)), ("both", (2.0**-64, 2.0**-63))):
                for p in (0, k // 2 + 3, k - 2):
                    rng = np.random.default_rng(n + p)
                    a, w = rng.standard_normal((m, k)).astype(np.float32), _bf16_exact(rng, n, k)
                    a[m - 1] = 0.0
                    if where == "w":
                        a[m - 1, p], a[m - 1, p + 1], w[n - 1, p], w[n - 1, p + 1] = large, 2 * large, small, small
                    else:
                        a[m - 1, p], a[m - 1, p + 1], w[n - 1, p], w[n - 1, p + 1] = small, small, large, 2 * large
                    want = oracle.nan_canon(oracle.gemm_rows(a, w, oracle.OP_NT))
                    yield "%s %s %s %s" % (kind, (m, n, k, gl), where, p), lambda a=a, w=w, kind=kind, gl=gl: _run(a, w, kind, plan=torch_ops.PLAN_STREAM, group_leaves=gl), want


def test_windows_that_need_the_flushed_step_get_it():
    for name, run, want in forcing_cases():
        assert np.array_equal(_bits(run()), want.view(np.int32)), name


CHILD = r"""
import sys
sys.path[:0] = [%(root)r, %(root)r + "/tests"]
import numpy as np
import test_gpu_stream as t
print("RIGHT", [name for name, run, want in t.forcing_cases() if np.array_equal(t._bits(run()), want.view(np.int32))])
"""


def test_admit_always_build_fails_every_forcing_case():
    from mojolearn_b200.csrc import build as cuda_build
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", CHILD % {"root": root}], env=dict(os.environ, MOJOLEARN_B200_LIB=cuda_build.build(sabotage=True)), capture_output=True,
                         text=True, timeout=600)
    assert run.returncode == 0 and run.stdout.strip().endswith("RIGHT []"), run.stdout + run.stderr[-2000:]


@pytest.mark.parametrize("m,n,k,gl,kind", [(17, 64, 256, 1, linalg.W_F32), (8, 64, 2048, 8, linalg.W_F32), (8, 64, 250, 1, linalg.W_F32), (8, 64, 16512, 2, linalg.W_BF16)])
def test_refusals(m, n, k, gl, kind):
    """More than sixteen rows, groups of more than four leaves, a depth that is no multiple of sixteen, more than 64 groups."""
    a, w = np.zeros((m, k), np.float32), np.zeros((n, k), np.float32)
    with pytest.raises(Exception):
        _run(a, w, kind, plan=torch_ops.PLAN_STREAM, group_leaves=gl)
