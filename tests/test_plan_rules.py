"""The host arithmetic of the product's plans, without a GPU: what the automatic choice takes, and the shared memory that the
rows plan lays out for it."""
import ctypes

import pytest

from mojolearn_b200 import _native
from mojolearn_b200.linalg import OP_NN, OP_NT, OP_TN, W_BF16, W_F32, W_INT8_EXP, W_INT8_SCALE, leaf_count
from mojolearn_b200.torch_ops import PLAN_BAND, PLAN_DECODE, PLAN_ROWS, PLAN_SKINNY, PLAN_STREAM

SMEM_LIMIT = 225 * 1024  # of a CTA of the rows plan; the device's own limit is 227 KB
KINDS = [W_F32, W_BF16, W_INT8_EXP, W_INT8_SCALE]


def auto_plan(m, n, k, op=OP_NT, wkind=W_F32, sms=148, ws=-1):
    leaves = ctypes.c_int64()
    return _native.lib().b200i_auto_plan(m, n, k, op, wkind, sms, ws, ctypes.byref(leaves)), leaves.value


def rows_stages(m, n, k, wkind, group_leaves, sms=148):
    smem = ctypes.c_int64()
    return _native.lib().b200i_rows_plan_stages(m, n, k, wkind, group_leaves, sms, ctypes.byref(smem)), smem.value


@pytest.mark.parametrize("kind", [W_INT8_EXP, W_INT8_SCALE])
@pytest.mark.parametrize("n,k", [(1144930, 4096), (278498, 16384), (61890, 65536), (65536, 50304), (151936, 32768), (300000, 16384), (100000, 65536),
                                 (131072, 65536), (2000000000, 4096)])
def test_weights_whose_factors_leave_no_ring_keep_the_skinny_plan(n, k, kind):
    for m in (5, 8):
        assert auto_plan(m, n, k, wkind=kind)[0] == PLAN_SKINNY
        run = 8
        while -(-leaf_count(k) // run) > 64:
            run *= 2
        assert rows_stages(m, n, k, kind, run)[0] == 0


@pytest.mark.parametrize("sms", [148, 132, 16, 1])
@pytest.mark.parametrize("kind", KINDS)
def test_the_rows_plan_always_has_two_stages(kind, sms):
    """Whatever the rule takes and whatever may be asked for by hand: a ring of two or three stages inside the limit, or a refusal."""
    taken = 0
    for m in (4, 5, 8, 9, 16):
        for k in (16, 128, 144, 768, 2048, 2064, 3072, 4096, 8192, 16384, 32768, 50304, 65536, 131072):
            for n in (1, 2, 24, 305, 768, 2304, 2369, 3072, 11008, 50304, 61890, 278498, 1144929, 1144930, 30000000, 2000000000):
                plan, leaves = auto_plan(m, n, k, wkind=kind, sms=sms)
                if plan == PLAN_ROWS:
                    taken += 1
                    stages, smem = rows_stages(m, n, k, kind, leaves, sms)
                    assert stages in (2, 3) and smem <= SMEM_LIMIT, (m, n, k, stages, smem)
                for run in (1, 2, 4, 8, 16, 32):
                    stages, smem = rows_stages(m, n, k, kind, run, sms)
                    assert stages in (0, 2, 3) and (stages == 0 or smem <= SMEM_LIMIT), (m, n, k, run, stages, smem)
    assert taken > 50


@pytest.mark.parametrize("m,n,k,plan", [(4, 220000, 4096, PLAN_ROWS), (4, 400000, 4096, PLAN_ROWS), (31, 178374, 12208, PLAN_BAND), (31, 165405, 1536, PLAN_BAND)])
def test_a_workspace_that_holds_the_skinny_plan_only_gets_the_skinny_plan(m, n, k, plan):
    """These sizes are unsplit in the skinny plan, which needs no workspace, and split in the plan that the rule prefers."""
    got, leaves = auto_plan(m, n, k)
    assert got == plan and leaves < leaf_count(k)
    need = -(-leaf_count(k) // leaves) * m * n * 4
    assert auto_plan(m, n, k, ws=need)[0] == plan
    for ws in (0, need - 1):
        got, leaves = auto_plan(m, n, k, ws=ws)
        assert got != plan and leaves >= leaf_count(k)


@pytest.mark.parametrize("m,n,k,before", [(8, 220000, 4096, PLAN_ROWS), (14, 178374, 12208, PLAN_BAND)])
def test_a_workspace_that_does_not_hold_the_stream_plan_gets_the_plan_before_it(m, n, k, before):
    got, leaves = auto_plan(m, n, k)
    need = -(-leaf_count(k) // leaves) * m * n * 4
    assert got == PLAN_STREAM and auto_plan(m, n, k, ws=need) == (got, leaves)
    got, leaves = auto_plan(m, n, k, ws=need - 1)
    assert got == before and -(-leaf_count(k) // leaves) * m * n * 4 < need
    assert auto_plan(m, n, k, ws=0) == (PLAN_SKINNY, leaf_count(k))


def test_workspace_by_op_and_storage():
    """Enough for the automatic plan, never more than the answer that knows neither op nor storage, and no node per leaf for an
    op that the tall plan does not take."""
    lib = _native.lib()
    for m, n, k in [(128, 128, 131072), (32, 32, 1000000), (27, 27, 3001), (8, 768, 3072), (8, 11008, 4096), (32, 16384, 2048), (300, 5136, 4096),
                    (128, 11008, 4096), (1000, 1000, 1000), (1, 64, 2048), (5, 7, 50), (31, 165405, 1536)]:
        for op in (OP_NN, OP_NT, OP_TN):
            for kind in KINDS if op == OP_NT else (W_F32, W_BF16):
                plan, leaves = auto_plan(m, n, k, op=op, wkind=kind)
                need = int(lib.b200i_product_workspace_bytes(m, n, k, op, kind))
                assert auto_plan(m, n, k, op=op, wkind=kind, ws=need) == (plan, leaves)
                assert need <= int(lib.b200i_workspace_bytes(m, n, k))
    assert int(lib.b200i_product_workspace_bytes(128, 128, 131072, OP_TN, W_F32)) == 1024 * 128 * 128 * 4
    for op, kind in ((OP_NN, W_F32), (OP_NT, W_F32), (OP_NT, W_BF16), (OP_TN, W_BF16)):
        assert int(lib.b200i_product_workspace_bytes(128, 128, 131072, op, kind)) <= 64 * 128 * 128 * 4


@pytest.mark.parametrize("m,n,k,kind,plan", [
    (8, 2304, 768, W_F32, PLAN_ROWS), (8, 11008, 4096, W_F32, PLAN_STREAM), (4, 11008, 4096, W_F32, PLAN_ROWS), (8, 2304, 768, W_INT8_EXP, PLAN_ROWS),
    (8, 11008, 4096, W_INT8_EXP, PLAN_ROWS), (12, 2304, 768, W_F32, PLAN_ROWS), (8, 1536, 6160, W_F32, PLAN_STREAM), (8, 32000, 1792, W_F32, PLAN_STREAM),
    (8, 1536, 6160, W_BF16, PLAN_SKINNY), (8, 1536, 6160, W_INT8_EXP, PLAN_SKINNY), (16, 1536, 6160, W_F32, PLAN_STREAM), (16, 5120, 4096, W_F32, PLAN_STREAM),
    (16, 8192, 1792, W_F32, PLAN_STREAM), (16, 16384, 2048, W_F32, PLAN_STREAM), (32, 16384, 2048, W_F32, PLAN_BAND),
    (4, 11008, 4096, W_BF16, PLAN_DECODE), (5, 11008, 4096, W_BF16, PLAN_STREAM), (16, 11008, 4096, W_BF16, PLAN_STREAM), (17, 11008, 4096, W_BF16, PLAN_SKINNY),
    (17, 11008, 4096, W_F32, PLAN_BAND), (5, 4800, 1872, W_F32, PLAN_ROWS), (5, 4800, 1888, W_F32, PLAN_STREAM), (16, 4800, 1888, W_F32, PLAN_STREAM),
    (16, 4800, 1872, W_F32, PLAN_SKINNY), (8, 7300, 4096, W_BF16, PLAN_SKINNY), (8, 7340, 4096, W_BF16, PLAN_STREAM), (9, 10240, 4096, W_BF16, PLAN_SKINNY),
    (9, 10288, 4096, W_BF16, PLAN_STREAM), (8, 4736, 1920, W_F32, PLAN_ROWS), (8, 9216, 1024, W_F32, PLAN_ROWS), (9, 44000, 1040, W_BF16, PLAN_SKINNY),
    (8, 220000, 4112 * 16, W_F32, PLAN_ROWS)])
def test_small_batches_take_the_plan_that_measured_faster(m, n, k, kind, plan):
    """Both sides of the rules' lines: depths whose last group or strip is nearly empty keep the skinny plan; from nine million
    words (bf16 30 and 42) the stream plan, but where a rows plan comes out even or the columns and leaves divide badly."""
    assert auto_plan(m, n, k, wkind=kind)[0] == plan
