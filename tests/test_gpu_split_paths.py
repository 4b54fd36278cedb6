"""GPU parity of the kernels that split a product by leaves, warps or SM pairs, at the sizes where a split can go wrong:
tile and strip edges, ragged last leaves and windows, failed admission, the largest and smallest of each range. The bar
is the CPU oracle's words."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from mojolearn_b200 import _native, linalg, torch_ops  # noqa: E402


def _same(got, want):
    return got.cpu().numpy().tobytes() == want.tobytes()


@pytest.mark.parametrize("m,n,k", [(32, 32, 20000), (27, 27, 3001), (1, 5, 2049), (128, 128, 2100), (33, 97, 140000), (4, 64, 257), (36, 36, 131088)])
def test_tall_products(m, n, k):
    """One warp per leaf and tile, both copy widths, leaves of 128 and longer ones, a ragged last leaf."""
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((k, m)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    a[k // 2, 0], b[k - 1, n - 1], a[0, m - 1] = 1e-41, 3e-39, np.inf  # leaves that fail admission
    want = oracle.nan_canon(oracle.gemm_rows(a, b, oracle.OP_TN))
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    assert _same(torch_ops.product(da, db, op=linalg.OP_TN, plan=torch_ops.PLAN_TALL), want)
    assert _same(torch_ops.matmul(da, db, transpose_a=True), want)
    if m % 4 == 0 and n % 4 == 0:  # rows of whole quads that do not start on 16 bytes
        pad = torch.empty(k * m + 1, device="cuda")
        pad[1:] = da.reshape(-1)
        assert _same(torch_ops.product(pad[1:].view(k, m), db, op=linalg.OP_TN, plan=torch_ops.PLAN_TALL), want)


def _weight(rng, n, k, kind):
    if kind == linalg.W_F32:
        w = rng.standard_normal((n, k)).astype(np.float32)
        return w, None, w
    if kind == linalg.W_BF16:
        bits = oracle.to_bf16(rng.standard_normal((n, k)).astype(np.float32))
        return bits, None, oracle.from_bf16(bits)
    codes = rng.integers(-127, 128, (n, k)).astype(np.int8)
    if kind == linalg.W_INT8_EXP:
        e = rng.integers(-13, -9, n).astype(np.int32)
        e[0], e[n // 2], e[n - 1] = -100, 118, -140  # factors past the short spellings
        return codes, e, oracle.dequantize_int8(codes, e)
    s = rng.uniform(0.001, 0.02, n).astype(np.float32)
    s[0] = 1e-36
    return codes, s, oracle.dequantize_int8_scaled(codes, s)


ROWS_SHAPES = [(2, 16), (24, 128), (768, 768), (305, 784), (1186, 144), (770, 3072), (300, 5136), (9600, 256), (20001, 128)]


@pytest.mark.parametrize("kind", [linalg.W_F32, linalg.W_BF16, linalg.W_INT8_EXP, linalg.W_INT8_SCALE])
@pytest.mark.parametrize("m", [1, 5, 8, 9, 16])
def test_rows_plan(m, kind):
    """A column's whole contraction in one CTA: every strip width, runs of one to four leaves, leaf groups past 4096 / 2048
    steps, strips past the last column, rows past m."""
    for n, k in ROWS_SHAPES:
        rng = np.random.default_rng(m * 31 + n + k + kind)
        w, scale, dense = _weight(rng, n, k, kind)
        a = rng.standard_normal((m, k)).astype(np.float32)
        a[m // 2, k // 3] = 1e-41
        want = oracle.nan_canon(oracle.gemm_rows(a, dense, oracle.OP_NT))
        da, dw = torch.from_numpy(a).cuda(), torch.from_numpy(w).cuda()
        ds = torch.from_numpy(scale).cuda() if scale is not None else None
        cap = 32 if m <= 8 else 16
        gl = cap if oracle.leaf_count(k) > cap else 0
        assert _same(torch_ops.product(da, dw, ds, kind, linalg.OP_NT, plan=torch_ops.PLAN_ROWS, group_leaves=gl), want), (n, k)
        assert _same(torch_ops.product(da, dw, ds, kind, linalg.OP_NT), want), (n, k)


@pytest.mark.parametrize("m", [9, 16, 17, 32])
@pytest.mark.parametrize("n,k", [(24, 128), (770, 784), (255, 16), (1001, 144), (300, 5136)])
def test_band_plan(m, n, k):
    """256-column tiles with ragged edges, leaf groups, a chunk of activations restaged every two leaves."""
    rng = np.random.default_rng(m + n + k)
    a, w = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    a[m // 2, k // 3], w[n - 1, k - 1], w[7, 3] = 1e-41, np.inf, 3e-39
    want = oracle.nan_canon(oracle.gemm_rows(a, w, oracle.OP_NT))
    da, dw = torch.from_numpy(a).cuda(), torch.from_numpy(w).cuda()
    for gl in (0, 1, 4):
        if gl <= oracle.leaf_count(k):
            assert _same(torch_ops.product(da, dw, None, linalg.W_F32, linalg.OP_NT, plan=torch_ops.PLAN_BAND, group_leaves=gl), want), gl


@pytest.mark.parametrize("act", [torch_ops.ACT_GELU_ERF, torch_ops.ACT_SILU, torch_ops.ACT_PAIR_SWIGLU, torch_ops.ACT_PAIR_GEGLU_TANH])
@pytest.mark.parametrize("n,k", [(1000, 768), (48, 5136)])
def test_rows_plan_store_epilogues(n, k, act):
    rng = np.random.default_rng(n + act)
    a, w = torch.from_numpy(rng.standard_normal((7, k)).astype(np.float32)).cuda(), torch.from_numpy(rng.standard_normal((n, k)).astype(np.float32)).cuda()
    bias = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    gl = 32 if k > 4096 else 0
    want = torch_ops.product(a, w, None, linalg.W_F32, linalg.OP_NT, plan=torch_ops.PLAN_SKINNY, bias=bias, act=act)
    got = torch_ops.product(a, w, None, linalg.W_F32, linalg.OP_NT, plan=torch_ops.PLAN_ROWS, group_leaves=gl, bias=bias, act=act)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("rows,cols", [(1, 4), (9, 1024), (8, 1028), (5, 2052), (3, 4096), (2, 8192), (3, 8196), (7, 7), (4, 1001)])
def test_quantised_rows(rows, cols):
    rng = np.random.default_rng(cols)
    x = (rng.standard_normal((rows, cols)) * np.exp2(rng.integers(-140, 120, (rows, 1)))).astype(np.float32)
    x[0, :3] = [np.nan, 1e-41, -np.inf][:3]
    x[rows - 1] = 0.0
    q, e = torch_ops.quantize_int8(torch.from_numpy(x).cuda())
    qo, eo = oracle.quantize_int8(x)
    assert _same(q, qo) and _same(e, eo)


@pytest.mark.parametrize("m,n,k", [(2304, 2304, 144), (2500, 2060, 272), (130, 38000, 128), (4000, 2600, 16)])
def test_int8_products_on_sm_pairs(m, n, k):
    """Whole tiles, the halved last round, rows and columns past the edge, k below and across a stage."""
    rng = np.random.default_rng(m)
    qa, qb = rng.integers(-127, 128, (m, k)).astype(np.int8), rng.integers(-127, 128, (n, k)).astype(np.int8)
    ea, eb = rng.integers(-60, 30, m).astype(np.int32), rng.integers(-60, 30, n).astype(np.int32)
    got = torch_ops.matmul_int8(*(torch.from_numpy(t).cuda() for t in (qa, ea, qb, eb))).cpu().numpy()
    rows = np.unique(np.r_[0, 127, 128, 255, 256, m - 1, rng.integers(0, m, 24)] % m)
    want = oracle.nan_canon(oracle.gemm_int8(np.ascontiguousarray(qa[rows]), ea[rows], qb, eb))
    assert got[rows].tobytes() == want.tobytes()
    assert _native.lib().b200i_decode_status(-1) == 0


@pytest.mark.parametrize("m,n,k", [(1100, 17000, 144), (1030, 17003, 16), (40, 151600, 1008), (2056, 8960, 512)])
def test_int8_products_with_a_short_contraction(m, n, k):
    """One CTA a tile: at least four 128 x 256 tiles per SM and k below 1024; whole and ragged rows of 16-byte stores, exponents
    inside and outside the short conversion's range."""
    assert -(-m // 128) * -(-n // 256) >= 4 * torch.cuda.get_device_properties(0).multi_processor_count and k < 1024
    rng = np.random.default_rng(n)
    qa, qb = rng.integers(-127, 128, (m, k)).astype(np.int8), rng.integers(-127, 128, (n, k)).astype(np.int8)
    ea, eb = rng.integers(-60, 30, m).astype(np.int32), rng.integers(-60, 30, n).astype(np.int32)
    eb[n // 2 :] += 40
    got = torch_ops.matmul_int8(*(torch.from_numpy(t).cuda() for t in (qa, ea, qb, eb))).cpu().numpy()
    rows = np.unique(np.r_[0, 31, 127, 128, m - 1, rng.integers(0, m, 12)] % m)
    want = oracle.nan_canon(oracle.gemm_int8(np.ascontiguousarray(qa[rows]), ea[rows], qb, eb))
    assert got[rows].tobytes() == want.tobytes()
    assert _native.lib().b200i_decode_status(-1) == 0


@pytest.mark.parametrize("m,n,k,opname", [(96, 2304, 1500, "NT"), (1100, 1000, 1030, "NN"), (40, 1500, 3000, "NN"), (2000, 70, 900, "TN")])
def test_host_arrays_through_the_copy_threads(m, n, k, opname):
    """Megabytes of pageable arrays: both ways of cutting the product, and the plain path."""
    op = {"NN": linalg.OP_NN, "NT": linalg.OP_NT, "TN": linalg.OP_TN}[opname]
    rng = np.random.default_rng(k)
    a = rng.standard_normal((k, m) if opname == "TN" else (m, k)).astype(np.float32)
    b = rng.standard_normal((n, k) if opname == "NT" else (k, n)).astype(np.float32)
    want = torch_ops.product(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), op=op).cpu().numpy()
    for _ in range(2):
        got = linalg.matmul(a, b, transpose_a=opname == "TN", transpose_b=opname == "NT")
        assert got.tobytes() == want.tobytes()


def test_gated_activation_layouts_agree():
    """Four outputs a thread on aligned rows against one output a thread on the same values off the 16-byte grid."""
    import ctypes
    rng = np.random.default_rng(5)
    for kind in (0, 4, 5):
        gu = torch.from_numpy((rng.standard_normal((5, 2 * 72)) * 4).astype(np.float32)).cuda()
        gu[0, :4] = torch.tensor([float("inf"), float("nan"), 1e-41, -1e-40], device="cuda")
        off = torch.empty(gu.numel() + 1, device="cuda")
        off[1:] = gu.reshape(-1)
        outs = []
        for src in (gu.data_ptr(), off.data_ptr() + 4):
            out = torch.empty((5, 72), device="cuda")
            _native.call("b200i_act_mul", 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(src), None,
                         5, 72, 144, kind, 1)
            outs.append(out.view(torch.int32))
        assert torch.equal(*outs)


ACTS = [torch_ops.ACT_NONE, torch_ops.ACT_GELU_ERF, torch_ops.ACT_SILU]


@pytest.mark.parametrize("m", [9, 16, 17, 32])
@pytest.mark.parametrize("n,k", [(1001, 144), (770, 2064), (516, 1040)])
def test_band_plan_store_epilogues(m, n, k):
    """Bias, activations and (whole quads of columns) gated stores, in the kernel's own store and in the fold of its groups."""
    rng = np.random.default_rng(m + n + k)
    a, w = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda(), torch.from_numpy(rng.standard_normal((n, k)).astype(np.float32)).cuda()
    bias = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    for act in ACTS + ([torch_ops.ACT_PAIR_SWIGLU, torch_ops.ACT_PAIR_GEGLU_TANH] if n % 4 == 0 else []):
        want = torch_ops.product(a, w, None, linalg.W_F32, linalg.OP_NT, plan=torch_ops.PLAN_SKINNY, bias=bias, act=act)
        for gl in (0, 4):
            if gl < oracle.leaf_count(k):
                got = torch_ops.product(a, w, None, linalg.W_F32, linalg.OP_NT, plan=torch_ops.PLAN_BAND, group_leaves=gl, bias=bias, act=act)
                assert torch.equal(got.view(torch.int32), want.view(torch.int32)), (act, gl)


@pytest.mark.parametrize("m,n,k", [(33, 40, 20000), (27, 5, 140000)])
def test_tall_plan_store_epilogues(m, n, k):
    """Both depths of the node fold (up to 256 nodes, and more), which is where the tall plan applies them."""
    rng = np.random.default_rng(k)
    a, b = torch.from_numpy(rng.standard_normal((k, m)).astype(np.float32)).cuda(), torch.from_numpy(rng.standard_normal((k, n)).astype(np.float32)).cuda()
    bias = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    for act in ACTS:
        got, want = (torch_ops.product(a, b, op=linalg.OP_TN, plan=p, bias=bias, act=act) for p in (torch_ops.PLAN_TALL, torch_ops.PLAN_FLAT))
        assert torch.equal(got.view(torch.int32), want.view(torch.int32)), act


@pytest.mark.parametrize("m", [9, 16, 17, 32])
def test_band_plan_by_the_rule(m):
    """Float32 weights of a size that the rule gives to the band plan, ragged columns: the automatic split and its workspace (at 9
    to 16 rows a depth whose leaves the stream plan has no groups for)."""
    n, k = (301, 33808) if m <= 16 else (4901, 2048)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert _native.lib().b200i_auto_plan(m, n, k, linalg.OP_NT, linalg.W_F32, sms, -1, None) == torch_ops.PLAN_BAND
    rng = np.random.default_rng(m)
    a, w = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    a[m - 1, k // 3], w[n - 1, 5] = 1e-41, 3e-39
    rows = np.unique([0, m // 2, m - 1])
    want = oracle.nan_canon(oracle.gemm_rows(np.ascontiguousarray(a[rows]), w, oracle.OP_NT))
    got = torch_ops.matmul(torch.from_numpy(a).cuda(), torch.from_numpy(w).cuda(), transpose_b=True).cpu().numpy()
    assert got[rows].tobytes() == want.tobytes()


@pytest.mark.parametrize("kind", [linalg.W_F32, linalg.W_INT8_EXP])
def test_rows_plan_with_many_columns_and_several_leaf_groups(kind):
    """Hundreds of columns in a CTA beside five groups of eight leaves, the last one ragged."""
    m, n, k = 7, 30001, 4112
    rng = np.random.default_rng(kind)
    w, scale, dense = _weight(rng, n, k, kind)
    a = rng.standard_normal((m, k)).astype(np.float32)
    want = oracle.nan_canon(oracle.gemm_rows(a, dense, oracle.OP_NT))
    ds = torch.from_numpy(scale).cuda() if scale is not None else None
    got = torch_ops.product(torch.from_numpy(a).cuda(), torch.from_numpy(w).cuda(), ds, kind, linalg.OP_NT, plan=torch_ops.PLAN_ROWS, group_leaves=8)
    assert _same(got, want)


SPECIALS = [1e-41, -3e-39, 2.0**-64, -(2.0**-63), np.inf, np.nan]


@pytest.mark.parametrize("m,n,k", [(128, 300, 1044), (37, 130, 396), (1, 129, 20), (65, 256, 2048)])
def test_packed_plan_reading_b_in_place(m, n, k):
    """One row of tiles over float32 rows of whole quads, ragged last stages, split and unsplit: subnormal, tiny and non-finite
    words in the first, a middle and the last stage of 32 steps."""
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    for p in (0, (k // 2) // 32 * 32 + 7, k - 4):
        for i, v in enumerate(SPECIALS):
            b[(i * 37 + p) % n, p + (i & 3)] = v
            a[(i * 11) % m, p + (i & 3)] = SPECIALS[i - 1] if i < 4 else v
    want = oracle.nan_canon(oracle.gemm_rows(a, b, oracle.OP_NT))
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    for gl in (0, 2):
        if gl < oracle.leaf_count(k):
            assert _same(torch_ops.product(da, db, None, linalg.W_F32, linalg.OP_NT, plan=torch_ops.PLAN_PACKED, group_leaves=gl), want), gl


def forcing_cases():
    """(name, product, oracle's words): products with ONE window in which bare steps give another word than flushed ones, the words
    that force it in the weight only, in the activations only, or in both; in the first, a middle and the last window.
    The last row is zero but for two steps, whose products are 2^-127 (flushed away) and 2^-126. `ragged` in a name: the steps lie
    in a window that is not whole, which every kernel walks flushed."""
    def build(m, n, k, where, p, exps=False):
        rng = np.random.default_rng(m * 7 + n + k + p)
        a, w = rng.standard_normal((m, k)).astype(np.float32), rng.integers(-127, 128, (n, k)).astype(np.float32) / 64
        a[m - 1] = 0.0
        small, large = {"w": (2.0**-120, 2.0**-7), "a": (2.0**-120, 2.0**-7), "both": (2.0**-64, 2.0**-63)}[where]
        if where == "w":
            a[m - 1, p], a[m - 1, p + 1], w[n - 1, p], w[n - 1, p + 1] = large, 2 * large, small, small
        else:
            a[m - 1, p], a[m - 1, p + 1], w[n - 1, p], w[n - 1, p + 1] = small, small, large, 2 * large
        e = np.full(n, -6, np.int32)
        if exps:  # a row of codes has one exponent: the whole column is as small as its two words
            e[n - 1] = int(np.log2(small if where == "w" else large))
            w[n - 1] = np.where(np.arange(k) < p, 3, 5) * np.exp2(e[n - 1].astype(np.float64))
            w[n - 1, p] = np.exp2(float(e[n - 1]))
            w[n - 1, p + 1] = w[n - 1, p] * (1 if where == "w" else 2)
        return a, w, e

    def case(name, a, w, e, kind, op, plan, gl):
        stored, scale = w, None
        if kind == linalg.W_BF16:
            stored = oracle.to_bf16(w)
        elif kind in (linalg.W_INT8_EXP, linalg.W_INT8_SCALE):
            stored = np.rint(w / np.exp2(e.astype(np.float64))[:, None]).astype(np.int8)
            scale = e if kind == linalg.W_INT8_EXP else np.exp2(e.astype(np.float64)).astype(np.float32)
        want = oracle.nan_canon(oracle.gemm_rows(a, w, op))

        def run():
            up = lambda t: torch.from_numpy(t).cuda() if t is not None else None  # noqa: E731
            return torch_ops.product(up(a), up(stored), up(scale), kind, op, plan=plan, group_leaves=gl)
        return name, run, want

    for where in ("w", "a", "both"):
        for m, n, k, plan, gls in ((128, 300, 1044, torch_ops.PLAN_PACKED, (0, 2)), (37, 130, 396, torch_ops.PLAN_PACKED, (0,)), (16, 770, 784, torch_ops.PLAN_BAND, (0, 4)),
                                   (32, 300, 528, torch_ops.PLAN_BAND, (0,)), (8, 305, 784, torch_ops.PLAN_ROWS, (0, 4)), (16, 40, 256, torch_ops.PLAN_ROWS, (0,))):
            kinds = [linalg.W_F32, linalg.W_BF16, linalg.W_INT8_EXP, linalg.W_INT8_SCALE] if plan == torch_ops.PLAN_ROWS else [linalg.W_F32]
            for p in (0, k // 2 + 3, k // 32 * 32 - 2, k - 2):
                for kind in kinds:
                    a, w, e = build(m, n, k, where, p, kind in (linalg.W_INT8_EXP, linalg.W_INT8_SCALE))
                    for gl in gls:
                        ragged = " ragged" if p == k - 2 and k % 32 else ""
                        yield case("%s %s %s %s %s%s" % (plan, (m, n, k, gl), where, p, kind, ragged), a, w, e, kind, linalg.OP_NT, plan, gl)
        for m, n, k in ((32, 64, 2100), (27, 33, 20001)):
            for p in (0, k // 2 + 3, k // 128 * 128 - 19, k - 2):
                a, w, e = build(m, n, k, where, p)
                yield case("tall %s %s %s%s" % ((m, n, k), where, p, " ragged" if p == k - 2 else ""), np.ascontiguousarray(a.T), np.ascontiguousarray(w.T), e, linalg.W_F32, linalg.OP_TN,
                           torch_ops.PLAN_TALL, 0)


def test_windows_that_need_the_flushed_step_get_it():
    for name, run, want in forcing_cases():
        assert _same(run(), want), name


@pytest.mark.parametrize("m", [2176, 2500, 3970])
def test_packed_plan_walks_a_whole_band_of_tiles_and_a_part_of_one(m):
    """17, 20 and 32 rows of tiles: bands of sixteen, the last one short or whole."""
    n, k = 300, 200
    rng = np.random.default_rng(m)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    want = oracle.nan_canon(oracle.gemm_rows(a, b, oracle.OP_NN))
    got = torch_ops.product(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), op=linalg.OP_NN, plan=torch_ops.PLAN_PACKED)
    assert _same(got, want)
