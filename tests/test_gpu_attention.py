"""The attention entry points against the CPU oracle at serving sizes.

`b200i_attention` and `b200i_attention_at` (the position read from a device word, as a replayed CUDA graph needs it)
with 1, 2, 4 and 8 query rows per sequence -- the decode-step kernels -- at head_dim 128 and 64, on caches of
31 ... 1279 positions: around the edges of a 32-key tile, past the point where the value ring refills a slot (more
than 96 keys), and at the serving benchmark's lengths; with and without a sliding window, with grouped-query heads,
and with operands that make a late tile fail the admission test of the bare multiply-add, so that the flushed chain
has to take over in the middle of a row. Bit for bit, against oracle/decoder_oracle.c's dec_attention, which follows
transformer/checks/transformer_oracle.mojo:2373-2546 of the reference (S11-S19).
"""
import ctypes

import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from mojolearn_b200 import _native  # noqa: E402

KEYS = (31, 32, 33, 95, 96, 97, 129, 1030, 1279)


def _vp(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _run(q, kc, vc, l, used, window, at, softcap=0.0):
    """ctx through the C ABI; `at` = the device-position twin."""
    b, nkv, cap, hd = kc.shape
    nh = q.shape[1]
    dq, dk, dv = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (q, kc, vc))
    ctx = torch.full((b * l, nh * hd), np.float32(-777.0), device="cuda")
    if at:
        smax = min(cap, window - 1 + l) if window else cap
        scores = torch.empty((b * nh * l * smax,), device="cuda")
        pos = torch.tensor([used - l], dtype=torch.int32, device="cuda")
        _native.call("b200i_attention_at", 0, None, _vp(ctx), _vp(dq), _vp(dk), _vp(dv), _vp(scores), b, l, nh, nkv, hd, cap,
                     _vp(pos), window, softcap)
    else:
        s = used - (max(0, used - l - (window - 1)) if window else 0)
        scores = torch.empty((b * nh * l * s,), device="cuda")
        _native.call("b200i_attention", 0, None, _vp(ctx), _vp(dq), _vp(dk), _vp(dv), _vp(scores), b, l, nh, nkv, hd, cap, used,
                     window, softcap)
    torch.cuda.synchronize()
    assert _native.lib().b200i_decode_status(0) == 0
    return ctx.cpu().numpy()


def _operands(rng, b, l, nh, nkv, hd, cap, scale_q=1.0):
    q = (rng.standard_normal((b * l, nh, hd)) * scale_q).astype(np.float32)
    kc = rng.standard_normal((b, nkv, cap, hd)).astype(np.float32)
    vc = rng.standard_normal((b, nkv, cap, hd)).astype(np.float32)
    return q, kc, vc


@pytest.mark.parametrize("hd", (128, 64))
@pytest.mark.parametrize("l", (1, 2, 4, 8))
def test_decode_step_attention_at_tile_edges_and_serving_lengths(l, hd):
    rng = np.random.default_rng(1000 * l + hd)
    b, nh, nkv, cap = 2, 4, 4, 1280
    q, kc, vc = _operands(rng, b, l, nh, nkv, hd, cap, 0.3)
    for used in KEYS:
        if used < l:
            continue
        want = oracle.attention(q, kc, vc, l, used)
        for at in (False, True):
            got = _run(q, kc, vc, l, used, 0, at)
            assert got.tobytes() == want.tobytes(), (l, hd, used, at)


@pytest.mark.parametrize("hd", (128, 64))
def test_decode_step_attention_window_and_grouped_heads(hd):
    rng = np.random.default_rng(7 + hd)
    b, nh, nkv, cap = 3, 6, 2, 1100
    for l in (1, 4):
        q, kc, vc = _operands(rng, b, l, nh, nkv, hd, cap, 0.3)
        for used, window in ((33, 0), (97, 40), (129, 100), (1030, 0), (1030, 333), (1030, 31), (1099, 64)):
            want = oracle.attention(q, kc, vc, l, used, window)
            for at in (False, True):
                got = _run(q, kc, vc, l, used, window, at)
                assert got.tobytes() == want.tobytes(), (l, hd, used, window, at)


@pytest.mark.parametrize("l", (1, 8))
def test_decode_step_attention_admission_fails_in_a_late_tile(l):
    """Subnormal-forcing operands in the last tiles only: tiny values (the value chain's products fall below 2^-126)
    and tiny keys (the score chain's), after hundreds of ordinary keys; and one subnormal word in the middle."""
    rng = np.random.default_rng(99 + l)
    b, nh, nkv, hd, cap, used = 2, 2, 1, 128, 1100, 1030
    q, kc, vc = _operands(rng, b, l, nh, nkv, hd, cap, 0.3)
    tiny = np.float32(2.0 ** -100)
    for variant in range(4):
        k2, v2, q2 = kc.copy(), vc.copy(), q.copy()
        if variant == 0:
            v2[:, :, 990:, :] *= tiny
        elif variant == 1:
            k2[:, :, 1000:, :] *= tiny
            q2 *= np.float32(2.0 ** -40)
        elif variant == 2:
            v2[0, 0, 517, 5] = np.float32(1e-41)
            k2[1, 0, 700, 77] = np.float32(-1e-42)
        else:
            v2[:, :, 64:96, :] *= np.float32(2.0 ** -120)  # a whole middle tile, ordinary tiles on both sides
        want = oracle.attention(q2, k2, v2, l, used)
        for at in (False, True):
            got = _run(q2, k2, v2, l, used, 0, at)
            assert got.tobytes() == want.tobytes(), (l, variant, at)


def value_chain_cases():
    """One decode row's chains with one feature zero but for a tile of words so small that each weighted one is flushed, the other
    features ordinary: the first, a middle and the last whole tile, with few rows (256 threads a row) and many (128)."""
    for hd in (64, 128):
        for b, nh in ((1, 2), (10, 32)):
            rng = np.random.default_rng(hd + b)
            used, d = 672, hd - 5
            q, kc, vc = _operands(rng, b, 1, nh, 1, hd, used, 0.01)
            for tile in (0, 10, 20):
                v2 = vc.copy()
                v2[:, :, :, d] = 0.0
                v2[:, :, 32 * tile:32 * tile + 32, d] = np.float32(2.0 ** -118)
                yield "head_dim %d, %d rows, tile %d" % (hd, b * nh, tile), d, q, kc, v2, used


def value_chain_right():
    """name -> whether all words are right, over the cases above; the walked feature's and the others' apart."""
    out = {}
    for name, d, q, kc, vc, used in value_chain_cases():
        want = oracle.attention(q, kc, vc, 1, used)
        hd = vc.shape[3]
        assert not want.reshape(-1, hd)[:, d].any(), name  # every weighted word is below 2^-126
        for at in (False, True):
            same = (_run(q, kc, vc, 1, used, 0, at).view(np.int32) == want.view(np.int32)).reshape(-1, hd)
            out["%s, at %d" % (name, at)] = (bool(same[:, d].all()), bool(np.delete(same, d, axis=1).all()))
    return out


def test_a_value_chain_takes_the_flushed_step_by_its_own_words():
    assert set(value_chain_right().values()) == {(True, True)}


def test_prefill_attention_against_the_oracle_at_head_dim_128_and_64():
    """A prompt-sized call (l > 8 takes the tiled kernels): 200 and 77 positions on an empty and on a part-filled cache."""
    rng = np.random.default_rng(5)
    for hd, l, used, window in ((128, 200, 200, 0), (64, 77, 300, 0), (128, 130, 130, 50), (64, 33, 1030, 0)):
        b, nh, nkv, cap = 2, 4, 2, max(used, 64)
        q, kc, vc = _operands(rng, b, l, nh, nkv, hd, cap, 0.3)
        want = oracle.attention(q, kc, vc, l, used, window)
        got = _run(q, kc, vc, l, used, window, False)
        assert got.tobytes() == want.tobytes(), (hd, l, used, window)


@pytest.mark.parametrize("l,hd,cap,used", [(1, 128, 8192, 8192), (1, 128, 7150, 7140), (1, 128, 10240, 8288), (2, 64, 2700, 2690), (2, 128, 8192, 8100),
                                           (4, 128, 1300, 1285), (4, 64, 8192, 6000), (8, 64, 600, 580), (8, 128, 4096, 3200)])
def test_few_rows_on_a_long_cache(l, hd, cap, used):
    """A lone sequence on a long cache: the launch spends an SM's whole shared memory on its score rows and its ring."""
    rng = np.random.default_rng(cap + l)
    q, kc, vc = _operands(rng, 1, l, 2, 1, hd, cap, 0.3)
    want = oracle.attention(q, kc, vc, l, used)
    for at in (False, True):
        got = _run(q, kc, vc, l, used, 0, at)
        assert got.tobytes() == want.tobytes(), at
