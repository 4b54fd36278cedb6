"""The decode attention kernels divide an SM's shared memory among the CTAs of a wave (ATT_SM_BYTES, ATT_CTA_BYTES): what a CTA has
beside its dynamic part has to fit the bytes that are set aside for it. Read from the sources, without a GPU."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mojolearn_b200", "csrc")
SM_TOTAL, SYSTEM = 228 * 1024, 1024  # bytes of an SM, and of them what the system takes for each CTA
STATIC = 384                         # static arrays of the largest of the two kernels (attn_decode_kernel<8>)


def _sources():
    return {os.path.basename(p): re.sub(r"//[^\n]*", "", open(p).read()) for p in glob.glob(os.path.join(CSRC, "*.cu*"))}


def _constant(text, name):
    value = re.search(r"\b%s = ([0-9 *]+)[,;]" % name, text).group(1)
    out = 1
    for factor in value.split("*"):
        out *= int(factor)
    return out


def test_a_wave_of_decode_attention_fits_an_sm():
    """The static arrays of every kernel of the library are rounded up to the strictest alignment that any of its kernels asks of
    its dynamic shared memory."""
    strictest = 16
    for name, text in _sources().items():
        for a in re.findall(r"extern __shared__ __align__\((\w+)\)", text):
            strictest = max(strictest, int(a) if a.isdigit() else _constant(text, a))
    text = _sources()["decoder.cuh"]
    sm, cta = _constant(text, "ATT_SM_BYTES"), _constant(text, "ATT_CTA_BYTES")
    static = -(-STATIC // strictest) * strictest
    for ctas in (1, 2, 3, 4):
        assert ctas * (sm // ctas - cta + static + SYSTEM) <= SM_TOTAL, (strictest, ctas)
