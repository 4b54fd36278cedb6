"""The order of copies and waits of the streaming kernel's rings (csrc/stream_ring.cuh), with the host compiler: a barrier is armed
once a phase, every copy is waited for in its own phase, and after a wait that ran out nothing is asked for and nothing is left in
flight."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mojolearn_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "stream_ring.cuh"
struct Barrier { unsigned phase = 0; bool armed = false; }; // the phase that its next completion ends
int main(int argc, char **argv) {
    const int stages = atoi(argv[1]), copies = atoi(argv[2]), fails_at = atoi(argv[3]); // the wait of this number runs out, its copy lands later
    std::vector<Barrier> bar(stages);
    std::vector<int> holds(stages, -1);
    int asked = 0, read = 0, waits = 0;
    bool lost = false;
    auto fill = [&](int slot) {
        if (asked == copies) return false;
        if (lost) { puts("a copy after the wait ran out"); exit(1); }
        if (bar[slot].armed) { puts("a barrier armed twice in a phase"); exit(1); }
        bar[slot].armed = true;
        holds[slot] = asked++;
        return true;
    };
    auto wait = [&](int slot, unsigned phase) {
        if (!bar[slot].armed || bar[slot].phase != phase) { puts("a wait for a phase that nothing completes"); exit(1); }
        if (waits++ == fails_at) { lost = true; return false; }
        bar[slot].armed = false;
        bar[slot].phase ^= 1u;
        return true;
    };
    b200i::StreamRing ring{stages};
    ring.start(fill);
    while (read < copies) {
        if (!wait(ring.slot, ring.phase)) { ring.drain(wait); break; }
        if (holds[ring.slot] != read) { puts("copies out of order"); return 1; }
        read++;
        ring.release(fill);
    }
    for (const Barrier &b : bar) if (b.armed) { puts("a copy left in flight"); return 1; }
    if (lost != (fails_at < copies) || read != (lost ? fails_at : copies)) { puts("counts"); return 1; }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    (d / "ring.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / "ring.cpp"), "-o", str(d / "ring")], check=True)
    return str(d / "ring")


@pytest.mark.parametrize("stages", [1, 2, 3])
def test_every_copy_is_waited_for_once_and_in_order(program, stages):
    for copies in (0, 1, 2, 3, 4, 7, 32):
        for fails_at in {0, 1, 2, 3, 5, copies - 1, copies} - {-1}:
            run = subprocess.run([program, str(stages), str(copies), str(fails_at)], capture_output=True, text=True)
            assert run.returncode == 0, (copies, fails_at, run.stdout)


def test_the_streaming_kernel_waits_as_a_warp():
    """Its one wait is voted on, and it goes through the ring."""
    with open(os.path.join(CSRC, "gemm_stream.cuh")) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    assert code.count("mbar_wait(") == code.count("__all_sync(0xFFFFFFFFu, mbar_wait(") == 1
    assert code.count("t8_tma_load(") == 1 and "flow.start(fill)" in code and "flow.drain(StreamWait{full})" in code and "flow.release(fill)" in code


def test_the_value_rings_of_decode_attention_fill_nothing_after_a_lost_wait():
    """Whichever thread's wait runs out reports it and ends there; the thread that fills the slots drains its copies first."""
    with open(os.path.join(CSRC, "decoder.cuh")) as f:
        code = re.sub(r"\s+", " ", re.sub(r"//[^\n]*", "", f.read()))
    fillers = re.findall(r"if \(!mbar_wait\([^{};]*\)\) \{ value_ring_lost\(full, tid == (\w+), k, stages, nstages\); return; \}", code)
    assert fillers == ["issuer", "0"]
    assert code.count("mbar_wait(") == 3  # those two, and the drain's own
    assert "else if (refill && tid == issuer) copy_bulk(" in code and "if (tid == 0 && k < nstages) {" in code
