"""The exits of the batched projection's load warps (csrc/gemm_turns.hpp), followed on the host: wherever a warp stops, what it waits for is what may still be in flight."""
import ctypes
import itertools
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quintrit_b200", "csrc")


@pytest.fixture(scope="module")
def turns(tmp_path_factory):
    d = tmp_path_factory.mktemp("turns")
    (d / "turns.cpp").write_text('#include "gemm_turns.hpp"\nextern "C" int drain_from(int until, int stages) { return qtb::gemm_drain_from(until, stages); }\n'
                                 'extern "C" int load_warps() { return qtb::kGemmLoadWarps; }\n')
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "turns.so"), str(d / "turns.cpp")], check=True)
    return ctypes.CDLL(str(d / "turns.so"))


@pytest.mark.parametrize("stages", [4, 5, 7, 12])
@pytest.mark.parametrize("total", [1, 3, 13, 30])
def test_load_warps_that_stop_anywhere_wait_for_their_own_copies(turns, stages, total):
    """Either warp stops in front of any stage or behind the last, in the middle of an item too: together they wait for what may be in flight, and only at buffers that have
    not been used again (a barrier two phases on would never show the phase that is waited for)."""
    warps = turns.load_warps()
    stops = range(total + warps)
    for ends in itertools.product(stops, repeat=warps):
        issued = sorted(it for w in range(warps) for it in range(w, min(ends[w], total), warps))
        gap = next((it for it in range(total) if it not in issued), total)  # the products get no further than the first stage that is missing
        if any(it - stages >= gap for it in issued):
            continue  # a stage is issued when the one in its buffer has been multiplied
        until = [max((it + 1 for it in issued if it % warps == w), default=0) for w in range(warps)]
        read = max((it - stages for it in issued), default=-1)  # seen done by one warp or the other
        waited = [it for w in range(warps) for it in range(turns.drain_from(max(until), stages), until[w]) if it % warps == w]
        assert {it for it in issued if it > read} == set(waited)
        for it in waited:
            assert it + stages not in issued
