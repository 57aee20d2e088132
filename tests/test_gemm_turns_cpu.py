"""The exits of the batched projection's load warps (csrc/gemm_turns.hpp), followed on the host: wherever a warp stops, what it waits for is what may still be in flight."""
import ctypes
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


def stages_of(warp, warps, total):
    return range(warp, total, warps)


@pytest.mark.parametrize("stages", [4, 5, 12])
@pytest.mark.parametrize("items,per", [(1, 3), (1, 90), (2, 90), (3, 12), (5, 1)])
def test_a_load_warp_that_stops_anywhere_waits_for_its_own_copies(turns, stages, items, per):
    """The warp stops in front of any stage (in the middle of an item of 90 stages too, of which only a few are in flight) or behind the last."""
    warps, total = turns.load_warps(), items * per
    for warp in range(warps):
        mine = list(stages_of(warp, warps, total))
        for stop in range(len(mine) + 1):
            issued = mine[:stop]
            until = issued[-1] + 1 if issued else 0
            # the products of stage i - stages were seen done before i was issued, and with them everything up to it
            read = max((i - stages for i in issued), default=-1)
            in_flight = {i for i in issued if i > read}
            waited = {i for i in range(turns.drain_from(until, stages), until) if i % warps == warp}
            assert waited == in_flight
            assert len({i % stages for i in waited}) == len(waited)  # every buffer's barrier once: its last use
