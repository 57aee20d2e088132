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
                                 'extern "C" int announced(int it, int until) { return qtb::gemm_announced(it, until); }\n'
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


class Barrier:
    """An mbarrier with one arrival a phase: the phase ends when that arrival has come and all announced bytes have."""

    def __init__(self):
        self.phase, self.arrived, self.bytes = 0, False, 0

    def _turn(self):
        if self.arrived and self.bytes == 0:
            self.phase, self.arrived = self.phase + 1, False

    def announce(self, n):
        assert not self.arrived
        self.arrived, self.bytes = True, self.bytes + n
        self._turn()

    def land(self, n):
        self.bytes -= n
        self._turn()


@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("stages,total", [(4, 4), (4, 9), (5, 11), (7, 9)])
def test_the_second_blocks_copies_are_seen_by_the_first(turns, stages, total, late):
    """The barriers in the first block on which the second one's activations complete: through the phases of whole runs, and where any load warp of either block stops at any
    stage, with copies that land at once (before they are announced) or, what has not been multiplied, only at the very end."""
    warps, act, tried = turns.load_warps(), 100, 0
    for ends in itertools.product(range(total + 1), repeat=2 * warps):
        if any(e != total and (e - k) % warps for k, e in enumerate(ends)):
            continue  # (a warp stops in front of a stage of its own)
        issued = [{it for it in range(total) if it < ends[block * warps + it % warps]} for block in (0, 1)]
        gap = next((it for it in range(total) if it not in issued[0] or it not in issued[1]), total)
        if any(it - stages >= gap for it in issued[0] | issued[1]):
            continue
        tried += 1
        bars, in_flight = [Barrier() for _ in range(stages)], []
        for it in range(total):
            if it in issued[1]:
                if late and it >= gap:
                    in_flight.append(it)
                else:
                    bars[it % stages].land(act)
            if it in issued[0]:
                bars[it % stages].announce(act)
            assert (bars[it % stages].phase == it // stages + 1) == (it in issued[0] and it in issued[1] and it not in in_flight)
        until = [[max((it + 1 for it in issued[block] if it % warps == w), default=0) for w in range(warps)] for block in (0, 1)]
        waited = []
        for w in range(warps):
            for it in range(turns.drain_from(max(until[1]), stages), until[1][w]):
                if it % warps == w:
                    if not turns.announced(it, until[0][w]):
                        bars[it % stages].announce(act)
                    waited.append(it)
        assert {it for it in issued[1] if it >= gap} <= set(waited)
        for it in in_flight:
            assert bars[it % stages].phase == it // stages  # (not taken for landed before it has)
            bars[it % stages].land(act)
        for it in waited:
            assert bars[it % stages].phase == it // stages + 1  # the phase behind the copies: its parity shows them
    assert tried > 10
