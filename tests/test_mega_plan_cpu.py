"""The token kernel's shared-memory plan (csrc/mega_plan.hpp) on the host: which models take the kernel, and that what they need is there."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quintrit_b200", "csrc")
LIMIT = 227 * 1024  # shared memory a block may ask for

SOURCE = """
#include <initializer_list>

#include "mega_plan.hpp"
using namespace qtb;
extern "C" long plan(int ctx, int gqa, int hd, int hidden, int maxvec, int layers, int v2) {
    return static_cast<long>(mega_smem_bytes(mega_attn_region(ctx, gqa, hd, hidden, v2 != 0), maxvec, hidden, layers));
}
extern "C" long charge(int ctx, int gqa, int hd, int hidden, int maxvec, int layers, int v2) { return static_cast<long>(mega_charge(ctx, gqa, hd, hidden, maxvec, layers, v2 != 0)); }
// the most by which the plan exceeds what is charged, over all contexts, groups and head sizes that the kernel takes
extern "C" long worst() {
    long w = -(1L << 40);
    for (int hd = 64; hd <= 256; hd *= 2)
        for (int gqa = 1; gqa <= 16; ++gqa)
            for (int ctx = 8; ctx <= 8192; ctx += 8)
                for (int v2 = 0; v2 < (gqa <= kV2MaxGqa && ctx <= kV2MaxCtx ? 2 : 1); ++v2)
                    for (int hidden : {32, 64, 1024, 2560, 5120, 9600})
                        for (int layers : {1, 2, 40})
                            for (int maxvec = hidden; maxvec <= hidden + 2048; maxvec += 2048) {
                                const long c = charge(ctx, gqa, hd, hidden, maxvec, layers, v2), d = plan(ctx, gqa, hd, hidden, maxvec, layers, v2) - c;
                                if (c <= 227 * 1024 && d > w) w = d;
                            }
    return w;
}
extern "C" int dead_bytes_needed() { return kMegaMaxHeads * 12 * 4; }
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "plan.so"), str(d / "plan.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "plan.so"))
    lib.plan.restype = lib.charge.restype = lib.worst.restype = ctypes.c_long
    return lib


def form(plan, ctx, gqa, hidden, layers, hd=128):
    """2, 1: the token kernel with the second or first form of the attention's second half; 0: one kernel per step."""
    if gqa <= 7 and ctx <= 4096 and plan.charge(ctx, gqa, hd, hidden, hidden, layers, 1) <= LIMIT:
        return 2
    return 1 if plan.charge(ctx, gqa, hd, hidden, hidden, layers, 0) <= LIMIT else 0


def test_what_is_charged_is_there(plan):
    assert plan.worst() <= 0


@pytest.mark.parametrize("gqa,hidden,layers,ctx,want", [
    (4, 4096, 32, 2816, 2), (4, 4096, 40, 2816, 2), (3, 5120, 40, 3072, 2), (7, 4096, 32, 2048, 2),  # just inside the second form
    (4, 2048, 40, 8192, 1), (3, 4096, 32, 8192, 1),                                                  # just inside the kernel
    (4, 4096, 32, 3072, 1), (7, 4096, 32, 2304, 1), (4, 4096, 40, 8192, 0), (3, 8192, 32, 8192, 0),  # and outside
    (3, 3072, 40, 1280, 2), (4, 2560, 30, 4096, 1), (1, 3072, 40, 8192, 1)])
def test_models_at_the_edge_take_the_kernel_they_took(plan, gqa, hidden, layers, ctx, want):
    assert form(plan, ctx, gqa, hidden, layers) == want


def test_the_factors_lie_in_front_of_the_tables_first_zero_row(plan):
    """Between two GEMVs the chunk-combine factors of 64 heads use the table's rows before row 27, the first that is never written."""
    assert plan.dead_bytes_needed() <= 27 * 256
