"""Output and down projection of few tokens, whose tiles are shared by the blocks of a cluster (dense_gemm_tc_kernel, SPLIT): two, four and eight blocks, a K that
does not divide evenly, a boundary between the two products inside a block's range, a second row tile that is mostly padding, widths that are
no multiple of four, token counts around a block's share and around a tile."""
import numpy as np
import pytest

from oracle import layered as plain
from quintrit_b200 import model_folder as mf
from quintrit_b200.runtime import Model

pytestmark = pytest.mark.gpu

M, H = mf.mamba2, mf.hgrn2
CASES = [
    (200, [M(16, 64, 32, groups=2, conv=3, norm_groups=4, ff=3200)]),   # 16 + 50 slices on eight blocks
    (130, [H(8, 32, 64, ff=1100), M(6, 64, 32, groups=1, conv=2, norm_groups=2, ff=700)]),  # 8 + 18 on two; 6 + 11 on two
    (96, [M(20, 64, 16, groups=1, conv=2, norm_groups=1, ff=1000)]),    # 20 + 16 on four
    (136, [M(33, 64, 16, groups=1, conv=2, norm_groups=1)]),            # one product alone: 33 on four
]


@pytest.mark.parametrize("tokens", [9, 17, 128, 143])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_shared_tiles(tmp_path, case, tokens):
    width, layers = CASES[case]
    config = mf.lasosun_config(layers, width, 41, 300, eps=3e-5)
    bits = mf.random_lasosun(config, 31 + case)
    w = {k: mf.bf16_floats(v) for k, v in bits.items()}
    model = Model.load(mf.write_folder(str(tmp_path / "m"), config, bits), context=300)
    ids = np.random.default_rng(tokens).integers(0, 41, tokens)
    want = plain.lasosun(config, w, ids)
    d = np.asarray(model.new_session().feed(ids, range(tokens)), np.float64) - want
    d -= d.mean(-1, keepdims=True)
    base = want - want.mean(-1, keepdims=True)
    assert (np.sqrt((d * d).mean(-1)) / np.sqrt((base * base).mean())).max() < 5e-2  # the tolerance of bfloat16 models (test_layered_gpu.py)


A = mf.attention
SHARED = mf.experts(8, 2, 96, 1100, groups=2, keep=1)
RET = mf.retention(8, 64, 128)
# (design, width, layers): attention and retention give a place the same bits whatever follows it, so that between a prompt and the beginning of a
# longer one only the split of the sums differs
PREFIXES = {
    "two products on eight blocks": ("lasosun", 1024, [A(8, 2, 128, 128, 64, 16, ff=3200)]),  # 16 + 50 slices
    "boundary inside a range": ("lasosun", 1024, [A(8, 2, 128, 128, 64, 16, ff=700)]),        # 16 + 11 on two blocks
    "one product": ("lasosun", 1024, [A(16, 4, 64, 72, 64, 16)]),                             # 18 on two
    "gate of a token": ("tosevik", 1024, [mf.retention_layer(RET, SHARED)]),                  # the shared expert: 18 on two; retention's output: 16 on two
}


@pytest.mark.parametrize("tokens", [9, 128, 200])
@pytest.mark.parametrize("name", PREFIXES)
def test_shared_tiles_equal_whole_ones(tmp_path, name, tokens):
    """A prompt of few tokens (tiles shared by a cluster) against the same places of one of 1152 (72 tiles, a block each). The sums differ in the order
    in which 32-bit partial results are added (some 1e-7 of them); rounded to bfloat16 behind that, a value now and then takes the other neighbour,
    2^-8 away. In a vector of 1024 values one that is three times the usual size moves the result by 3 * 2^-8 / 32 = 3.7e-4: that is the head's input,
    the one vector behind the sums of a Lasosun layer. Behind a layer with experts there are also an expert's 96 channels, where one such value is 1.2e-3
    of that expert's result. A missing slice of K or gate is 0.05 and more."""
    design, width, layers = PREFIXES[name]
    most = 5e-4 if design == "lasosun" else 2e-3
    if design == "lasosun":
        config = mf.lasosun_config(layers, width, 41, 1200, eps=3e-5)
        bits = mf.random_lasosun(config, 7)
    else:
        config = mf.tosevik_config(layers, width, 41, eps=3e-5)
        bits = mf.random_tosevik(config, 7)
    model = Model.load(mf.write_folder(str(tmp_path / "m"), config, bits), context=1200)
    ids = np.random.default_rng(5).integers(0, 41, 1152)
    whole = np.asarray(model.new_session().feed(ids, range(tokens), keep_context=False), np.float64)
    got = np.asarray(model.new_session().feed(ids[:tokens], range(tokens), keep_context=False), np.float64)
    e = np.sqrt(((got - whole) ** 2).mean(-1)) / np.sqrt((whole * whole).mean())
    assert e.max() < most, f"place {int(e.argmax())}: {e.max():.2e}"


@pytest.mark.parametrize("width,tokens", [(2048, 2000), (2560, 2048)])  # one wave of 256-token tiles; a block's second tile waits for its one set of accumulators
def test_wide_tiles_of_two_products(tmp_path, width, tokens):
    """The dual form with 256-token tiles against the same prompt in portions that take 128-token tiles: every sum runs over K in the same order, so
    the logits are equal to the bit. The 32-bit mode pins the values."""
    config = mf.lasosun_config([A(4, 1, 64, 64, 64, 16, ff=160), A(2, 2, 64, 64, 64, 16, ff=96)], width, 41, 2100, eps=3e-5)
    path = mf.write_folder(str(tmp_path / "m"), config, mf.random_lasosun(config, 11))
    model = Model.load(path, context=2100)
    ids = np.random.default_rng(6).integers(0, 41, tokens)
    got = np.asarray(model.new_session().feed(ids, range(tokens), keep_context=False))
    one = model.new_session()
    portions = [np.asarray(one.feed(ids[i:i + 1024], range(len(ids[i:i + 1024])))) for i in range(0, tokens, 1024)]
    exact = Model.load(path, context=2100, dtype="float32").new_session().feed(ids, range(tokens), keep_context=False)
    e = np.sqrt(((got - np.asarray(exact, np.float64)) ** 2).mean(-1)) / np.sqrt((np.asarray(exact, np.float64) ** 2).mean())
    assert e.max() < 2e-2, f"place {int(e.argmax())}: {e.max():.2e}"  # a few roundings to bfloat16, 2^-9 each
    assert np.array_equal(got.view(np.uint32), np.concatenate(portions).view(np.uint32))
