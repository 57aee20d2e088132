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
