"""The recurrences of a prompt in segments that scan side by side (chunk_scan_kernel with segments, chunk_carry_kernel): state sizes of every
instantiation, lengths at which the number of segments changes or the last one is short, a second portion that starts from a state, against
the same prompt in portions too short for segments (those the oracle pins: test_layered_gpu.py). Both are the same sums in another order, rounded
in the same places, so their logits are about as close as two roundings to bfloat16 of the mixer's output: a tenth of the tolerance against the
oracle holds them together."""
import numpy as np
import pytest

from quintrit_b200 import model_folder as mf
from quintrit_b200.runtime import Model

pytestmark = pytest.mark.gpu

M, H = mf.mamba2, mf.hgrn2
LAYERS = {
    "mamba2 20": M(6, 24, 20, groups=3, conv=3, norm_groups=4, ff=72),
    "mamba2 64": M(2, 80, 64, groups=2, conv=4, norm_groups=2),
    "mamba2 100": M(3, 64, 100, groups=1, conv=2, norm_groups=1, ff=40),
    "hgrn2 24": H(5, 24, 40, ff=56),
    "hgrn2 60": H(2, 60, 130),
    "hgrn2 128": H(3, 128, 64, ff=40),
}


@pytest.mark.parametrize("name", LAYERS)
def test_segments_equal_short_portions(tmp_path, name):
    layer, vocab = LAYERS[name], 53
    config = mf.lasosun_config([layer, layer], 64, vocab, 3000, eps=3e-5, embed_scale=1.3)
    model = Model.load(mf.write_folder(str(tmp_path / "m"), config, mf.random_lasosun(config, 5)), context=3000)
    ids = np.random.default_rng(3).integers(0, vocab, 2400)
    a, b = model.new_session(), model.new_session()
    at = 0
    for n in (384, 385, 1000, 631):  # 24 chunks: three segments of eight; 25: the last is short; 63; 40
        got = a.feed(ids[at:at + n], range(n))
        want = np.concatenate([b.feed(ids[i:min(i + 100, at + n)], range(min(100, at + n - i))) for i in range(at, at + n, 100)])
        d = np.asarray(got, np.float64) - want
        e = np.sqrt((d * d).mean(-1)) / np.sqrt((np.asarray(want, np.float64) ** 2).mean())
        assert e.max() < 5e-3, f"portion of {n} at {at}, place {int(e.argmax())}: {e.max():.2e}"
        at += n
