"""Attention of prompt chunks, eight tokens of a KV head to a block (attention_tile_kernel), against single steps, whose attention the
oracle pins (test_decoder_gpu.py): group sizes, head sizes and numerics of every instantiation, portions that start and end inside a
tile of eight tokens and inside a tile of 64 cache rows, across the position (512) where the cache is divided into four chunks and the
multiples of 256 where the division changes. Equality of bits."""
import numpy as np
import pytest

import quintrit_b200 as q
from quintrit_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32_values", [False, True])
@pytest.mark.parametrize("group,head_dim", [(1, 64), (2, 64), (3, 64), (4, 64), (1, 128), (2, 128), (3, 128), (4, 128), (1, 256), (2, 256), (3, 256), (4, 256)])
def test_portions_equal_single_steps(group, head_dim, f32_values):
    kv_heads = 1 if head_dim == 256 else 2
    spec = synth.make_model(q.ARCH_LLAMA, f32_values, 256, 512, 1, group * kv_heads, kv_heads, head_dim, 300, 1024, 500000.0, 1e-5, config=90 + group, random_norms=True)
    spec["scales"] = (spec["scales"] * np.float32(0.06)).astype(np.float32)  # scores of a few units: weights spread over many positions
    portions = (45, 300, 200, 70, 290, 33)  # 256 of the 300 and of the 290, the 200 (they cross position 512) and the 70 take that kernel
    tokens = synth.prompt_tokens(9, sum(portions), spec["vocab"])
    a, b = q.Decoder(spec), q.Decoder(spec)
    pos = 0
    for n in portions:
        for i in range(n):
            want, want_next = a.forward(int(tokens[pos + i]), pos + i, want_logits=i == n - 1)
        got, got_next = b.prefill(tokens[pos:pos + n], pos=pos)
        pos += n
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and got_next == want_next, pos
    for step in range(2):  # the caches are the same
        (x, tx), (y, ty) = a.forward(want_next, pos + step), b.forward(got_next, pos + step)
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)) and tx == ty
        want_next = got_next = tx


@pytest.mark.parametrize("f32_values", [False, True])
@pytest.mark.parametrize("group,head_dim", [(1, 64), (4, 64), (2, 128), (3, 128), (1, 256), (3, 256), (3, 32), (2, 96), (3, 96), (3, 224)])
def test_short_portions_behind_long_contexts(group, head_dim, f32_values):
    """Portions too short for tiles of tokens (attention_rows_kernel, for the head sizes it does not take attention_gqa_kernel: a block per token, KV head and chunk) where a
    chunk takes more than one round of 256 positions, with a round of one position (chunks of 320 and 576: rounds of 64; position 1281 leaves one row in the last chunk),
    against single steps."""
    kv_heads = 1 if head_dim == 256 else 2
    spec = synth.make_model(q.ARCH_LLAMA, f32_values, 256, 512, 1, group * kv_heads, kv_heads, head_dim, 300, 2304, 500000.0, 1e-5, config=70 + group, random_norms=True)
    spec["scales"] = (spec["scales"] * np.float32(0.06)).astype(np.float32)  # scores of a few units: weights spread over many positions
    tokens = synth.prompt_tokens(11, 2304, spec["vocab"])
    a, b = q.Decoder(spec), q.Decoder(spec)
    for before, n in [(1000, 24), (1279, 5), (1540, 2), (2290, 14)]:
        for d in (a, b):
            d.prefill(tokens[:before])
        for i in range(n):
            want, want_next = a.forward(int(tokens[before + i]), before + i, want_logits=i == n - 1)
        got, got_next = b.prefill(tokens[before:before + n], pos=before)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and got_next == want_next, before
