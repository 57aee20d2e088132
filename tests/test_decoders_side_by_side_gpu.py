"""Several decoders open in one process. How much dynamic shared memory a kernel may ask for is a property of the kernel and not of a decoder:
creating a small model must not lower it under a larger one that is open."""
import numpy as np
import pytest

import quintrit_b200 as q
from quintrit_b200 import gguf_io, synth

pytestmark = pytest.mark.gpu


def _block_scaled(hidden, inter):
    spec = synth.make_model(q.ARCH_LLAMA, True, hidden, inter, 1, 2, 1, 64, 300, 256, 500000.0, 1e-5, config=7, random_norms=True)
    shapes = [(128, hidden), (64, hidden), (64, hidden), (hidden, 128), (inter, hidden), (inter, hidden), (hidden, inter)]
    payloads = [(q.SRC_Q2_0, gguf_io.encode_q2_0(synth.trits(synth.seed_for(7, 0, p, 0), r * c).reshape(r, c), np.full(r * c // 64, 0.7, np.float16))) for p, (r, c) in enumerate(shapes)]
    return dict(spec, weights=payloads)


def _use(decoder, tokens):
    """Prompt, steps one by one and a step of several sequences; the logits of all of them."""
    out = [decoder.prefill(tokens)[0]]
    out += [decoder.forward(int(t), len(tokens) + i)[0] for i, t in enumerate(tokens[:2])]
    batch = q.Batch(decoder, 3)
    out.append(batch.step(None, tokens[:3], want_logits=True)[1])
    batch.free()
    return out


@pytest.mark.parametrize("blocks", [True, False], ids=["block-scaled", "per-tensor"])
def test_a_small_model_beside_a_large_one(blocks):
    spec = synth.make_model(q.ARCH_LLAMA, False, 2080, 2112, 3, 4, 2, 64, 300, 512, 500000.0, 1e-5, config=44, random_norms=True)  # (no multiple of 128: heads token by token)
    tokens = synth.prompt_tokens(3, 9, spec["vocab"])
    large = q.Decoder(spec)
    want = _use(large, tokens)
    small = q.Decoder(_block_scaled(64, 704) if blocks else synth.make_model(q.ARCH_LLAMA, False, 64, 96, 1, 2, 1, 64, 300, 256, 500000.0, 1e-5, config=45))
    small.forward(1, 0)
    for a, b in zip(_use(large, tokens), want):
        assert np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32))


def test_a_large_block_scaled_model_beside_a_small_one():
    spec = _block_scaled(12352, 64)  # 49 KB vectors: more than a kernel may ask for unless it is allowed to
    large = q.Decoder(spec)
    want = [large.forward(t, i)[0] for i, t in enumerate((5, 9, 2))]
    q.Decoder(_block_scaled(64, 704)).forward(1, 0)
    for i, t in enumerate((5, 9, 2)):
        assert np.array_equal(large.forward(t, i)[0].view(np.uint32), want[i].view(np.uint32))
