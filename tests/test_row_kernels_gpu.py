"""The steps between the batched projections (norm_quant_rows_kernel, attn_finish_rows_kernel, act_quant_rows_kernel) against single steps, whose
kernels the oracle pins: vector lengths that leave lanes of a warp, blocks of a cluster or turns of a thread without elements, with and
without sub-norms. Equality of bits."""
import numpy as np
import pytest

import quintrit_b200 as q
from quintrit_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arch,hidden,inter,heads,kv_heads,head_dim", [
    (q.ARCH_LLAMA, 96, 32, 2, 1, 64),        # one element quad in each block of a cluster
    (q.ARCH_LLAMA, 160, 1056, 3, 1, 64),     # lengths that are no multiples of 128
    (q.ARCH_BITNET, 544, 8224, 3, 1, 96),    # a second turn of the activation's threads, sub-norms, a head size that is no power of two
    (q.ARCH_LLAMA, 4128, 16416, 5, 1, 256),  # a second turn of the norm's threads, a third of the activation's
    (q.ARCH_LLAMA, 128, 24608, 34, 2, 128),  # a second turn of the attention's threads, a fourth of the activation's
    (q.ARCH_BITNET, 128, 32800, 2, 1, 64),   # the activation step with blocks of 512 threads
    (q.ARCH_BITNET, 128, 51200, 2, 1, 64),   # the longest vector a model may have: a fourth turn of those
    (q.ARCH_LLAMA, 8224, 64, 2, 1, 64),      # a third turn of the norm's threads
    (q.ARCH_LLAMA, 128, 128, 68, 17, 128),   # a third turn of the attention's threads
])
def test_prompt_equals_single_steps(arch, hidden, inter, heads, kv_heads, head_dim):
    spec = synth.make_model(arch, False, hidden, inter, 2, heads, kv_heads, head_dim, 300, 1024, 500000.0, 1e-5, config=hidden % 97, random_norms=True, tied=arch == q.ARCH_BITNET)
    n = 530 if inter < 1100 else 9  # the first two past position 512, where the cache is divided into four chunks
    tokens = synth.prompt_tokens(11, n, spec["vocab"])
    a, b = q.Decoder(spec), q.Decoder(spec)
    for pos, t in enumerate(tokens):
        want, want_next = a.forward(int(t), pos, want_logits=pos == n - 1)
    got, got_next = b.prefill(tokens)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and got_next == want_next
    (x, tx), (y, ty) = a.forward(want_next, n), b.forward(got_next, n)
    assert np.array_equal(x.view(np.uint32), y.view(np.uint32)) and tx == ty


@pytest.mark.parametrize("hidden", [64, 960, 4160])  # lanes of a warp without elements, several warps, a second turn of the threads
def test_block_scaled_steps(oracle, hidden):
    """The norm of a block-scaled model's step (norm_quant_rows_kernel with BLOCKS) against the oracle."""
    from quintrit_b200 import gguf_io

    spec = synth.make_model(q.ARCH_LLAMA, True, hidden, 704, 2, 4, 2, 64, 300, 256, 500000.0, 1e-5, config=hidden % 89, random_norms=True)
    shapes = [(256, hidden), (128, hidden), (128, hidden), (hidden, 256), (704, hidden), (704, hidden), (hidden, 704)]
    rng = np.random.default_rng(hidden)
    payloads, block_scales = [], []
    for l in range(2):
        for p, (r, c) in enumerate(shapes):
            sc = rng.uniform(0.5, 2.0, r * c // 64).astype(np.float16)
            payloads.append((q.SRC_Q2_0, gguf_io.encode_q2_0(synth.trits(synth.seed_for(hidden % 89, l, p, 0), r * c).reshape(r, c), sc)))
            block_scales.append(sc.astype(np.float32))
    dec, ref = q.Decoder(dict(spec, weights=payloads)), oracle.Model(dict(spec, block_scales=block_scales))
    for pos, tok in enumerate(synth.prompt_tokens(5, 4, spec["vocab"])):
        want, got = ref.forward(int(tok), pos), dec.forward(int(tok), pos)[0]
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), pos
