"""The output head of several tokens (lm_head_batch_kernel) and of one (lm_head_kernel) against single steps through the token kernel,
whose logits the oracle pins: group sizes of 8, 16 and 32 tokens and the remainders beside them, vocabularies that end inside a tile of
rows, hidden sizes of one and more column blocks and one that only the single-token kernel takes, both table types. Equality of bits."""
import numpy as np
import pytest

import quintrit_b200 as q
from quintrit_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("hidden,vocab", [(128, 300), (384, 1027), (896, 129), (352, 515)])
def test_logits_of_a_batch_equal_single_steps(hidden, vocab, bf16):
    spec = synth.make_model(q.ARCH_LLAMA, False, hidden, 256, 1, 2, 1, 64, vocab, 256, 500000.0, 1e-5, config=110 + hidden, random_norms=True, bf16_tables=bf16)
    one, many = q.Decoder(spec), q.Decoder(spec)
    tokens = np.arange(40, dtype=np.uint32) * 7 % vocab
    want = [one.forward(int(t), 0) for t in tokens]
    for n in (1, 2, 7, 8, 9, 16, 17, 32, 33, 40):
        batch = q.Batch(many, n)
        got, logits = batch.step(None, tokens[:n], want_logits=True)
        for z in range(n):
            assert np.array_equal(logits[z].view(np.uint32), want[z][0].view(np.uint32)), (n, z)
            assert got[z] == want[z][1]
        batch.free()
    for pos, t in enumerate(tokens[:9]):
        last, _ = one.forward(int(t), pos)
    assert np.array_equal(many.prefill(tokens[:9])[0].view(np.uint32), last.view(np.uint32))


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("hidden", [128, 384])
def test_a_vocabulary_of_several_tiles_a_block(hidden, bf16):
    """40037 rows: with 148 blocks every block of lm_head_batch_kernel walks two tiles of 128 rows, four of 64 or eight of 32 and more, some blocks one
    more than others, and lm_head_kernel's blocks a second round; the last tile is short. One column block and three."""
    vocab = 40037
    spec = synth.make_model(q.ARCH_LLAMA, False, hidden, 128, 1, 2, 1, 64, vocab, 256, 500000.0, 1e-5, config=120 + hidden, random_norms=True, bf16_tables=bf16)
    one, many = q.Decoder(spec), q.Decoder(spec)
    tokens = np.arange(33, dtype=np.uint32) * 1201 % vocab
    want = [one.forward(int(t), 0) for t in tokens]
    for n in (1, 2, 9, 17, 33):
        batch = q.Batch(many, n)
        got, logits = batch.step(None, tokens[:n], want_logits=True)
        for z in range(n):
            assert np.array_equal(logits[z].view(np.uint32), want[z][0].view(np.uint32)), (n, z)
            assert got[z] == want[z][1]
        batch.free()
