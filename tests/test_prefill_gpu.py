"""Prompt ingestion in chunks (quintrit_b200_decoder_prefill: batched projections on the tensor cores, the other steps with a token index in the
grid) against token-by-token decoding: the reference ingests a prompt one token at a time (quintrit-c/src/runtime.rs:430-436), so a batched pass has
to leave the same KV cache, position, logits and greedy choice, bit for bit."""
import numpy as np
import pytest

import oracle
import quintrit_b200 as q
from quintrit_b200 import synth

pytestmark = pytest.mark.gpu


def _spec(arch, f32_values, config, ctx=512, **kw):
    return synth.make_model(arch, f32_values, 256, 512, 2, 4, 2, 64, 300, ctx, 500000.0, 1e-5, config=config, random_norms=True, **kw)


@pytest.mark.parametrize("arch,f32_values,n", [(q.ARCH_LLAMA, False, 40), (q.ARCH_LLAMA, True, 17), (q.ARCH_BITNET, False, 33), (q.ARCH_LLAMA, False, 300)])
def test_chunked_ingestion_equals_single_steps(arch, f32_values, n):
    spec = _spec(arch, f32_values, 21 + n, tied=arch == q.ARCH_BITNET)
    tokens = synth.prompt_tokens(3, n, spec["vocab"])
    a, b = q.Decoder(spec), q.Decoder(spec)
    want = None
    for pos, t in enumerate(tokens):
        want, want_next = a.forward(int(t), pos)
    got, got_next = b.prefill(tokens)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and got_next == want_next
    # both continue identically (the cache and the position are the same)
    for step in range(6):
        la, ta = a.forward(want_next, n + step)
        lb, tb = b.forward(got_next, n + step)
        assert np.array_equal(la.view(np.uint32), lb.view(np.uint32)) and ta == tb
        want_next = got_next = ta
    # and the oracle agrees with the last logits
    ref = oracle.Model(spec)
    for pos, t in enumerate(tokens):
        r = ref.forward(int(t), pos)
    assert np.array_equal(got.view(np.uint32), r.view(np.uint32))


@pytest.mark.parametrize("heads,kv_heads,off", [(8, 1, False), (4, 2, True)])
def test_chunks_with_one_query_head_per_attention_block(monkeypatch, heads, kv_heads, off):
    """Where no attention kernel for the whole group of query heads exists (eight heads per KV head) or it is switched off, the
    kernel with one query head per block serves the tokens of a chunk, each at its own position."""
    if off:
        monkeypatch.setenv("QUINTRIT_B200_ATTN_GQA_OFF", "1")
    spec = synth.make_model(q.ARCH_LLAMA, False, 256, 512, 2, heads, kv_heads, 64, 300, 1024, 500000.0, 1e-5, config=41 + heads, random_norms=True)
    tokens = synth.prompt_tokens(7, 600, spec["vocab"])  # past 512 positions: all four KV chunks in use
    a, b = q.Decoder(spec), q.Decoder(spec)
    for pos, t in enumerate(tokens):
        want, want_next = a.forward(int(t), pos, want_logits=pos == len(tokens) - 1)
    got, got_next = b.prefill(tokens)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and got_next == want_next


def test_ingestion_in_two_calls_and_after_decoding():
    spec = _spec(q.ARCH_LLAMA, False, 77)
    tokens = synth.prompt_tokens(5, 90, spec["vocab"])
    a, b = q.Decoder(spec), q.Decoder(spec)
    for pos, t in enumerate(tokens):
        want, want_next = a.forward(int(t), pos)
    b.prefill(tokens[:50])
    lg, _ = b.forward(int(tokens[50]), 50)  # a single step in between
    got, got_next = b.prefill(tokens[51:], pos=51)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and got_next == want_next
    # rewriting from a shorter prefix (engine_gpu.rs:40-45)
    got2, _ = b.prefill(tokens[10:], pos=10)
    assert np.array_equal(got2.view(np.uint32), want.view(np.uint32))


def test_arguments():
    spec = _spec(q.ARCH_LLAMA, False, 78, ctx=256)
    d = q.Decoder(spec)
    with pytest.raises(q.QuintritError) as e:
        d.prefill(np.zeros(300, np.uint32))
    assert e.value.code == 11
    with pytest.raises(q.QuintritError) as e:
        d.prefill([5], pos=3)  # skips positions
    assert e.value.code == 2
    with pytest.raises(q.QuintritError) as e:
        d.prefill([100000])
    assert e.value.code == 2
    with pytest.raises(q.QuintritError) as e:
        d.prefill([])
    assert e.value.code == 2


@pytest.mark.parametrize("arch", [q.ARCH_LLAMA, q.ARCH_BITNET])
def test_many_chunks_replay_one_graph(arch):
    """From the third full pass on the launches of a pass are replayed as a CUDA graph: 3200 tokens = 3 full passes of 1024 (as they are, captured, replayed) and a tail, then
    another prompt on the same decoder, whose full passes are all replays. Against single steps, which take none of it."""
    spec = _spec(arch, arch == q.ARCH_BITNET, 79, ctx=4096, tied=arch == q.ARCH_BITNET)
    a, b = q.Decoder(spec), q.Decoder(spec)
    launches = []
    for seed, n in ((6, 3200), (7, 3100)):
        tokens = synth.prompt_tokens(seed, n, spec["vocab"])
        for pos, t in enumerate(tokens):
            want, want_next = a.forward(int(t), pos, want_logits=pos == n - 1)
        before = q.launch_count()
        got, got_next = b.prefill(tokens)
        launches.append(q.launch_count() - before)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and got_next == want_next
        for step in range(2):  # the caches are the same
            la, ta = a.forward(want_next, n + step)
            lb, tb = b.forward(got_next, n + step)
            assert np.array_equal(la.view(np.uint32), lb.view(np.uint32)) and ta == tb
            want_next = got_next = ta
    assert launches[1] < launches[0] / 2  # a replay launches nothing one by one: of the second prompt only the tail and the head



@pytest.mark.parametrize("arch,inter,n", [(q.ARCH_LLAMA, 512, 513), (q.ARCH_LLAMA, 4128, 1000), (q.ARCH_BITNET, 512, 1025), (q.ARCH_LLAMA, 512, 1600)])
def test_long_passes_equal_short_ones(arch, inter, n):
    """Passes of up to 1024 tokens, their feed-forward half in portions of 512, products over several token tiles: a portion of one token, ragged
    tiles, a second pass of one token and a longer one, against calls of at most 200 tokens (one token tile, one portion)."""
    spec = synth.make_model(arch, arch == q.ARCH_BITNET, 256, inter, 2, 4, 2, 64, 300, 1792, 500000.0, 1e-5, config=n, random_norms=True, tied=arch == q.ARCH_BITNET)
    tokens = synth.prompt_tokens(9, n, spec["vocab"])
    a, b = q.Decoder(spec), q.Decoder(spec)
    for at in range(0, n, 200):
        want, want_next = a.prefill(tokens[at:at + 200], at)
    got, got_next = b.prefill(tokens)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and got_next == want_next
    for step in range(3):  # the caches are the same
        la, ta = a.forward(want_next, n + step)
        lb, tb = b.forward(got_next, n + step)
        assert np.array_equal(la.view(np.uint32), lb.view(np.uint32)) and ta == tb
        want_next = got_next = ta


@pytest.mark.parametrize("arch,rope_dims", [(q.ARCH_LLAMA, 64), (q.ARCH_LLAMA, 32), (q.ARCH_LLAMA, 20), (q.ARCH_BITNET, 64), (q.ARCH_BITNET, 40), (q.ARCH_BITNET, 12)])
def test_rotated_dimensions_of_a_chunk(arch, rope_dims):
    """Heads rotated whole, in part (whole eights: rope_kv_rows_kernel; others: rope_kv_kernel), neighbouring and distant pairs, against single steps."""
    spec = _spec(arch, arch == q.ARCH_BITNET, 3 + rope_dims, tied=arch == q.ARCH_BITNET)
    spec["rope_dims"] = rope_dims
    tokens = synth.prompt_tokens(13, 45, spec["vocab"])
    a, b = q.Decoder(spec), q.Decoder(spec)
    for pos, t in enumerate(tokens):
        want, want_next = a.forward(int(t), pos)
    got, got_next = b.prefill(tokens)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and got_next == want_next
    la, lb = a.forward(want_next, 45)[0], b.forward(got_next, 45)[0]
    assert np.array_equal(la.view(np.uint32), lb.view(np.uint32))
