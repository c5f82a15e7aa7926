"""The decode step of two launches a block (block_step.cu, head_row.cu) against the oracle and against the other forms of a step."""
import numpy as np
import pytest

import ferrum_cpu_b200 as fcb
from ferrum_cpu_b200 import _lib, synth
from ferrum_cpu_b200.llama import CudaLlama
from tests import oracle as O

pytestmark = pytest.mark.gpu


# rows that do not fill a warp's units or the threads' shares, two and three hidden units a warp, one to sixteen slices of them,
# clusters with fewer positions than CTAs, and contexts their shares do not divide
@pytest.mark.parametrize("d,heads,ff,ctx,prompt,new,vocab", [(512, 8, 2048, 40, 1, 30, 515), (640, 10, 2560, 61, 3, 50, 515), (768, 12, 3072, 24, 9, 14, 4099),
                                                             (896, 14, 4608, 200, 190, 9, 515), (1024, 16, 256, 70, 8, 40, 515)])
def test_tokens_and_probabilities(d, heads, ff, ctx, prompt, new, vocab):
    sm = synth.SynthModel(2, d, heads, ff, ctx, vocab, seed=d + ff, perturb=True)
    om, gm = O.OracleModel(sm), fcb.CudaSlm(sm.config, sm.weights)
    ids = synth.token_ids(4, prompt, vocab)
    want, margin = om.generate_greedy(ids, new)
    fcb.take_launch_count()
    got, _ = gm.generate_tokens(ids, new)
    assert fcb.take_launch_count() < 8 * new + 100          # seven launches a step: two a block, embedding, head, pick
    for i, (a, b) in enumerate(zip(got, want)):
        assert a == b or margin[i] < 1e-4, i
        if a != b:
            break
    gm.set_decode_mode(1)                                   # feeds take the same step
    om.prime(ids), gm.prime(ids)
    for t in want[: min(len(want), ctx - prompt)]:
        assert np.abs(gm.feed(t) - om.feed(t)).max() < 2e-5
    gm.close()
    om.close()


# one CTA of the head and as many as the chip has, a last span that is not full, rows that no CTA reaches a second time
@pytest.mark.parametrize("vocab", [31, 515, 4736, 9501])
@pytest.mark.parametrize("rows", ["ties", "flat", "nan"])
def test_pick_reads_the_rows_that_reach_the_largest(vocab, rows):
    """Equal rows all over the head: the first of them is picked. Rows that all lie within the bound, and rows without mass: the first."""
    sm = synth.SynthModel(1, 512, 8, 2048, 32, vocab, seed=vocab, perturb=True)
    table = synth.q8_0_dequantize(sm.token_embd, vocab * 512).reshape(vocab, 512)
    if rows == "ties":
        table = table[np.arange(vocab) % 131]
    elif rows == "flat":
        table[:] = table[0]
    else:
        sm.out_norm_g[:] = np.nan
    sm.token_embd[:] = synth.q8_0_quantize(table)
    om, gm = O.OracleModel(sm), fcb.CudaSlm(sm.config, sm.weights)
    ids = synth.token_ids(4, 3, vocab)
    want = om.generate_greedy(ids, 12)[0]
    assert (want < min(vocab, 131) if rows == "ties" else want == 0).all()
    gm.set_decode_mode(1)                                   # the prompt by the same step, not by the persistent kernel
    assert np.array_equal(gm.generate_tokens(ids, 12)[0], want)
    gm.close()
    om.close()


# the persistent kernel, the chain, what a new stream takes (a prompt on the persistent kernel, or as a window), and streams in lock step;
# widths whose heads give a CTA fewer strips than an item holds, and more
@pytest.mark.parametrize("d,heads", [(128, 2), (512, 8), (768, 12)])
@pytest.mark.parametrize("vocab", [515, 4736, 9501, 50257])
@pytest.mark.parametrize("mode,prompt", [(0, 3), (1, 3), (2, 3), (2, 80), ("batch", 5)])
def test_the_first_of_equal_rows_is_picked(d, heads, vocab, mode, prompt):
    sm = synth.SynthModel(1, d, heads, 256, 128, vocab, seed=vocab, perturb=True)
    blocks = sm.token_embd.reshape(vocab, d // 32 * 34)
    blocks[:] = blocks[np.arange(vocab) % 131]
    gm = fcb.CudaSlm(sm.config, sm.weights)
    ids = synth.token_ids(4, 2 * prompt, vocab).reshape(2, prompt)
    if mode == "batch":
        got = np.concatenate(gm.decode_batch(ids, 12))
    else:
        gm.set_decode_mode(mode)
        got = gm.generate_tokens(ids[0], 12)[0]
    assert (got < min(vocab, 131)).all()
    gm.close()


def test_scores_of_minus_infinity_and_huge_rows():
    """A row without a finite logit ends as it does in the step of five launches: no id beyond the vocabulary, no hang."""
    sm = synth.SynthModel(1, 512, 8, 2048, 32, 515, seed=3)
    sm.position_embd[:] = np.float32(3e38)
    gm = fcb.CudaSlm(sm.config, sm.weights)
    got, _ = gm.generate_tokens(synth.token_ids(1, 2, 515), 5)
    assert ((got >= 0) & (got < 515)).all()
    gm.close()


def test_a_wait_that_runs_out_feeds_nothing():
    sm = synth.SynthModel(2, 512, 8, 2048, 64, 515, seed=5, perturb=True)
    om, gm = O.OracleModel(sm), fcb.CudaSlm(sm.config, sm.weights)
    gm.set_decode_mode(1)
    ids = synth.token_ids(2, 3, 515)
    om.prime(ids), gm.prime(ids)
    _lib.check(_lib.lib().fc_debug_set_wait_budget(200000, 1))
    try:
        with pytest.raises(fcb.FerrumCudaError) as e:
            gm.feed(7)
    finally:
        _lib.check(_lib.lib().fc_debug_set_wait_budget(4000000000, 0))
    assert e.value.code == _lib.FC_E_TIMEOUT and gm.cached_len() == 3
    assert np.abs(gm.feed(7) - om.feed(7)).max() < 2e-5
    gm.close()
    om.close()


@pytest.mark.parametrize("kind", ["gpt2", "llama", "levels"])
def test_hidden_units_that_never_come_feed_nothing(kind):
    """The wait inside the MLP half runs out in every warp of a cluster; the step fails as a whole and the next one is as if it had not been."""
    if kind == "gpt2":
        sm = synth.SynthModel(2, 512, 8, 2048, 64, 515, seed=5, perturb=True)
        om, gm = O.OracleModel(sm), fcb.CudaSlm(sm.config, sm.weights)
        gm.set_decode_mode(1)
        gpu, cpu = gm.feed, om.feed
    else:
        prec = {"llama": None, "levels": 0}[kind]
        sm = synth.SynthLlama(515, 512, 2, 8, 2, 64, 2048, 64, seed=5, perturb=True)
        om, gm = O.OracleLlama(sm, threads=4, **({} if prec is None else {"prec": prec})), CudaLlama.from_synth(sm, prec=prec)
        cache = gm.new_cache()
        om.clear()
        gpu, cpu = lambda t: gm.forward_one(t, cache), om.forward_one
    for t in (3, 11):
        gpu(t), cpu(t)
    _lib.check(_lib.lib().fc_debug_set_wait_budget(200000, 2))
    try:
        with pytest.raises(fcb.FerrumCudaError) as e:
            gpu(7)
    finally:
        _lib.check(_lib.lib().fc_debug_set_wait_budget(4000000000, 0))
    assert e.value.code == _lib.FC_E_TIMEOUT
    got, want = gpu(7), cpu(7)
    assert np.abs(got - want).max() < (2e-5 if kind == "gpt2" else 2e-4 * max(1.0, float(np.abs(want).max())))
    gm.close()
    om.close()


# both pairings of the rotation with and without a tail that is not rotated, grouped heads, weights as stored and on rows of levels,
# and caches longer than a CTA of a head holds
@pytest.mark.parametrize("d,heads,kv,ff,ctx,rope_dim,rope_type,prec", [(512, 8, 2, 2048, 40, 64, 0, None), (512, 8, 8, 1024, 33, 48, 1, 0),
                                                                       (640, 10, 1, 1280, 50, 64, 1, 1), (768, 12, 4, 3072, 40, 64, 0, 0),
                                                                       (1024, 16, 4, 3072, 24, 64, 0, None)])
def test_llama_steps(d, heads, kv, ff, ctx, rope_dim, rope_type, prec):
    sm = synth.SynthLlama(515, d, 2, heads, kv, 64, ff, ctx, seed=d + kv, perturb=True, rope_dim=rope_dim, rope_type=rope_type)
    om, gm = O.OracleLlama(sm, threads=4, **({} if prec is None else {"prec": prec})), CudaLlama.from_synth(sm, prec=prec)
    cache = gm.new_cache()
    om.clear()
    for t, tok in enumerate(synth.token_ids(2, ctx, 515)):
        if t == 1:
            fcb.take_launch_count()
        got, want = gm.forward_one(tok, cache), om.forward_one(tok)
        assert np.abs(got - want).max() < 2e-4 * max(1.0, float(np.abs(want).max())), t
        if t == 1:
            assert fcb.take_launch_count() <= 8             # embedding, two a block, head, advance, state
    gm.close()


def test_llama_steps_past_the_held_rows():
    sm = synth.SynthLlama(515, 512, 1, 8, 2, 64, 512, 1400, seed=9, perturb=True, rope_dim=64, rope_type=0)
    om, gm = O.OracleLlama(sm, threads=4), CudaLlama.from_synth(sm)
    ids = synth.token_ids(2, 1300, 515)
    cache = gm.new_cache()
    om.clear()
    for t, tok in enumerate(ids):
        want = om.forward_one(tok)
        got = gm.forward_one(tok, cache)
        if t % 97 == 0 or t > 1290:
            assert np.abs(got - want).max() < 2e-4, t
    gm.close()


@pytest.mark.parametrize("prec", [None, 0])
@pytest.mark.parametrize("what", ["forward_one", "prime", "generate"])
def test_a_llama_wait_that_runs_out_feeds_nothing(what, prec):
    """The row never comes: the call says so, the cache ends where its last whole step left it, and goes on from there."""
    sm = synth.SynthLlama(515, 512, 2, 8, 2, 64, 2048, 64, seed=5, perturb=True)
    om, gm = O.OracleLlama(sm, threads=4, **({} if prec is None else {"prec": prec})), CudaLlama.from_synth(sm, prec=prec)
    cache = gm.new_cache()
    ids = [3, 11, 5]
    om.clear()
    for t in ids:
        gm.forward_one(t, cache), om.forward_one(t)
    greedy = _lib.FcSampling(0.0, 0, 1.0, 1.0)
    gm.generate(ids, 12, greedy, cache=cache)               # with graphs of every kind
    gm.prime(ids, cache)
    calls = {"forward_one": lambda: gm.forward_one(7, cache), "prime": lambda: gm.prime(ids, cache), "generate": lambda: gm.generate(ids, 12, greedy, cache=cache)}
    _lib.check(_lib.lib().fc_debug_set_wait_budget(200000, 1))
    try:
        with pytest.raises(fcb.FerrumCudaError) as e:
            calls[what]()
    finally:
        _lib.check(_lib.lib().fc_debug_set_wait_budget(4000000000, 0))
    assert e.value.code == _lib.FC_E_TIMEOUT and "wait" in str(e.value)
    assert cache.pos() == (3 if what == "forward_one" else 0)
    if what != "forward_one":
        for t in ids:
            gm.forward_one(t, cache)
    got, want = gm.forward_one(7, cache), om.forward_one(7)
    assert np.abs(got - want).max() < 2e-4 * max(1.0, float(np.abs(want).max()))
    gm.close()
    om.close()
