"""The chain of dependent launches that decodes one token (gemv_row.cu, attn_step.cu, the pick), against the oracle."""
import numpy as np
import pytest

import ferrum_cpu_b200 as fcb
from ferrum_cpu_b200 import synth
from ferrum_cpu_b200.llama import CudaLlama
from tests import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,heads,ff,ctx,prompt,new", [(32, 1, 64, 16, 1, 14), (96, 3, 160, 64, 60, 9), (64, 1, 96, 512, 345, 20),
                                                      (256, 4, 4128, 40, 17, 20), (64, 1, 96, 1024, 889, 12), (96, 3, 64, 1024, 1010, 10)])
def test_decode_chain_at_its_edges(d, heads, ff, ctx, prompt, new):
    """Greedy tokens of the decode chain against the oracle: heads of 32 and 64, the first positions, caches long enough
    for several CTAs a head, a window that slides, rows wider than one slice and odd vocabularies."""
    sm = synth.SynthModel(2, d, heads, ff, ctx, 515, seed=d + ff, perturb=True)
    om, gm = O.OracleModel(sm), fcb.CudaSlm(sm.config, sm.weights)
    window, want = list(synth.token_ids(4, prompt, 515)), []
    dist = om.prime(window)
    for _ in range(new):
        want.append(int(np.argmax(dist)))
        window.append(want[-1])
        if len(window) > ctx:
            window = window[-(ctx // 2):]
            dist = om.prime(window)
        else:
            dist = om.feed(want[-1])
    got, _ = gm.generate_tokens(synth.token_ids(4, prompt, 515), new)
    assert list(got) == want
    gm.close()
    om.close()


@pytest.mark.parametrize("hd,heads,kv,rope_dim,rope_type", [(128, 2, 1, 128, 0), (128, 2, 2, 96, 1), (32, 3, 1, 30, 0), (64, 8, 2, 64, 1)])
def test_rotary_steps_match_the_oracle_past_the_held_rows(hd, heads, kv, rope_dim, rope_type):
    sm = synth.SynthLlama(515, 96, 2, heads, kv, hd, 160, 416, seed=hd + kv, perturb=True, rope_dim=rope_dim, rope_type=rope_type)
    om, gm = O.OracleLlama(sm, threads=4), CudaLlama.from_synth(sm)
    cache = gm.new_cache()
    om.clear()
    for t, tok in enumerate(synth.token_ids(2, 400, 515)):
        got, want = gm.forward_one(tok, cache), om.forward_one(tok)
        assert np.abs(got - want).max() < 2e-4, t


def test_generation_runs_in_the_mode_it_was_asked_for():
    """fc_stream_set_mode holds for generations: one cooperative launch per batch of tokens, or a chain of launches per token; a
    new stream takes the chain, and the persistent kernel while its timeline is recorded."""
    sm = synth.named("tiny", seed=0, perturb=True)
    gm = fcb.CudaSlm(sm.config, sm.weights)
    prompt = synth.token_ids(17, 9, sm.dims[5])          # primed as a window: every traced token is a generated one
    tokens, launches = {}, {}
    gm.reset()                                           # makes the stream
    for mode in (None, 0, 1, 2):
        if mode is not None:
            gm.set_decode_mode(mode)
        fcb.take_launch_count()
        tokens[mode] = list(gm.generate_tokens(prompt, 24)[0])
        launches[mode] = fcb.take_launch_count()
    assert tokens[None] == tokens[0] == tokens[1] == tokens[2]
    per_token = 5 * sm.dims[0] + 3                       # embedding, five a block, head, pick
    assert launches[None] == launches[1] == launches[2] >= 24 * per_token
    assert launches[1] - launches[0] >= 23 * per_token   # 24 feeds in one launch
    for mode, traced in ((2, True), (0, True), (1, False)):
        gm.set_decode_mode(mode)
        gm.set_trace(True)
        fcb.take_launch_count()
        gm.generate_tokens(prompt, 24)
        gm.set_trace(False)
        assert (fcb.take_launch_count() < launches[1]) == traced
    gm.close()


@pytest.mark.parametrize("rows", ["nan", "minus infinity"])
def test_pick_on_rows_that_are_not_finite(rows):
    """A row of NaN has no largest probability: ln(max(p, 1e-12)) is the floor everywhere and index 0 is picked. Logits of -inf
    have probability 0, wherever they stand."""
    sm = synth.SynthModel(1, 64, 1, 96, 64, 1031, seed=9, perturb=True)
    if rows == "nan":
        sm.out_norm_g[:] = np.nan
    else:
        # the first 300 rows meet -3e38 with a weight of 2, the others with 0
        table = synth.q8_0_dequantize(sm.token_embd, 1031 * 64).reshape(1031, 64)
        table[:300, 0], table[300:, 0] = 2.0, 0.0
        sm.token_embd[:] = synth.q8_0_quantize(table)
        sm.out_norm_g[0], sm.out_norm_b[0] = 0.0, -3e38
    om, gm = O.OracleModel(sm), fcb.CudaSlm(sm.config, sm.weights)
    prompt = synth.token_ids(8, 12, 1031)
    want = om.generate_greedy(prompt, 12)[0]
    assert (want == 0).all() if rows == "nan" else (want >= 300).all()
    gm.set_decode_mode(1)
    assert np.array_equal(gm.generate_tokens(prompt, 12)[0], want)
    if rows == "nan":
        gm.set_decode_mode(0)
        assert np.array_equal(gm.generate_tokens(prompt, 12)[0], want)
    else:
        assert np.array_equal(gm.generate_sampled(prompt, 12, fcb.sampling(temperature=0.0), 1)[0], want)
    gm.close()
    om.close()


@pytest.mark.parametrize("heads,kv,hd,ctx,prompt", [(2, 1, 128, 2048, 1640), (4, 1, 32, 6144, 5500)])
def test_shared_heads_past_the_held_rows(heads, kv, hd, ctx, prompt):
    """Positions at which even the parts of a shared head outgrow its CTAs' shared memory: 8 of them hold about 188 rows each of
    width 128, about 650 of width 32."""
    sm = synth.SynthLlama(515, 96, 1, heads, kv, hd, 160, ctx, seed=hd, perturb=True)
    om, gm = O.OracleLlama(sm, threads=4), CudaLlama.from_synth(sm)
    cache, ids = gm.new_cache(), synth.token_ids(2, prompt + 3, 515)
    om.clear()
    for tok in ids[:prompt]:
        om.forward_one(tok)
    gm.prime(ids[:prompt], cache, want_logits=False)
    for tok in ids[prompt:]:
        assert np.abs(gm.forward_one(tok, cache) - om.forward_one(tok)).max() < 2e-4
