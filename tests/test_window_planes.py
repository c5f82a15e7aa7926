"""Window forwards of models whose activations have parts far apart in size. An element that no weight reads (its column of levels is
zero) or that GELU turns into zero leaves the function as it is, whatever its size: only what the products hold of the others may change."""
import ctypes as C

import numpy as np
import pytest

import ferrum_cpu_b200 as fcb
from ferrum_cpu_b200 import _lib, synth

pytestmark = pytest.mark.gpu


def _clear_column(raw, n, k, col):
    """Levels of input column `col` of a Q8_0 matrix [n][k] to zero."""
    raw.reshape(n, k // 32, 34)[:, col // 32, 2 + col % 32] = 0


def _logprobs(sm, ids):
    gm = fcb.CudaSlm(sm.config, sm.weights)
    lp = gm.score_sequences(ids)[1]
    gm.close()
    return lp


def _spread(d, heads, ff, where, size, math_mode):
    """Two blocks; `size` is the element nobody reads: 0 in the plain model."""
    sm = synth.SynthModel(2, d, heads, ff, 64, 515, seed=d, perturb=True, math_mode=math_mode)
    L = sm.layers[1]
    if where in ("ln1_b", "ln1_g"):
        _clear_column(L["attn_qkv_q8"], 3 * d, d, 5)
        L[where][5] = size
    elif where in ("ln2_b", "ln2_g"):
        _clear_column(L["ffn_up_q8"], ff, d, 5)
        L[where][5] = size
    elif where == "attn_qkv_b":                        # a value element
        _clear_column(L["attn_out_q8"], d, d, 5)
        L[where][2 * d + 5] = size
    elif where == "ffn_up_b":                          # a hidden unit that is always off
        L[where][5] = -100.0 - abs(size)
    else:
        _clear_column(sm.token_embd, 515, d, 5)
        sm.out_norm_b[5] = size
    return sm


PLACES = ["ln1_b", "ln1_g", "ln2_b", "ln2_g", "attn_qkv_b", "ffn_up_b", "out_norm_b"]


@pytest.mark.parametrize("where", PLACES)
def test_f32_mode_holds_every_element(where):
    """Activations of the f32 mode reach the products with all of their bits: not one bit of a log-probability moves."""
    ids = synth.token_ids(1, 3 * 64, 515).reshape(3, 64)
    plain, wide = (_logprobs(_spread(512, 8, 2048, where, size, fcb.FC_MATH_FP32), ids) for size in (0.0, 1e8))
    assert np.array_equal(plain, wide)


@pytest.mark.parametrize("size", [0.0, 1e4, 1e6, 1e8, 1e12])
@pytest.mark.parametrize("where", PLACES)
def test_two_plane_mode_keeps_its_precision(where, size):
    """Activations to 2^-17 of each element (f16 planes hold more, where a scale of all elements allows it) behind whatever nobody reads. An element
    is off by 2^-17 / sqrt(3) at random, so is a logit (they have a size of 1/2), nine products in a row add up to 3 times that, and 4.5 times
    it is what 192 rows show; behind f16 planes alone 1e12 is off by 0.2."""
    ids = synth.token_ids(1, 3 * 64, 515).reshape(3, 64)
    want = _logprobs(_spread(512, 8, 2048, where, 0.0, fcb.FC_MATH_FP32), ids)
    got = _logprobs(_spread(512, 8, 2048, where, size, fcb.FC_MATH_BF16X3), ids)
    assert np.abs(got - want).max() < 4.5 * 3 * 2.0**-17 / np.sqrt(3) / 2


def test_planes_make_room():
    """A workspace, a stream or a batch that finds no memory gets that of the f16 planes; forwards go on without them."""
    ids = synth.token_ids(1, 4 * 64, 515).reshape(4, 64)
    sm = _spread(512, 8, 2048, "ln1_b", 0.0, fcb.FC_MATH_BF16X3)
    want = _logprobs(_spread(512, 8, 2048, "ln1_b", 0.0, fcb.FC_MATH_FP32), ids)

    def stream(gm):
        s = C.c_void_p()
        _lib.check(_lib.lib().fc_stream_create(gm._m, C.byref(s)))
        _lib.lib().fc_stream_free(s)

    uses = [lambda gm: gm.score_sequences(ids), stream, lambda gm: gm.decode_batch(ids[:, :4], 3)]
    left = []
    for use in uses:
        gm = fcb.CudaSlm(sm.config, sm.weights)
        few = gm.score_sequences(ids[:1])[1]
        _lib.check(_lib.lib().fc_debug_withhold_scratch(2))
        try:
            use(gm)
        finally:
            _lib.check(_lib.lib().fc_debug_withhold_scratch(0))
        left.append(gm.score_sequences(ids)[1])
        assert not np.array_equal(left[-1][:1], few)             # no longer on f16 planes
        gm.close()
    assert all(np.array_equal(lp, left[0]) for lp in left[1:])
    assert np.abs(left[0] - want).max() < 4.5 * 3 * 2.0**-17 / np.sqrt(3) / 2
