"""The resident-weight linears on device pointers as a program strings them together: one call's output as the next one's
operand on a stream."""
import ctypes as C

import numpy as np
import pytest

import ferrum_cpu_b200 as fcb
from ferrum_cpu_b200 import _lib, engine, synth

pytestmark = pytest.mark.gpu


def q8_weight(n, k, seed):
    wq = synth.q8_0_quantize((0.02 * np.random.default_rng(seed).standard_normal((n, k))).astype(np.float32))
    return fcb.QWeight(wq, n, k), synth.q8_0_dequantize(wq, n * k).reshape(n, k).astype(np.float64)


def rowq_weight(n, k, seed):
    w = (0.02 * np.random.default_rng(seed).standard_normal((k, n))).astype(np.float32)
    q, scales = engine.rowq_from_f32(w, _lib.FC_Q_INT8)
    return engine.RowQWeight(q, scales, k, n, _lib.FC_Q_INT8), engine.rowq_to_f32(q, scales, k, n, _lib.FC_Q_INT8).astype(np.float64).T


@pytest.mark.parametrize("make", [q8_weight, rowq_weight])
@pytest.mark.parametrize("n,k_long", [(4096, 12288), (300, 8192)])
def test_single_row_bias_is_the_output_of_the_call_ahead(make, n, k_long):
    """y1 = W1 x1 over a long row, then y2 = W2 x2 + y1 over a short one, on one stream: the second call is a programmatic
    dependent of the first and may not take its bias before the first has written it."""
    import torch

    (w1, f1), (w2, f2) = make(n, k_long, 1), make(n, 64, 2)
    rng = np.random.default_rng(n)
    x1, x2 = rng.standard_normal((24, k_long)).astype(np.float32), rng.standard_normal((24, 64)).astype(np.float32)
    d1, d2 = torch.from_numpy(x1).cuda(), torch.from_numpy(x2).cuda()
    zero, y1, y2 = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(24, n, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for i in range(24):
        w1.linear_dev(d1[i].data_ptr(), zero.data_ptr(), y1.data_ptr(), 1, stream=stream)
        w2.linear_dev(d2[i].data_ptr(), y1.data_ptr(), y2[i].data_ptr(), 1, stream=stream)
    want = x1.astype(np.float64) @ f1.T + x2.astype(np.float64) @ f2.T
    # f32 sums of up to 12288 products: 24 roundings of a tree of that depth, relative to the largest result
    assert np.abs(y2.cpu().numpy() - want).max() <= 24 * 2.0 ** -24 * 4 * np.abs(want).max()
    w1.close()
    w2.close()
