"""The tensor-core Q8_0 product at the edges of its tilings: a pair tile is 256 weight rows x up to 160 activation rows, a
single one 128 x up to 128, k-blocks are 32 wide (two per pipeline stage) and few rows split K over a cluster."""
import numpy as np
import pytest

from ferrum_cpu_b200 import engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("math_mode,tol", [(0, 2e-6), (1, 3e-5)])
@pytest.mark.parametrize("m,k,n", [
    (2, 32, 1), (3, 96, 515), (16, 64, 128), (17, 768, 129), (31, 4096, 256), (65, 160, 2304), (129, 256, 255), (161, 544, 257),
    (321, 1024, 768), (1000, 3072, 300), (2049, 96, 640),
])
def test_linear_matches_f64_at_tile_edges(m, k, n, math_mode, tol):
    rng = np.random.default_rng(m * 7919 + k * 31 + n)
    x = rng.standard_normal((m, k), dtype=np.float32)
    wq = synth.q8_0_quantize((0.02 * rng.standard_normal((n, k))).astype(np.float32))
    bias = (0.1 * rng.standard_normal(n)).astype(np.float32)
    want = x.astype(np.float64) @ synth.q8_0_dequantize(wq, n * k).reshape(n, k).astype(np.float64).T + bias
    got = engine.q8_0_linear(x, wq, bias, n, math_mode=math_mode)
    assert got.shape == (m, n)
    assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))


@pytest.mark.parametrize("m,k,n", [(2, 64, 1), (3, 128, 515), (16, 64, 128), (17, 768, 129), (31, 4096, 256), (64, 1024, 300)])
def test_few_rows_on_the_gemm_with_two_planes(m, k, n):
    """The allocation-free entry always takes the GEMM; the others have a kernel of their own for products this small."""
    import torch

    rng = np.random.default_rng(m + k + n)
    wq = synth.q8_0_quantize((0.02 * rng.standard_normal((n, k))).astype(np.float32))
    w, x = engine.QWeight(wq, n, k), torch.from_numpy(rng.standard_normal((m, k), dtype=np.float32)).cuda()
    y = torch.zeros(m, n, device="cuda")
    w.linear_dev_noalloc(x.data_ptr(), None, y.data_ptr(), m)
    want = x.double().cpu().numpy() @ synth.q8_0_dequantize(wq, n * k).reshape(n, k).astype(np.float64).T
    assert np.max(np.abs(y.cpu().numpy() - want)) <= 3e-5 * np.max(np.abs(want))
    w.close()


@pytest.mark.parametrize("m,k,n", [(2, 3104, 1), (3, 3136, 515), (16, 3200, 129), (33, 3136, 300), (64, 4096, 128)])
def test_few_rows_on_the_gemm_with_three_planes(m, k, n):
    """Rows wider than 3072 stay on the GEMM however few they are."""
    rng = np.random.default_rng(m + k + n)
    wq = synth.q8_0_quantize((0.02 * rng.standard_normal((n, k))).astype(np.float32))
    x, bias = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal(n, dtype=np.float32)
    want = x.astype(np.float64) @ synth.q8_0_dequantize(wq, n * k).reshape(n, k).astype(np.float64).T + bias
    assert np.max(np.abs(engine.q8_0_linear(x, wq, bias, n) - want)) <= 2e-6 * np.max(np.abs(want))
