"""The resident-weight linears on device pointers as a program strings them together: one call's output as the next one's
operand on a stream, calls on several streams, captured calls, and what they keep."""
import ctypes as C

import numpy as np
import pytest

import ferrum_cpu_b200 as fcb
from ferrum_cpu_b200 import _lib, engine, synth
from tests.test_timeouts import short_waits_without_producers

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


def run_linear(w, x, bias, y, math_mode, stream):
    args = (x.data_ptr(), bias.data_ptr(), y.data_ptr(), x.shape[0])
    s = C.c_void_p(stream.cuda_stream)
    w.linear_dev(*args, stream=s) if isinstance(w, engine.RowQWeight) else w.linear_dev(*args, math_mode, s)


# largest error over the largest result against f64, as test_gemm_tiles.py has it for the two math modes
KINDS = [(q8_weight, _lib.FC_MATH_FP32, 2e-6), (q8_weight, _lib.FC_MATH_BF16X3, 3e-5), (rowq_weight, None, 2e-6)]


def close_to(y, x, f, tol):
    want = x.double().cpu().numpy() @ f.T
    return np.abs(y.cpu().numpy() - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("make,math_mode,tol", KINDS)
def test_calls_on_two_streams_share_nothing(make, math_mode, tol):
    """The same weight on two streams without an order between them, with rows of their own."""
    import torch

    n, k, m = 640, 1024, 2048
    w, f = make(n, k, 3)
    xs = [[torch.randn(m, k, device="cuda") for _ in range(6)] for _ in range(2)]
    ys = [[torch.zeros(m, n, device="cuda") for _ in range(6)] for _ in range(2)]
    zero, streams = torch.zeros(n, device="cuda"), [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for i in range(6):
        for s in range(2):
            run_linear(w, xs[s][i], zero, ys[s][i], math_mode, streams[s])
    torch.cuda.synchronize()
    assert all(close_to(ys[s][i], xs[s][i], f, tol) for s in range(2) for i in range(6))
    w.close()


@pytest.mark.parametrize("make,math_mode,tol", KINDS)
def test_first_call_may_be_captured(make, math_mode, tol):
    import torch

    n, k, m = 300, 512, 277
    w, f = make(n, k, 4)
    x, zero, y = torch.randn(m, k, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(m, n, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run_linear(w, x, zero, y, math_mode, torch.cuda.current_stream())
    for _ in range(3):
        x.normal_()
        graph.replay()
        run_linear(w, torch.randn(4 * m, k, device="cuda"), zero, torch.empty(4 * m, n, device="cuda"), math_mode, torch.cuda.current_stream())
        torch.cuda.synchronize()
        assert close_to(y, x, f, tol)
    del graph
    w.close()


@pytest.mark.parametrize("make,math_mode,tol", KINDS)
@pytest.mark.parametrize("rows_k", [544, 3104])
def test_without_memory_for_scratch_the_rows_need_none(make, math_mode, tol, rows_k):
    import torch

    n, k, m = 1290, rows_k, 45
    w, f = make(n, k, 5)
    x, zero, y = torch.randn(m, k, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(m, n, device="cuda")
    _lib.lib().fc_debug_withhold_scratch(1)
    try:
        run_linear(w, x, zero, y, math_mode, torch.cuda.current_stream())
    finally:
        _lib.lib().fc_debug_withhold_scratch(0)
    torch.cuda.synchronize()
    assert close_to(y, x, f, tol)
    w.close()


def test_weights_share_a_bounded_scratch():
    """Eight weights of 96 MiB of scratch a call: what stays allocated is the pool's 256 MiB at most, not a buffer per weight."""
    import torch

    n, k, m = 32, 4096, 4096
    weights = [q8_weight(n, k, 6)[0] for _ in range(8)]
    x, zero, y = torch.randn(m, k, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(m, n, device="cuda")
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    for w in weights:
        run_linear(w, x, zero, y, _lib.FC_MATH_FP32, torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= (256 + 32) << 20
    for w in weights:
        w.close()


@pytest.mark.parametrize("make,math_mode,tol", KINDS)
def test_a_wait_that_ran_out_is_reported_by_the_next_call(make, math_mode, tol):
    import torch

    n, k, m = 256, 768, 300
    w, f = make(n, k, 7)
    x, zero, y = torch.randn(m, k, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(m, n, device="cuda")
    stream = torch.cuda.current_stream()
    with short_waits_without_producers():
        run_linear(w, x, zero, y, math_mode, stream)
        torch.cuda.synchronize()                             # the kernel has returned; the context is intact
    with pytest.raises(fcb.FerrumCudaError) as e:
        run_linear(w, x, zero, y, math_mode, stream)
    assert e.value.code == _lib.FC_E_TIMEOUT
    run_linear(w, x, zero, y, math_mode, stream)
    torch.cuda.synchronize()
    assert close_to(y, x, f, tol)
    w.close()


def test_host_entry_reports_a_wait_that_ran_out():
    w, f = rowq_weight(256, 768, 8)
    x = np.random.default_rng(8).standard_normal((300, 768)).astype(np.float32)
    with short_waits_without_producers():
        with pytest.raises(fcb.FerrumCudaError) as e:
            w.linear(x, np.zeros(256, np.float32))
        assert e.value.code == _lib.FC_E_TIMEOUT
    want = x.astype(np.float64) @ f.T
    assert np.abs(w.linear(x, np.zeros(256, np.float32)) - want).max() <= 2e-6 * np.abs(want).max()
    w.close()


@pytest.mark.parametrize("make", [q8_weight, rowq_weight])
@pytest.mark.parametrize("n,k", [(4096, 96), (4097, 32), (4130, 4128), (8191, 768), (16383, 512), (16384, 512), (16390, 544), (24575, 544),
                                 (24576, 544), (24579, 1056), (50257, 96)])
def test_single_row_against_matrices_of_many_rows(make, n, k):
    """The sizes at which the row product changes its kernel, last rows that fill no half warp, rows of fewer chunks than lanes and
    no multiple of them; the bias is the output of the call ahead."""
    import torch

    w, f = make(n, k, n + k)
    x = torch.from_numpy(np.random.default_rng(k).standard_normal((2, k)).astype(np.float32)).cuda()
    zero, y1, y2 = torch.zeros(n, device="cuda"), torch.full((n,), np.nan, device="cuda"), torch.full((n + 64,), np.nan, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    w.linear_dev(x[0].data_ptr(), zero.data_ptr(), y1.data_ptr(), 1, stream=stream)
    w.linear_dev(x[1].data_ptr(), y1.data_ptr(), y2.data_ptr(), 1, stream=stream)
    want = x.double().cpu().numpy().sum(axis=0) @ f.T
    assert np.abs(y2[:n].cpu().numpy() - want).max() <= 24 * 2.0 ** -24 * 4 * np.abs(want).max()
    assert torch.isnan(y2[n:]).all()
    w.close()


@pytest.mark.parametrize("make", [q8_weight, rowq_weight])
@pytest.mark.parametrize("m,n,k", [(2, 1, 32), (2, 4097, 288), (3, 515, 96), (4, 33, 3072), (4, 2050, 544), (5, 129, 256), (7, 31, 1056), (13, 700, 800),
                                   (64, 500, 96), (3, 300, 3104), (30, 4096, 256), (33, 4096, 256)])
def test_few_rows_without_scratch(make, m, n, k):
    """Rows that fill no block of four, weight rows that fill no half warp, chunks that fill no lane, and the sizes on either side of
    the change to the GEMM; the bias is the output of the call ahead."""
    import torch

    w, f = make(n, k, n + k)
    x = torch.from_numpy(np.random.default_rng(m).standard_normal((m, k)).astype(np.float32)).cuda()
    zero, y1 = torch.zeros(n, device="cuda"), torch.full((n,), np.nan, device="cuda")
    y = torch.full((m * n + 64,), np.nan, device="cuda")
    stream = torch.cuda.current_stream()
    run_linear(w, x[:1], zero, y1, _lib.FC_MATH_FP32, stream)
    w_args = (x.data_ptr(), y1.data_ptr(), y.data_ptr(), m)
    s = C.c_void_p(stream.cuda_stream)
    w.linear_dev(*w_args, stream=s) if isinstance(w, engine.RowQWeight) else w.linear_dev(*w_args, _lib.FC_MATH_FP32, s)
    xs = x.double().cpu().numpy()
    want = xs @ f.T + xs[0] @ f.T
    assert np.abs(y[:m * n].cpu().numpy().reshape(m, n) - want).max() <= 2e-6 * np.abs(want).max()
    assert torch.isnan(y[m * n:]).all()
    w.close()
