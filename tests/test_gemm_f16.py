"""The two-plane product on f16 planes (gemm_f16.cu) against 64-bit sums: tiles and their remainders, the magnitudes the row scales
have to carry, weights at the ends of f16, and what must not change with the rows beside a row."""
import numpy as np
import pytest

import ferrum_cpu_b200 as fcb

pytestmark = pytest.mark.gpu


def _weight(n, k, seed, scales=None):
    rng = np.random.RandomState(seed)
    q = rng.randint(-127, 128, (n, k // 32, 32)).astype(np.int8)
    d = (rng.uniform(0.5, 2.0, (n, k // 32)) * 1e-3 if scales is None else rng.choice(scales, (n, k // 32))).astype(np.float16)
    raw = np.concatenate([d[..., None].view(np.uint8), q.view(np.uint8)], axis=2).reshape(-1)
    return raw, (d.astype(np.float64)[..., None] * q).reshape(n, k)


def _bound(x, w, k):
    # per element, of sum |x||w|: 24 truncations of 2^-23 in a group (up to 384 k, then 192), one rounding a group, three plane terms and the
    # bias; the small terms' truncations are 2^-11 of that
    s = np.abs(x).astype(np.float64) @ np.abs(w).T
    return (24 * 2.0**-23 + (k / 192 + 6) * 2.0**-24) * s


def _run(qw, x, n, bias=None):
    import torch
    xd, y = torch.from_numpy(x).cuda(), torch.full((x.shape[0], n), float("nan"), device="cuda")
    b = torch.from_numpy(bias).cuda() if bias is not None else None
    fcb.take_launch_count()
    qw.linear_dev(xd.data_ptr(), b.data_ptr() if b is not None else None, y.data_ptr(), x.shape[0], fcb.FC_MATH_BF16X3)
    # small products run on f32 FMA, in one launch; the tensor core's have a launch for the planes
    small = qw.k <= 3072 and x.shape[0] * n * ((qw.k + 255) // 256 * 256) < 2**25
    assert fcb.take_launch_count() == (1 if small else 2)
    torch.cuda.synchronize()
    return y.cpu().numpy()


@pytest.mark.parametrize("m,n,k", [(512, 1, 64), (513, 127, 128), (575, 129, 320), (769, 257, 256), (1024, 1000, 768), (2305, 300, 832),
                                   (4096, 2048, 64), (131072, 1, 64), (2050, 1, 4096), (1600, 127, 3136), (2080, 128, 192)])
def test_matches_64_bit_sums(m, n, k):
    raw, w = _weight(n, k, 1)
    x = np.random.RandomState(2).standard_normal((m, k)).astype(np.float32)
    bias = np.random.RandomState(3).standard_normal(n).astype(np.float32)
    qw = fcb.QWeight(raw, n, k)
    want = x.astype(np.float64) @ w.T + bias
    got = _run(qw, x, n, bias)
    assert (np.abs(got - want) <= _bound(x, w, k) + 2.0**-24 * np.abs(want)).all()
    # no bf16 planes, which leave 2.5e-6
    assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want)
    qw.close()


@pytest.mark.parametrize("n", [160, 264])                # on f32 FMA, and on f16 planes
def test_rows_of_any_magnitude_and_their_neighbours(n):
    k, m = 128, 600
    raw, w = _weight(n, k, 4)
    x = np.random.RandomState(5).standard_normal((m, k)).astype(np.float32)
    x *= np.float32(10.0) ** np.random.RandomState(6).randint(-30, 31, (m, 1)).astype(np.float32)
    x[7] = 0.0
    x[11, 3] = np.nan
    x[13] *= np.exp(np.random.RandomState(7).standard_normal(k) * 4).astype(np.float32)
    qw = fcb.QWeight(raw, n, k)
    got = _run(qw, x, n)
    want = x.astype(np.float64) @ w.T
    ok = np.arange(m) != 11
    assert np.isnan(got[11]).all() and (got[7] == 0.0).all()
    assert (np.abs(got[ok] - want[ok]) <= _bound(x[ok], w, k)).all()
    alone = _run(qw, np.ascontiguousarray(x[: m - 64]), n)
    assert np.array_equal(alone[ok[: m - 64]], got[: m - 64][ok[: m - 64]])
    qw.close()


@pytest.mark.parametrize("n", [130, 258])                # on f32 FMA, and on the tensor core
@pytest.mark.parametrize("scales", [(2.0**-24, 3 * 2.0**-24, 1.5 * 2.0**-14), (511.5, 400.0), (512.0, 600.0, 1e-3)])
def test_scales_at_the_ends_of_f16(scales, n):
    """Subnormal scales, the largest that f16 planes hold, and scales beyond (which the level kernel takes)."""
    k, m = 192, 512
    raw, w = _weight(n, k, 8, np.array(scales))
    x = np.random.RandomState(9).standard_normal((m, k)).astype(np.float32)
    qw = fcb.QWeight(raw, n, k)
    want, got = x.astype(np.float64) @ w.T, _run(qw, x, n)
    # the level kernel splits x to 2^-17, each term of a product once more
    bound = _bound(x, w, k) if max(scales) < 512 else 2.0**-16 * (np.abs(x).astype(np.float64) @ np.abs(w).T)
    assert (np.abs(got - want) <= bound).all()
    # on f16 planes if these hold the weights, else on levels and bf16 planes
    assert n < 258 or (np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want)) == (max(scales) < 512)
    qw.close()


# stages of 64: the last small terms behind the first ones, one and two groups, a group of one stage
@pytest.mark.parametrize("k", [192, 256, 384, 448, 640, 704, 1024])
def test_orders_of_a_tile(k):
    n, m = 300, 1100
    raw, w = _weight(n, k, 10)
    x = np.random.RandomState(11).standard_normal((m, k)).astype(np.float32)
    qw = fcb.QWeight(raw, n, k)
    assert (np.abs(_run(qw, x, n) - x.astype(np.float64) @ w.T) <= _bound(x, w, k)).all()
    qw.close()


@pytest.mark.parametrize("k", [128, 1024])
def test_sums_that_need_no_rounding_are_exact(k):
    """One element of few bits a row: its product, rounded once. Whole numbers on one scale: their sum."""
    n, m = 256, 1024
    raw, w = _weight(n, k, 12)
    qw = fcb.QWeight(raw, n, k)
    x = np.zeros((m, k), np.float32)
    x[np.arange(m), np.arange(m) % k] = 1.375 * 2.0 ** (np.arange(m) % 9 - 4)
    assert np.array_equal(_run(qw, x, n), (x.astype(np.float64) @ w.T).astype(np.float32))
    qw.close()
    raw, w = _weight(n, k, 13, np.array([2.0**-10]))
    qw = fcb.QWeight(raw, n, k)
    x = np.random.RandomState(14).randint(-3, 4, (m, k)).astype(np.float32)
    assert np.array_equal(_run(qw, x, n), x.astype(np.float64) @ w.T)
    qw.close()


@pytest.mark.parametrize("size", [1e4, 1e6, 1e8])
def test_an_element_that_no_weight_reads(size):
    """However large it is, the others keep their bits: 2^-36 of the row's scale, which is at most 2^14 / size, is 2^-23 of an element of 1."""
    n, k, m = 200, 256, 700
    raw, w = _weight(n, k, 15)
    raw.reshape(n, k // 32, 34)[:, 2, 2 + 9] = 0
    w[:, 73] = 0.0
    x = np.random.RandomState(16).standard_normal((m, k)).astype(np.float32)
    x[:, 73] = size
    qw = fcb.QWeight(raw, n, k)
    got, want = _run(qw, x, n), x.astype(np.float64) @ w.T
    x[:, 73] = 0.0
    assert (np.abs(got - want) <= _bound(x, w, k) + 2.0**-36 * size * 2.0**-14 * np.abs(w).sum(1)).all()
    qw.close()
