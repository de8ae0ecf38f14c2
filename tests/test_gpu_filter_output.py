"""The row filter, binning and byte-output kernels at the sizes where their
vector paths, runs and fallbacks begin and end."""
import numpy as np
import pytest
import torch

from autom2_b200 import tiltrec as T

pytestmark = pytest.mark.gpu


def _cuda(a, misaligned):
    """The array on the GPU, 4 bytes past a 16-byte boundary when misaligned."""
    t = torch.empty(a.size + 1, device="cuda")[int(misaligned):][:a.size].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


def _bytes(v, slab, alpha):
    """The byte mapping in numpy, in the precisions the reference uses."""
    out = np.zeros(v.size, np.uint8)
    gm = gs = np.float32(0)
    a = np.float32(alpha)
    for s0 in range(0, v.size, slab):
        x = v[s0:s0 + slab]
        mean = np.float32(x.astype(np.float64).sum() / x.size)
        d = x - mean
        sd = np.sqrt(np.float32((d * d).astype(np.float64).sum() / x.size))
        gm = a * gm + (np.float32(1) - a) * mean
        gs = a * gs + (np.float32(1) - a) * sd
        with np.errstate(all="ignore"):
            y = np.maximum(np.float32(-10), np.fmin(np.float32(10), (x - gm) / gs))
        y = ((y + np.float32(10)) / np.float32(20)) * np.float32(255)
        n4 = x.size // 4 * 4
        out[s0:s0 + n4] = y[:n4].astype(np.uint8)
    return out


@pytest.mark.parametrize("misaligned", [False, True])
@pytest.mark.parametrize("n,slab,alpha", [(4096, 4096, 0.0), (100003, 10007, 0.9),
                                          (65536, 1000, 0.9), (262147, 262147, 0.0), (7, 3, 0.5),
                                          (30000, 6, 0.9)])
def test_bytes(engine, n, slab, alpha, misaligned):
    rng = np.random.default_rng(n + slab)
    v = (rng.normal(size=n) * 3 + 1).astype(np.float32)
    v[::97] *= 20  # beyond ten deviations
    got = engine.volume_to_bytes(_cuda(v, misaligned), slab, alpha).cpu().numpy()
    np.testing.assert_array_equal(got, _bytes(v, slab, alpha))


def test_bytes_of_a_constant_and_of_values_that_are_not_finite(engine):
    flat = torch.full((1024,), 2.5, device="cuda")  # deviation 0: 0/0 maps as NaN does
    assert int(engine.volume_to_bytes(flat, 1024, 0.0).min()) == 255
    v = np.random.default_rng(0).normal(size=4096).astype(np.float32)
    w = v.copy()
    w[5], w[9] = np.inf, np.nan
    # statistics of the second slab only (alpha 0), so that the first one's are finite
    got = engine.volume_to_bytes(_cuda(np.concatenate([v, w]), False), 8192 // 2, 0.0).cpu().numpy()
    np.testing.assert_array_equal(got[:4096], _bytes(v, 4096, 0.0))


@pytest.mark.parametrize("misaligned", [False, True])
@pytest.mark.parametrize("shape,factor", [((2, 37, 1025), 1), ((1, 130, 4100), 4), ((2, 127, 127), 64),
                                          ((1, 64, 2052), 3), ((3, 9, 12), 5), ((1, 200, 4096), 64)])
def test_binning(restatement, shape, factor, misaligned):
    a = np.random.default_rng(sum(shape)).normal(size=shape).astype(np.float32)
    got = T.resample_bin(_cuda(a, misaligned), factor).cpu().numpy()
    nt, ny, nx = shape
    def axis(n):
        d = n // factor
        e = np.arange(d + 1) * (n / d)
        i = np.arange(n)
        o = np.minimum(e[1:, None], i + 1) - np.maximum(e[:-1, None], i)
        return np.clip(o, 0, None) / (n / d)
    want = np.einsum("jy,tyx,ix->tji", axis(ny), a.astype(np.float64), axis(nx))
    # one rounding to float of sums of magnitude max|a|
    assert np.abs(got - want).max() <= 2 ** -23 * np.abs(a).max()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("nx", [2, 7, 255, 257, 2049, 26000])
def test_fbp_rows(engine, restatement, nx, mode):
    rng = np.random.default_rng(nx)
    p = rng.normal(size=(3, 2, nx)).astype(np.float32)
    c8 = restatement.coeffs(np.array([-10, 0, 10], np.float32), 0, 0, 0)
    engine.set_problem(nx, 2, 3, 1, c8, T.LAYOUT_Y)
    d = _cuda(p, False)
    engine.filter_fbp(d, mode)
    want = restatement.filter_fbp(p.copy(), mode)
    want = want[0] if isinstance(want, tuple) else want
    # FP64 sums of the same float taps on both sides, one rounding to float each
    assert np.abs(d.cpu().numpy() - want).max() <= 2 ** -22 * np.abs(want).max()
