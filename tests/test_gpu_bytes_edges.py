"""Byte output where the mapping's divisions are not avoided: statistics that are not
finite, that overflow or that vanish, against the float mapping in NumPy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _map(x, mean, sd):
    with np.errstate(all="ignore"):
        y = np.maximum(np.float32(-10), np.fmin(np.float32(10), (x - mean) / sd))
    return (((y + np.float32(10)) / np.float32(20)) * np.float32(255)).astype(np.uint8)


def _bytes(x):
    """One slab with its own statistics."""
    with np.errstate(all="ignore"):
        mean = np.float32(x.astype(np.float64).sum() / x.size)
        d = x - mean
        sd = np.sqrt(np.float32((d * d).astype(np.float64).sum() / x.size))
    return _map(x, mean, sd)


def _run(engine, x, slab):
    return engine.volume_to_bytes(torch.from_numpy(x).cuda(), slab, 0.0).cpu().numpy()


def test_a_slab_with_values_that_are_not_finite(engine):
    """Its statistics are not numbers, so all its bytes are those of NaN, and as the
    averages run on (g = alpha g + (1 - alpha) stat, 0 x NaN with alpha 0) those of the
    slabs after it; the slabs before it keep theirs."""
    v = np.random.default_rng(0).normal(size=(3, 4096)).astype(np.float32)
    v[1, 5], v[1, 9] = np.inf, np.nan
    got = _run(engine, v.ravel(), 4096).reshape(3, 4096)
    np.testing.assert_array_equal(got[0], _bytes(v[0]))
    assert (got[1:] == 255).all()


@pytest.mark.parametrize("big", [3.0e38, 3.4e38])
def test_a_deviation_that_overflows(engine, big):
    """Infinite deviation: every difference maps to the middle, one that overflows
    itself to the byte of NaN."""
    v = np.random.default_rng(1).normal(size=4096).astype(np.float32)
    v[3:2000:2] = big
    v[2001], v[2002] = -big, -big
    np.testing.assert_array_equal(_run(engine, v, 4096), _bytes(v))


@pytest.mark.parametrize("scale", [1e-45, 1e-30, 1e-22, 1e17])
def test_deviations_that_vanish_or_are_large(engine, scale):
    v = (np.random.default_rng(2).normal(size=4096) * scale).astype(np.float32)
    np.testing.assert_array_equal(_run(engine, v, 4096), _bytes(v))


def test_values_beside_the_edges_of_bytes(engine):
    """Values that map to whole numbers, and the floats beside them: those the
    division-free form leaves to the exact one."""
    steps = np.arange(1, 255, dtype=np.float64) / 12.75 - 10
    edge = np.concatenate([steps, steps, steps]).astype(np.float32)
    edge[254:508] = np.nextafter(edge[254:508], np.float32(100))
    edge[508:] = np.nextafter(edge[508:], np.float32(-100))
    # mean 0 and deviation 1, up to rounding: the edges, their negatives and noise
    v = np.concatenate([edge, -edge])
    rest = np.random.default_rng(3).normal(size=1 << 20).astype(np.float32)
    rest *= np.float32(np.sqrt((rest.size - (v.astype(np.float64) ** 2 - 1).sum()) /
                               (rest.astype(np.float64) ** 2).sum()))
    v = np.concatenate([v, rest - rest.mean(dtype=np.float64).astype(np.float32)])
    v = v[:v.size // 4 * 4].astype(np.float32)
    np.testing.assert_array_equal(_run(engine, v, v.size), _bytes(v))
