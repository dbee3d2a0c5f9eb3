"""The tracking's FP32 test that a scatter cannot come before the flight's end (scatter_may_win in
imc_device.cuh) against the full path it skips, in the same precisions on the CPU: whenever
p = 1 - u >= sigma s (1 + 1e-6) the FP64 series test must also rule the scatter out (sigma s < 0.01),
and otherwise the FP32 distance -ln(u) / sigma, off by the 2^-21 (relative) that its logarithm and
quotient may be off by, must not be below s.  Every sampled uniform is near the limit p = sigma s,
where the two could differ.
"""
import numpy as np
import pytest

F = np.float32


@pytest.mark.parametrize("lo,hi", [(1e-12, 1e-7), (1e-7, 1e-5), (1e-5, 0.0099), (0.0099, 0.0101), (0.0101, 0.99)])
def test_early_rejection_agrees_with_full_test(lo, hi):
    rng = np.random.default_rng(17)
    n = 400_000
    sig = F(10.0) ** rng.uniform(-6, 6, n).astype(F)
    t = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    s = (t / sig).astype(F)
    # odd multiples of 2^-24 within a few steps of p = t, and the two smallest p there are
    k = np.maximum(np.rint(t * 2.0 ** 23).astype(np.int64) + rng.integers(-3, 4, n), 0)
    k[:1000] = rng.integers(0, 2, 1000)
    k = np.minimum(k, 2 ** 23 - 1)
    u = F(1.0) - ((2 * k + 1) * 2.0 ** -24).astype(F)
    assert np.array_equal(1.0 - u.astype(np.float64), (2 * k + 1) * 2.0 ** -24)  # u is exact
    reject = (F(1.0) - u) >= (sig * s).astype(F) * F(1.000001)
    assert reject.any()
    td = sig.astype(np.float64) * s.astype(np.float64)
    small = td < 0.01
    may = u.astype(np.float64) > 1.0 - td * (1.0 - td * (0.5 - td * (1.0 / 6.0)))
    assert not np.any(reject & small & may)
    dist = -np.log(u.astype(np.float64)) / sig * (1.0 - 2.0 ** -21)
    assert not np.any(reject & ~small & (dist < s))
