"""The parity kernels' exp(-x) without double precision (rg_render.cu, exp_neg_slab): t + tail rounds to
the correctly rounded value wherever its remainder is not within d of half an ulp.  Restated in
float32 (each fused step once through float64, whose extra rounding stays far inside d)."""
import numpy as np
import pytest

F = np.float32


@pytest.mark.parametrize("lo,hi", [(2.0e-4, 1e-3), (1e-3, 1.0 / 16), (1.0 / 16, 0.25)])
def test_rounding_decision_is_exact(lo, hi):
    x = np.random.default_rng(3).uniform(lo, hi, 2_000_000).astype(F)
    s = F(1) - x
    sl = (F(1) - s) - x
    x2 = x * x
    x2l = (x.astype(np.float64) * x - x2).astype(F)
    P = np.full_like(x, F(1 / 40320))
    for c in (-1 / 5040, 1 / 720, -1 / 120, 1 / 24, -1 / 6):
        P = (x.astype(np.float64) * P + np.float64(F(c))).astype(F)
    h, x3 = F(0.5) * x2, x2 * x
    t = s + h
    e = (s - t) + h
    tail = (x3.astype(np.float64) * P + (((x2l.astype(np.float64) * 0.5 + sl).astype(F)) + e)).astype(F)
    r = t + tail
    rest = tail - (r - t)
    d = (x3.astype(np.float64) * F(5e-8) + 2.0 ** -43).astype(F)
    sure = np.abs(rest) + d <= F(2.0 ** -25)
    true = np.exp(-x.astype(np.float64))
    assert np.abs((t.astype(np.float64) + tail) - true).max() <= d.max()
    assert np.array_equal(r[sure], true.astype(F)[sure])
    # remainders are spread evenly over +-2^-25: the share handed on is that of the band d at its ends
    assert (~sure).mean() <= 1.2 * (d.astype(np.float64) / 2.0 ** -25).mean() + 1e-4
