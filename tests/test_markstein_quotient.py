"""MarksteinDiv of wam_b200/csrc/devmath.cuh restated on the host: two corrections
by the exact residual from a rounded reciprocal end in the IEEE quotient."""
import numpy as np


def test_two_corrections_give_the_ieee_quotient():
    rng = np.random.default_rng(3)
    f32, f64 = np.float32, np.float64
    a = (rng.random(2000000) * 10.0 ** rng.uniform(-12, 6, 2000000)).astype(f32)
    b = (rng.uniform(0.5, 2.0, a.size) * 2.0 ** rng.integers(-20, 20, a.size)).astype(f32)
    y = f32(1) / b
    q = a * y
    for _ in range(2):
        # fmaf(-q, b, a): the residual is exact in single precision
        r = (f64(a) - f64(q) * f64(b)).astype(f32)
        # fmaf(r, y, q): r*y is exact in double, the sum nearly so
        q = (f64(q) + f64(r) * f64(y)).astype(f32)
    assert (q == a / b).all()
