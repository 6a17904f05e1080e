"""The exact mode's flights leave out the terms of zero accelerations where
they cannot change a sum: labels, rows, last rows and margins must be the
oracle's for zeros of either sign, planes already reached, backward flights,
no and reversed gravity, and numbers far outside a beamline's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g", [9.81, 0.0, -9.81, 1e-70, 1e80])
def test_flights_equal_the_oracle(g):
    import ctraj
    from ctraj.compiler import compile_beamline
    from ctraj.engine import Engine
    from oracle import oracle

    cb = compile_beamline(ctraj.Beamline([
        ctraj.CircularAperture(name="A1", z0=0.30, L=1e-3, d=0.5),
        ctraj.RectangularAperture(name="R1", z0=0.50, L=0.0, w=0.4, h=0.4),
        ctraj.CircularAperture(name="Detection plane", z0=1.0, L=0.0, d=float("inf")),
    ]))
    rng = np.random.default_rng(5)
    special = [0.0, -0.0, 1e-3, -1e-3, 1e-310, -1e-310, 1e200]
    n = 4096
    ics = np.zeros((6, n))
    for k in (0, 1):
        ics[k] = rng.choice(special[:6], n) + np.where(rng.random(n) < 0.5, 0.0, rng.standard_normal(n) * 1e-3)
        ics[3 + k] = rng.choice(special, n, p=[0.3, 0.3, 0.1, 0.1, 0.09, 0.09, 0.02])
        ics[3 + k] += np.where(rng.random(n) < 0.5, -0.0, rng.standard_normal(n))
    ics[2] = rng.choice([0.0, -0.0, 0.30, 0.4, -1e-310], n)
    ics[5] = rng.choice([184.0, -184.0, 1e-3, 1e70, 1e-70, 0.0, -0.0], n, p=[0.5, 0.1, 0.1, 0.1, 0.1, 0.05, 0.05])
    want = oracle.run(cb, np.ascontiguousarray(ics), g=g)
    eng = Engine(0)
    try:
        got = eng.run(cb, n, precision=64, ics=ics, outputs=True, g=g)
    finally:
        eng.close()
    np.testing.assert_array_equal(got.label, want["label"])
    np.testing.assert_array_equal(got.rows, want["rows"])
    np.testing.assert_array_equal(got.margin, want["margin"])
    np.testing.assert_array_equal(got.final, want["final"])
    np.testing.assert_array_equal(np.signbit(got.final[:6]) & ~np.isnan(want["final"][:6]),
                                  np.signbit(want["final"][:6]) & ~np.isnan(want["final"][:6]))
