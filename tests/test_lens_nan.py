"""A molecule whose position is not a number passes every test (a comparison
with NaN is false) and leaves its margin alone: the persistent FP32 lens pass,
which notes one margin per group of steps, must give it the chunked pass's,
which notes one per step, however full its CTA is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compiled(table):
    import ctraj
    from ctraj.compiler import compile_beamline

    force = ctraj.hexapole_force(V=30e3, R=17.5e-3, n_knots=200 if table == "quadratic" else 4096)
    if table == "radial":
        force = ctraj.reference_radial_table(ctraj.TwoLevelStark(6.7e9, 4.2, 1.0), V=27.6e3, d=0.035)
    elif table == "stark1":
        force = ctraj.StarkForce(force.knots, force.coef, V=27.6e3, R=17.5e-3, field_order=1)
    return compile_beamline(ctraj.Beamline([
        ctraj.ElectrostaticLens(name="ES lens", z0=0.80, L=0.30, d=35e-3, dt=1e-6, dz=1e-3, a_interp=force),
        ctraj.CircularAperture(name="Detection plane", z0=3.0, L=0.0, d=float("inf"))]))


@pytest.mark.parametrize("table", ["linear", "quadratic", "stark1", "radial"])
@pytest.mark.parametrize("n", [1, 33, 5_000, 90_001])
def test_margin_of_a_position_that_is_not_a_number(table, n):
    from ctraj import _abi
    from ctraj.engine import Engine

    cb = _compiled(table)
    g = np.random.default_rng(n)
    ics = g.standard_normal((6, n)) * np.array([2e-3, 2e-3, 0, 4.0, 4.0, 16.0])[:, None]
    ics[5] += 184.0
    nan = np.arange(0, n, 7)
    ics[g.integers(0, 5, nan.size), nan] = np.nan  # x, y, z, vx or vy
    eng = Engine(0)
    try:
        eng.set_tuning(lens_mode=_abi.LENS_CHUNKED)
        ref = eng.run(cb, n, ics=ics, outputs=True)
        assert np.isposinf(ref.margin[nan]).all()
        eng.set_tuning()
        r = eng.run(cb, n, ics=ics, outputs=True)
        for k in ("label", "rows", "margin"):
            np.testing.assert_array_equal(getattr(r, k), getattr(ref, k), err_msg=k)
        np.testing.assert_array_equal(r.final, ref.final)
        np.testing.assert_array_equal(eng.run(cb, n, ics=ics).counts, ref.counts)
    finally:
        eng.close()
