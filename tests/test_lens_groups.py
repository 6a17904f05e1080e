"""The persistent FP32 lens pass takes its steps in groups, loads table pieces
ahead when few warps have molecules, spreads short queues over the CTAs and
picks its CTA size by the queue; none of it may change a result.  Against the
chunked pass, which looks at every molecule after every step: every table
form, steps too wide to extrapolate, and queues around the sizes where the
pass changes its ways (a warp, a CTA's four warps, 512 lanes per CTA)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compiled(table, dt, V=30e3):
    import ctraj
    from ctraj.compiler import compile_beamline

    force = ctraj.hexapole_force(V=V, R=17.5e-3, low_field_seeker=table == "focus",
                                 n_knots=200 if table == "quadratic" else 4096)
    if table == "radial":
        force = ctraj.reference_radial_table(ctraj.TwoLevelStark(6.7e9, 4.2, 1.0), V=27.6e3, d=0.035)
    elif table == "stark1":
        force = ctraj.StarkForce(force.knots, force.coef, V=27.6e3, R=17.5e-3, field_order=1)
    return compile_beamline(ctraj.Beamline([
        ctraj.ElectrostaticLens(name="ES lens", z0=0.80, L=0.30, d=35e-3, dt=dt, dz=1e-3, a_interp=force),
        ctraj.CircularAperture(name="Detection plane", z0=3.0, L=0.0, d=float("inf"))]))


def _ics(n, spread):
    g = np.random.default_rng(n)
    ics = g.standard_normal((6, n)) * np.array([2e-3, 2e-3, 0, spread, spread, 16.0])[:, None]
    ics[5] += 184.0
    if n > 40:
        ics[:2, :2] = ics[3:5, :2] = 0.0  # on the axis
    return ics


@pytest.mark.parametrize("table,dt,n,spread", [
    ("linear", 1e-6, 1, 1.0), ("linear", 1e-6, 33, 4.0), ("focus", 1e-6, 5_000, 4.0), ("linear", 2e-5, 3_000, 4.0),
    ("focus", None, 19_457, 4.0), ("linear", 1e-6, 77_824, 2.0), ("linear", 2e-6, 77_825, 2.0), ("focus", 2e-6, 300_000, 4.0),
    ("quadratic", 1e-6, 5_000, 4.0), ("stark1", None, 20_000, 4.0), ("radial", None, 33, 4.0), ("radial", 2e-6, 90_000, 4.0)])
def test_persistent_equals_chunked(table, dt, n, spread):
    from ctraj import _abi
    from ctraj.engine import Engine

    cb, ics = _compiled(table, dt), _ics(n, spread)
    eng = Engine(0)
    try:
        eng.set_tuning(lens_mode=_abi.LENS_CHUNKED)
        ref = eng.run(cb, n, ics=ics, outputs=True)
        for lanes in (512, 1024):
            eng.set_tuning(lens_threads=lanes, batch_lens_threads=lanes, batch_group=2)
            r = eng.run(cb, n, ics=ics, outputs=True)
            for k in ("label", "rows", "margin"):
                assert np.array_equal(getattr(r, k), getattr(ref, k)), k
            assert np.array_equal(r.final, ref.final, equal_nan=True)
            plain = eng.run(cb, n, ics=ics)
            runs = eng.run_batch(cb, n, None, ics=[ics, ics])
            for p in (plain, *runs):
                assert np.array_equal(p.counts, ref.counts)
                assert (p.molecule_steps, p.lens_steps) == (ref.molecule_steps, ref.lens_steps)
    finally:
        eng.close()
