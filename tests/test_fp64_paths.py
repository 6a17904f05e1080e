"""The exact mode's lens pass away from its usual tables: records too large to
stage, tables and lenses that the four-lane kernel leaves to the general one,
lookups below and above the table, and two lenses in a row; queues that take
four lanes per molecule (up to 10 000) and one.  Against the FP64 oracle, bit
for bit."""
import numpy as np
import pytest
from scipy.interpolate import interp1d

pytestmark = pytest.mark.gpu


def _force(kind):
    import ctraj

    hexapole = dict(V=30e3, R=17.5e-3)
    if kind == "unstaged":  # 8192 records of 32 bytes: read through L2
        return ctraj.hexapole_force(n_knots=8192, **hexapole)
    if kind == "unstaged radial":
        r = np.linspace(0.0, 0.02, 7000)
        return interp1d(r, -3e4 * r)
    if kind == "last staged":  # 6 400 records fill what a CTA stages
        return ctraj.hexapole_force(n_knots=6400, **hexapole)
    f = ctraj.hexapole_force(n_knots=1024, **hexapole)
    if kind == "order 1, unstaged":
        f = ctraj.hexapole_force(n_knots=8192, **hexapole)
        return ctraj.StarkForce(f.knots, f.coef, V=27.6e3, R=17.5e-3, field_order=1)
    if kind == "negative knot":
        E = np.linspace(-1e4, 1e7, 1024)
        return ctraj.StarkForce.from_spline(ctraj.stark.CubicSpline(E, ctraj.TwoLevelStark(6.7e9, 4.2, -1.0)(E)), **hexapole)
    if kind == "negative V":
        return ctraj.hexapole_force(V=-30e3, R=17.5e-3, n_knots=1024)
    if kind == "light":
        return ctraj.StarkForce(f.knots, f.coef * 1e-70, mass=f.mass * 1e-70, **hexapole)
    if kind == "infinite entry":  # in an interval that no molecule reaches
        c = f.coef.copy()
        c[-1, 0] = np.inf
        return ctraj.StarkForce(f.knots, c, **hexapole)
    if kind == "radial below zero":
        r = np.linspace(-0.001, 0.02, 300)
        return interp1d(r, -3e4 * r)
    if kind == "short of both ends":  # |E| from 0 to 5.1e6 in the bore
        E = np.linspace(1e5, 2e6, 512)
        return ctraj.StarkForce.from_spline(ctraj.stark.CubicSpline(E, ctraj.TwoLevelStark(6.7e9, 4.2, -1.0)(E)), **hexapole)
    raise KeyError(kind)


def _ics(n, spread=4.0):
    g = np.random.default_rng(n)
    ics = g.standard_normal((6, n)) * np.array([1e-3, 1e-3, 0, spread, spread, 16.0])[:, None]
    ics[5] += 184.0
    ics[:2, :2] = ics[3:5, :2] = 0.0  # on the axis but for gravity
    return ics


def _compare(cb, ics, enters):
    from ctraj.engine import Engine
    from oracle import oracle

    n = ics.shape[1]
    ref = oracle.run(cb, np.ascontiguousarray(ics), threads=8)
    assert n - ref["counts"][cb.labels.index("Lens entrance")] > enters  # of the first lens: they decide the lanes
    eng = Engine(0)
    try:
        r = eng.run(cb, n, precision=64, ics=ics, outputs=True)
        plain = eng.run(cb, n, precision=64, ics=ics)
    finally:
        eng.close()
    for k in ("label", "rows", "margin", "final"):
        np.testing.assert_array_equal(getattr(r, k), ref[k], err_msg=k)
    np.testing.assert_array_equal(plain.counts, ref["counts"])
    assert plain.lens_steps == ref["lens_steps"] == r.lens_steps
    return ref, r


@pytest.mark.parametrize("n", [1_001, 12_001])
@pytest.mark.parametrize("kind", ["unstaged", "unstaged radial", "last staged", "order 1, unstaged", "negative knot",
                                  "negative V", "light", "infinite entry", "radial below zero", "short of both ends"])
def test_lens_equals_the_oracle(kind, n):
    import ctraj
    from ctraj.compiler import compile_beamline

    cb = compile_beamline(ctraj.Beamline([
        ctraj.ElectrostaticLens(name="ES lens", z0=0.80, L=0.10, d=35e-3, dt=2e-6, dz=5e-4, a_interp=_force(kind)),
        ctraj.CircularAperture(name="Detection plane", z0=3.0, L=0.0, d=float("inf"))]))
    ref, r = _compare(cb, _ics(n, 2.0), 10_000 if n > 10_000 else 0)
    assert (r.table_range > 0) == (ref["table_range"] > 0) == (kind in ("short of both ends", "negative V"))


# more than 10 000 molecules in the first lens, of which the second has more and fewer
@pytest.mark.parametrize("n,spread,at_second", [(1_500, 2.0, 0), (14_001, 1.0, 10_000), (16_001, 4.0, 0)])
@pytest.mark.parametrize("kinds", [("unstaged", "negative knot"), ("negative V", "last staged"), ("unstaged radial", "unstaged")])
def test_two_lenses_equal_the_oracle(kinds, n, spread, at_second):
    import ctraj
    from ctraj.compiler import compile_beamline

    first, second = (_force(k) for k in kinds)
    cb = compile_beamline(ctraj.Beamline([
        ctraj.ElectrostaticLens(name="ES lens", z0=0.40, L=0.06, d=35e-3, dt=2e-6, a_interp=first),
        ctraj.CircularAperture(name="A1", z0=0.60, L=1e-3, d=30e-3),
        ctraj.ElectrostaticLens(name="ES lens 2", z0=0.80, L=0.05, d=33e-3, dt=3e-6, scheme="classic", a_interp=second),
        ctraj.CircularAperture(name="Detection plane", z0=3.0, L=0.0, d=float("inf"))]))
    ref, _ = _compare(cb, _ics(n, spread), 10_000 if n > 10_000 else 0)
    both = (ref["rows"] > 150 + 60).sum()  # steps of the first lens and more
    assert both > at_second


# a radial table that ends inside the bore or begins off the axis: a molecule that looks outside is lost at that step
# and the run raises
@pytest.mark.parametrize("n", [1_001, 12_001])
@pytest.mark.parametrize("first,last", [(0.0, 0.009), (2e-4, 0.02)])
def test_lookups_outside_a_radial_table(first, last, n):
    import ctraj
    import torch
    from ctraj.compiler import compile_beamline
    from ctraj.engine import Engine
    from oracle import oracle

    r = np.linspace(first, last, 200)
    cb = compile_beamline(ctraj.Beamline([
        ctraj.ElectrostaticLens(name="ES lens", z0=0.80, L=0.10, d=35e-3, dt=2e-6, a_interp=interp1d(r, 1e5 * r)),
        ctraj.CircularAperture(name="Detection plane", z0=3.0, L=0.0, d=float("inf"))]))
    ics = _ics(n, 0.6)
    ref = oracle.run(cb, np.ascontiguousarray(ics), threads=8)
    assert 0 < ref["errors"] < n and n - ref["counts"][cb.labels.index("Lens entrance")] > (10_000 if n > 10_000 else 0)
    out = {"label": torch.zeros(n, dtype=torch.int32, device="cuda"), "rows": torch.zeros(n, dtype=torch.int32, device="cuda"),
           "margin": torch.zeros(n, dtype=torch.float64, device="cuda"),
           "final": torch.zeros((10, n), dtype=torch.float64, device="cuda")}
    eng = Engine(0)
    try:
        with pytest.raises(ValueError, match=f"{ref['errors']} molecules"):
            eng.run(cb, n, precision=64, ics=ics, device_outputs=out)
    finally:
        eng.close()
    for k in out:
        np.testing.assert_array_equal(out[k].cpu().numpy(), ref[k], err_msg=k)
