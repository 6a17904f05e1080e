"""The persistent FP32 lens pass picks the form of its steps by the table, the
lens and how full its CTAs are: the quadratic form's one at a time (full CTAs in
a lens that pushes outward) or in groups, the linear form's with table pieces
loaded ahead or without (by the steps through the lens and the molecules per
warp).  Every choice gives the chunked pass's results, and the runs' own ends
those of the deferred ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS_WARPS = 152 * 4  # warps that a short queue is spread over


def _compiled(force, **step):
    import ctraj
    from ctraj.compiler import compile_beamline

    return compile_beamline(ctraj.Beamline([
        ctraj.ElectrostaticLens(name="ES lens", z0=0.80, L=0.60, d=35e-3, a_interp=force, **step),
        ctraj.CircularAperture(name="Detection plane", z0=3.0, L=0.0, d=float("inf"))]))


def _ics(n, spread):
    g = np.random.default_rng(n)
    ics = g.standard_normal((6, n)) * np.array([2e-3, 2e-3, 0, spread, spread, 16.0])[:, None]
    ics[5] += 184.0
    if n > 40:
        ics[:2, :2] = ics[3:5, :2] = 0.0  # on the axis
        ics[0, 2:4] = np.nan
    return ics


def _equal_to_chunked(cb, n, spread):
    from ctraj import _abi
    from ctraj.engine import Engine

    ics = _ics(n, spread)
    eng = Engine(0)
    try:
        eng.set_tuning(lens_mode=_abi.LENS_CHUNKED)
        ref = eng.run(cb, n, ics=ics, outputs=True)
        for tuning in (dict(), dict(lens_service=24, lens_interval=40), dict(lens_threads=1024, batch_lens_threads=768)):
            eng.set_tuning(batch_group=2, **tuning)
            r = eng.run(cb, n, ics=ics, outputs=True)
            for k in ("label", "rows", "margin", "final"):
                np.testing.assert_array_equal(getattr(r, k), getattr(ref, k), err_msg=k)
            for p in (eng.run(cb, n, ics=ics), *eng.run_batch(cb, n, None, ics=[ics, ics])):
                np.testing.assert_array_equal(p.counts, ref.counts)
                assert (p.molecule_steps, p.lens_steps) == (ref.molecule_steps, ref.lens_steps)
    finally:
        eng.close()


# tables of 200 knots (staged) and of 8192 (read through L1), a lens that loses most and one that keeps most; a warp, a
# queue spread over the SMs, one of just over 512 lanes per SM and one of several rounds
@pytest.mark.parametrize("knots", [200, 8192])
@pytest.mark.parametrize("low", [False, True])
@pytest.mark.parametrize("n", [33, 20_000, 77_825, 200_001])
def test_quadratic_form(knots, low, n):
    import ctraj

    force = ctraj.hexapole_force(V=10e3 if low else 30e3, R=17.5e-3, low_field_seeker=low, n_knots=knots)
    _equal_to_chunked(_compiled(force, dz=3e-3), n, 2.0)


# 600, 300 and 240 steps through the lens: pieces ahead up to 6, 1 and 1 molecules per warp
@pytest.mark.parametrize("dz,n", [(1e-3, 6 * SMS_WARPS), (1e-3, 6 * SMS_WARPS + 1), (1e-3, 30 * SMS_WARPS), (2e-3, SMS_WARPS),
                                  (2e-3, SMS_WARPS + 1), (2.5e-3, 1), (2.6e-3, 1), (2e-4, 27 * SMS_WARPS)])
@pytest.mark.parametrize("low", [False, True])
def test_pieces_ahead(dz, n, low):
    import ctraj

    force = ctraj.hexapole_force(V=10e3 if low else 30e3, R=17.5e-3, low_field_seeker=low)
    _equal_to_chunked(_compiled(force, dz=dz), n, 3.0)
