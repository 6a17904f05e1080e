"""The FP32 fronts: the packed Box-Muller pair gives box_muller's normals for
every word, and a sweep's front, whose warps walk contiguous ranges of
molecules, counts each configuration's molecules whatever their number, and
the molecules that the front screens by x and vy are those that the walk stops."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_box_muller_pair_is_two_box_mullers():
    from bench_kernels.build import build as build_probes

    lib = ctypes.CDLL(str(build_probes()))
    lib.ctraj_peak_bm_pair_check.argtypes = [ctypes.POINTER(ctypes.c_ulonglong)]
    bad = ctypes.c_ulonglong(1)
    assert lib.ctraj_peak_bm_pair_check(ctypes.byref(bad)) == 0
    assert bad.value == 0


# empty configurations at the ends, alone and in a row, and boundaries in, at and across a warp's 32 molecules
@pytest.mark.parametrize("numbers", [
    [0, 1, 31, 32, 33, 0, 0, 65, 5000, 0], [1, 0, 0, 0, 0, 0, 0, 0, 0, 0], [0, 0, 0, 0, 0, 0, 0, 0, 0, 7],
    [40_000, 0, 1, 1, 1, 1, 200_000, 3, 0, 90_001], [64, 32, 96, 0, 32, 1, 31, 0, 32, 32]])
def test_sweep_front_counts_every_configuration(numbers):
    from ctraj.engine import default_engine
    from ctraj.stark import hexapole_force
    from ctraj.sweep import SweepConfigs, config_beamlines, loop_sweep, run_sweep
    from ctraj.workloads import lens_beamline, source

    forces = [hexapole_force(V=30e3, splitting_hz=a, n_knots=256) for a in (6.7e9, 20.0e9)]
    cfg = SweepConfigs(voltages=np.linspace(0, 30e3, 5), forces=forces, n_molecules=np.array(numbers).reshape(2, 5))
    bl = lens_beamline()
    xs, vs = source()
    kw = dict(xdist=xs, vdist=vs, seed=3, offset=17, engine=default_engine())
    r = run_sweep(bl, cfg, **kw)
    cbs = config_beamlines(bl, cfg)
    loop = loop_sweep(cbs, cfg, **kw)
    first = cbs[0].labels.index(bl.elements[0].name)
    np.testing.assert_array_equal(r.counts.sum(-1), cfg.n_molecules)
    np.testing.assert_array_equal(r.counts[..., first], loop[..., first])
    # at the bore to within the rounding of the two forms of the force
    assert np.abs(r.counts - loop).sum(-1).max() <= 2


# (first element, sigma of y, sigma of vy, g): planes in and off the beam's centre, y from nothing to more than the
# aperture, vy from nothing up, gravity of either sign and strong enough to decide, and apertures that stop all or none
@pytest.mark.parametrize("element,sigma_y,sigma_vy,g", [
    ("circle", 1.5e-3, 20.0, 9.81), ("circle", 0.0, 20.0, 9.81), ("circle", 20e-3, 1.0, -9.81), ("wide", 1.5e-3, 20.0, 9.81),
    ("closed", 1.5e-3, 20.0, 9.81), ("square", 1.5e-3, 20.0, 9.81), ("strip", 0.5e-3, 20.0, -9.81),
    ("above", 1e-3, 10.0, 9.81), ("above", 0.0, 0.0, -2e4), ("circle", 0.0, 0.0, 4e3), ("circle", 1.5e-3, 20.0, 1e31)])
def test_screened_molecules_are_those_the_walk_stops(element, sigma_y, sigma_vy, g):
    import ctraj
    from ctraj.compiler import compile_beamline
    from ctraj.distributions import device_spec
    from ctraj.engine import default_engine

    first = {"circle": ctraj.CircularAperture(name="A1", z0=0.30, L=1e-3, d=12e-3),
             "wide": ctraj.CircularAperture(name="A1", z0=0.30, L=1e-3, d=2.0),
             "closed": ctraj.CircularAperture(name="A1", z0=0.30, L=1e-3, d=0.0),
             "square": ctraj.RectangularAperture(name="A1", z0=0.30, L=1e-3, w=12e-3, h=12e-3),
             "strip": ctraj.RectangularAperture(name="A1", z0=0.30, L=1e-3, w=0.5, h=2e-3),
             "above": ctraj.RectangularAperture(name="A1", z0=0.30, L=1e-3, y0=30e-3, w=20e-3, h=10e-3)}[element]
    cb = compile_beamline(ctraj.Beamline([first, ctraj.CircularAperture(name="A2", z0=0.8, L=1e-3, d=30e-3)]))
    n = 300_001
    xs = device_spec(ctraj.GaussianPositionDistribution(sigmax=1.5e-3, sigmay=sigma_y, z=0.0), "position")
    vs = device_spec(ctraj.CeNTREXVelocityDistribution(sigmax=20.0, sigmay=sigma_vy), "velocity")
    kw = dict(xdist=xs, vdist=vs, seed=7, offset=3, g=g)
    eng = default_engine()
    plain = eng.run(cb, n, **kw)
    walked = eng.run(cb, n, outputs=True, **kw)  # per-molecule outputs: every molecule walks
    np.testing.assert_array_equal(plain.counts, walked.counts)
    assert plain.molecule_steps == walked.molecule_steps
