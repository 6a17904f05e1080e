"""A set number of lanes per CTA (tuning lens_threads, batch_lens_threads) is
the one that runs, for every queue: one lens pass is launched.  0, the default,
leaves the choice to the queue's length, which may take more launches.  Results
are the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SET = (512, 768, 1024)


@pytest.fixture(scope="module")
def engine():
    from ctraj.engine import Engine

    eng = Engine(0)
    yield eng
    eng.close()


def _args(sigma=20.0, table="linear"):
    import ctraj
    from ctraj.compiler import compile_beamline
    from ctraj.distributions import device_spec
    from ctraj.workloads import lens_beamline

    bl = lens_beamline()
    if table == "quadratic":
        bl.elements[1].a_interp = ctraj.hexapole_force(V=30e3, R=17.5e-3, n_knots=200)
    xs = device_spec(ctraj.GaussianPositionDistribution(sigmax=1.5e-3, sigmay=1.5e-3, z=0.0), "position")
    vs = device_spec(ctraj.CeNTREXVelocityDistribution(sigmax=sigma, sigmay=sigma), "velocity")
    return compile_beamline(bl), dict(xdist=xs, vdist=vs)


def test_default_is_by_the_queue(engine):
    engine.set_tuning()
    t = engine.get_tuning()
    assert (t["lens_threads"], t["batch_lens_threads"]) == (0, 0)
    for bad in (dict(lens_threads=256), dict(batch_lens_threads=640), dict(lens_threads=-512)):
        with pytest.raises(ValueError):
            engine.set_tuning(**bad)


# few molecules in the lens; a queue most of the molecules fill; one long enough for the wider passes by itself
@pytest.mark.parametrize("table,n,sigma", [("linear", 10_001, 20.0), ("linear", 2_000_001, 2.0), ("linear", 21_000_001, 15.0),
                                           ("quadratic", 300_001, 2.0)])
def test_single_runs(engine, table, n, sigma):
    cb, kw = _args(sigma, table)
    engine.set_tuning()
    ref = engine.run(cb, n, seed=4, **kw)
    for lanes in SET:
        engine.set_tuning(lens_threads=lanes)
        r = engine.run(cb, n, seed=4, **kw)
        assert r.counts.tolist() == ref.counts.tolist() and r.lens_steps == ref.lens_steps
        assert r.kernels == 6  # front, three of the order, the pass, the ends


def test_runs_with_outputs_launch_one_pass(engine):
    cb, kw = _args()
    for lanes in (0,) + SET:
        engine.set_tuning(lens_threads=lanes)
        assert engine.run(cb, 50_001, seed=4, outputs=True, **kw).kernels == 5


@pytest.mark.parametrize("table", ["linear", "quadratic"])
def test_batches(engine, table):
    cb, kw = _args(2.0, table)
    seeds = [1, 2, 3, 4]
    engine.set_tuning()
    ref = engine.run_batch(cb, 40_001, seeds, **kw)
    for lanes in SET:
        engine.set_tuning(batch_lens_threads=lanes)
        rs = engine.run_batch(cb, 40_001, seeds, **kw)
        assert [r.counts.tolist() for r in rs] == [r.counts.tolist() for r in ref]
        assert sum(r.kernels for r in rs) == len(seeds) + 5


def test_sweeps(engine):
    from ctraj.stark import hexapole_force
    from ctraj.sweep import SweepConfigs, run_sweep
    from ctraj.workloads import lens_beamline, source

    cfg = SweepConfigs(voltages=np.linspace(1e3, 30e3, 5), forces=[hexapole_force(V=30e3, splitting_hz=a) for a in (6.7e9, 20.0e9)],
                       n_molecules=np.full((2, 5), 20_001))
    xs, vs = source()
    kw = dict(xdist=xs, vdist=vs, seed=3, engine=engine)
    engine.set_tuning()
    ref = run_sweep(lens_beamline(), cfg, **kw)
    for graph in (True, False):
        for lanes, launches in ((0, 7), (512, 6), (0, 7), (768, 6), (1024, 6), (512, 6)):
            engine.set_tuning(lens_threads=lanes)
            for _ in range(2):
                r = run_sweep(lens_beamline(), cfg, use_graph=graph, **kw)
                np.testing.assert_array_equal(r.counts, ref.counts)
                assert r.kernels == launches, lanes
