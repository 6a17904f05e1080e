"""At the tuning's defaults the linear lens pass takes 512, 768 or 1024 lanes
per CTA by the queue's length (on the device, or for a single run also by the
molecules that may fill it): every choice gives the counts and steps of the
pass with a set number of lanes."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from ctraj.engine import Engine

    eng = Engine(0)
    yield eng
    eng.close()


def _args(sigma):
    import ctraj
    from ctraj.compiler import compile_beamline
    from ctraj.distributions import device_spec
    from ctraj.workloads import lens_beamline

    xs = device_spec(ctraj.GaussianPositionDistribution(sigmax=1.5e-3, sigmay=1.5e-3, z=0.0), "position")
    vs = device_spec(ctraj.CeNTREXVelocityDistribution(sigmax=sigma, sigmay=sigma), "velocity")
    return compile_beamline(lens_beamline()), dict(xdist=xs, vdist=vs)


# groups of four runs: queues of less than 1, of 1 to 3 (some CTAs thin), of 3 to 8, of 8 to 32 and of more than 32 rounds
# of 512 lanes on 152 SMs
@pytest.mark.parametrize("n", [10_001, 19_470, 40_001, 57_001, 100_001, 250_001, 900_001])
def test_batch_equals_single_runs(engine, n):
    cb, kw = _args(2.0)
    seeds = [3, 4, 5, 6]
    engine.set_tuning()
    batch = engine.run_batch(cb, n, seeds, **kw)
    engine.set_tuning(lens_threads=768)
    for seed, b in zip(seeds, batch):
        r = engine.run(cb, n, seed=seed, **kw)
        assert b.counts.tolist() == r.counts.tolist() and b.lens_steps == r.lens_steps


# queues of a few, of 8 to 32 and of more than 32 rounds: the default's 512, 768 and 1024 lanes
@pytest.mark.parametrize("n,sigma", [(1_000_001, 2.0), (21_000_001, 15.0), (81_000_001, 15.0)])
def test_long_queues_equal_set_lanes(engine, n, sigma):
    cb, kw = _args(sigma)
    engine.set_tuning()
    r = engine.run(cb, n, seed=9, **kw)
    for lanes in (768, 1024):
        engine.set_tuning(lens_threads=lanes)
        o = engine.run(cb, n, seed=9, **kw)
        assert o.counts.tolist() == r.counts.tolist() and o.lens_steps == r.lens_steps
