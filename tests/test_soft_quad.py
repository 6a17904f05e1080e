"""The FP64 soft lens pass gives a molecule four lanes while the queue is short
(k_soft_lens_quad) and one beyond: a run whose queue is long must equal the sum
of its parts whose queues are short, counts exactly, loss and gradient to the
rounding of their sums; without whole eights between checkpoints every queue
takes the one-lane pass.  The FP32 pass's edge test (soft_test_r2) must give
the general one's values."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("low,detector,dt_scale", [(False, float("inf"), 1.0), (True, 10e-3, 3.0)])
def test_long_queue_equals_its_parts(low, detector, dt_scale):
    from ctraj.adjoint import SoftProblem, soft_transmission
    from ctraj.engine import Engine
    from ctraj.workloads import lens_beamline

    bl = lens_beamline(V=10e3 if low else 30e3, low_field_seeker=low, detector_d=detector)
    bl.elements[1].dt *= dt_scale
    eng = Engine(0)

    def run(n, offset, checkpoint=64, grad=True):
        prob = SoftProblem.from_beamline(bl, n=n, aperture="A1", precision=64, seed=5, offset=offset, checkpoint=checkpoint)
        return soft_transmission(prob, prob.initial_params(), want_grad=grad, engine=eng)

    try:
        n = 480_000
        whole = run(n, 0)
        assert whole.lens_molecules > 10_000
        parts = [run(n // 2, 0), run(n // 4, n // 2), run(n // 4, 3 * n // 4)]
        assert max(p.lens_molecules for p in parts) <= 10_000
        for k in ("lens_molecules", "lens_steps", "dropped"):
            assert sum(getattr(p, k) for p in parts) == getattr(whole, k), k
        w = np.array([0.5, 0.25, 0.25])
        assert abs(w @ [p.loss for p in parts] - whole.loss) <= 1e-13 * whole.loss
        g = sum(wk * p.grad for wk, p in zip(w, parts))
        assert np.abs(g - whole.grad).max() <= 1e-11 * np.abs(whole.grad).max()
        # a tail of molecules per warp, the forward pass alone, and the one-lane pass by the checkpoint interval
        a, b, c = run(3_333, 7), run(3_333, 7, grad=False), run(3_333, 7, checkpoint=60)
        assert a.loss == b.loss and (a.lens_steps, a.dropped) == (b.lens_steps, b.dropped)
        assert abs(a.loss - c.loss) <= 1e-13 * c.loss and a.lens_molecules == c.lens_molecules
        assert np.abs(a.grad - c.grad).max() <= 1e-10 * np.abs(c.grad).max()
    finally:
        eng.close()


# widths from a ten-thousandth of the radius to a hundred times it, and an edge of radius 0: every float radius, of which
# the smallest have a square below the normal numbers
@pytest.mark.parametrize("radius,inv_w", [(0.0222, 5e3), (0.0175, 1.0), (1e-3, 1e7), (1.0, 1e2), (0.0, 1.0)])
def test_the_lens_pass_edge_test_is_the_general_one(radius, inv_w):
    from bench_kernels.build import build as build_probes

    lib = ctypes.CDLL(str(build_probes()))
    lib.ctraj_peak_soft_test_check.argtypes = [ctypes.c_float, ctypes.c_float, ctypes.POINTER(ctypes.c_ulonglong)]
    bad = ctypes.c_ulonglong(1)
    assert lib.ctraj_peak_soft_test_check(radius, inv_w, ctypes.byref(bad)) == 0
    assert bad.value == 0


# queues whose tests have warps of their own (up to two eights of molecules per SM) against one that has not: one
# molecule, an incomplete eight, the last such queue, and step counts that are not whole blocks (dt)
@pytest.mark.parametrize("low,dt_scale,part", [(False, 1.0, 20_000), (True, 1.0, 40_000), (True, 7.3, 13_337), (False, 3.1, 84_000)])
def test_tests_in_their_own_warps(low, dt_scale, part):
    from ctraj.adjoint import SoftProblem, soft_transmission
    from ctraj.engine import Engine
    from ctraj.workloads import lens_beamline

    bl = lens_beamline(V=10e3 if low else 30e3, low_field_seeker=low, detector_d=12e-3)
    bl.elements[1].dt *= dt_scale
    eng = Engine(0)

    def run(n, offset, grad=True):
        prob = SoftProblem.from_beamline(bl, n=n, aperture="A1", precision=64, seed=8, offset=offset)
        return soft_transmission(prob, prob.initial_params(), want_grad=grad, engine=eng)

    try:
        k = 240_000 // part
        whole, parts = run(k * part, 0), [run(part, j * part) for j in range(k)]
        assert 2_432 < whole.lens_molecules <= 10_000 and max(p.lens_molecules for p in parts) <= 2_432
        for f in ("lens_molecules", "lens_steps", "dropped"):
            assert sum(getattr(p, f) for p in parts) == getattr(whole, f), f
        assert abs(sum(p.loss for p in parts) / k - whole.loss) <= 1e-13 * whole.loss
        g = sum(p.grad for p in parts) / k
        assert np.abs(g - whole.grad).max() <= 1e-11 * np.abs(whole.grad).max()
        a, b = run(37, 0), run(37, 0, grad=False)  # about one molecule in the queue
        assert a.loss == b.loss and (a.lens_steps, a.dropped) == (b.lens_steps, b.dropped)
    finally:
        eng.close()
