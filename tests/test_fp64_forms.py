"""The exact mode forms its square roots and quotients from fewer FP64
instructions (csrc/fp64.cuh); every one must be the IEEE operation's result,
bit for bit.  Its lens kernel takes four lanes per molecule up to a queue
size and one beyond: both against the FP64 oracle, with the table kinds,
schemes and step rules it accepts."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 2])
def test_forms_equal_the_ieee_operations(seed):
    from bench_kernels.build import build as build_probes

    lib = ctypes.CDLL(str(build_probes()))
    lib.ctraj_peak_fp64_check.restype = ctypes.c_int
    lib.ctraj_peak_fp64_check.argtypes = [ctypes.c_longlong, ctypes.c_ulonglong, ctypes.POINTER(ctypes.c_ulonglong)]
    n = 400_000_000
    bad = (ctypes.c_ulonglong * 4)(1, 1, 1, 1)
    assert lib.ctraj_peak_fp64_check(n, seed, bad) == 0
    assert list(bad)[:3] == [0, 0, 0]
    assert bad[3] < 3 * n / 8 * 1e-4  # unsure: near a tie or a power of two, 2^-17 + 2^-19 of random operands each


def test_the_fp32_root_is_sqrtf():
    from bench_kernels.build import build as build_probes

    lib = ctypes.CDLL(str(build_probes()))
    lib.ctraj_peak_sqrt32_check.argtypes = [ctypes.POINTER(ctypes.c_ulonglong)]
    bad = ctypes.c_ulonglong(1)
    assert lib.ctraj_peak_sqrt32_check(ctypes.byref(bad)) == 0
    assert bad.value == 0


def _beamline(table, scheme, dt):
    import ctraj

    force = ctraj.hexapole_force(V=30e3, R=17.5e-3)
    if table == "radial":
        force = ctraj.reference_radial_table(ctraj.TwoLevelStark(6.7e9, 4.2, 1.0), V=27.6e3, d=0.035)
    elif table == "stark1":
        force = ctraj.StarkForce(force.knots, force.coef, V=27.6e3, R=17.5e-3, field_order=1)
    elif table == "zero":  # no field: every force quotient is a zero
        force = ctraj.hexapole_force(V=0.0, R=17.5e-3)
    return ctraj.Beamline([
        ctraj.CircularAperture(name="A1", z0=0.30, L=1e-3, d=12e-3),
        ctraj.ElectrostaticLens(name="ES lens", z0=0.80, L=0.10, d=35e-3, dt=dt, dz=5e-4, a_interp=force, scheme=scheme),
        ctraj.CircularAperture(name="Detection plane", z0=3.0, L=0.0, d=float("inf")),
    ])


# the queue takes 2 % of a wide beam and all of a narrow one: 1 molecule, a part of a quad's warp, 9 999 and 10 000
# (four lanes each), 10 001 (one lane each) and a queue of several batches per warp
@pytest.mark.parametrize("table,scheme,dt,n", [
    ("stark2", "reference", 1e-6, 1), ("stark2", "classic", 1e-6, 13), ("stark2", "reference", None, 9_999),
    ("stark1", "reference", None, 2_000), ("radial", "reference", 2e-6, 2_001), ("radial", "classic", None, 10_001),
    ("zero", "reference", 2e-6, 999), ("stark2", "reference", 2e-6, 10_000), ("stark2", "classic", 2e-6, 10_001),
    ("stark1", "classic", 2e-6, 12_345), ("stark2", "reference", None, 90_001)])
def test_lens_equals_the_oracle(table, scheme, dt, n):
    from ctraj.compiler import compile_beamline
    from ctraj.engine import Engine
    from oracle import oracle

    cb = compile_beamline(_beamline(table, scheme, dt))
    g = np.random.default_rng(n)
    ics = g.standard_normal((6, n)) * np.array([1e-3, 1e-3, 0, 4.0, 4.0, 16.0])[:, None]
    ics[5] += 184.0
    if n > 20:  # on the axis: r = 0, and one component zero throughout the horizontal plane
        ics[:2, :3] = 0.0
        ics[3:5, :3] = 0.0
        ics[0, 3:6] = ics[3, 3:6] = 0.0
    ref = oracle.run(cb, np.ascontiguousarray(ics))
    eng = Engine(0)
    try:
        r = eng.run(cb, n, precision=64, ics=ics, outputs=True)
    finally:
        eng.close()
    assert np.array_equal(r.label, ref["label"])
    assert np.array_equal(r.final, ref["final"], equal_nan=True)
    assert np.array_equal(r.margin, ref["margin"])
    assert np.array_equal(r.rows, ref["rows"])
