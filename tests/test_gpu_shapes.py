"""Shapes and counts at which the steps take other launches than at the sizes of
the other tests.

Tolerances: FP64 1e-10 against the oracle and between two boxes that hold the
same flow (the bound of the FP64 path); mixed 1e-5 on the velocity field and
1e-4 on particle velocities, and 1e-4 on an electrolyte's spectra (the bounds of
the mixed path)."""
import os
import sys

import numpy as np
import pytest

from oracle import spm, udf

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def rel(a, b):
    n = np.linalg.norm(b)
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / (n if n > 0 else 1.0)


def _spheres(np_xyz, n, seed, a=3.0):
    from kapsel_old_b200 import workload

    return workload.place_spheres(n, [1 << p for p in np_xyz], a, 0.5, seed)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("np_xyz,axis,copies", [((5, 4, 5), 0, 4), ((5, 4, 5), 0, 8), ((4, 5, 6), 2, 4),
                                                ((4, 5, 5), 2, 2)])
def test_lees_edwards_box_of_copies(np_xyz, axis, copies, precision):
    """The sheared step at NX = 128 and 256 and at NZ = 32 and 256: a box that holds
    a shorter box's flow and spheres several times over along x or z moves as the
    shorter one does (NX = 32 and NZ = 64 are held to recorded runs).  No thermal
    kicks; the grid is reset in the third step."""
    import kapsel_old_b200 as kg

    N = 1 << np_xyz[axis]
    xs = _spheres(np_xyz, 2, 31)
    xs[0, 1] = 0.3  # its profile reaches across the sheared boundary
    shift = np.zeros(3)
    shift[axis] = N
    many = np.concatenate([xs + c * shift for c in range(copies)])
    runs = []
    for x in (xs, many):
        npx = list(np_xyz)
        npx[axis] += int(np.log2(len(x) // len(xs)))
        s = kg.Simulation({"eq": "Shear_Navier_Stokes_Lees_Edwards", "np_xyz": tuple(npx), "a": 3.0, "a_xi": 2.0,
                           "kbt": 0.0, "dt": 0.01, "shear_rate": 0.1,
                           "particles": [{"x": tuple(map(float, p))} for p in x]}, precision=precision)
        s.set_oblique(0.9975, 0.1)
        s.step(5)
        runs.append((s.velocity(), s.particles(), s.oblique()))
        s.close()
    (u, p, o), (um, pm, om) = runs
    assert rel(um, np.concatenate([u] * copies, axis=1 + axis)) < (1e-5 if precision else 1e-10)
    tol = 1e-4 if precision else 1e-10
    for c in range(copies):
        part = slice(c * len(xs), (c + 1) * len(xs))
        assert rel(pm["v"][part], p["v"]) < tol and rel(pm["omega"][part], p["omega"]) < tol
        d = pm["x"][part] - p["x"]
        assert np.abs(d - N * np.round(d / N) * (shift > 0)).max() < tol  # the shorter box wraps sooner
    assert om["degree_oblique"] == o["degree_oblique"] < 0.1
    assert rel(om["shear_rate_eff"], o["shear_rate_eff"]) < tol


def test_recorded_lees_edwards_steps_are_what_their_script_writes():
    sys.path.insert(0, GOLDEN)
    try:
        import make_le_steps
    finally:
        sys.path.remove(GOLDEN)
    want, got = np.load(os.path.join(GOLDEN, "le_steps.npz")), make_le_steps.record()
    assert set(want.files) == set(got)
    for k in got:
        assert rel(got[k], want[k]) < 1e-10, k


@pytest.mark.parametrize("np_xyz", [(5, 4, 4), (5, 4, 5), (4, 5, 6), (5, 4, 7), (4, 6, 8), (7, 4, 5), (8, 4, 5)])
def test_electrolyte_step_shapes_mixed(np_xyz):
    """The 32-bit fused charge, flux and Coulomb passes at every NZ, and the x
    passes."""
    import kapsel_old_b200 as kg

    cfg = udf.electrolyte_config(np_xyz, 2, seed=8, surface_charge=-50.0, efield=(0.05, 0.02, 0.0), a=3.0)
    g, o = kg.Simulation(cfg, precision=1), spm.ElectrolyteOracle(cfg)
    g.step(2)
    o.step()
    o.step()
    z = spm.SpmOracle.to_ooura(np.stack([o.S.truncate(o.zeta[d]) for d in range(2)]))
    c = spm.SpmOracle.to_ooura(np.stack([o.S.truncate(o.conc_k[n]) for n in range(2)]))
    assert rel(g.zeta(), z) < 1e-4 and rel(g.concentration(), c) < 1e-4
    assert rel(g.particles()["v"], o.p.v) < 1e-4


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1023, 1024, 1025])
def test_gather_and_scatter_at_a_thousand_spheres(n, precision):
    """Either side of where gather and scatter take fewer threads and blocks a
    sphere (1024), and where the scatter's candidates come from the neighbour
    lists (above 1024)."""
    import kapsel_old_b200 as kg

    np_xyz = (6, 6, 6)
    cfg = {"eq": "Navier_Stokes", "np_xyz": np_xyz, "a": 2.0, "a_xi": 2.0, "kbt": 1e-3, "dt": 0.01,
           "particles": [{"x": tuple(map(float, x))} for x in _spheres(np_xyz, n, 29, a=2.0)]}
    g, o = kg.Simulation(cfg, precision=precision), spm.SpmOracle(cfg)
    for _ in range(2):
        g.step(1)
        o.step()
    z = spm.SpmOracle.to_ooura(np.stack([o.S.truncate(o.zeta[d]) for d in range(2)]))
    tol, p = (1e-5 if precision else 1e-10), g.particles()
    assert rel(g.zeta(), z) < tol
    assert rel(p["v"], o.p.v) < tol and rel(p["omega"], o.p.omega) < tol


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("np_xyz", [(4, 5, 6), (4, 4, 5)])
def test_block_level_x_passes_of_sixteen_points(np_xyz, precision):
    import ctypes

    import kapsel_old_b200 as kg

    cfg = {"eq": "Navier_Stokes", "np_xyz": np_xyz, "a": 3.0, "a_xi": 2.0, "kbt": 1e-3, "dt": 0.01,
           "particles": [{"x": tuple(map(float, x))} for x in _spheres(np_xyz, 2, 33)]}
    a, b = (kg.Simulation(cfg, precision=precision) for _ in range(2))
    fn = b.L.kapsel_gpu_set_x_split
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int]
    assert fn(b.h, 1) == 0
    a.step(4)
    b.step(4, graph=True)
    assert rel(b.zeta(), a.zeta()) < (1e-5 if precision else 1e-12)


@pytest.mark.parametrize("np_xyz,precision,planes", [
    # one plane an SM: half a wave, 1.3 waves, 2.6 waves
    ((5, 6, 8), 0, False), ((6, 6, 8), 0, False), ((7, 6, 8), 0, True),
    ((4, 7, 7), 0, False), ((6, 7, 7), 0, False), ((7, 7, 7), 0, True),
    ((6, 5, 8), 0, True), ((4, 6, 7), 0, True),  # more than one
    ((6, 6, 6), 1, True), ((6, 6, 8), 1, False)])
def test_where_the_plane_kernels_are_the_default(np_xyz, precision, planes):
    import kapsel_old_b200 as kg

    cfg = {"eq": "Navier_Stokes", "np_xyz": np_xyz, "a": 3.0, "a_xi": 2.0, "kbt": 0.0, "dt": 0.01,
           "particles": [{"x": (9.0, 9.0, 9.0)}]}
    s = kg.Simulation(cfg, precision=precision)
    assert (s.step_kernel_names()[6] == "k_yzw_c2r") == planes
    # either way the other form is there and gives the same bits
    s.step(2)
    t = kg.Simulation(cfg, precision=precision)
    assert t.L.kapsel_gpu_set_pass_variant(t.h, 0, 0 if planes else 3) == 0
    t.step(2)
    assert np.array_equal(s.zeta(), t.zeta())
