"""The transform passes and the point operations fused into them, at the edges
of the shapes each is compiled for; the stencil and its overlaps; repeated
network calls.

Tolerances: FP64 1e-10 against the oracle and the recorded runs (the bound of
the FP64 path), 1e-12 between two sets of kernels over three steps; mixed 1e-5
on the fluid (the bound of the mixed path)."""
import os

import numpy as np
import pytest

from oracle import spm, udf

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "le_steps.npz")


def rel(a, b):
    n = np.linalg.norm(b)
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / (n if n > 0 else 1.0)


def _spheres(np_xyz, n, seed, a=3.0):
    from kapsel_old_b200 import workload

    xs = workload.place_spheres(n, [1 << p for p in np_xyz], a, 0.5, seed)
    return [{"x": tuple(map(float, x))} for x in xs]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("np_xyz", [(4, 5, 6), (4, 6, 7), (4, 7, 8), (4, 8, 6), (5, 6, 8), (4, 6, 5)])
def test_warp_passes_match_block_passes(np_xyz, precision):
    """NZ = 32..256 and NY = 32..256, the lengths of the warp-level z passes and
    of the tile y passes, against the block-level ones."""
    import kapsel_old_b200 as kg

    cfg = {"eq": "Navier_Stokes", "np_xyz": np_xyz, "a": 3.0, "a_xi": 2.0, "kbt": 1e-3, "dt": 0.01,
           "particles": _spheres(np_xyz, 3, 21)}
    zeta = []
    for z, y in ((0, 0), (1, 1)):
        s = kg.Simulation(cfg, precision=precision)
        assert s.L.kapsel_gpu_set_pass_variant(s.h, z, y) == 0
        s.step(3)
        zeta.append(s.zeta())
    assert rel(zeta[0], zeta[1]) < (1e-5 if precision else 1e-12)


def _against_oracle(cfg, precision, steps=2):
    import kapsel_old_b200 as kg

    g, o = kg.Simulation(cfg, precision=precision), spm.SpmOracle(cfg)
    for _ in range(steps):
        g.step(1)
        o.step()
    z = spm.SpmOracle.to_ooura(np.stack([o.S.truncate(o.zeta[d]) for d in range(2)]))
    tol = 1e-5 if precision else 1e-10
    p = g.particles()
    assert rel(g.zeta(), z) < tol
    assert rel(p["v"], o.p.v) < tol and rel(p["omega"], o.p.omega) < tol


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("lx", [4, 5, 6, 7, 8])
def test_x_pass_lengths(lx, precision):
    """The x passes at every length, with a ragged last tile of columns."""
    np_xyz = (lx, 4, 5)
    _against_oracle({"eq": "Navier_Stokes", "np_xyz": np_xyz, "a": 3.0, "a_xi": 2.0, "kbt": 1e-3, "dt": 0.01,
                     "particles": _spheres(np_xyz, 2, 22)}, precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [32, 33, 148, 149])
def test_gather_shapes(n, precision):
    """Either side of the particle counts where the gather's blocks change: a
    cluster per particle, blocks of 1024 threads, of 512."""
    np_xyz = (6, 6, 6)
    _against_oracle({"eq": "Navier_Stokes", "np_xyz": np_xyz, "a": 3.0, "a_xi": 2.0, "kbt": 1e-3, "dt": 0.01,
                     "particles": _spheres(np_xyz, n, 23)}, precision)


@pytest.mark.parametrize("np_xyz", [(5, 4, 4), (5, 4, 5), (4, 5, 6), (5, 4, 7), (4, 6, 8), (7, 4, 5), (8, 4, 5)])
def test_electrolyte_step_shapes(np_xyz):
    """Fused charge, flux and Coulomb passes (NZ >= 32) and the separate ones
    (NZ = 16), with the full-spectrum gradient's Nyquist planes, and the x
    passes; NX = 128 and 256 are where loads of the rigidity force's x pass had
    moved in front of the wait for the kernel that writes it."""
    import kapsel_old_b200 as kg

    cfg = udf.electrolyte_config(np_xyz, 2, seed=8, surface_charge=-50.0, efield=(0.05, 0.02, 0.0), a=3.0)
    g, o = kg.Simulation(cfg, precision=0), spm.ElectrolyteOracle(cfg)
    g.step(2)
    o.step()
    o.step()
    z = spm.SpmOracle.to_ooura(np.stack([o.S.truncate(o.zeta[d]) for d in range(2)]))
    c = spm.SpmOracle.to_ooura(np.stack([o.S.truncate(o.conc_k[n]) for n in range(2)]))
    assert rel(g.zeta(), z) < 1e-10 and rel(g.concentration(), c) < 1e-10
    assert rel(g.particles()["v"], o.p.v) < 1e-10


@pytest.mark.parametrize("name,np_xyz", [("z64", (4, 5, 6)), ("z128", (5, 4, 7))])
def test_lees_edwards_recorded_steps(name, np_xyz):
    """Six FP64 steps across the grid reset, against a run recorded from the
    separate Lees-Edwards kernels that were pinned to the reference."""
    import kapsel_old_b200 as kg

    d = np.load(GOLDEN)
    cfg = {"eq": "Shear_Navier_Stokes_Lees_Edwards", "np_xyz": np_xyz, "a": 3.0, "a_xi": 2.0, "kbt": 1e-3, "dt": 0.01,
           "shear_rate": 0.1, "particles": [{"x": tuple(map(float, x))} for x in d[name + "_x0"]]}
    s = kg.Simulation(cfg, precision=0)
    s.set_oblique(0.9975, 0.1)
    s.step(6)
    p, o = s.particles(), s.oblique()
    for k in ("x", "v", "omega", "q"):
        assert rel(p[k], d[f"{name}_{k}"]) < 1e-10, k
    assert rel(s.zeta(), d[name + "_zeta"]) < 1e-10
    assert o["degree_oblique"] == d[name + "_obl"][0]
    assert rel([o["shear_rate_eff"], o["strain"]], d[name + "_obl"][1:]) < 1e-10


@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (1, 1e-5)])
@pytest.mark.parametrize("np_xyz,a", [((4, 4, 4), 5.0), ((5, 5, 5), 5.0), ((6, 6, 6), 4.3)])
def test_overlapping_profiles(np_xyz, a, precision, tol):
    """phi and phi u_p of overlapping spheres: a support that nearly spans the
    box (the whole offset list), neighbours whose offsets wrap, and ones whose
    do not."""
    import kapsel_old_b200 as kg

    L = 1 << np_xyz[0]
    rng = np.random.Generator(np.random.PCG64(4))
    xs = np.mod(np.array([[0.3, 0.2, L - 0.1], [5.1, 0.4, 1.2], [2.2, 6.0, L - 2.0], [L / 2, L / 2, L / 2]]), L)
    cfg = {"eq": "Navier_Stokes", "np_xyz": np_xyz, "a": a, "a_xi": 2.0, "kbt": 0.0, "dt": 0.01,
           "particles": [{"x": tuple(map(float, x))} for x in xs]}
    s = kg.Simulation(cfg, precision=precision)
    st = s.particles()
    st["v"], st["omega"] = rng.normal(size=(4, 3)), rng.normal(size=(4, 3))
    s.set_particle_state(st)
    phi, up = s.make_phi_u()
    ro, uo = spm.SpmOracle(cfg).phi_up(xs, st["v"], st["omega"])
    assert np.abs(phi - ro).max() < tol
    assert np.abs(up - uo).max() < tol * np.abs(uo).max()


def test_network_calls_of_changing_size():
    """The rows an object keeps on the device serve larger and smaller calls."""
    from kapsel_old_b200 import nearcontact as nc

    rng = np.random.Generator(np.random.PCG64(6))
    params, w = nc.init_params(3), np.ones(16, np.float32)
    kept = nc.NearContactNet(params)
    for n in (300, 64, 1000, 1, 129):
        x, y = rng.normal(size=(n, 16)).astype(np.float32), rng.normal(size=(n, 16)).astype(np.float32)
        fresh = nc.NearContactNet(params)
        assert np.array_equal(kept.forward(x), fresh.forward(x))
        (ga, la), (gb, lb) = kept.gradient(x, y, w), fresh.gradient(x, y, w)
        # the same products, added by atomics in any order
        assert rel(ga, gb) < 1e-5 and abs(la - lb) < 1e-5 * abs(lb)


def test_network_rows_grow_without_waiting_for_other_streams():
    """A call with more rows than any before takes its memory in its own stream's
    order: it is back while another stream's work (a device-side sleep of about
    half a second, here) is still running."""
    import torch

    from kapsel_old_b200 import nearcontact as nc

    rng = np.random.Generator(np.random.PCG64(8))
    x, w = rng.normal(size=(4096, 16)).astype(np.float32), np.ones(16, np.float32)
    net = nc.NearContactNet(nc.init_params(3))
    other, done = torch.cuda.Stream(), torch.cuda.Event()
    net.gradient(x[:64], x[:64], w)
    net.forward(x[:64])
    with torch.cuda.stream(other):
        torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        torch.cuda._sleep(10 ** 9)
        done.record()
    net.gradient(x[:2048], x[:2048], w)
    net.forward(x)
    still_running = not done.query()
    torch.cuda.synchronize()
    assert still_running
