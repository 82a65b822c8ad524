"""Writes le_steps.npz: six FP64 Lees-Edwards steps across the grid reset on two
boxes, one sphere's profile reaching across the sheared boundary.

    python tests/golden/make_le_steps.py [out.npz]

The committed file was recorded with the step's former kernels (separate
launches for the cross product, the force and its interpolation), which
tests/test_gpu_obl.py had compared with the reference's own run.  A present
build writes the same file to roundoff; test_lees_edwards_recorded_steps holds
it to that.  Needs a GPU."""
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(os.path.dirname(HERE)))

# name, log2 of the grid, spheres
BOXES = [("z64", (4, 5, 6), 3), ("z128", (5, 4, 7), 4)]


def config(np_xyz, xs):
    return {"eq": "Shear_Navier_Stokes_Lees_Edwards", "np_xyz": np_xyz, "a": 3.0, "a_xi": 2.0, "kbt": 1e-3,
            "dt": 0.01, "shear_rate": 0.1, "particles": [{"x": tuple(map(float, x))} for x in xs]}


def record():
    import kapsel_old_b200 as kg
    from kapsel_old_b200 import workload

    out = {}
    for name, np_xyz, n in BOXES:
        xs = workload.place_spheres(n, [1 << p for p in np_xyz], 4.0, 0.5, 9)
        xs[0, 1] = 0.3
        s = kg.Simulation(config(np_xyz, xs), precision=kg.FP64)
        s.set_oblique(0.9975, 0.1)
        s.step(6)
        p, o = s.particles(), s.oblique()
        out[name + "_x0"] = xs
        for k in ("x", "v", "omega", "q"):
            out[f"{name}_{k}"] = p[k]
        out[name + "_zeta"] = s.zeta()
        out[name + "_obl"] = np.array([o["degree_oblique"], o["shear_rate_eff"], o["strain"]])
    return out


if __name__ == "__main__":
    np.savez_compressed(sys.argv[1] if len(sys.argv) > 1 else os.path.join(HERE, "le_steps.npz"), **record())
