"""bench.py's byte counts against what the present kernels read and write.

The scatter forms the rigidity force: it reads u* and stores the force at the
points under a sphere's profile, and the force's forward z pass reads those three
fields and clears them there."""
import math
import os
import re

import pytest

import bench
from kapsel_old_b200 import workload

CFG = workload.mixed_128_256()
N = 128 ** 3
I1, I2, ZETA = 128 * 85 * 43, 128 * 128 * 43, 2 * 85 * 85 * 43  # complex values
PART = 256 * 26 * 8


def test_points_under_a_profile():
    # the mean number of grid points within a + xi/2 of a centre, below the
    # 1256 offsets that can be there for some centre and the 1935 of the list
    assert bench.support_points(CFG) == round(4.0 / 3.0 * math.pi * 6.0 ** 3) == 905


@pytest.mark.parametrize("R", [4, 8])
def test_bytes_of_the_force_and_particle_kernels(R):
    kb, pts = bench.kernel_bytes(CFG, R), 256 * 905
    assert kb["k_particles_hydro_velocity"] == 3 * pts * R + 2 * PART
    assert kb["k_particles_scatter"] == (3 + 3) * pts * R + PART
    assert kb["k_z_force"] == 3 * N * R + 3 * pts * R + 3 * I2 * 2 * R
    assert kb["k_zyw_r2c"] == 3 * N * R + 3 * pts * R + 3 * I1 * 2 * R


@pytest.mark.parametrize("R", [4, 8])
def test_step_bytes_are_those_of_the_steady_launches(R):
    C, pts = 2 * R, 256 * 905
    transforms = (3 * (I1 + I2) + 8 * I2 + 5 * (I2 + I1)      # y, products, y
                  + (8 * I1 + 2 * ZETA) + 3 * I1 + 3 * I1     # x, into and out of the planes
                  + (6 * I1 + 2 * ZETA)) * C                  # x, with the next step's u_k
    fields = (3 * N + 3 * N) * R                              # u* written, the force read
    points = (3 + 6 + 3) * pts * R                            # gather; scatter; clear
    assert bench.step_bytes(CFG, R) == transforms + fields + points + (2 + 2 + 1) * PART


def test_every_slot_of_a_step_has_its_bytes():
    src = open(os.path.join(os.path.dirname(__file__), "..", "kapsel_old_b200", "csrc", "kapsel_gpu.cu")).read()
    names = re.findall(r'"(k_\w+(?:<\w+>)?)"', re.search(r"kKernelNames\[\w*\]\s*=\s*\{(.*?)\};", src, re.S).group(1))
    assert len(names) == 13
    kb = bench.kernel_bytes(CFG, 4)
    assert all(n in kb for n in bench.slot_labels(names) + ["k_yzw_c2r", "k_zyw_r2c"])
