"""apic_restore and apic_set_particles into a handle that already holds as many
particles: the buffers and the recorded update graph stay in place.  What a
handle does after it must be what a fresh handle does that loads the same
state for the first time."""
import numpy as np
import pytest

import apic_gb300 as A
from parity_helpers import eq

pytestmark = pytest.mark.gpu
FIELDS = A.PARTICLE_FIELDS + ["u", "v", "pressure"]


def scene(n_cut, seed=3):
    p = A.generate_scene(A.scene_params(A.SCENE_DAM_BREAK, 64, cell_size=1 / 64, sub=2, seed=seed, fluid_x=0.4,
                                        fluid_y=0.6))
    return [a[:len(a) - n_cut] for a in p]


def make(parts, mode):
    g = A.Apic(64, 64, 1 / 64, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    g.set_particles(*parts)
    g.set_solver(mode, 1e-6, 500)
    return g


def run(g, k=3):
    for _ in range(k):
        g.update(A.DebugOptions(), 1 / 120)
    return {f: g.read_field(f) for f in FIELDS}


@pytest.mark.parametrize("mode", [A.SOLVER_REFERENCE, A.SOLVER_REL_MIXED])
@pytest.mark.parametrize("n_cut", [0, 3])
def test_restore_again(gpu_lib, mode, n_cut):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    g = make(scene(n_cut), mode)
    run(g, 2)
    g.add_radial_force(0.3, 0.2, 0.1, 5.0)
    blob = g.snapshot()
    first = run(g)
    fresh = make(scene(0, seed=4), mode)   # another state, another count when n_cut > 0
    run(fresh, 1)
    for sim in (g, fresh, g):
        if sim is g:
            bits = sim.read_field("obstacle_bits")
            sim.write_field("obstacle_bits", bits ^ np.uint64(1 << 40))  # the snapshot's world differs
        sim.restore(blob)
        assert sim.snapshot() == blob
        got = run(sim)
        for f in FIELDS:
            eq(got[f], first[f], f)


def test_set_particles_again(gpu_lib):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    for n_cut in (0, 5):
        g = make(scene(n_cut, seed=7), A.SOLVER_REL_MIXED)
        run(g, 3)
        g.set_particles(*scene(n_cut, seed=8))
        h = make(scene(n_cut, seed=8), A.SOLVER_REL_MIXED)
        for f in A.PARTICLE_FIELDS:
            eq(g.read_field(f), h.read_field(f), f)
