"""A write that apic_write_field refuses changes nothing: the residual, which lies
in one of two buffers after a solve, still reads as before."""
import ctypes

import numpy as np
import pytest

import apic_gb300 as A
from parity_helpers import eq

pytestmark = pytest.mark.gpu
SIDE = 64


@pytest.mark.parametrize("iterations", [1, 2])
def test_refused_residual_write(gpu_lib, iterations):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    # the reference mode leaves the residual where its last iteration wrote it;
    # the exit (max |r| < solve_error) is set so that it takes the wanted count
    for solve_error in np.geomspace(1e-5, 1e3, 60):
        g = A.Apic(SIDE, SIDE, 1 / SIDE, A.WorldProperties(-9.81, 0.1, 5.0, float(solve_error)))
        g.set_particles(*A.generate_scene(A.scene_params(A.SCENE_NOISE, SIDE, cell_size=1 / SIDE, sub=2, seed=5,
                                                         noise_period=1 / 9, noise_threshold=0.5, vel_sigma=0.5)))
        for stage in ("p2g", "forces", "build", "mg", "pcg"):
            g.run_stage(stage, 1 / 1000)
        if g.stats().pcg_iterations == iterations:
            break
        g.close()
    assert g.stats().pcg_iterations == iterations
    before = g.read_field("residual")
    data = np.zeros(before.size + 1, np.float32)
    rc = gpu_lib.apic_write_field(g._h, A.FIELDS["residual"], data.ctypes.data_as(ctypes.c_void_p), data.nbytes)
    assert rc == 1 and "size mismatch" in gpu_lib.apic_last_error().decode()
    assert gpu_lib.apic_write_field(g._h, A.FIELDS["residual"], None, before.nbytes) == 1
    eq(g.read_field("residual"), before, "residual")
    g.write_field("residual", before + np.float32(1))
    eq(g.read_field("residual"), before + np.float32(1), "residual written")
