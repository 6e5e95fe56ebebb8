"""The V-cycle's tile kernels (32 x 16 cells and a halo of two) at grids that
cut tiles in every way: narrower and lower than a tile, one column or row
beyond a tile, rows that are no multiple of a mask word, tiles without fluid.
In the reference solver mode the V-cycle (no update), then the whole solve (the
update in the down kernel, the residual alternating between its buffers) equal
the oracle's bit for bit."""
import pytest

import apic_gb300 as A
from parity_helpers import eq, fluid_padded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,threshold", [(14, 10, 0.0), (32, 16, 0.0), (34, 18, 0.0), (66, 34, 0.3), (64, 98, 0.5),
                                           (100, 44, 0.5), (200, 136, 0.6), (256, 64, 0.4)])
def test_tiles_equal_oracle(gpu_lib, oracle_mod, w, h, threshold):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    props = A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)
    parts = A.generate_scene(A.scene_params(A.SCENE_NOISE, w, h, cell_size=1 / w, sub=2, seed=5, noise_period=1 / 5,
                                            noise_threshold=threshold, vel_sigma=0.5))
    g, o = A.Apic(w, h, 1 / w, props), oracle_mod.OracleSim(w, h, 1 / w, props)
    for sim in (g, o):
        sim.set_particles(*parts)
        for stage in ("p2g", "forces", "build", "mg", "vcycle"):
            sim.run_stage(stage, 1 / 1000)
    fl = fluid_padded(o)
    eq(g.read_field("fluid_list"), o.read_field("fluid_list"), "fluid list")
    eq(g.read_field("residual")[fl], o.read_field("residual")[fl], "right-hand side")
    eq(g.read_field("error")[fl], o.read_field("error")[fl], "vcycle z")
    for sim in (g, o):
        sim.run_stage("pcg", 1 / 1000)
    assert g.stats().pcg_iterations == o.stats().pcg_iterations > 0
    eq(g.read_field("pressure")[fl - w], o.read_field("pressure")[fl - w], "pressure")
    eq(g.read_field("residual")[fl], o.read_field("residual")[fl], "residual")
