"""The SpMV's form for rows of whole vectors (four cells a lane) and the one for
a cell a lane, on both sides of the rule that picks one: grids above 256^2 cells
whose widths are and are not multiples of four, whose last mask word is cut, thin
and wide.  In the reference solver mode (its sums have their own order) the
solve equals the oracle's bit for bit."""
import pytest

import apic_gb300 as A
from parity_helpers import eq, fluid_padded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(256, 256), (256, 258), (260, 254), (262, 258), (36, 2050), (2052, 34), (300, 226)])
def test_solve_equals_oracle(gpu_lib, oracle_mod, w, h):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    props = A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)
    parts = A.generate_scene(A.scene_params(A.SCENE_NOISE, w, h, cell_size=1 / w, sub=2, seed=5, noise_period=1 / 9,
                                            noise_threshold=0.5, vel_sigma=0.5))
    g, o = A.Apic(w, h, 1 / w, props), oracle_mod.OracleSim(w, h, 1 / w, props)
    for sim in (g, o):
        sim.set_particles(*parts)
        for stage in ("p2g", "forces", "build", "mg", "pcg"):
            sim.run_stage(stage, 1 / 1000)
    fl = fluid_padded(o)
    assert g.stats().pcg_iterations == o.stats().pcg_iterations > 0
    eq(g.read_field("pressure")[fl - w], o.read_field("pressure")[fl - w], "pressure")
    eq(g.read_field("residual")[fl], o.read_field("residual")[fl], "residual")
