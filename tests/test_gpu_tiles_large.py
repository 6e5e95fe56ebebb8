"""The tile kernels on a level of more than 2048 tiles read fluid cells only; a
smaller one's reads go ahead of the mask.  Both sides of the rule, with tiles
cut on every side, in the reference solver mode: V-cycle and solve equal the
oracle's bit for bit."""
import pytest

import apic_gb300 as A
from parity_helpers import eq, fluid_padded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1024, 1024), (1040, 1016)])
def test_both_forms_equal_oracle(gpu_lib, oracle_mod, w, h):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    props = A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)
    parts = A.generate_scene(A.scene_params(A.SCENE_NOISE, w, h, cell_size=1 / w, sub=2, seed=5, noise_period=1 / 9,
                                            noise_threshold=0.6, vel_sigma=0.5))
    g, o = A.Apic(w, h, 1 / w, props), oracle_mod.OracleSim(w, h, 1 / w, props)
    for sim in (g, o):
        sim.set_particles(*parts)
        for stage in ("p2g", "forces", "build", "mg", "vcycle"):
            sim.run_stage(stage, 1 / 1000)
    fl = fluid_padded(o)
    eq(g.read_field("error")[fl], o.read_field("error")[fl], "vcycle z")
    for sim in (g, o):
        sim.run_stage("pcg", 1 / 1000)
    assert g.stats().pcg_iterations == o.stats().pcg_iterations > 0
    eq(g.read_field("pressure")[fl - w], o.read_field("pressure")[fl - w], "pressure")
