"""The coarsest level's CG over the sizes at which its form changes: one warp,
several warps, two and four cells per thread, cells in memory, and levels too
large for the shared-memory tail (with all and with a few of their arrays in
shared memory).  In the reference solver mode one V-cycle on a noise scene
equals the oracle's bit for bit.  (In the relative modes the oracle sums in
FP32: a CG that its iteration cap cuts short differs by up to 3e-4.)"""
import numpy as np
import pytest

import apic_gb300 as A
from parity_helpers import eq, fluid_padded

pytestmark = pytest.mark.gpu


# grid sides; the coarsest level's cells
SIZES = [(40, 40, 25), (88, 88, 121), (248, 120, 465), (256, 248, 1984), (264, 264, 1089), (488, 488, 3721),
         (146, 146, 5329), (250, 150, 9375), (302, 302, 22801), (442, 442, 48841)]


def scene_of(w, h):
    return A.generate_scene(A.scene_params(A.SCENE_NOISE, w, h, cell_size=1 / w, sub=2, seed=2, noise_period=1 / 6,
                                           noise_threshold=0.3, vel_sigma=0.5))


@pytest.mark.parametrize("w,h,cells", SIZES)
def test_vcycle_coarsest_equals_oracle(gpu_lib, oracle_mod, w, h, cells):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    props = A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)
    g, o = A.Apic(w, h, 1 / w, props), oracle_mod.OracleSim(w, h, 1 / w, props)
    for sim in (g, o):
        sim.set_particles(*scene_of(w, h))
        for stage in ("p2g", "forces", "build", "mg", "vcycle"):
            sim.run_stage(stage, 1 / 1000)
    bits = g.read_field(A.mg_field("fluid_bits", g.info().mg_levels - 1))
    fluid = int(np.unpackbits(bits.view(np.uint8)).sum())
    assert 0.2 * cells < fluid <= cells
    fl = fluid_padded(o)
    eq(g.read_field("error")[fl], o.read_field("error")[fl], "vcycle z")
