"""apic_restore rebuilds the open-face masks from the snapshot's obstacles also
where a caller wrote the mask fields by hand: the handle then goes on as a fresh
one that loads the same snapshot."""
import numpy as np
import pytest

import apic_gb300 as A
from parity_helpers import eq

pytestmark = pytest.mark.gpu
SIDE = 64


def make():
    g = A.Apic(SIDE, SIDE, 1 / SIDE, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    g.set_particles(*A.generate_scene(A.scene_params(A.SCENE_DAM_BREAK, SIDE, cell_size=1 / SIDE, sub=2, seed=3,
                                                     fluid_x=0.4, fluid_y=0.6)))
    return g


@pytest.mark.parametrize("field", ["u_open_bits", "v_open_bits"])
def test_restore_after_written_mask(gpu_lib, field):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    g, fresh = make(), make()
    g.update(A.DebugOptions(), 1 / 120)
    blob = g.snapshot()
    for _ in range(2):  # (the second time the handle has restored before)
        g.write_field(field, np.zeros_like(g.read_field(field)))
        g.restore(blob)
        eq(g.read_field(field), fresh.read_field(field), field)
    fresh.restore(blob)
    for sim in (g, fresh):
        sim.update(A.DebugOptions(), 1 / 60)
    for f in A.PARTICLE_FIELDS + ["u", "v"]:
        eq(g.read_field(f), fresh.read_field(f), f)
