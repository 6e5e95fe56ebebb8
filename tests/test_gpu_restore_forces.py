"""apic_restore replaces the forces a handle has gathered by the snapshot's: a force
added after the restore acts alone, as in a fresh handle."""
import pytest

import apic_gb300 as A
from parity_helpers import eq

pytestmark = pytest.mark.gpu
SIDE = 64


@pytest.mark.parametrize("strength", [5.0, -5.0])  # post (repelling) and external
@pytest.mark.parametrize("saved", [False, True])
def test_pending_forces(gpu_lib, strength, saved):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    sims = [A.Apic(SIDE, SIDE, 1 / SIDE, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)) for _ in range(2)]
    g, fresh = sims
    if saved:
        g.add_radial_force(0.3, 0.2, 0.1, strength)
    blob = g.snapshot()
    g.add_radial_force(0.5, 0.3, 0.2, strength)
    for sim in sims:
        sim.restore(blob)
        sim.add_radial_force(0.4, 0.2, 0.1, strength)
    for f in ("ext_force_u", "ext_force_v", "post_force_u", "post_force_v"):
        eq(g.read_field(f), fresh.read_field(f), f)
    for sim in sims:
        sim.update(A.DebugOptions(), 1 / 60)
    for f in A.PARTICLE_FIELDS:
        eq(g.read_field(f), fresh.read_field(f), f)
