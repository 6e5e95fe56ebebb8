"""Particle sets of changing counts in one handle, across the counts at which the
sorts change their tile size (fewer particles can take more tiles): the buffers
of the largest set serve every smaller one, and both sorts and P2G do what they do
in a fresh handle."""
import numpy as np
import pytest

import apic_gb300 as A
from parity_helpers import eq

pytestmark = pytest.mark.gpu
SIDE = 256


def sorted_and_transferred(g, n):
    rng = np.random.default_rng(n)
    g.set_particles(*(rng.uniform(0.05, 0.95, n).astype(np.float32) for _ in range(2)),
                    *(rng.normal(0, 0.3, n).astype(np.float32) for _ in range(2)))
    for stage in ("sort", "p2g"):
        g.run_stage(stage, 1 / 500)
    return {f: g.read_field(f) for f in A.PARTICLE_FIELDS + ["sort_keys", "sort_vals", "u", "v", "density"]}


@pytest.mark.parametrize("counts", [(262145, 262144, 65537, 65536, 8, 262145), (65537, 65536, 1, 65536, 65537),
                                    (65536, 262144, 1, 262144)])
def test_counts(gpu_lib, counts):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    props = A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)
    g = A.Apic(SIDE, SIDE, 1 / SIDE, props)
    g.set_particles([], [])
    for n in counts:
        got, want = sorted_and_transferred(g, n), sorted_and_transferred(A.Apic(SIDE, SIDE, 1 / SIDE, props), n)
        for f in want:
            eq(got[f], want[f], f"{n}: {f}")
