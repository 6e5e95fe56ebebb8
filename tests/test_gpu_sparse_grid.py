"""P2G of a few particles on a large grid: what each cell costs (its run emptied,
its faces written) is spread over the whole chip, so a thousand particles do not
take longer than a million."""
import time

import numpy as np
import pytest

import apic_gb300 as A

pytestmark = pytest.mark.gpu
SIDE = 4096


@pytest.mark.parametrize("mode", [A.SOLVER_REFERENCE, A.SOLVER_REL_MIXED])
def test_few_particles_cost_no_more(gpu_lib, mode):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    g = A.Apic(SIDE, SIDE, 1 / SIDE, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    g.set_solver(mode, 1e-6, 500)
    rng = np.random.default_rng(1)
    best = {}
    for n in (1000, 1000000):
        g.set_particles(*(rng.uniform(0.1, 0.9, n).astype(np.float32) for _ in range(2)))
        best[n] = np.inf
        for _ in range(12):
            t0 = time.perf_counter()
            g.run_stage("p2g", 1 / 1000)
            best[n] = min(best[n], time.perf_counter() - t0)
    assert best[1000] <= best[1000000], best
