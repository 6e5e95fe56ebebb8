"""Views of few particles in a large frame: a tile without a quad costs its
pixels' background and nothing else, so a frame without particles takes less than
half of one whose particles touch every other tile."""
import time

import numpy as np
import pytest

import apic_gb300 as A

pytestmark = pytest.mark.gpu


def test_empty_tiles(gpu_lib, oracle_mod):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(1)
    p = A.render_params(3840, 2160, scale=2160.0, background=(10, 200, 30))
    best = {}
    for n in (0, 20000):
        g = A.Apic(64, 64, 1 / 64, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
        px, py = (rng.uniform(0, s, n).astype(np.float32) for s in (3840 / 2160, 1))
        g.set_particles(px, py)
        want, _ = oracle_mod.render(px, py, np.zeros_like(px), np.zeros_like(px), p)
        assert np.array_equal(g.render(p)[0], want)
        best[n] = np.inf
        for _ in range(20):
            t0 = time.perf_counter()
            g.render(p, read=False)
            best[n] = min(best[n], time.perf_counter() - t0)
    assert best[0] < 0.5 * best[20000], best
