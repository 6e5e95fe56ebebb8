"""The raster's windows: more quads over a warp's 8 x 4 pixels than one window
holds (512), exactly as many, around the groups of 128 that are loaded at once,
quads of every size, and frames that end inside a tile.  Byte for byte the
oracle's draw loop."""
import numpy as np
import pytest

import apic_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,radius,spread", [(1, 0.4, 0.0), (127, 3.0, 2.0), (128, 3.0, 2.0), (129, 7.0, 4.0),
                                             (512, 3.0, 0.5), (513, 3.0, 0.5), (2600, 1.3, 6.0), (5000, 7.0, 3.0)])
@pytest.mark.parametrize("size", [(64, 48), (61, 35)])
def test_dense_pixels(gpu_lib, oracle_mod, n, radius, spread, size):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    w, h = size
    rng = np.random.default_rng(n)
    # a cluster around a corner of four tiles, some single particles elsewhere
    px = np.concatenate([(16 + spread * rng.standard_normal(n)), rng.uniform(-60, w + 60, 40)]) / w
    py = np.concatenate([(h - 16 + spread * rng.standard_normal(n)), rng.uniform(-60, h + 60, 40)]) / w
    px, py = px.astype(np.float32), py.astype(np.float32)
    vx, vy = (8 * rng.standard_normal((2, n + 40))).astype(np.float32)
    g = A.Apic(64, 64, 1 / 64, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    g.set_particles(px, py, vx, vy)
    p = A.render_params(w, h, scale=float(w), draw_radius=radius, background=(10, 200, 30))
    frame, st = g.render(p)
    want, sw = oracle_mod.render(px, py, vx, vy, p)
    assert np.array_equal(frame, want)
    assert (st.valid, st.nan, st.out_of_bounds) == (sw.valid, sw.nan, sw.out_of_bounds)
