"""The SpMV kernels of the relative solver modes (four cells a lane on rows of whole
vectors, a cell a lane elsewhere) on both sides of the rule that picks one: grids
above 256^2 cells whose widths are and are not multiples of four, whose last mask
word is cut, thin and wide.  After a few iterations the norm of the recursive
residual, which the SpMV makes, is that of b - A p in FP64, up to the rounding of
the iterations: each one rounds A s (five operations a cell), the residual and the
pressure once."""
import numpy as np
import pytest

import apic_gb300 as A
from parity_helpers import fluid_padded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(256, 256), (256, 258), (260, 254), (262, 258), (36, 2050), (2052, 34), (300, 226)])
@pytest.mark.parametrize("iterations", [1, 2, 4])
def test_recursive_residual(gpu_lib, w, h, iterations):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    g = A.Apic(w, h, 1 / w, A.WorldProperties(-9.81, 0.1, 1e9, 1e-5))
    g.set_particles(*A.generate_scene(A.scene_params(A.SCENE_NOISE, w, h, cell_size=1 / w, sub=2, seed=5,
                                                     noise_period=1 / 9, noise_threshold=0.5, vel_sigma=0.5)))
    g.set_solver(A.SOLVER_REL_FP32, 1e-30, iterations)
    g.update(A.DebugOptions(), 1 / 1000)
    st = g.stats()
    assert st.substeps == 1 and st.pcg_iterations == iterations
    # |A| |p| of the final pressure, and b = r + A p
    fl = fluid_padded(g)
    on = np.zeros(w * h + 2 * w, bool)
    on[fl] = True
    p = np.zeros(on.size)
    p[fl] = g.read_field("pressure")[fl - w]
    d, px, py, r = (g.read_field(n).astype(np.float64) for n in ("diag", "plus_x", "plus_y", "residual"))
    ap, mag = d[fl] * p[fl], np.abs(d[fl] * p[fl])
    for n, k in ((fl + 1, px[fl]), (fl - 1, px[fl - 1]), (fl + w, py[fl]), (fl - w, py[fl - w])):
        t = np.where(on[n], k * p[n], 0.0)
        ap, mag = ap + t, mag + np.abs(t)
    b = np.linalg.norm(r[fl] + ap)
    rounding = 2.0 ** -24 * iterations * (7 * np.linalg.norm(mag) + 2 * b) / b
    assert abs(st.residual_rel - st.true_residual_rel) <= rounding
    assert st.true_residual_rel < 0.9
