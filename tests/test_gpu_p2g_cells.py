"""Cell-order P2G: particles whose stencils lie inside the grids take a form of
their own (a select per position), the others (beside the walls, outside the
grid, not finite) the general one, and a power-of-two cell size is divided by
with its reciprocal.  Against FP64 sums of the same terms, formed by the
reference's index and weight arithmetic: FP32 sums of k terms differ by at
most k * 2^-24 of the sum of their magnitudes, and each term carries about 16
roundings."""
import numpy as np
import pytest

import apic_gb300 as A

pytestmark = pytest.mark.gpu


def sums(px, py, w, h, dx, ox, oy, sw, sh, value):
    """Weight, momentum and magnitude sums of a staggered grid, and the terms per node."""
    f = np.float32
    gx, gy = (px / f(dx)).astype(np.float64) - ox, (py / f(dx)).astype(np.float64) - oy
    bx, by = np.floor(gx), np.floor(gy)
    tx, ty = gx - bx, gy - by
    wt = 0.75 ** 3 * 2.1875
    out = np.zeros((4, sh * sw))
    for j, wy in ((0, 1 - ty), (1, ty)):
        for i, wx in ((0, 1 - tx), (1, tx)):
            node = np.clip(by + j, 0, sh - 1).astype(int) * sw + np.clip(bx + i, 0, sw - 1).astype(int)
            wgt = wx * wy * wt
            for k, q in enumerate((wgt, wgt * value, np.abs(wgt * value), np.ones_like(wgt))):
                np.add.at(out[k], node, q)
    return out


@pytest.mark.parametrize("w,h,dx", [(64, 48, 1 / 64), (64, 48, 0.075), (34, 10, 1.0), (128, 32, 1 / 128), (40, 40, 0.3)])
def test_cell_order_sums(gpu_lib, w, h, dx):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(w)
    n = 5 * w * h
    px = (rng.uniform(-1, w + 1, n) * dx).astype(np.float32)  # some outside, some in the wall cells
    py = (rng.uniform(-1, h + 1, n) * dx).astype(np.float32)
    edge = rng.integers(0, n, n // 8)
    px[edge] = (np.round(px[edge] / dx * 2) / 2 * dx).astype(np.float32)  # on cell edges and centres
    vx, vy = rng.standard_normal((2, n)).astype(np.float32)
    g = A.Apic(w, h, dx, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    g.set_particles(px, py, vx, vy)
    g.set_option(A.OPT_P2G_ORDER, 2)
    g.run_stage("p2g", 1 / 1000)
    eps = 2.0 ** -24
    for name, ox, oy, sw, sh, val in (("u", 0.0, 0.5, w + 1, h, vx), ("v", 0.5, 0.0, w, h + 1, vy)):
        wgt, mom, mag, k = sums(px, py, w, h, dx, ox, oy, sw, sh, val)
        got = g.read_field(name).astype(np.float64)
        ok = wgt > 1e-3  # (a face that only grazing weights reach amplifies their rounding)
        want = mom[ok] / wgt[ok]
        bound = (2 * k[ok] + 40) * eps * (mag[ok] / wgt[ok]) + 64 * eps * max(w, h) * mag[ok] / wgt[ok]
        assert np.all(np.abs(got[ok] - want) <= bound), name
        assert np.all(got[wgt == 0] == 0)
    wgt, _, _, k = sums(px, py, w, h, dx, 0.5, 0.5, w, h, np.ones_like(px))
    got = g.read_field("density").astype(np.float64)
    assert np.all(np.abs(got - wgt) <= (2 * k + 40) * eps * wgt + 64 * eps * max(w, h) * np.maximum(k, 1))
