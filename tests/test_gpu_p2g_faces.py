"""Reference-order P2G: faces merge the runs of their four stencil bases from a
stage of limited size.  Grids that cut tiles in every way, densities that need
bands of rows or exceed the stage altogether, slots in random order, particles
beside the walls and outside the grid (the form that reads global memory): all
sums equal the oracle's bit for bit."""
import numpy as np
import pytest

import apic_gb300 as A
from parity_helpers import eq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,per_cell,spread", [
    (16, 8, 4, "inside"), (34, 10, 9, "inside"), (64, 48, 9, "all"), (130, 70, 3, "inside"), (40, 26, 20, "inside"),
    (30, 20, 45, "inside"), (32, 16, 2, "outside"), (48, 24, 6, "corner"), (18, 34, 1, "one cell")])
def test_reference_order_equals_oracle(gpu_lib, oracle_mod, w, h, per_cell, spread):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(w + h)
    n = per_cell * w * h + 5
    lo, hi = {"inside": (1.001, -1.001), "all": (0, 0), "outside": (-2, 2), "corner": (1.001, -1.001),
              "one cell": (1.001, -1.001)}[spread]
    x, y = rng.uniform(lo, w + hi, n), rng.uniform(lo, h + hi, n)
    if spread == "corner":  # half of the particles in a few cells: one band fits the stage, another does not
        x[::2], y[::2] = rng.uniform(4, 9, len(x[::2])), rng.uniform(8.5, 12, len(x[::2]))
    if spread == "one cell":
        x[:], y[:] = rng.uniform(7.2, 7.9, n), rng.uniform(5.2, 5.9, n)
    edge = rng.integers(0, n, n // 8)
    x[edge] = np.clip(np.round(x[edge] * 2) / 2, 1.5, w - 1.5)  # on cell edges and centres
    dx = 1 / w
    px, py = (x * dx).astype(np.float32), (y * dx).astype(np.float32)
    vx, vy = rng.standard_normal((2, n)).astype(np.float32)
    props = A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)
    g, o = A.Apic(w, h, dx, props), oracle_mod.OracleSim(w, h, dx, props)
    for sim in (g, o):
        sim.set_particles(px, py, vx, vy)
        sim.run_stage("p2g", 1 / 1000)
    for name in ("u", "v", "density"):
        eq(g.read_field(name), o.read_field(name), name)
