"""The pressure system's setup on both sides of its rules: the base list by one
CTA or by blocks, tile lists in the coarse levels' kernel or by their own, the
three smoothing passes on tiles of two sizes, grids that cut tiles and mask words
in every way, an empty grid, obstacles.  Lists, smoothed density, system and
one V-cycle equal the oracle's bit for bit."""
import numpy as np
import pytest

import apic_gb300 as A
from parity_helpers import eq, fluid_padded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,threshold", [(6, 6, 0.0), (14, 10, 0.0), (34, 18, 0.4), (66, 130, 0.5), (256, 256, 0.6),
                                           (512, 512, 0.7), (514, 512, 0.7), (64, 48, 2.0)])
def test_setup_equals_oracle(gpu_lib, oracle_mod, w, h, threshold):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    props = A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)
    x, y, vx, vy = A.generate_scene(A.scene_params(A.SCENE_NOISE, w, h, cell_size=1 / w, sub=2, seed=4, noise_period=1 / 7,
                                                   noise_threshold=min(threshold, 0.9), vel_sigma=0.5))
    if threshold > 1 or len(x) == 0:  # one particle
        x, y, vx, vy = (np.full(1, v, np.float32) for v in (2.5 / w, 2.5 / w, 0.1, 0.2))
    g, o = A.Apic(w, h, 1 / w, props), oracle_mod.OracleSim(w, h, 1 / w, props)
    bits = o.read_field("obstacle_bits")
    flat = np.unpackbits(bits.view(np.uint8), bitorder="little")
    flat[(h // 2) * w + w // 2] = 1  # a solid cell inside
    bits = np.packbits(flat, bitorder="little").view(bits.dtype)
    for sim in (g, o):
        sim.write_field("obstacle_bits", bits)
        sim.set_particles(x, y, vx, vy)
        for stage in ("p2g", "forces", "build"):
            sim.run_stage(stage, 1 / 1000)
    eq(g.read_field("fluid_bits"), o.read_field("fluid_bits"), "fluid bits")
    eq(g.read_field("fluid_list"), o.read_field("fluid_list"), "fluid list")
    eq(g.read_field("smoothed_density"), o.read_field("smoothed_density"), "smoothed density")
    fl = fluid_padded(o)
    for f in ("residual", "diag", "inv_diag", "plus_x", "plus_y"):
        eq(g.read_field(f)[fl], o.read_field(f)[fl], f)
    for sim in (g, o):
        for stage in ("mg", "vcycle"):
            sim.run_stage(stage, 1 / 1000)
    eq(g.read_field("error")[fl], o.read_field("error")[fl], "vcycle z")
