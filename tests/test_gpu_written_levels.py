"""Coarse levels that a caller wrote (APIC_F_MG_*): the V-cycle takes what the
written mask says, also where fluid cells' couplings point at cells that the mask
leaves out and where a cell is left out whose finer cells are fluid.  The bits
are those of the reference's V-cycle in numpy, for the levels held by one CTA,
by a cluster, and by the stand-alone coarse solve."""
import numpy as np
import pytest

import apic_gb300 as A
import vcycle_numpy as V
from parity_helpers import eq, fluid_padded

pytestmark = pytest.mark.gpu
NAMES = ("diag", "inv_diag", "plus_x", "plus_y")


def sides(w, h, level):
    return w >> (level + 1), h >> (level + 1)


def make(w, h):
    g = A.Apic(w, h, 1 / w, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    g.set_particles(*A.generate_scene(A.scene_params(A.SCENE_NOISE, w, h, cell_size=1 / w, sub=2, seed=2,
                                                     noise_period=1 / 6, noise_threshold=0.3, vel_sigma=0.5)))
    for stage in ("p2g", "forces", "build", "mg"):
        g.run_stage(stage, 1 / 1000)
    return g


def read_levels(g, w, h):
    """[(bits, {coefficient})] of the coarse levels."""
    return [(g.read_field(A.mg_field("fluid_bits", l)), {n: g.read_field(A.mg_field(n, l)) for n in NAMES})
            for l in range(g.info().mg_levels)]


def expected(g, w, h, written):
    base = V.Level(w, h, g.read_field("fluid_bits"), *(g.read_field(n) for n in NAMES))
    levels = [base] + [V.Level(*sides(w, h, l), bits, *(co[n] for n in NAMES)) for l, (bits, co) in enumerate(written)]
    return V.vcycle(levels, g.read_field("residual"))


GRIDS = [(64, 64), (128, 128), (250, 150)]


@pytest.mark.parametrize("w,h", GRIDS)
def test_levels_as_built(gpu_lib, w, h):
    """(the numpy V-cycle on what the setup built)"""
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    g = make(w, h)
    want = expected(g, w, h, read_levels(g, w, h))
    g.run_stage("vcycle", 1 / 1000)
    fl = fluid_padded(g)
    eq(g.read_field("error")[fl], want[fl], "z")


@pytest.mark.parametrize("w,h", GRIDS)
def test_written_masks(gpu_lib, w, h):
    """Masks with cells taken out, the coefficients of the others as they were."""
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    g, rng = make(w, h), np.random.default_rng(1)
    written = read_levels(g, w, h)
    for l, (bits, _) in enumerate(written):
        cells = sides(w, h, l)[0] * sides(w, h, l)[1]
        on = np.unpackbits(bits.view(np.uint8), bitorder="little")
        on[:cells] &= rng.random(cells) > 0.2
        written[l] = (np.packbits(on, bitorder="little").view(np.uint64), written[l][1])
        g.write_field(A.mg_field("fluid_bits", l), written[l][0])
    want = expected(g, w, h, written)
    g.run_stage("vcycle", 1 / 1000)
    fl = fluid_padded(g)
    eq(g.read_field("error")[fl], want[fl], "z")


@pytest.mark.parametrize("w,h", GRIDS)
def test_coefficients_before_masks(gpu_lib, w, h):
    """The order of the writes does not matter, and what was written stays, also
    outside the mask and after a V-cycle."""
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    g, rng = make(w, h), np.random.default_rng(2)
    built = read_levels(g, w, h)
    for l, (bits, _) in enumerate(built):  # a first mask without any cell
        g.write_field(A.mg_field("fluid_bits", l), np.zeros_like(bits))
    for l, (bits, co) in enumerate(built):
        lw, lh = sides(w, h, l)
        out = ~V.Level(lw, lh, bits, *(co[n] for n in NAMES)).on
        for n in NAMES:  # values outside the mask that nothing may read
            co[n] = np.where(out, rng.uniform(1, 2, co[n].size), co[n]).astype(np.float32)
            g.write_field(A.mg_field(n, l), co[n])
        g.write_field(A.mg_field("fluid_bits", l), bits)
    want = expected(g, w, h, built)
    g.run_stage("vcycle", 1 / 1000)
    fl = fluid_padded(g)
    eq(g.read_field("error")[fl], want[fl], "z")
    for l, (bits, co) in enumerate(built):
        eq(g.read_field(A.mg_field("fluid_bits", l)), bits, f"level {l} mask")
        for n in NAMES:
            eq(g.read_field(A.mg_field(n, l)), co[n], f"level {l} {n}")
