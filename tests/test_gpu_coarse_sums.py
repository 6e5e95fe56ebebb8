"""The coarsest level's CG in the relative modes sums its dot products as exactly
as FP64 does: where a sum lies nearer to a rounding boundary than a double-float
resolves, and where it leaves the FP32 range (the step is then zero, as with an
infinite FP64 sum).  Two-level grids whose base level passes the residual on
unchanged, at the sizes of the CG's forms; the expected error is the CG's in
numpy with FP64 sums."""
import numpy as np
import pytest

import apic_gb300 as A
import vcycle_numpy as V
from parity_helpers import eq

pytestmark = pytest.mark.gpu
F = np.float32


def total64(q):
    with np.errstate(over="ignore"):
        return F(q.astype(np.float64).sum())


@pytest.mark.parametrize("side", [18, 74, 130, 162, 206])  # 81 .. 10609 coarsest cells
@pytest.mark.parametrize("case", ["boundary", "overflow"])
def test_sums_as_fp64(gpu_lib, side, case):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    half = side // 2
    if case == "boundary":  # r.r = 2^-18 (1 + 2^-24 + 2^-50)
        r, d = [2.0 ** -9, 2.0 ** -21, 2.0 ** -34], [4.0, 8.0, 4.0]
    else:                   # r.r = 2e38, r.Ar = 6e38
        r, d = [1e19, 1e19], [3.0, 3.0]
    cells = np.random.default_rng(side).choice((half - 2) ** 2, len(r), replace=False)
    cx, cy = cells % (half - 2) + 1, cells // (half - 2) + 1
    g = A.Apic(side, side, 1 / side, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    g.set_solver(A.SOLVER_REL_FP32, 1e-6, 100)
    bits = np.zeros(g.read_field("fluid_bits").size * 64, np.uint8)
    inside = np.zeros((side, side), np.uint8)
    inside[1:-1, 1:-1] = 1
    bits[:side * side] = inside.ravel()
    g.write_field("fluid_bits", np.packbits(bits, bitorder="little").view(np.uint64))
    for name in ("diag", "inv_diag", "plus_x", "plus_y"):
        g.write_field(name, np.zeros(side * side + 2 * side, F))
    res = np.zeros(side * side + 2 * side, F)
    fine = 2 * cy * side + 2 * cx + side
    res[fine] = r
    g.write_field("residual", res)
    assert g.info().mg_levels == 1
    bits = np.zeros(g.read_field(A.mg_field("fluid_bits", 0)).size * 64, np.uint8)
    bits[:half * half] = 1
    words = np.packbits(bits, bitorder="little").view(np.uint64)
    g.write_field(A.mg_field("fluid_bits", 0), words)
    zero = np.zeros(half * half + 2 * half, F)
    diag = zero.copy()
    diag[half:-half] = 1
    diag[cy * half + cx + half] = d
    for name, data in (("diag", diag), ("inv_diag", zero), ("plus_x", zero), ("plus_y", zero)):
        g.write_field(A.mg_field(name, 0), data)
    coarse = V.Level(half, half, words, diag, zero, zero, zero)
    coarse.res[cy * half + cx + half] = r
    with np.errstate(over="ignore"):
        coarse.solve(total64)
    g.run_stage("vcycle", 1 / 1000)
    eq(g.read_field("error")[fine], coarse.err[cy * half + cx + half], "coarse error")
