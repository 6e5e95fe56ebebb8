"""A solve whose r.z becomes zero while the residual does not ends: the kernel
after the update takes the loop decision also where the update itself ended
the solve.  A crowded cell walled in on all sides has a volume error that no
pressure can correct (its row of the matrix is zero) beside open fluid whose
residual shrinks until its squares underflow; whole updates return, in each
form of the kernel after the update, with a result or with the error that
non-finite velocities earn."""
import numpy as np
import pytest

import apic_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,dsm", [(32, 1), (64, 1), (128, 1), (128, 0), (30, 1)])
@pytest.mark.parametrize("mode", [A.SOLVER_REL_FP32, A.SOLVER_REL_MIXED])
def test_enclosed_dense_cell(gpu_lib, side, dsm, mode):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(side)
    g = A.Apic(side, side, 1 / side, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    g.set_option(A.OPT_DSM_VCYCLE, dsm)
    g.set_solver(mode, 1e-6, 500)
    bits = g.read_field("obstacle_bits")
    flat = np.unpackbits(bits.view(np.uint8), bitorder="little")
    for y in (9, 10, 11):
        for x in (9, 10, 11):
            if (x, y) != (10, 10):
                flat[y * side + x] = 1
    g.write_field("obstacle_bits", np.packbits(flat, bitorder="little").view(bits.dtype))
    x = np.concatenate([10 + rng.uniform(0.3, 0.7, 60), rng.uniform(15, 19, 40)]).astype(np.float32) / np.float32(side)
    y = np.concatenate([10 + rng.uniform(0.3, 0.7, 60), rng.uniform(15, 19, 40)]).astype(np.float32) / np.float32(side)
    g.set_particles(x, y, np.zeros(100, np.float32), np.zeros(100, np.float32))
    for _ in range(3):
        try:
            g.update(A.DebugOptions(), 1 / 500)
        except A.ApicError as e:
            assert e.code == 5  # APIC_ERR_NONFINITE
            break
        assert g.stats().substeps >= 1
