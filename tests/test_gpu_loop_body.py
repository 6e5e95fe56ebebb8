"""The PCG loop's graph body holds several iterations; those after the last one
do nothing.  Whole updates with solves that end at the iteration cap (odd and
even) or by the residual test equal, bit for bit, those of the profiling
mode, whose host loop launches one iteration at a time."""
import numpy as np
import pytest

import apic_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [32, 64, 136, 128])
@pytest.mark.parametrize("mode", [A.SOLVER_REL_FP32, A.SOLVER_REL_MIXED, A.SOLVER_REFERENCE])
@pytest.mark.parametrize("cap", [1, 2, 3, 4, 500])
def test_body_equals_single_iterations(gpu_lib, side, mode, cap):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    props = A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)
    parts = A.generate_scene(A.scene_params(A.SCENE_DAM_BREAK, side, cell_size=1 / side, seed=3, fluid_x=0.4, fluid_y=0.5))
    runs = []
    for profiling in (False, True):
        g = A.Apic(side, side, 1 / side, props)
        g.set_solver(mode, 1e-6, cap)
        g.set_particles(*parts)
        g.set_profiling(profiling)
        for _ in range(3):
            g.update(A.DebugOptions(), 1 / 240)
        st = g.stats()
        runs.append((st.substeps, st.pcg_iterations, st.pcg_iterations_total, st.refinement_steps, st.not_converged))
        runs.append([g.read_field(f) for f in ("pos_x", "pos_y", "vel_x", "vel_y")])
    assert runs[0] == runs[2]
    for a, b in zip(runs[1], runs[3]):
        assert np.array_equal(a, b)
