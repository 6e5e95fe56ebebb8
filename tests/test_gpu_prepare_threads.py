"""The server prepares scenes on several threads at once.  Scenes of different
sizes sort with different digit widths, hence different shared-memory sizes of
one kernel: recording one scene's graph must not disturb another's.  Every
burst finishes with the same positions."""
import numpy as np
import pytest

import apic_gb300 as A

pytestmark = pytest.mark.gpu


def test_bursts_of_uneven_scenes(gpu_lib):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    props = A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)
    scenes = [A.scene_params(A.SCENE_DAM_BREAK, n, cell_size=1 / n, seed=n, fluid_x=0.4, fluid_y=0.5)
              for n in (64, 72, 100, 128, 150, 90, 80, 136)]
    first = None
    for _ in range(40):
        server = A.Server(8 << 30, 64, keep_results=True)
        ids = [server.submit(s, props, 1, 1 / 240) for s in scenes]
        while server.step().completed or server.stats().completed + server.stats().failed < len(ids):
            pass
        assert server.stats().failed == 0
        got = [server.result_positions(i) for i in ids]
        server.close()
        first = first or got
        for a, b in zip(first, got):
            assert np.array_equal(a, b)
