"""An empty particle set, given as arrays of no elements (their addresses are
not null), is accepted before and after a set with particles."""
import ctypes

import numpy as np
import pytest

import apic_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", [0, 5])
def test_empty_set(gpu_lib, before):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    g = A.Apic(32, 16, 1 / 32, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    if before:
        x = np.full(before, 0.3, np.float32)
        g.set_particles(x, x, x, x)
    some = np.zeros(1, np.float32)
    p = some.ctypes.data_as(ctypes.POINTER(ctypes.c_float))
    assert A.load_library().apic_set_particles(g._h, 0, p, p, p, p) == A.OK
    assert g.num_particles == 0
    g.update(A.DebugOptions(), 1 / 240)
