"""Extrapolation reads any non-zero validity byte as valid and writes 1, on tiles
whose faces are all valid as on mixed ones."""
import numpy as np
import pytest

import apic_gb300 as A
from parity_helpers import eq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [64, 600])
@pytest.mark.parametrize("flag", [2, 255])
def test_flags_are_one(gpu_lib, side, flag):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    g = A.Apic(side, side, 1 / side, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    for name in ("valid_u", "valid_v"):
        g.write_field(name, np.full(g.read_field(name).size, flag, np.uint8))
    g.run_stage("extrap", 1 / 1000)
    for name in ("valid_u", "valid_v"):
        got = g.read_field(name)
        eq(got, np.ones_like(got), name)
