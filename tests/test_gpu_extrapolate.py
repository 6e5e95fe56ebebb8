"""Velocity extrapolation on tiles with a halo: grids that cut tiles in every
way and on both sides of the tile size's rule, valid faces sparse, in blobs,
everywhere and nowhere.  Four sweeps equal the oracle's bit for bit."""
import numpy as np
import pytest

import apic_gb300 as A
from parity_helpers import eq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(14, 10), (32, 8), (34, 16), (66, 42), (130, 70), (512, 512), (516, 514), (640, 450)])
@pytest.mark.parametrize("share", [0.0, 0.002, 0.3, 1.0])
def test_four_sweeps(gpu_lib, oracle_mod, w, h, share):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(w * h)
    props = A.WorldProperties(-9.81, 0.1, 5.0, 1e-5)
    g, o = A.Apic(w, h, 1 / w, props), oracle_mod.OracleSim(w, h, 1 / w, props)
    fields = {}
    for name, n in (("u", (w + 1) * h), ("v", w * (h + 1))):
        ok = rng.random(n) < share
        if share == 0.3:  # a blob instead of single faces
            k = np.arange(n)
            ok = (k % (w + 1) < w // 2) & (k < n // 2)
        fields[name] = rng.standard_normal(n).astype(np.float32)
        fields["valid_" + name] = ok.astype(np.uint8)
    for sim in (g, o):
        for name, v in fields.items():
            sim.write_field(name, v)
        sim.run_stage("extrap", 1 / 1000)
    for name in ("u", "v"):
        eq(g.read_field(name), o.read_field(name), name)
