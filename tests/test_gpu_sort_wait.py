"""A sort tile whose wait for the tiles before it runs out counts their keys
itself.  A build in which every wait runs out at once (APIC_SORT_SPIN_LIMIT 0)
gives the same bits as the default one in every caller of the sort: the
no-allocation sort, the scene's two sorts, the particle view."""
import os
import subprocess
import sys

import numpy as np
import pytest

import apic_gb300 as A
from apic_gb300 import build as gpu_build
from parity_helpers import eq

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def run_all():
    import torch
    out = {}
    for n, w, h in ((20000, 64, 64), (200000, 1000, 600), (1 << 20, 1024, 1024), (1 << 20, 65536, 65536)):
        rng = np.random.default_rng(n + w)
        x, y = (torch.from_numpy(rng.uniform(0, s, n).astype(np.float32)).cuda() for s in (w, h))
        k, v = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
        rc = A.load_library().apic_morton_sort_noalloc(x.data_ptr(), y.data_ptr(), n, w, h, 1.0, k.data_ptr(),
                                                       v.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == A.OK
        out[f"noalloc {n} {w} keys"], out[f"noalloc {n} {w} slots"] = k.cpu().numpy(), v.cpu().numpy()
    side, n = 512, 400000
    rng = np.random.default_rng(3)
    g = A.Apic(side, side, 1 / side, A.WorldProperties(-9.81, 0.1, 5.0, 1e-5))
    g.set_particles(*(rng.uniform(0.05, 0.95, n).astype(np.float32) for _ in range(2)))
    for stage in ("sort", "p2g"):
        g.run_stage(stage, 1 / 500)
    for f in ("sort_keys", "sort_vals", "u", "v", "density"):
        out[f] = g.read_field(f)
    g.update(A.DebugOptions(), 1 / 2000)
    out["pos_x"] = g.read_field("pos_x")
    out["view"] = g.render(A.render_params(800, 800, scale=800.0))[0]
    return out


def test_waits_that_run_out(gpu_lib, tmp_path):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    pytest.importorskip("torch")
    obj, lib, res = (str(tmp_path / f) for f in ("sort.o", "libapic_gpu_wait.so", "wait.npz"))
    nvcc = gpu_build._nvcc()
    gpu_build._run([nvcc] + gpu_build.NVCC_FLAGS + ["-DAPIC_SORT_SPIN_LIMIT=0u", "-c",
                                                    os.path.join(gpu_build.CSRC, "sort.cu"), "-o", obj])
    objs = [obj if s == "sort.cu" else os.path.join(gpu_build.BUILD_DIR, s + ".o")
            for s in gpu_build.CUDA_SOURCES + gpu_build.CXX_SOURCES]
    gpu_build._run([nvcc] + gpu_build.ARCH + ["-shared", "-cudart", "static", "-o", lib] + objs +
                   ["-lpthread", "-ldl", "-lrt"])
    env = dict(os.environ)
    env["PYTHONPATH"] = os.pathsep.join([HERE, os.path.dirname(A.__file__) + "/.."] +
                                        ([env["PYTHONPATH"]] if env.get("PYTHONPATH") else []))
    r = subprocess.run([sys.executable, os.path.abspath(__file__), lib, res], capture_output=True, text=True, env=env,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    want, got = run_all(), np.load(res)
    assert sorted(got.files) == sorted(want)
    for k in want:
        eq(got[k].ravel(), np.asarray(want[k]).ravel(), k)


if __name__ == "__main__":
    A.load_library(sys.argv[1])
    np.savez(sys.argv[2], **run_all())
