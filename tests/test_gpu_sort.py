"""The radix sort at the sizes where its form changes: one tile, one pair more,
the limits of the tile sizes, few and many digit values, one to four passes
(an odd number starts in the scratch), all keys equal, sorted and reversed.
Keys and slots equal numpy's stable sort of the same Morton codes."""
import numpy as np
import pytest

import apic_gb300 as A

pytestmark = pytest.mark.gpu


def spread(v):
    v = v.astype(np.uint64)
    for s, m in ((8, 0x00FF00FF), (4, 0x0F0F0F0F), (2, 0x33333333), (1, 0x55555555)):
        v = (v | (v << np.uint64(s))) & np.uint64(m)
    return v


GRIDS = [(1, 1), (8, 4), (32, 32), (23, 61), (1024, 1024), (2048, 512), (65536, 65536)]
SIZES = [1, 31, 1023, 1024, 1025, 65536, 65537, 262144, 262145, 1 << 20]
CASES = [("random", n, w, h) for n in SIZES for w, h in GRIDS] + \
        [(o, n, w, h) for o in ("equal", "sorted", "reversed") for n in (1025, 262145) for w, h in GRIDS]


@pytest.mark.parametrize("order,n,w,h", CASES)
def test_stable_sort(gpu_lib, order, n, w, h):
    if A.device_count() == 0:
        pytest.skip("no CUDA device")
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + w)
    x, y = rng.integers(0, w, n), rng.integers(0, h, n)
    if order == "equal":
        x[:], y[:] = w // 2, h // 2
    keys = spread(x) | (spread(y) << np.uint64(1))
    if order in ("sorted", "reversed"):
        at = np.argsort(keys, kind="stable")
        at = at[::-1] if order == "reversed" else at
        x, y, keys = x[at], y[at], keys[at]
    want = np.argsort(keys, kind="stable")
    px = torch.from_numpy((x + 0.5).astype(np.float32)).cuda()
    py = torch.from_numpy((y + 0.5).astype(np.float32)).cuda()
    k = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    v = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    rc = A.load_library().apic_morton_sort_noalloc(px.data_ptr(), py.data_ptr(), n, w, h, 1.0, k.data_ptr(),
                                                   v.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == A.OK
    assert np.array_equal(k.cpu().numpy().view(np.uint32), keys[want].astype(np.uint32))
    assert np.array_equal(v.cpu().numpy(), want)
