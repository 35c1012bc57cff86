"""State read into host arrays that are page-locked only in part: the gather
kernel may store into a caller's array only where all of it is mapped, so
these go through the handle's staging buffer, wherever in the array the
registered range lies."""
import numpy as np
import pytest

import titan_gb300 as tg
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

PAGE = 65536  # of the largest page size in use


@pytest.mark.parametrize("first,count", [(0, 1), (0, 3), (1, 2), (3, 1), (0, 4)])
def test_arrays_registered_in_part(first, count):
    torch = pytest.importorskip("torch")
    rt = torch.cuda.cudart()
    s = wl.make_sim(wl.actuated_lattice(22), tg.FP32C)  # 255,552 bytes an array: 3.9 pages
    s.step(5)
    want = s.get_state()
    raw = np.zeros(3 * 5 * PAGE, np.uint8)
    off = -raw.ctypes.data % PAGE
    pages = raw[off:off + 2 * 4 * PAGE]
    out = {k: pages[q * 4 * PAGE:][:s.n * 24].view(np.float64).reshape(s.n, 3) for q, k in enumerate(("pos", "vel"))}
    at = pages.ctypes.data + first * PAGE
    assert int(rt.cudaHostRegister(at, count * PAGE, 0)) == 0
    try:
        got = s.get_state(out=out)
        assert got["pos"] is out["pos"]
        assert all(np.array_equal(out[k], want[k]) for k in out)
    finally:
        assert int(rt.cudaHostUnregister(at)) == 0
