"""Single steps while the caller captures the handle's stream, on scenes whose
other calls run on the resident grid, as its single pass, or on tables for
calls of a few steps: the captured step leaves the bits of a plain one."""
import pytest

import titan_gb300 as tg
from tests.test_resident_grid_gpu import same, scene
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["grid", "bodies", "bodies prepared"])
@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32C])
def test_captured_single_step(prec, kind):
    torch = pytest.importorskip("torch")
    sc = scene(9, 8, 13, seed=6, fixed=0.05) if kind == "grid" else wl.robot_batch(310, side_range=(6, 7), seed=1)
    a, b = wl.make_sim(sc, prec), wl.make_sim(sc, prec)
    if kind == "bodies prepared":
        a.prepare_steps(1)
    for s in (a, b):
        s.step(3)
        s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(a.stream), capture_error_mode="thread_local"):
        a.step(1)
    g.replay()
    torch.cuda.synchronize()
    b.step(1)
    for s in (a, b):
        s.step(4)
        s.step(1)
    same(a.get_state(acc=True, T=True), b.get_state(acc=True, T=True))
