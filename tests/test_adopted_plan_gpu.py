"""adopt_plan between handles whose settings give different default plans: the
handle starts with the plan that its own settings give, as a fresh one does;
with the same settings, or an explicit tile size, it takes the template's."""
import numpy as np
import pytest

import titan_gb300 as tg
from tests.test_resident_grid_gpu import same
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def handle(sc, prec, **kw):
    s = tg.Sim(prec)
    wl.load(s, dict(sc, integrator=kw.pop("integ", tg.EULER)), start=False, **kw)
    return s


@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32C])
@pytest.mark.parametrize("kind", ["lattice", "bodies"])
@pytest.mark.parametrize("own", [dict(), dict(integ=tg.VERLET), dict(resident=(0, 0, 0)), dict(threads=256)])
@pytest.mark.parametrize("tile", [0, 128])
def test_plan_of_the_handles_own_settings(prec, kind, own, tile):
    sc = wl.actuated_lattice(13) if kind == "lattice" else wl.robot_batch(310, side_range=(5, 7), seed=2)
    template = handle(sc, prec)
    template.plan_host(tile)
    a, f = handle(sc, prec, **own), handle(sc, prec, **own)
    a.adopt_plan(template)
    for s in (a, f):
        s.start(tile)
        s.step(3)
        s.step(1)
    pa, pf = a.plan_info(), f.plan_info()
    assert pa == pf
    assert a.kernel_info() == f.kernel_info() and a.grid_info() == f.grid_info()
    same(a.get_state(acc=True, T=True), f.get_state(acc=True, T=True))
