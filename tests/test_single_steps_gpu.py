"""Calls of a single step on scenes cut for the resident grid: in the FP32
forms a pass of that kernel that may start while the step before drains
(launch_grid_single), against the per-step kernels bit for bit.  Tiles of one
and two per SM and above the size it takes; both integrators with state of
their own; new spring parameters, mass state, time and integrator in between,
with no wait of the host."""
import numpy as np
import pytest

import titan_gb300 as tg
from tests.test_resident_grid_gpu import same, scene
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


# tiles: a few, one or two per SM, above the single pass's size
@pytest.mark.parametrize("shape,single", [((7, 6, 6), 1), ((9, 8, 13), 1), ((18, 17, 15), 1), ((31, 30, 29), 0)])
@pytest.mark.parametrize("integ", [tg.EULER, tg.VERLET, tg.RK2])
@pytest.mark.parametrize("prec", [tg.FP32, tg.FP32C])
def test_bits_of_the_per_step_kernels(prec, integ, shape, single):
    sc = scene(*shape, seed=sum(shape), fixed=0.05, act=0.2)
    sc["integrator"] = integ
    got = []
    for resident in (None, (0, 0, 0)):
        s = wl.make_sim(sc, prec, resident=resident)
        info = s.grid_info()
        assert (info["active"], info["single"]) == ((1, single) if resident is None else (0, 0))
        for n, kind in ((1, 2 * single), (1, 2 * single), (5, 1), (1, 2 * single), (1, 2 * single), (2, 1)):
            s.step(n)
            assert s.grid_info()["last"] == (kind if resident is None else 0)
        for _ in range(20):
            s.step(1)
        got.append(s.get_state(acc=True, T=True))
        assert np.isfinite(got[-1]["pos"]).all()
    same(*got)


@pytest.mark.parametrize("prec", [tg.FP32, tg.FP32C])
def test_changes_between_single_steps(prec):
    sc = scene(14, 13, 12, seed=3, act=0.3, hub=150)
    rng = np.random.default_rng(4)
    ns = sc["left"].size
    new = [dict(k=np.exp(rng.uniform(6, 9, ns)), phase=rng.uniform(-3, 3, ns)) for _ in range(6)]
    idx = np.arange(0, 300, 7)
    got = []
    for resident in (None, (0, 0, 0)):
        s = wl.make_sim(sc, prec, resident=resident)
        for q, par in enumerate(new):
            s.step(1)
            s.set_spring_params(None, **par)
            s.step(1)
            s.set_mass_state(idx, pos=sc["pos"][idx] + 0.001 * q)
            s.step(1)
            s.set_time_step(1e-4 / (1 + q))
            s.step(1)
            if q == 2:
                s.set_integrator(tg.VERLET)
            if q == 4:
                s.set_integrator(tg.RK2)
        s.set_time(0.5)
        s.step(1)
        assert s.grid_info()["last"] == (2 if resident is None else 0)
        got.append(s.get_state(acc=True, T=True))
    same(*got)
