"""Calls of a few steps on scenes of many bodies whose whole bodies above the
per-step tile size are resident in longer calls (short_limit): the same masses
in tiles of the per-step kernel's size, against handles without resident tiles
bit for bit -- calls on both sides of the limit mixed, and new spring
parameters (all, by index, other types), mass state and time in between."""
import numpy as np
import pytest

import titan_gb300 as tg
from tests.test_resident_grid_gpu import same
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


# all resident and small, all resident, some bodies too large to be resident; and the limit of each
@pytest.mark.parametrize("bodies,sides,limit", [(310, (6, 6), 1), (310, (5, 8), 4), (310, (6, 9), 12)])
@pytest.mark.parametrize("prec", [tg.FP32, tg.FP32C])
def test_bits_of_the_per_step_kernels(prec, bodies, sides, limit):
    sc = wl.robot_batch(bodies, side_range=sides, seed=5)
    rng = np.random.default_rng(2)
    sc["vel"] = rng.normal(scale=0.2, size=sc["pos"].shape)
    sc["fixed"] = (rng.random(sc["pos"].shape[0]) < 0.02).astype(np.uint8)
    ns = sc["left"].size
    k2 = np.exp(rng.uniform(6, 9, ns))
    idx = np.arange(0, ns, 13)
    types = np.where(sc["type"] >= 2, rng.integers(2, 4, ns), sc["type"]).astype(np.int32)
    rows = np.arange(0, 5000, 3)
    got = []
    for resident in (None, (0, 0, 0)):
        s = wl.make_sim(sc, prec, resident=resident)

        def step(*calls):
            for n in calls:
                s.step(n)
                assert s.grid_info()["last"] == (3 if resident is None and n <= limit else 0)

        s.prepare_steps(1)
        if resident is None:
            assert s.resident_info()["active"] == 2
        step(limit + 1, 1, limit, limit + 3)
        got.append(s.get_state(acc=True, T=True))
        s.set_spring_params(None, k=k2)
        step(1, 9)
        s.set_spring_params(idx, damping=np.full(idx.size, 0.2))
        step(1, limit + 1)
        s.set_spring_params(None, type=types)
        s.prepare_steps(1)
        step(1)
        s.set_mass_state(rows, pos=sc["pos"][rows] + 0.001)
        step(limit, 8)
        s.set_time(0.4)
        step(1, 1)
        got.append(s.get_state(acc=True, T=True))
        assert s.time == pytest.approx(0.4 + 2e-4)
    assert np.isfinite(got[3]["pos"]).all()
    same(got[0], got[2])
    same(got[1], got[3])


def test_integrator_change_after_short_calls():
    sc = wl.robot_batch(310, side_range=(6, 8), seed=9)
    got = []
    for resident in (None, (0, 0, 0)):
        s = wl.make_sim(sc, tg.FP32C, resident=resident)
        s.prepare_steps(2)
        for n in (1, 20, 2):
            s.step(n)
        s.set_integrator(tg.VERLET)
        s.step(3)
        s.step(1)
        s.set_integrator(tg.EULER)
        s.step(1)
        got.append(s.get_state(acc=True, T=True))
    same(*got)


def test_repeated_short_calls_get_their_tables():
    """The first 64 calls run on the resident bodies, the others on the tables
    made then."""
    sc = wl.robot_batch(310, side_range=(6, 6), seed=9)
    got = []
    for resident in (None, (0, 0, 0)):
        s = wl.make_sim(sc, tg.FP32C, resident=resident)
        for q in range(70):
            s.step(1)
            assert s.grid_info()["last"] == (3 if resident is None and q >= 64 else 0)
        got.append(s.get_state(acc=True, T=True))
    same(*got)


def test_mass_attributes_set_after_the_tables():
    """The tables made before hold no copy of what later calls replace: masses,
    loads and the arrays of local constraints, which are uploaded with them."""
    sc = wl.robot_batch(310, side_range=(6, 7), seed=3)
    n = sc["pos"].shape[0]
    rng = np.random.default_rng(8)
    on = rng.random(n) < 0.1
    sc["lc_ptr"] = np.concatenate([[0], np.cumsum(on)]).astype(np.int64)
    sc["lc_type"] = np.zeros(int(on.sum()), np.int32)
    sc["lc_vec"] = np.tile([0.0, 0.0, 1.0], (int(on.sum()), 1))
    sc["lc_num"] = np.full(int(on.sum()), 0.1)
    ext, m = rng.normal(size=(n, 3)), rng.uniform(0.05, 0.2, n)
    got = []
    for resident in (None, (0, 0, 0)):
        s = wl.make_sim(sc, tg.FP32C, resident=resident)
        s.prepare_steps(1)
        for q in range(3):
            s.set_mass_state(None, ext=ext * q, m=m * (1 + q))
            for c in (1, 1, 9, 1):
                s.step(c)
        got.append(s.get_state(acc=True, T=True))
    same(*got)
