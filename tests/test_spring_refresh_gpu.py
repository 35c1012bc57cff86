"""Spring parameters of a started scene rewritten on the device
(refresh_entries): whole arrays, one at a time and together, against a fresh
handle that was started with them -- the records are the same bits -- and the
diagnostics, which share the device's spring arrays, after each change."""
import numpy as np
import pytest

import titan_gb300 as tg
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

CHANGES = [("k",), ("rest", "damping"), ("omega", "phase"), ("amp",), ("k", "rest", "damping", "omega", "amp", "phase"),
           ("k", "type")]


@pytest.mark.parametrize("side", [3, 11])  # one halo-free tile (FP32 forms); many tiles
@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32, tg.FP32C])
def test_refreshed_records_equal_a_fresh_start(prec, side):
    sc = wl.rollout_request(side, 1)
    s = wl.make_sim(sc, prec)
    rng = np.random.default_rng(side)
    ns = sc["left"].size
    s.step(3)
    for q, names in enumerate(CHANGES):
        new = {"k": np.exp(rng.uniform(5, 9, ns)), "rest": sc["rest"] * rng.uniform(0.9, 1.1, ns),
               "damping": rng.uniform(0, 0.3, ns), "omega": rng.uniform(1, 30, ns), "amp": rng.uniform(-0.2, 0.2, ns),
               "phase": rng.uniform(-4, 4, ns),
               "type": np.where(sc["type"] >= 2, rng.integers(2, 4, ns), sc["type"]).astype(np.int32)}
        new = {k: new[k] for k in names}
        sc = dict(sc, **new)
        s.set_spring_params(None, **new)
        if q == 3:  # and a few by index
            idx = np.arange(0, ns, 7)
            sc["k"] = sc["k"].copy()
            sc["k"][idx] *= 1.5
            s.set_spring_params(idx, k=sc["k"][idx])
        s.set_mass_state(None, pos=sc["pos"], vel=sc["vel"])
        s.set_time(0.25 * q)
        f = wl.make_sim(sc, prec)
        f.set_time(0.25 * q)
        s.step(5)
        f.step(5)
        a, b = s.get_state(acc=True), f.get_state(acc=True)
        assert all(np.array_equal(a[k], b[k]) for k in ("pos", "vel", "acc")), names
        da, db = s.diagnostics(), f.diagnostics()
        assert da["spring_pe"] == db["spring_pe"] and da["total"] == db["total"], names


def test_state_into_page_locked_and_other_buffers():
    sc = wl.actuated_lattice(9)
    s = wl.make_sim(sc, tg.FP32C)
    s.step(4)
    want = s.get_state(acc=True)
    pin = {k: tg.pinned_empty((s.n, 3)) for k in ("pos", "acc")}
    got = s.get_state(acc=True, out=pin)
    assert got["pos"] is pin["pos"]
    assert all(np.array_equal(got[k], want[k]) for k in ("pos", "vel", "acc"))
    odd = tg.pinned_empty((3 * s.n + 1,))[1:].reshape(s.n, 3)  # not 16-byte aligned
    assert np.array_equal(s.get_state(vel=False, out={"pos": odd})["pos"], want["pos"])
    idx = np.array([5, 3, 700, 0])
    sub = s.get_masses(idx, acc=True)
    assert all(np.array_equal(sub[k], want[k][idx]) for k in ("pos", "vel", "acc"))
