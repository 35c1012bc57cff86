"""New spring parameters of a started scene, for all springs, for some by
index, for a prefix, and twice for one spring: the kernel that rewrites the
slab's records has to leave those that a fresh handle has, also where the
parameters given are few and the scene small."""
import numpy as np
import pytest

import titan_gb300 as tg
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

NAMES = ("k", "rest", "damping", "omega", "amp", "phase")


@pytest.mark.parametrize("side", [4, 6, 10])  # 400, 2,100 and 11,000 springs
@pytest.mark.parametrize("names", [("k",), ("phase", "amp"), NAMES])
@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32, tg.FP32C])
def test_records_of_a_fresh_start(prec, names, side):
    sc = wl.rollout_request(side, 1)
    s = wl.make_sim(sc, prec)
    rng = np.random.default_rng(side)
    ns = sc["left"].size
    for q in range(4):
        new = {"k": np.exp(rng.uniform(5, 9, ns)), "rest": sc["rest"] * rng.uniform(0.9, 1.1, ns),
               "damping": rng.uniform(0, 0.3, ns), "omega": rng.uniform(1, 30, ns), "amp": rng.uniform(-0.2, 0.2, ns),
               "phase": rng.uniform(-4, 4, ns)}
        # all; some; a prefix in order without an index; one twice (the last value holds)
        idx = [None, rng.permutation(ns)[:ns // 3], np.arange(ns // 2), np.array([7, 3, 7])][q]
        given = {k: new[k][:idx.size] if idx is not None else new[k] for k in names}
        sc = {k: v.copy() if k in names else v for k, v in sc.items()}
        for k in names:
            if idx is None:
                sc[k] = given[k]
            else:
                for i, v in zip(idx, given[k]):
                    sc[k][i] = v
        s.step(1)
        s.set_spring_params(idx, **given)
        s.set_mass_state(None, pos=sc["pos"], vel=sc["vel"])
        s.set_time(0.1 * q)
        f = wl.make_sim(sc, prec)
        f.set_time(0.1 * q)
        for x in (s, f):
            x.step(1)
            x.step(4)
        a, b = s.get_state(acc=True), f.get_state(acc=True)
        assert all(np.array_equal(a[k], b[k]) for k in ("pos", "vel", "acc")), (names, q)
        da, db = s.diagnostics(), f.diagnostics()
        assert da["spring_pe"] == db["spring_pe"] and da["total"] == db["total"], (names, q)
        f.close()
