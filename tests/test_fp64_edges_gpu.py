"""FP64 contact, friction, drag, ball and division by the mass at operands that
the integer-unit functions take (ordinary, and exponents near their limits of
+-250) and refuse (subnormal, huge, overflowing): single masses without
springs, each body on its own plane and all against a ball, two steps and
more, against the oracle bit for bit.  In tiles of few masses (the resident
grid's lanes), in tiles of many (its thread per mass), and by the per-step
kernel."""
import numpy as np
import pytest

import titan_gb300 as tg
from oracle import pyoracle as po
from tests.test_fp64_alu_gpu import values
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

# exponents; squares and products of two stay finite
RANGES = {"ordinary": (-4, 3), "edges": (-249, 120), "outside": (-1023, 400)}


def masses(kind, n, seed):
    """n masses with positions, velocities and loads of the given range of
    exponents, and springs of no stiffness between those farthest apart (so
    that tiles have halos)."""
    rng = np.random.default_rng(seed)
    lo, hi = RANGES[kind]
    sc = wl.empty_scene(1e-4, (0.3, -0.2, -9.81))
    pos = values(rng, 3 * n, lo, hi).reshape(n, 3)
    left = pos.argmin(0).astype(np.int32)
    right = pos.argmax(0).astype(np.int32)
    ns = left.size
    sc.update(pos=pos, vel=values(rng, 3 * n, lo, hi).reshape(n, 3),
              m=np.abs(values(rng, n, max(lo, -200), min(hi, 60), zeros=0.0)),
              ext=values(rng, 3 * n, lo, hi).reshape(n, 3), drag=np.where(rng.random(n) < 0.5, 3.0, 0.0),
              left=left, right=right, k=np.zeros(ns), rest=np.ones(ns), damping=np.zeros(ns), type=np.zeros(ns, np.int32),
              omega=np.zeros(ns), amp=np.full(ns, 0.2), phase=np.zeros(ns))
    sc["planes"].append(((0.0, 0.0, 1.0), 0.125, 0.4, 0.6))
    sc["planes"].append(((0.6, 0.0, 0.8), -0.5, 0.0, 0.5))
    sc["balls"].append(((0.25, 0.0, -0.5), 1.5))
    return sc


@pytest.mark.parametrize("how", ["lanes", "threads", "per step"])
@pytest.mark.parametrize("kind", list(RANGES))
def test_masses_bitwise(kind, how):
    sc = masses(kind, 5000, list(RANGES).index(kind) + 10)
    s = wl.make_sim(sc, tg.FP64, 128 if how == "threads" else 0, resident=(0, 0, 0) if how == "per step" else None)
    o = po.OracleSim(sc)
    for n in (2, 3):
        s.step(n)
        info = s.grid_info()
        assert (info["last"], info["lanes"]) == {"lanes": (1, 1), "threads": (1, 0), "per step": (0, 0)}[how]
        o.step(n, po.ASCENDING)
        st = s.get_state(acc=True)
        # the oracle adds terms with a factor of zero that the engine does not
        # have, which are NaN at infinite velocities: masses whose state has
        # overflowed are left out
        seen = np.isfinite(np.concatenate([o.pos, o.vel, o.acc], 1)).all(1)
        assert seen.mean() > 0.5
        for got, want in ((st["acc"], o.acc), (st["vel"], o.vel), (st["pos"], o.pos)):
            assert np.array_equal(got[seen], want[seen]), n
        if kind == "ordinary":
            assert seen.all()
