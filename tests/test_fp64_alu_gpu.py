"""FP64 entry forces on the integer units (fp64_alu.cuh) against the oracle.

Independent pairs of masses, one spring each, so that every spring force is
seen alone in the accelerations.  The square root, divisions and products
have to give the IEEE results, so the bar is the oracle's bits: at ordinary
operands, at the edges of the range the integer path takes (exponents of
+-250) and outside it (subnormals, huge values, overflow to infinity and
NaN), where the FP64 instructions take over.
"""
import numpy as np
import pytest

import titan_gb300 as tg
from oracle import pyoracle as po
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def values(rng, n, lo, hi, zeros=0.1):
    """Random signed doubles with exponents in [lo, hi]: full, short and all-ones significands, some zeros."""
    f = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    cut = rng.integers(0, 52, n, dtype=np.uint64)
    kind = rng.integers(0, 4, n)
    one = np.uint64(1)
    f = np.where(kind == 1, f & ~((one << cut) - one), f)
    f = np.where(kind == 2, f | ((one << cut) - one), f)
    f = np.where(kind == 3, (np.uint64(1 << 52) - one) - (f & np.uint64(7)), f)
    e = rng.integers(lo + 1023, hi + 1024, n).astype(np.uint64)
    x = ((rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63)) | (e << np.uint64(52)) | f).view(np.float64)
    return np.where(rng.random(n) < zeros, 0.0, x)


RANGES = {
    "ordinary": ((-4, 3), (-2, 17), (-6, 1)),
    "edges": ((-249, 120), (-250, 120), (-250, 60)),
    "outside": ((-1023, 600), (-1023, 400), (-1023, 300)),
}


@pytest.mark.parametrize("kernel", [1, 4])
@pytest.mark.parametrize("kind", list(RANGES))
def test_pair_forces_bitwise(kind, kernel):
    (xlo, xhi), (klo, khi), (dlo, dhi) = RANGES[kind]
    rng = np.random.default_rng(list(RANGES).index(kind))
    pairs = 3001
    n = 2 * pairs
    sc = wl.empty_scene(1e-4, (0.0, 0.0, 0.0))
    pos = values(rng, 3 * n, xlo, xhi).reshape(n, 3)
    near = rng.random(pairs) < 0.5  # half the pairs close together (short differences)
    pos[1::2][near] = pos[0::2][near] * (1.0 + rng.normal(scale=1e-3, size=(int(near.sum()), 3)))
    rest = np.abs(values(rng, pairs, xlo, xhi))
    with np.errstate(all="ignore"):
        rest[::5] = np.sqrt(((pos[1::2] - pos[0::2]) ** 2).sum(1))[::5]  # some at rest
    rest[~np.isfinite(rest)] = 1.0
    sc.update(pos=pos, vel=values(rng, 3 * n, xlo, xhi).reshape(n, 3), m=np.full(n, 0.1),
              left=np.arange(0, n, 2, dtype=np.int32), right=np.arange(1, n, 2, dtype=np.int32),
              k=np.abs(values(rng, pairs, klo, khi)), rest=rest,
              damping=np.abs(values(rng, pairs, dlo, dhi, zeros=0.3)), type=np.zeros(pairs, np.int32),
              omega=np.zeros(pairs), amp=np.full(pairs, 0.2), phase=np.zeros(pairs))
    s = wl.make_sim(sc, tg.FP64, 64, kernel=kernel)
    s.step(1)
    st = s.get_state(acc=True)
    o = po.OracleSim(sc)
    o.step(1, po.ASCENDING)
    # the oracle adds terms with a factor of zero that the engine does not
    # have: the drag of masses without any, 0 |v|^2 (NaN where |v|^2
    # overflows), and the damping of springs without any, 0 w.d / |d| (NaN
    # where |d| underflows to 0)
    with np.errstate(all="ignore"):
        seen = np.isfinite((sc["vel"] ** 2).sum(1))
        seen &= np.repeat((sc["damping"] != 0) | (((pos[1::2] - pos[0::2]) ** 2).sum(1) > 0), 2)
    for got, want in ((st["acc"], o.acc), (st["vel"], o.vel), (st["pos"], o.pos)):
        assert np.array_equal(got[seen], want[seen], equal_nan=True)


@pytest.mark.parametrize("lo,hi", [(-40, -20), (-12, 12), (26, 34)])
def test_actuated_rest_length(lo, hi):
    """The sine of actuated rest lengths: angles below, inside and above the
    integer path's range (2^-24 to 2^30), both actuation types, amplitudes on
    either side of its limit of 4.  A spring at rest length 1 whose ends are 1
    apart has the force k (scale - 1), whose error against libm's sine is
    bounded by the two sines' errors (below 2 units in the last place each)
    and the roundings of amp sin and 1 -+ amp sin."""
    rng = np.random.default_rng(100 + hi)
    pairs = 3001
    n = 2 * pairs
    pos = np.zeros((n, 3))
    pos[:, 1] = np.repeat(np.arange(pairs) * 2.0, 2)
    pos[1::2, 0] = 1.0
    th = values(rng, pairs, lo, hi, zeros=0.02)
    th[::7] = np.round(th[::7] / np.pi) * np.pi  # near the sine's zeros
    amp = np.where(rng.random(pairs) < 0.2, rng.uniform(4.0, 9.0, pairs), rng.uniform(-0.3, 0.3, pairs))
    sc = wl.empty_scene(1e-4, (0.0, 0.0, 0.0))
    sc.update(pos=pos, vel=np.zeros((n, 3)), m=np.ones(n), left=np.arange(0, n, 2, dtype=np.int32),
              right=np.arange(1, n, 2, dtype=np.int32), k=np.ones(pairs), rest=np.ones(pairs), damping=np.zeros(pairs),
              type=rng.integers(2, 4, pairs).astype(np.int32), omega=np.zeros(pairs), amp=amp, phase=th)
    s = wl.make_sim(sc, tg.FP64, 64)
    s.step(1)
    got = s.get_state(acc=True)["acc"][1::2, 0]
    want = (1.0 + np.where(sc["type"] == 2, -amp, amp) * np.sin(th)) - 1.0
    scale = np.maximum(1.0, np.abs(1.0 + want))
    assert np.all(np.abs(got - want) <= (5 * np.abs(amp) + 2 * scale) * 2.0 ** -52)
