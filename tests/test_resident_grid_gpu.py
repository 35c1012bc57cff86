"""All tiles at once (resident_grid.cu) against the per-step kernels and the
oracle, bit for bit: the default handle runs calls of two steps and more in
one cooperative launch, set_resident(0) keeps the per-step kernels."""
import numpy as np
import pytest

import titan_gb300 as tg
from oracle import pyoracle as po
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

CHUNKS = [2, 1, 3, 7, 1, 1, 20]  # single steps (per-step kernels) between grid launches


def scene(nx, ny, nz, seed, fixed=0.0, act=0.0, hub=0):
    """An irregular lattice on a frictional plane beside a ball: random
    stiffness and velocities, some fixed, loaded, dragged and locally
    constrained masses, springs removed; hub: springs from one mass to that
    many others (more than 96: a heavy mass)."""
    rng = np.random.default_rng(seed)
    sc = wl.lattice_scene((0, 0, 0.05 * nz), (0.1 * nx, 0.1 * ny, 0.1 * nz), nx, ny, nz, damping=0.1)
    n = sc["pos"].shape[0]
    keep = rng.random(sc["left"].size) > 0.05
    for k in ("left", "right", "rest", "k", "damping", "type", "omega", "amp", "phase"):
        sc[k] = sc[k][keep]
    if hub:
        other = rng.permutation(np.arange(1, n))[:hub].astype(np.int32)
        d = np.linalg.norm(sc["pos"][other] - sc["pos"][0], axis=1)
        for k, v in (("left", np.zeros(hub, np.int32)), ("right", other), ("rest", d), ("k", np.full(hub, 50.0)),
                     ("damping", np.zeros(hub)), ("type", np.zeros(hub, np.int32)), ("omega", np.zeros(hub)),
                     ("amp", np.full(hub, 0.2)), ("phase", np.zeros(hub))):
            sc[k] = np.concatenate([sc[k], v])
    ns = sc["left"].size
    sc["k"] = sc["k"] * np.exp(rng.uniform(-2, 1, ns))
    sc["vel"] = rng.normal(scale=0.3, size=(n, 3))
    if act:
        wl.actuate(sc, rng, act, 0.1)
    sc["fixed"] = (rng.random(n) < fixed).astype(np.uint8)
    sc["ext"] = np.where(rng.random((n, 1)) < 0.1, rng.normal(size=(n, 3)), 0.0)
    sc["drag"] = np.where(rng.random(n) < 0.1, 2.0, 0.0)
    lc = rng.random(n) < 0.02
    sc["lc_ptr"] = np.concatenate([[0], np.cumsum(lc)]).astype(np.int64)
    sc["lc_type"] = np.zeros(int(lc.sum()), np.int32)
    sc["lc_vec"] = np.tile([0.0, 0.0, 1.0], (int(lc.sum()), 1))
    sc["lc_num"] = np.full(int(lc.sum()), 0.1)
    sc["planes"].append(((0.0, 0.0, 1.0), 0.0, 0.4, 0.6))
    sc["balls"].append(((0.0, 0.0, -0.2), 0.25))
    return sc


def run(sc, prec, resident):
    s = wl.make_sim(sc, prec, resident=resident)
    for c in CHUNKS:
        s.step(c)
    return s, s.get_state(acc=True, T=True)


def same(a, b):
    for k in ("pos", "vel", "acc", "T"):
        assert np.array_equal(a[k], b[k]), k


# tiles: 4, about one per SM, about two per SM, more than the grid takes (FP64)
@pytest.mark.parametrize("shape", [(3, 4, 5), (9, 8, 13), (23, 17, 12), (31, 30, 29)])
@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32, tg.FP32C])
def test_bits_of_the_per_step_kernels(prec, shape):
    sc = scene(*shape, seed=sum(shape), fixed=0.05, act=0.2 if prec != tg.FP64 else 0.0)
    s, st = run(sc, prec, None)
    _, ref = run(sc, prec, (0, 0, 0))
    same(st, ref)
    if prec == tg.FP64 and sc["pos"].shape[0] < 2000:
        o = po.OracleSim(sc)
        o.step(sum(CHUNKS), po.ASCENDING)
        for k, w in (("pos", o.pos), ("vel", o.vel), ("acc", o.acc), ("T", o.T)):
            assert np.array_equal(st[k], w), k
        assert s.time == o.time


@pytest.mark.parametrize("integ", [tg.VERLET, tg.RK2])
@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32, tg.FP32C])
def test_integrators(prec, integ):
    sc = scene(13, 9, 11, seed=5, fixed=0.05)
    sc["integrator"] = integ
    _, st = run(sc, prec, None)
    _, ref = run(sc, prec, (0, 0, 0))
    same(st, ref)


@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32C])
def test_heavy_mass_and_uneven_bodies(prec):
    sc = scene(12, 11, 10, seed=8, hub=300)
    _, st = run(sc, prec, None)
    _, ref = run(sc, prec, (0, 0, 0))
    same(st, ref)
    sc = wl.robot_batch(24, side_range=(2, 9))  # some bodies are one tile (no halo), others several
    sc["pos"][:, 2] -= 0.06  # into their ground planes
    sc["vel"] = np.random.default_rng(1).normal(scale=0.2, size=sc["pos"].shape)
    _, st = run(sc, prec, None)
    _, ref = run(sc, prec, (0, 0, 0))
    same(st, ref)


def test_state_changes_between_launches_and_two_handles():
    """Uploads, a fix / unfix rebuild, a time step change and an integrator
    change between launches, with another handle's launches in flight."""
    sc, sc2 = scene(14, 13, 12, seed=3), scene(10, 9, 30, seed=4)
    res = []
    for resident in (None, (0, 0, 0)):
        a, b = wl.make_sim(sc, tg.FP32C, resident=resident), wl.make_sim(sc2, tg.FP64, resident=resident)
        a.step(30)
        b.step(40)
        a.step(11)
        idx = np.arange(0, 200, 3)
        a.set_mass_state(idx, pos=sc["pos"][idx] + 0.01, vel=np.zeros((idx.size, 3)))
        a.step(9)
        b.set_time_step(5e-5)
        b.step(8)
        a.set_mass_state(idx, fixed=np.ones(idx.size, np.uint8))
        a.step(9)
        a.set_integrator(tg.VERLET)
        a.step(6)
        b.set_integrator(tg.RK2)
        b.step(5)
        res.append((a.get_state(acc=True, T=True), b.get_state(acc=True, T=True)))
    same(res[0][0], res[1][0])
    same(res[0][1], res[1][1])


@pytest.mark.parametrize("sides", [(3, 9), (6, 9)])
@pytest.mark.parametrize("prec", [tg.FP32, tg.FP32C])
def test_many_bodies_in_size_groups(prec, sides):
    """More bodies than two per SM: whole bodies of up to 512 masses run as
    resident tiles in size groups, larger ones on the per-step kernels beside
    them.  Where all are above the per-step tile size, a switch to VERLET keeps
    state and accelerations as between the per-step kernels."""
    sc = wl.robot_batch(320, side_range=sides, seed=5)
    sc["vel"] = np.random.default_rng(2).normal(scale=0.2, size=sc["pos"].shape)
    s, st = run(sc, prec, None)
    assert s.resident_info()["active"] == 2 and s.resident_info()["cap"] == 512
    r, ref = run(sc, prec, (0, 0, 0))
    same(st, ref)
    if sides[0] < 6:
        return
    for x in (s, r):
        x.set_integrator(tg.VERLET)
        x.step(4)
    same(s.get_state(acc=True, T=True), r.get_state(acc=True, T=True))


@pytest.mark.parametrize("integ", [tg.EULER, tg.VERLET, tg.RK2])
@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32C])
def test_long_calls_in_several_launches(prec, integ):
    """Calls on both sides of the launches' 512 steps, and odd remainders."""
    sc = scene(6, 7, 8, seed=4, fixed=0.05, act=0.2 if prec != tg.FP64 else 0.0)
    sc["integrator"] = integ
    got = []
    for resident in (None, (0, 0, 0)):
        s = wl.make_sim(sc, prec, resident=resident)
        for n in (512, 513, 1027):
            s.step(n)
        got.append(s.get_state(acc=True, T=True))
    assert np.isfinite(got[1]["pos"]).all()
    same(*got)
