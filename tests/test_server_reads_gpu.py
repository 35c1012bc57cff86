"""Transfers of one scene while the request loop steps another: the loop
holds two CTAs on every SM, and the kernels behind get_state, get_masses,
set_mass_state, set_spring_params and export_vertices have to fit beside
them -- a read that waited for the loop to leave would hold the host (and
with it every admission) until a second after the last rollout."""
import numpy as np
import pytest

import titan_gb300 as tg
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


# long: steps of about a second of the loop's time
@pytest.mark.parametrize("prec,tile,long", [(tg.FP64, 128, 60000), (tg.FP32, 208, 150000), (tg.FP32C, 208, 150000)])
def test_transfers_run_beside_the_loop(prec, tile, long):
    def make(side, seed):
        return wl.make_sim(wl.rollout_request(side, seed), prec, tile, kernel=1, resident=(0, 0, 0))

    sc = wl.rollout_request(9, 2)
    a, b, ref = make(5, 1), make(9, 2), make(9, 2)
    ref.step(20)
    want = ref.get_state(acc=True)
    idx = np.array([700, 3, 31, 32])
    pin = {"pos": tg.pinned_empty((b.n, 3))}
    with tg.Server(prec, max_slots=4) as srv:
        t_long = srv.submit(a, long)
        srv.wait(srv.submit(b, 20))
        got = b.get_state(acc=True)
        sub = b.get_masses(idx, acc=True)
        b.get_state(vel=False, out=pin)
        vert = b.export_vertices()
        b.set_spring_params(None, k=2 * sc["k"])
        b.set_mass_state(None, pos=sc["pos"], vel=sc["vel"])
        back = b.get_state()
        assert not srv.poll(t_long)  # still running: nothing above waited for the loop to leave
        srv.wait(t_long)
    for k in ("pos", "vel", "acc"):
        assert np.array_equal(got[k], want[k]) and np.array_equal(sub[k], want[k][idx]), k
    assert np.array_equal(pin["pos"], want["pos"])
    assert np.array_equal(vert, want["pos"].astype(np.float32).reshape(vert.shape))
    if prec == tg.FP64:
        assert np.array_equal(back["pos"], sc["pos"]) and np.array_equal(back["vel"], sc["vel"])
