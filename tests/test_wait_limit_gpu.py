"""The resident grid's bounded wait for other tiles' masses: with a limit of
one poll it runs out in a scene of some hundred tiles (a tile would have to
find all its neighbours' records there at the first look, in every pass), the
kernel returns with its error flag, and the handle refuses steps until a whole
state is uploaded; it then steps as a fresh one."""
import numpy as np
import pytest

import titan_gb300 as tg
from tests.test_resident_grid_gpu import same
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integ", [tg.EULER, tg.RK2])
@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32C])
def test_a_wait_that_runs_out(prec, integ):
    sc = wl.actuated_lattice(20)
    sc["integrator"] = integ
    s, f = wl.make_sim(sc, prec), wl.make_sim(sc, prec)
    s.set_wait_limit(1)
    s.step(200)
    assert s.grid_info()["last"] == 1 and s.grid_info()["tiles"] > 100
    with pytest.raises(tg.TitanError) as e:
        s.synchronize()
    assert e.value.code == 6 and "wait" in str(e.value)
    for call in (lambda: s.step(1), lambda: s.step(5)):
        with pytest.raises(tg.TitanError) as e:
            call()
        assert e.value.code == 6
    s.set_wait_limit(0)
    s.set_mass_state(None, pos=sc["pos"])  # not a whole state
    with pytest.raises(tg.TitanError):
        s.step(1)
    s.set_time(0.0)
    s.set_mass_state(None, pos=sc["pos"], vel=sc["vel"], T=np.zeros(s.n))
    for x in (s, f):
        x.step(1)
        x.step(30)
        x.step(1)
    same(s.get_state(acc=True, T=True), f.get_state(acc=True, T=True))
