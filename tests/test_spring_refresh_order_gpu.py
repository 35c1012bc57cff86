"""New spring parameters and the step right behind them: the warp-specialised
step may start while the kernel before it on the stream drains and reads the
slab records at once, so the launch behind the kernel that rewrites those
records has to wait for it.  A scene with more tiles than run at once, single
steps and a graph of them, against handles started with the parameters."""
import numpy as np
import pytest

import titan_gb300 as tg
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 3])
@pytest.mark.parametrize("prec", [tg.FP32, tg.FP32C])
def test_first_step_behind_new_parameters(prec, steps):
    sc = wl.actuated_lattice(41)
    rng = np.random.default_rng(7)
    ns = sc["left"].size
    s = wl.make_sim(sc, prec)
    assert s.kernel_info()["kernel"] == "warp-specialised"
    s.step(2)
    for _ in range(3):
        new = dict(k=np.exp(rng.uniform(7, 10, ns)), rest=sc["rest"] * rng.uniform(0.9, 1.1, ns),
                   phase=rng.uniform(-3, 3, ns))
        s.set_mass_state(None, pos=sc["pos"], vel=sc["vel"])
        s.set_time(0.0)
        s.set_spring_params(None, **new)
        s.step(steps)
        got = s.get_state(acc=True)
        f = wl.make_sim(dict(sc, **new), prec)
        f.step(steps)
        want = f.get_state(acc=True)
        f.close()
        assert all(np.array_equal(got[k], want[k]) for k in ("pos", "vel", "acc"))
