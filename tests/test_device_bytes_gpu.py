"""device_bytes as admission control uses it, read once after start(): the
first parameter updates of an engine, which every reuse of a pooled one makes,
add nothing to it, in any order; and the rollout server's record of a design
covers its engines."""
import pytest

import titan_gb300 as tg
from titan_gb300 import serving
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

NAMES = ("k", "rest", "damping", "omega", "amp", "phase")


@pytest.mark.parametrize("order", [[NAMES], [("amp",), ("k", "phase"), NAMES], [("rest",), ("omega", "damping"), ("k", "amp", "phase")]])
@pytest.mark.parametrize("side", [5, 14])
@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32C])
def test_parameter_updates_are_in_the_count(prec, side, order):
    sc = wl.rollout_request(side, 1)
    s = wl.make_sim(sc, prec)
    held = s.device_bytes()
    for names in order:
        s.set_spring_params(None, **{k: sc[k] for k in names})
        s.step(2)
        assert s.device_bytes() == held


def test_rollout_server_counts_reused_engines():
    reqs = [{"id": i, "arrival_s": 0.0, "side": 4 + 5 * (i % 2), "steps": 20, "seed": i} for i in range(12)]
    with serving.RolloutServer(tg.FP32C, max_active=3) as srv:
        _, stats = srv.run(reqs)
        assert stats["engines_built"] < len(reqs)
        for side, engines in srv.pool.items():
            assert engines and all(e.device_bytes() <= srv.bytes_of[side] for e in engines)
