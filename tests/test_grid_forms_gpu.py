"""Every form of the resident grid, named by what it reports, against the
per-step kernels bit for bit with actuated springs: CTAs of 128, 256 and 512
threads, tables in shared memory or not, FP64 with a lane per component or a
thread per mass, and scenes just above what it takes.  Each call has to have
run in the form that is compared."""
import numpy as np
import pytest

import titan_gb300 as tg
from tests.test_resident_grid_gpu import same, scene
from titan_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

# precision, masses per axis, tile size asked for, (threads, staged, lanes) or None: too large
FORMS = [
    (tg.FP64, (9, 8, 13), 0, (256, 1, 1)),
    (tg.FP64, (18, 17, 15), 0, (512, 1, 1)),
    (tg.FP64, (24, 24, 24), 0, (512, 1, 0)),
    (tg.FP64, (31, 30, 29), 0, (512, 0, 0)),
    (tg.FP64, (33, 32, 33), 0, (256, 0, 0)),
    (tg.FP64, (37, 37, 37), 0, None),
    (tg.FP32, (9, 8, 13), 0, (128, 1, 0)),
    (tg.FP32, (24, 24, 24), 0, (256, 1, 0)),
    (tg.FP32, (37, 37, 37), 0, (256, 0, 0)),
    (tg.FP32, (16, 15, 14), 288, (512, 1, 0)),
    (tg.FP32, (16, 15, 14), 400, (512, 0, 0)),
    (tg.FP32, (40, 40, 40), 0, None),
    (tg.FP32C, (9, 8, 13), 0, (128, 1, 0)),
    (tg.FP32C, (24, 24, 24), 0, (256, 1, 0)),
    (tg.FP32C, (39, 40, 39), 0, (256, 0, 0)),
    (tg.FP32C, (16, 15, 14), 512, (512, 0, 0)),
    (tg.FP32C, (40, 40, 40), 0, None),
]


@pytest.mark.parametrize("integ", [tg.EULER, tg.VERLET, tg.RK2])
@pytest.mark.parametrize("prec,shape,tile,form", FORMS)
def test_bits_of_the_per_step_kernels(prec, shape, tile, form, integ):
    sc = scene(*shape, seed=sum(shape), fixed=0.05, act=0.3)
    sc["integrator"] = integ
    got = []
    for resident in (None, (0, 0, 0)):
        s = wl.make_sim(sc, prec, tile, resident=resident)
        info = s.grid_info()
        here = resident is None and form is not None
        if here:
            assert (info["active"], info["threads"], info["staged"], info["lanes"]) == (1, *form)
        else:
            assert info["active"] == 0
        for n in (2, 1, 7, 3, 1, 12):
            s.step(n)
            assert s.grid_info()["last"] == (0 if not here else 1 if n > 1 else 2 * info["single"])
        got.append(s.get_state(acc=True, T=True))
        s.close()
    assert np.isfinite(got[1]["pos"]).all()
    same(*got)
