"""GPU: the batch autotuner keeps the choices of batches with and without the limiter apart:
their stage launches are different kernels."""
import pytest

from fr_sdg_b200 import FRSolver
from fr_sdg_b200.batch import DeviceBatch
from fr_sdg_b200.workloads import circular_explosion

pytestmark = pytest.mark.gpu


def test_limited_batches_are_timed_by_themselves(cuda):
    times = []
    for limit in (False, True, False):
        wl = circular_explosion(77, 4, "ideal", 1.4, (0.0, 0.0), 0.25, 0.1)
        wl.cfg.pp_limit = int(limit)
        with FRSolver(wl.cfg) as s:
            U = wl.init(cuda)
            db = DeviceBatch([(s, U, wl.time_step(U), 1.0)])
            db.run(1)
            times.append([(g["tile_variant"], g["stage_ms"]) for g in db.tuning()])
            db.close()
    assert times[0] == times[2]  # the same kernels: the choice is kept
    assert times[0] != times[1]  # a time of its own
