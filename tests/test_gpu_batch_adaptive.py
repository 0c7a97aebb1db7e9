"""GPU: adaptive steps of the batch engine in explosions with limited elements: the FP64 and the
mixed form bound the wave speed by the same nodes, so their clocks agree as far as their states."""
import pytest

from fr_sdg_b200.batch import BatchedInstances, load_manifest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [2, 6])
def test_both_forms_take_the_same_steps(steps, cuda):
    specs = [s for s in load_manifest() if s.n_elems <= 48][:24]
    times = []
    for mixed in (False, True):
        bi = BatchedInstances(specs, cuda, mixed=mixed)
        bi.run_persistent(0.25, n_steps=steps)
        times.append(bi.times)
        bi.close()
    # the states differ by FP32 rounding of the residual, 6e-8 of its terms a step
    assert all(abs(a - b) <= 1e-4 * b for a, b in zip(*times))
