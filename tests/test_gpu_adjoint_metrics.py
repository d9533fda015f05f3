"""What a handle reports after a reverse sweep is the state it is left in."""
import numpy as np
import pytest

from preprocess_src_b200 import configs
from tests.test_gpu_adjoint import _Run

pytestmark = pytest.mark.gpu


def test_metrics_after_a_binomial_sweep(native_lib):
    """The sweep steps the handle back and forth and leaves it at the run's end: the metrics read then are that state's."""
    from preprocess_src_b200.step import Simulation
    case = configs.small_duct(subdiv=2, radius=5.0, flow=32, width=20, g=2e-5, Gs=5e-3)
    with Simulation(case) as sim:
        run = _Run(sim, None, 12, 1)
        run.init.restore(sim)
        sim.adjoint_record_binomial(12, 1, 2)
        end = sim.cell_metrics()
        sim.adjoint_backward(run.r[0], run.r[1], run.r[2])
        after = sim.cell_metrics()
        # measured anew from the stored positions: FP64 sums over the wrapped positions, 1e-13 of the largest
        for k in ("volume", "area", "centroid"):
            np.testing.assert_allclose(after[k], end[k], rtol=0, atol=1e-12 * max(1.0, np.abs(end[k]).max()), err_msg=k)
