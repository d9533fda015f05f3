"""Gradients for cells of every block shape of the membrane's reverse solve and
for several cells, in runs whose volume corrections move, against central
differences (relative steps of 3e-2 for the drive, in which the positions are
nearly linear, and 1e-3 for the stiffnesses: round-off of the FP32 forward and
truncation stay below 6e-4 at these sizes).  The loss weighs the cells'
elongation, so that the derivatives do not cancel over the vertices."""
import dataclasses

import numpy as np
import pytest

from preprocess_src_b200 import configs
from tests.test_gpu_adjoint import REL_TOL, _Run
from tests.test_gpu_volume_moves import geodesic

pytestmark = pytest.mark.gpu


# 10 f^2 + 2 vertices: 642 (one vertex per thread of the reverse solve), 1212 (two), 2562 (three), 3242 (four)
@pytest.mark.parametrize("f,ncell", [(8, 3), (11, 1), (16, 1), (16, 2), (18, 1)])
def test_gradients_match_central_differences(native_lib, f, ncell):
    from preprocess_src_b200.step import Simulation
    v, t = geodesic(f)
    v = v * [5.0, 4.0, 3.0]
    base = configs.small_duct(subdiv=1, flow=16 + 16 * ncell, g=2e-5, Gs=5e-3)
    LZ = base.params["LZ"]
    x = np.concatenate([v + [0.3 - 0.2 * c, -0.2, -LZ / 2 + LZ * (c + 0.5) / ncell] for c in range(ncell)])
    case = dataclasses.replace(base, tri=t, xr=x.reshape(-1), ncell=ncell, vertex=len(v), element=len(t))
    mean = x.reshape(ncell, -1, 3).mean(1).repeat(len(v), axis=0)
    x0 = ((x - mean) * [1.03, 1 / 1.03, 1.0] + mean).T.copy()
    with Simulation(case) as sim:
        run = _Run(sim, x0, 12, 5)
        run.r = (x0 - mean.T) * np.array([1.0, -2.0, 0.5])[:, None] + 0.3
        adj = run.adjoint(want_x0=True)
        assert adj["flags"] == 0 and 2 <= sim.status()[1] <= 16   # moves of a correction, all reversed
        for k, i, rel in (("P", 0, 3e-2), ("B", 1, 1e-3), ("C_", 2, 1e-3)):
            h = rel * abs(run.theta0[k])
            fd = (run.loss(**{k: run.theta0[k] + h}) - run.loss(**{k: run.theta0[k] - h})) / (2 * h)
            print(f"d/d{k}: adjoint {adj['grad'][i]:.9e}  central {fd:.9e}  rel {abs(adj['grad'][i] - fd) / abs(fd):.2e}")
            assert abs(adj["grad"][i] - fd) <= REL_TOL * abs(fd), k
        d = run.r / np.abs(run.r).max()
        fd = (run.loss(x0=x0 + 3e-4 * d) - run.loss(x0=x0 - 3e-4 * d)) / 6e-4
        dx = float((adj["dx0"] * d).sum())
        print(f"dL/dx0 . d: adjoint {dx:.9e}  central {fd:.9e}  rel {abs(dx - fd) / abs(fd):.2e}")
        assert abs(dx - fd) <= REL_TOL * abs(fd)
