"""One measure of volume and area wherever the correction takes it: the pass
that also forms the normals (from the second iteration on), the first pass, the
measuring mode and the adjoint's replay, so that all of them judge a state the
same way.  A cell that a step's correction moved was measured by its last pass
(rbc_cell_metrics after the step); the same stored positions, handed back to
the handle, are measured by the measuring mode: equal bit for bit."""
import dataclasses

import numpy as np
import pytest

from preprocess_src_b200 import configs
from tests.test_gpu_volume_moves import geodesic

pytestmark = pytest.mark.gpu


# 42, 642 and 2562 vertices (normals kept from pass to pass), 3242 (not)
@pytest.mark.parametrize("f", [2, 8, 16, 18])
def test_last_pass_equals_measuring_mode(native_lib, f):
    from preprocess_src_b200.step import Simulation
    v, t = geodesic(f)
    n = 8
    base = configs.small_duct(subdiv=1, flow=24)
    rng = np.random.default_rng(f)
    ref = [v * rng.uniform(3.0, 5.0, 3) + rng.uniform(-2.0, 2.0, 3) for _ in range(n)]
    moved = np.concatenate([(x - x.mean(0)) * rng.uniform(1.0001, 1.0004) + x.mean(0) for x in ref])
    case = dataclasses.replace(base, tri=t, xr=np.concatenate(ref).reshape(-1), ncell=n, vertex=len(v), element=len(t))
    with Simulation(case) as sim:
        sim.import_cells(*moved.T.copy(), xd=moved.reshape(-1))
        sim.step(1)
        assert sim.status()[1] > 2   # moves
        step = sim.cell_metrics()
        c = sim.export_cells()
        sim.import_cells(x=c["x"], y=c["y"], z=c["z"])
        again = sim.cell_metrics()
        for k in ("volume", "area"):
            np.testing.assert_array_equal(again[k], step[k], err_msg=k)
