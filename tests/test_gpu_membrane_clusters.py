"""The membrane pass with a cell as one block's work and as a cluster's of two or
four (few cells of more than 1024 vertices): a vertex's arithmetic is the same in
all of them, so copies of one cell get the same forces bit for bit whatever the
number of cells, in both precisions, and those match the FP64 oracle."""
import dataclasses

import numpy as np
import pytest

from preprocess_src_b200 import configs
from tests.test_gpu_parity import rel_l2
from tests.test_gpu_volume_moves import geodesic

pytestmark = pytest.mark.gpu


def _cells(f, n, fp64):
    """n copies of a stretched geodesic ellipsoid (stress() sees each cell alone)."""
    v, t = geodesic(f)
    x = v * [5.0, 4.0, 3.0] + [0.3, -0.2, 1.0]
    base = configs.small_duct(subdiv=1, flow=24, membrane_fp64=fp64)
    case = dataclasses.replace(base, tri=t, xr=np.tile(x.reshape(-1), n), ncell=n, vertex=len(v), element=len(t))
    moved = (x - x.mean(0)) * [1.01, 0.997, 0.992] + x.mean(0)
    moved += 1e-3 * np.sin(7 * x[:, ::-1])
    return case, moved


# 1002 vertices: one block; 1212, 2562 and 3242: clusters of four for up to a fifth of the multiprocessors, of two for up to half
@pytest.mark.parametrize("fp64", [0, 1])
@pytest.mark.parametrize("f", [10, 11, 16, 18])
def test_forces_do_not_depend_on_the_number_of_cells(native_lib, oracle_mod, f, fp64):
    import torch
    from preprocess_src_b200.step import Simulation
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    first = None
    for n in (1, sms // 5, sms // 5 + 1, sms // 2, sms // 2 + 1):
        case, x = _cells(f, n, fp64)
        with Simulation(case) as sim:
            xs = [np.tile(x[:, k], n) for k in range(3)]
            sim.import_cells(x=xs[0], y=xs[1], z=xs[2], xd=np.tile(x.reshape(-1), n))
            sim.stress()
            c = sim.export_cells()
            assert sim.status()[0] == 0
        force = np.stack([c[k].reshape(n, -1) for k in ("fx", "fy", "fz")], axis=1)
        if first is None:
            first = force[0]
            o = oracle_mod.Oracle(case)
            for k, a in enumerate("xyz"):
                o.a[a][:] = x[:, k]
            o.a["xd"][:] = x.reshape(-1)
            o.stress()
            assert rel_l2(first, np.stack([o["cfx"], o["cfy"], o["cfz"]])) <= 7e-6   # as test_gpu_parity.py
        for k in range(n):
            np.testing.assert_array_equal(force[k], first, err_msg=f"{n} cells, cell {k}")
