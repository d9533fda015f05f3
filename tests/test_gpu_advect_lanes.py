"""The advection gives a vertex the same bits however its launch is cut: two or
four lanes per vertex, patches of any level (both follow the number of cells and
the device's multiprocessors), in one launch per simulation or one for a batch."""
import dataclasses

import numpy as np
import pytest

from preprocess_src_b200 import configs
from tests.test_gpu_volume_moves import geodesic

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("flow", ["duct", "shear"])
def test_two_lanes_equal_four(native_lib, flow):
    from preprocess_src_b200.step import Batch, Simulation
    n = 3 * _sms() // 16   # 16 patches of 41 vertices per cell: above two blocks per multiprocessor, at most three
    assert 2 * _sms() < 16 * n <= 3 * _sms()
    rng = np.random.default_rng(3)
    if flow == "duct":
        cases = [configs.small_duct(subdiv=3, flow=24, radius=4.0, seed=i, g=4e-5, Gs=float(rng.uniform(1e-3, 3e-3)))
                 for i in range(n)]
    else:
        cases = [configs.shear_case("s", 20, 18, 20, centers=[(9.3, 0.2, float(rng.uniform(-9, 9)))], sr=4e-3, subdiv=3,
                                    radius=4.0, seed=i, Gs=2e-3) for i in range(n)]
    alone = [Simulation(c) for c in cases]
    sims = [Simulation(c) for c in cases]
    batch = Batch(sims)
    assert batch.fused
    batch.step(7)
    for a, b in zip(alone, sims):
        a.step(7)
        ca, cb = a.export_cells(), b.export_cells()
        for k in ("x", "y", "z", "xd", "u", "v", "w"):
            np.testing.assert_array_equal(ca[k], cb[k], err_msg=k)
    batch.close()
    for s in alone + sims:
        s.close()


# 162, 642, 1212 and 2562 vertices; copies of one cell from a few blocks to more than eight per multiprocessor,
# either side of two and three blocks per multiprocessor at each patch level of 148 of them
@pytest.mark.parametrize("flow", ["duct", "shear"])
@pytest.mark.parametrize("f,counts", [(4, (1, 74, 75, 111, 112, 300, 1200)), (8, (1, 18, 19, 27, 28, 37, 38, 55, 60, 74, 110, 150, 300)),
                                      (11, (1, 20, 60, 112, 300)), (16, (1, 9, 10, 18, 20, 28, 38, 56, 100, 149, 150))])
def test_copies_of_a_cell_get_the_same_bits(native_lib, flow, f, counts):
    from preprocess_src_b200.step import Simulation
    v, t = geodesic(f)
    # in the shear box the cell lies across the periodic x and z
    x = v * [5.0, 4.0, 3.0] + ([9.0, 0.2, 11.0] if flow == "shear" else [0.3, -0.2, 1.0])
    base = configs.shear_case("s", 20, 18, 24, sr=4e-3) if flow == "shear" else configs.small_duct(subdiv=1, flow=24)
    fn = first = None
    for n in counts:
        case = dataclasses.replace(base, tri=t, xr=np.tile(x.reshape(-1), n), ncell=n, vertex=len(v), element=len(t))
        with Simulation(case) as sim:
            if fn is None:   # populations that make a rough velocity field
                fn = sim.export_lattice(fn=True, macro=False)["fn"]
                fn = fn * (1 + 0.2 * np.random.default_rng(1).standard_normal(fn.shape))
            p = case.params
            y = x.copy()
            for k, lo, hi, length in ((0, "xmin", "xmax", "LX"), (2, "zmin", "zmax", "LZ")):
                if k == 2 or flow == "shear":
                    y[:, k] = (y[:, k] - p[lo]) % p[length] + p[lo]
            sim.import_cells(*np.tile(y, (n, 1)).T.copy(), xd=np.tile(y.reshape(-1), n))
            sim.import_lattice(fn)
            sim.lbm_d3q19()
            sim.ibm_st2()
            c = sim.export_cells()
            got = np.stack([c[k].reshape(n, -1) for k in ("x", "y", "z", "u", "v", "w")], axis=1)
            assert sim.status()[0] == 0
        if first is None:
            first = got[0]
            assert np.abs(first[3:]).max() > 1e-3
        for k in range(n):
            np.testing.assert_array_equal(got[k], first, err_msg=f"{n} cells, cell {k}")
