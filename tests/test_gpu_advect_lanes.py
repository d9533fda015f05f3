"""The advection with two and with four lanes per vertex gives the same bits: the
same cells step as one batch (whose blocks, taken together, take two lanes) and
one by one (four lanes), in the channel and in the shear box."""
import numpy as np
import pytest

from preprocess_src_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flow", ["duct", "shear"])
def test_two_lanes_equal_four(native_lib, flow):
    from preprocess_src_b200.step import Batch, Simulation
    n = 24   # x 16 patches: more blocks than two per multiprocessor
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
