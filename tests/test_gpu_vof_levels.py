"""The front-tracking solve over the shapes its grid levels can take: a
coarsest level in shared memory and one that is too large for it (an odd
periodic length does not coarsen: 495 nodes at a length of 55, 513 at 57 and at
114), odd cross-sections, extents that coarsen
unevenly, and the shear box with its periodic x.  The volume fraction at
rbc_create against the FP64 oracle's solve of the same system, both to
|r| / |b| < 1e-12: 1e-9 leaves a condition number of 1e3."""
import numpy as np
import pytest

from preprocess_src_b200 import configs

pytestmark = pytest.mark.gpu

KW = dict(lambda1=3.0, vof_k=10, vof_residual=1e-12)


def _case(shape):
    kind, L, w, h = shape
    if kind == "shear":
        return configs.shear_case("levels", w, h, L, centers=[(0.3, -0.2, 0.4)], subdiv=2, radius=4.0, seed=3, **KW)
    return configs.duct_case("levels", L, w, h, centers_duct=[(L / 2 + 0.3, w / 2 - 0.2, h / 2 + 0.1)], subdiv=2,
                             radius=4.0, seed=3, **KW)


@pytest.mark.parametrize("shape", [("duct", 32, 20, 20), ("duct", 61, 21, 19), ("duct", 131, 20, 22), ("duct", 55, 20, 20), ("duct", 57, 20, 20), ("duct", 114, 20, 20), ("duct", 12, 17, 40),
                                   ("shear", 24, 22, 20), ("shear", 26, 21, 18)])
def test_front_tracking_matches_oracle(native_lib, oracle_mod, shape):
    from preprocess_src_b200.step import Simulation
    case = _case(shape)
    o = oracle_mod.Oracle(case)
    with Simulation(case) as sim:
        vf, _ = sim.export_vof()
        assert sim.status()[0] == 0
    err = np.abs(vf - o["vf"]).max()
    print(f"{shape}: max |dvf| {err:.2e}")
    assert err <= 1e-9
