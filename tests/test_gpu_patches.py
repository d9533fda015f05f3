"""Spread and advection over the surface patches a population is cut into.

The patches follow the number of cells (each launch takes the smallest ones
whose blocks are resident at once, the spread down to eight patches a cell), so
the same step is checked against the FP64 oracle for cells that stay whole, for
the smallest patches, and for populations on both sides of the lines.
Tolerances per step as in test_gpu_parity.py."""
import numpy as np
import pytest

from preprocess_src_b200 import configs
from tests.test_gpu_parity import comp, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("subdiv,ncell,flow", [(1, 1, 24), (2, 1, 24), (3, 2, 40), (4, 1, 32), (2, 70, 200), (3, 30, 200), (3, 60, 200)])
def test_step_matches_oracle(native_lib, oracle_mod, subdiv, ncell, flow):
    from preprocess_src_b200.step import Simulation
    if ncell <= 2:
        case = configs.small_duct(subdiv=subdiv, flow=flow, ncell=ncell, g=4e-5, Gs=2e-3)
    else:
        case = configs.suspension_case("patches", flow, 44, 44, ncell, subdiv=subdiv, radius=3.5, wall_margin=2.0,
                                       g=4e-5, Gs=2e-3, seed=8)
    o = oracle_mod.Oracle(case)
    o.step(6)
    with Simulation(case) as sim:
        sim.import_lattice(o.fn)
        sim.import_cells(x=o["x"], y=o["y"], z=o["z"], xd=o["xd"], nd=o["nd"], volume0=o["volume0"], gx=o["gx"])
        sim.iter = o.iter
        o.step(1)
        sim.step(1)
        cel, lat = sim.export_cells(), sim.export_lattice(fn=False)
        flags = sim.status()[0]
    m = comp(case)
    v = lambda d, k: np.concatenate([d[a][m] if k else d[a] for a in (("un", "vn", "wn") if k else "uvw")])  # noqa: E731
    dx = max(np.abs(cel[k] - o[k]).max() for k in "xyz")
    print(f"subdiv {subdiv}, {ncell} cells: velocity {rel_l2(v(lat, 1), v(o, 1)):.2e}, vertices {rel_l2(v(cel, 0), v(o, 0)):.2e}, dx {dx:.2e}")
    assert flags & 0xF == 0
    assert rel_l2(v(lat, 1), v(o, 1)) <= 8e-7
    assert rel_l2(v(cel, 0), v(o, 0)) <= 8e-7
    assert dx <= 3e-9
