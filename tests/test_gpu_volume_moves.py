"""The volume correction's moves over cell sizes: blocks narrower and wider than
the cell, several vertices per thread, and a cell whose unit normals do not fit
a block's shared memory beside its positions.  Each cell is scaled so that the
loop moves it a dozen times; iteration count and positions against the FP64
oracle (the same loop in FP64: 1e-9, as in test_gpu_parity.py)."""
import dataclasses

import numpy as np
import pytest

from preprocess_src_b200 import configs, mesh

pytestmark = pytest.mark.gpu


def geodesic(f):
    """Icosahedron with every face cut into f^2 triangles: 10 f^2 + 2 vertices of valence 5 or 6 on the unit sphere."""
    v0, t0 = mesh.icosahedron()
    ids, verts, tris = {}, [], []

    def vid(face, i, j):
        w = {}
        for n, k in zip(face, (f - i - j, i, j)):
            if k:
                w[int(n)] = k
        key = tuple(sorted(w.items()))
        if key not in ids:
            ids[key] = len(verts)
            p = sum(v0[n] * k for n, k in w.items())
            verts.append(p / np.linalg.norm(p))
        return ids[key]

    for face in t0:
        for i in range(f):
            for j in range(f - i):
                tris.append((vid(face, i, j), vid(face, i + 1, j), vid(face, i, j + 1)))
                if i + j < f - 1:
                    tris.append((vid(face, i + 1, j), vid(face, i + 1, j + 1), vid(face, i, j + 1)))
    v = np.array(verts)
    return v, mesh.orient_outward(v, np.array(tris, dtype=np.int32))


# 10 f^2 + 2 vertices: 12, 42, 1002 and 1212 (either side of 1024 threads), 3242 (normals do not fit)
@pytest.mark.parametrize("f", [1, 2, 10, 11, 18])
def test_moves_match_oracle(native_lib, oracle_mod, f):
    from preprocess_src_b200.step import Simulation
    v, t = geodesic(f)
    v = v * [1.0, 0.8, 0.6]
    base = configs.small_duct(subdiv=1, flow=24)
    x = v * 5.0 + [0.3, -0.2, 4.0]
    case = dataclasses.replace(base, tri=t, xr=x.reshape(-1), ncell=1, vertex=len(v), element=len(t))
    o = oracle_mod.Oracle(case)
    moved = (x - x.mean(0)) * 1.0004 + x.mean(0)
    for k, n in enumerate("xyz"):
        o.a[n][:] = moved[:, k]
    with Simulation(case) as sim:
        sim.import_cells(x=o["x"], y=o["y"], z=o["z"], gx=o["gx"])
        it_ref, it = o.volume_correction(), sim.volume_correction()
        got = sim.export_cells()
        assert it == it_ref and it > 5, (it, it_ref)
        assert max(np.abs(got[n] - o[n]).max() for n in "xyz") <= 1e-9
        assert sim.status()[0] == 0
