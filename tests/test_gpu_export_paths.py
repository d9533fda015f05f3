"""Exports into page-locked buffers (written by the layout kernel) and into
pageable ones (staged copies) give the same bytes, for every choice of arrays,
for a buffer that starts inside its allocation, and for one that is pageable
beside page-locked ones.  The launch counter tells the paths apart: one kernel
writes all page-locked arrays of the cells, the staged path runs one conversion
each for fem->xd, the velocities, the forces and the centroids and none for the
positions.  Up to three arrays are always staged."""
import ctypes as C

import numpy as np
import pytest

from preprocess_src_b200 import _native as N
from preprocess_src_b200 import configs

pytestmark = pytest.mark.gpu


def _p(a):
    return None if a is None else a.ctypes.data_as(N._DP)


@pytest.mark.parametrize("ncell", [1, 3])
def test_pinned_equals_pageable(native_lib, ncell):
    import torch
    from preprocess_src_b200.step import Simulation

    def pinned(n, shift=0):
        return torch.full((n + shift,), np.nan, dtype=torch.float64, pin_memory=True).numpy()[shift:]

    case = configs.small_duct(subdiv=2, flow=36, ncell=ncell, radius=4.0, g=4e-5, Gs=2e-3)
    with Simulation(case) as sim:
        sim.step(5)
        cel, lat = sim.export_cells(), sim.export_lattice(fn=False)
        nv, n = sim.nv, case.n
        keys = ("x", "y", "z", "xd", "u", "v", "w", "fx", "fy", "fz", "gx")
        sizes = [nv] * 3 + [3 * nv] + [nv] * 6 + [3 * ncell]
        for pick, conversions in ((range(11), 4), ((0, 1, 2, 3, 4, 7), 3), ((3, 6, 9, 10), 4), ((0, 1, 2), 0), ((3, 10), 2),
                                  ((4, 6, 9), 2), ((7,), 1)):
            for loose in (None, 0):
                out = [None] * 11
                for j, k in enumerate(pick):
                    out[k] = np.full(sizes[k], np.nan) if j == loose else pinned(sizes[k], shift=j)
                before = sim.launches
                sim._call("rbc_export_ref_cells", *map(_p, out))
                direct = loose is None and len(pick) > 3
                assert sim.launches - before == (1 if direct else conversions), (list(pick), loose)
                for k in pick:
                    np.testing.assert_array_equal(out[k], cel[keys[k]], err_msg=f"{keys[k]} of {list(pick)}")
        for loose in (None, 2):
            out = [np.full(n, np.nan) if k == loose else pinned(n, shift=k) for k in range(4)]
            sim._call("rbc_export_ref_lattice", None, *map(_p, out))
            for o, k in zip(out, ("dn", "un", "vn", "wn")):
                np.testing.assert_array_equal(o, lat[k], err_msg=k)
        # an address that no double is aligned to is staged, not written by a kernel
        raw = torch.zeros(8 * nv + 8, dtype=torch.uint8, pin_memory=True)
        odd = C.cast(raw.data_ptr() + 4, N._DP)
        rest = [pinned(n) for n in (nv, nv, 3 * nv, nv)]
        before = sim.launches
        sim._call("rbc_export_ref_cells", odd, *map(_p, rest), *[None] * 6)
        assert sim.launches - before == 2
        np.testing.assert_array_equal(rest[3], cel["u"])
        np.testing.assert_array_equal(np.frombuffer(raw.numpy()[4:4 + 8 * nv].tobytes()), cel["x"])
        assert sim.cell_metrics()["volume"].shape == (ncell,)
