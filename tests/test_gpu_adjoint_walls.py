"""The adjoint's store of the velocity field where a cell interpolates from
wall nodes that no collide-stream warp writes (a warp of wall nodes alone stores
nothing): the recomputation and the reverse sweep must read zero velocity there,
whatever the memory held before."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from preprocess_src_b200 import configs
from tests.test_gpu_adjoint import REL_TOL, _Run, _stretched

pytestmark = pytest.mark.gpu


def _leave_in_memory(byte, nbytes, blocks=48):
    """Freed device blocks of nbytes, all bytes the same, for the next allocations of that size to land in."""
    rt = C.CDLL("libcudart.so.12")
    ptrs = []
    for _ in range(blocks):
        p = C.c_void_p()
        assert rt.cudaMalloc(C.byref(p), C.c_size_t(nbytes)) == 0
        assert rt.cudaMemset(p, byte, C.c_size_t(nbytes)) == 0
        ptrs.append(p)
    assert rt.cudaDeviceSynchronize() == 0
    for p in ptrs:
        assert rt.cudaFree(p) == 0


# Widths whose wall rows hold warps of wall nodes alone (at 32 each row is one warp); the cell's
# lowest (highest) vertices lie 1.3 spacings from that row
@pytest.mark.parametrize("nsteps", [1, 2])
@pytest.mark.parametrize("width,top", [(32, False), (40, True)])
def test_wall_nodes_of_the_store(native_lib, width, top, nsteps):
    import torch
    from preprocess_src_b200.step import Simulation
    torch.zeros(1, device="cuda")   # the process's context and its CUDA runtime
    case = configs.duct_case("walls", 24, width, 20, centers_duct=[(12.0, width / 2.0, 10.0)], subdiv=2, radius=4.0, seed=2,
                             g=2e-5, Gs=5e-3)
    x0 = _stretched(case)
    hy = (case.params["ny"] - 1) / 2.0
    shift = np.array([0.0, hy - 1.3 - x0[1].max() if top else 1.3 - hy - x0[1].min(), 0.0])
    case = dataclasses.replace(case, xr=(case.xr.reshape(-1, 3) + shift).reshape(-1))
    x0 = x0 + shift[:, None]
    adj = []
    for byte in (0x00, 0x3F):   # velocities of 0 and of 0.75
        with Simulation(case) as sim:
            run = _Run(sim, x0, nsteps, nsteps)
            _leave_in_memory(byte, 2 * nsteps * 16 * 24 * width * 20)   # the store's two slots per step
            adj.append(run.adjoint(want_x0=True))
            d = np.random.default_rng(5).standard_normal(x0.shape)
            fd = (run.loss(x0=x0 + 1e-3 * d) - run.loss(x0=x0 - 1e-3 * d)) / 2e-3
    print(f"dL/dx0 . d: {[float((a['dx0'] * d).sum()) for a in adj]}, central {fd:.9e}; dL/dP {[a['grad'][0] for a in adj]}")
    for a in adj:
        assert abs(float((a["dx0"] * d).sum()) - fd) <= REL_TOL * abs(fd)
    # equal up to the order of the reverse sweep's FP32 atomics, as in test_gpu_adjoint.py
    np.testing.assert_allclose(adj[1]["grad"], adj[0]["grad"], rtol=2e-5)
    np.testing.assert_allclose(adj[1]["dx0"], adj[0]["dx0"], rtol=0, atol=2e-5 * np.abs(adj[0]["dx0"]).max())
