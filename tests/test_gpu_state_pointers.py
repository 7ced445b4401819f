"""States handed over as device, page-locked and pageable memory, of a small
grid (moved through the context's pinned array) and of a larger one: the same
bits."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("nx,ny", [(40, 33), (128, 128), (150, 140)])
def test_device_and_host_arrays_hold_the_same_state(cfsb, workloads, prec, nx, ny):
    import torch

    U = workloads.riemann_quadrants(nx, ny, seed=4).U0
    dev = torch.from_numpy(U.copy()).cuda()
    pin = torch.from_numpy(U.copy()).pin_memory()
    arrays = {"pageable": U.ctypes.data, "pinned": pin.data_ptr(), "device": dev.data_ptr()}
    outs = {"pageable": np.zeros_like(U), "pinned": torch.zeros(U.shape, dtype=torch.float64).pin_memory(),
            "device": torch.zeros(U.shape, dtype=torch.float64, device="cuda")}
    torch.cuda.synchronize()
    got = {}
    for name, src in arrays.items():
        out = outs[name]
        dst = out.ctypes.data if isinstance(out, np.ndarray) else out.data_ptr()
        with cfsb.Solver(nx, ny, precision=prec, rk=cfsb.RK_TVD2) as s:
            lib = cfsb.load_library()
            as_p = lambda a: ctypes.cast(a, ctypes.POINTER(ctypes.c_double))  # noqa: E731
            assert lib.cfs_set_state(s._ctx, as_p(src)) == 0
            s.step(1e-4)
            assert lib.cfs_get_state(s._ctx, as_p(dst)) == 0
        got[name] = out if isinstance(out, np.ndarray) else out.cpu().numpy()
    assert np.all(np.isfinite(got["pageable"])) and not np.array_equal(got["pageable"], U)
    assert np.array_equal(got["pinned"], got["pageable"]) and np.array_equal(got["device"], got["pageable"])
