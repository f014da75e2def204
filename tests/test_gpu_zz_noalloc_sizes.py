"""The allocation-free stab_green at sizes no lattice has (odd N, N below one
panel, remainders of every tile) and on buffers that are only 8-byte aligned,
against numpy's (I + UR DR VR VL DL UL)^-1.  D spans e^{+-1} and the
triangular factors are close to unit ones, so the dense inverse loses at most
three digits (condition below 1e3): 1e-12 relative for both."""
import ctypes as C

import numpy as np
import pytest

from z2_gauge_zfy_b200 import _ffi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 9, 13, 35, 36, 63, 100, 129, 143])
@pytest.mark.parametrize("nt", [3, 9])
def test_noalloc_any_size(N, nt):
    torch = pytest.importorskip("torch")
    lib = _ffi.load()
    rng = np.random.default_rng(N)
    UR, _ = np.linalg.qr(rng.standard_normal((N, N)))
    UL, _ = np.linalg.qr(rng.standard_normal((N, N)))
    DR, DL = (np.exp(rng.uniform(-1, 1, N)) for _ in range(2))
    VR, VL = (np.eye(N) + 0.1 * np.triu(rng.standard_normal((N, N)), 1) / np.sqrt(N) for _ in range(2))
    ref = np.linalg.inv(np.eye(N) + UR @ np.diag(DR) @ VR @ VL @ np.diag(DL) @ UL)
    # one element of padding in front: 8-byte aligned starts
    dev = []
    for a in (UR, DR, VR, UL, DL, VL):
        t = torch.zeros(a.size + 1, dtype=torch.float64, device="cuda")
        t[1:] = torch.tensor(np.ascontiguousarray(a.T).ravel(), device="cuda")
        dev.append(t)
    G = torch.full((N * N + 1,), float("nan"), dtype=torch.float64, device="cuda")
    rc = lib.z2_stab_green_noalloc(N, nt, 10, *[C.c_void_p(t.data_ptr() + 8) for t in dev],
                                   C.c_void_p(G.data_ptr() + 8), None)
    assert rc == 0
    torch.cuda.synchronize()
    got = G[1:].cpu().numpy().reshape(N, N).T
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
