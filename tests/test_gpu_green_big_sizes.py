"""The four blocks of z2_stab_green_big at the edges of the inverse's panels
and tiles (N = 16 ... 256) and above them (N = 288: the blocked LU), against the
dense formulas with B = UR DR VR, A = VL DL UL:
  G00 = (1 + A B)^-1, Gtt = (1 + B A)^-1, Gt0 = Gtt B, G0t = -G00 A.
D spans e^{+-1} and the V factors are close to unit triangles, so the dense
inverses lose at most three digits: 1e-12 relative to the largest entry."""
import numpy as np
import pytest

from z2_gauge_zfy_b200 import Chain, Z2Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly", [(4, 4), (4, 6), (6, 6), (10, 10), (8, 16), (10, 14), (12, 12),
                                   (12, 14), (16, 16), (16, 18)])
def test_blocks_match_dense(Lx, Ly):
    N = Lx * Ly
    rng = np.random.default_rng(N)
    UR, _ = np.linalg.qr(rng.standard_normal((N, N)))
    UL, _ = np.linalg.qr(rng.standard_normal((N, N)))
    DR, DL = (np.exp(rng.uniform(-1, 1, N)) for _ in range(2))
    VR, VL = (np.eye(N) + 0.1 * np.triu(rng.standard_normal((N, N)), 1) / np.sqrt(N) for _ in range(2))
    B, A = UR @ np.diag(DR) @ VR, VL @ np.diag(DL) @ UL
    G00 = np.linalg.inv(np.eye(N) + A @ B)
    Gtt = np.linalg.inv(np.eye(N) + B @ A)
    with Z2Batch([Chain(Nlx=Lx, Nly=Ly, Ltrot=2, beta=0.2, Nwrap=1, seed=3)]) as b:
        got = b.stab_green_big(0, UR, DR, VR, UL, DL, VL)
    for name, g, ref in zip(("G00", "G0t", "Gt0", "Gtt"), got, (G00, -G00 @ A, Gtt @ B, Gtt)):
        assert np.max(np.abs(g - ref)) <= 1e-12 * np.max(np.abs(ref)), name
