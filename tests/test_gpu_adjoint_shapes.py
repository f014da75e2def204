"""The adjoint of log det on every way its propagator and factorizations take:
rectangular lattices both ways (the group-2 partner of a bond is found from Lx and
Ly), sides of 2 and above 16 (group by group instead of by lines), G in global
memory (N = 160) and above the panel kernels (N = 288: the pivoted QR).  Against the
oracle's factor-by-factor gradient; bounds as at the square size
(tests/test_gpu_sizes.py)."""
import numpy as np
import pytest

from oracle import z2_oracle as zo
from z2_gauge_zfy_b200 import Chain, Z2Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly,Ltrot", [(4, 6, 20), (6, 4, 20), (8, 12, 20), (12, 8, 20), (2, 2, 20),
                                         (2, 8, 20), (8, 2, 20), (4, 20, 10), (18, 4, 10), (10, 16, 10),
                                         (16, 18, 10)])
def test_adjoint_matches_oracle(Lx, Ly, Ltrot):
    N = Lx * Ly
    rng = np.random.default_rng(N + Lx)
    rt = 1.0 + 0.05 * rng.standard_normal(2 * N)
    ch = Chain(RT=1.0, J=0.5, h=0.5, mu=0.1, Nlx=Lx, Nly=Ly, Ltrot=Ltrot, beta=0.1 * Ltrot, Nwrap=5,
               seed=515, rt_bond=rt)
    p = zo.Params(RT=rt, J=ch.J, h=ch.h, mu=ch.mu, Q=ch.Q, Nlx=Lx, Nly=Ly, Ltrot=Ltrot, beta=ch.beta,
                  Nwrap=5, absolute=ch.absolute)
    sig, _, _ = zo.seeded_config(p, zo.Lattice(Lx, Ly), ch.seed)
    ld_o, g_o, dmu_o = zo.logdet_grad_oracle(p, sig)
    with Z2Batch([ch]) as b:
        ld, g, dmu = b.logdet_grad(0)
    assert abs(ld - ld_o) <= 1e-10 * abs(ld_o)
    assert np.max(np.abs(g - g_o)) <= 1e-9 * np.max(np.abs(g_o))
    assert abs(dmu - dmu_o) <= 1e-10 * abs(dmu_o)
