"""Launches of more chains than the GPU has SMs on lattices of up to 64 sites
run on 128-thread blocks: the same chains in handles small enough for the
256-thread kernel (which the other parity tests pin against the oracle) give
the same decisions, links, ranf state and acceptance, and G and observables to
1e-10, through the start, a bin with the time-displaced pass, warm-up and
global moves.  Sizes at the tilings' edges (N = 16 ... 64), one and several
blocks per SM."""
import numpy as np
import pytest

from z2_gauge_zfy_b200 import Chain, Z2Batch

pytestmark = pytest.mark.gpu
RTOL = 1e-10
SIZES = [(4, 4), (4, 6), (2, 8), (4, 8), (6, 6), (4, 12), (6, 10), (8, 8), (4, 16)]


def _run(chains, tau):
    out = []
    with Z2Batch(chains, record=True, tau=tau) as b:
        acc = b.therm(2)
        b.pre()
        b.sweep_global(2)
        b.sweep(1, tau)
        obs = b.obs_equal_all()
        for i in range(len(chains)):
            out.append((acc[i], obs[i], b.green(i), b.decisions(i)[0], b.get_config(i),
                        b.global_stats(i), b.obs_tau(i) if tau else {}))
    return out


@pytest.mark.parametrize("n,sizes,tau", [(160, SIZES[:1], False), (333, SIZES, False),
                                         (700, SIZES[:4], False), (160, SIZES[4:], True)])
def test_small_blocks_match(n, sizes, tau):
    chains = [Chain(RT=1.0, J=0.5, h=0.3 + 0.5 * (i % 7) / 7, mu=0.2 if i % 3 == 0 else 0.0,
                    Nlx=sizes[i % len(sizes)][0], Nly=sizes[i % len(sizes)][1], Ltrot=10, beta=1.0,
                    Nwrap=5, seed=7001 + 2 * i) for i in range(n)]
    got = _run(chains, tau)
    ref = []
    for k in range(0, n, 100):
        ref += _run(chains[k:k + 100], tau)
    for ch, g, r in zip(chains, got, ref):
        tag = f"{ch.Nlx}x{ch.Nly} seed {ch.seed}"
        assert g[0] == r[0], tag
        assert np.array_equal(g[3], r[3]), tag
        assert np.array_equal(g[4][0], r[4][0]) and g[4][1] == r[4][1], tag
        assert g[5] == r[5], tag
        assert np.max(np.abs(g[2] - r[2])) <= RTOL * np.max(np.abs(r[2])), tag
        assert np.all(np.abs(g[1] - r[1]) <= RTOL * np.maximum(np.abs(r[1]), 1.0)), tag
        for k in r[6]:
            assert np.max(np.abs(g[6][k] - r[6][k])) <= RTOL * max(np.max(np.abs(r[6][k])), 1.0), (tag, k)
