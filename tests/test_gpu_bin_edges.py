"""Whole bins at the sizes where the chain kernel's tilings change: N at and
beside multiples of 8, 16, 32 and 64, the largest that keeps a thread per
proposal (N = 128: 256 bonds) and the first ones past it, the largest
register- and shared-memory-resident ones (N = 140, 144) and the first
beyond (N = 160, 196); delayed-update ranks from one pair upward.  Each chain
against the C restatement of the reference path (oracle/c/z2cpu.c) from the
same seed: decisions, links and ranf state identical, G and observables within
1e-10 relative (the bar of the other parity tests)."""
import numpy as np
import pytest

from oracle import z2cpu
from z2_gauge_zfy_b200 import Chain, Z2Batch

pytestmark = pytest.mark.gpu
RTOL = 1e-10
SIZES = [(4, 4), (4, 6), (4, 8), (6, 6), (6, 10), (8, 8), (4, 18), (8, 10), (6, 16), (10, 10),
         (8, 14), (8, 16), (10, 14), (12, 12), (10, 16), (14, 14)]


@pytest.mark.parametrize("delay_k,stab_exact",
                         [(0, False), (1, False), (3, False), (64, False), (0, True)])
def test_bins_match_c_port(delay_k, stab_exact):
    chains = [Chain(RT=1.0, J=0.5, h=0.3 + 0.05 * i, mu=0.0 if i % 2 else 0.2, Nlx=lx, Nly=ly,
                    Ltrot=20, beta=2.0, Nwrap=5 if i % 3 else 10, seed=4001 + 2 * i)
              for i, (lx, ly) in enumerate(SIZES)]
    with Z2Batch(chains, record=True, delay_k=delay_k, stab_exact=stab_exact) as b:
        b.pre()
        b.sweep(1, False)
        gpu = [(b.green(i), b.obs_equal(i), b.decisions(i)[0], b.get_config(i), b.stats(i))
               for i in range(len(chains))]
    for ch, (G, obs, dec, (sig, iseed), st) in zip(chains, gpu):
        c = z2cpu.CpuChain.from_chain(ch)
        c.pre()
        _, o, d = c.bin(record=True)
        ref = c.state()
        c.close()
        tag = f"{ch.Nlx}x{ch.Nly} k={delay_k}"
        assert np.array_equal(dec, d), tag
        assert np.array_equal(sig, ref["sigma"]) and iseed == ref["iseed"], tag
        assert st["accepted"] == d.sum(), tag
        assert np.max(np.abs(G - ref["G"])) <= RTOL * np.max(np.abs(ref["G"])), tag
        for q, name in enumerate(obs):
            assert abs(obs[name] - o[q]) <= RTOL * max(abs(o[q]), 1.0), (tag, name)
