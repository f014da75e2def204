"""Handles with different shared-memory needs side by side: a handle made later,
or a tuner call, leaves the launches of an earlier and larger one as they were
(both builds of the chain kernel)."""
import numpy as np
import pytest

from z2_gauge_zfy_b200 import Chain, Z2Batch, tune

pytestmark = pytest.mark.gpu


def _chains(n, Lx, Ly):
    return [Chain(RT=1.0, J=0.5, h=0.5, Nlx=Lx, Nly=Ly, Ltrot=10, beta=1.0, Nwrap=5, seed=901 + 2 * i)
            for i in range(n)]


def _small():
    return Z2Batch(_chains(1, 4, 4))


def _small_batch():
    return Z2Batch(_chains(160, 4, 4))


def _tuner():
    tune(_chains(1, 4, 4))


@pytest.mark.parametrize("n,L,delay_k", [(1, 10, 0), (1, 12, 0), (160, 8, 64)])
@pytest.mark.parametrize("later", [_small, _small_batch, _tuner])
def test_a_later_smaller_handle_changes_nothing(n, L, delay_k, later):
    with Z2Batch(_chains(n, L, L), delay_k=delay_k) as ref, Z2Batch(_chains(n, L, L), delay_k=delay_k) as b:
        ref.pre()
        ref.sweep(1)
        want = ref.obs_equal_all(), ref.green(n - 1)
        other = later()
        b.pre()
        b.sweep(1)
        assert np.array_equal(b.obs_equal_all(), want[0])
        assert np.array_equal(b.green(n - 1), want[1])
        if other is not None:
            other.close()
