"""Windowed production counts the attempts a chain spends in one (E_Delta, M)
bin in 32 bits and sends the count when the chain leaves the bin, or in time
before it could wrap.  MUCA_HOOK_AGED_RUN starts a launch's recording 1024
attempts before 2^32, so that a chain that stays where it is passes it;
MUCA_HOOK_FLUSH_ROWS sends the counts before every row.  Histograms must have
every entry (the reference kernel adds one per attempt to 64-bit bins,
produce2_multigpu.cu:490)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bin(ed, mag):
    ed, mag = np.asarray(ed, np.int64), np.asarray(mag, np.int64)
    return (ed * ed + 2 * ed + mag) // 2


def _sweep(muca, L, nch, lnw, lat, hooks, therm, nup):
    with muca.Engine(L, nchains=nch, mode=muca.MODE_PRODUCE) as e:
        e.set_weights(lnw)
        e.set_lattice(lat)
        e.set_test_hooks(hooks)
        e.sweep(1, 100, 1000, therm, nup)
        return e.histogram(), e.get_lattice(), e.chain_state()


# drawing warps (with and without whole groups per row), one to four warps of
# chains per SM, blocks of up to 512 chains, the row ring
SHAPES = [(8, 64), (10, 40), (24, 9728), (24, 14592), (16, 30000), (128, 40)]


@pytest.mark.parametrize("L,nch", [(8, 64), (10, 40), (16, 30000), (128, 40)])
def test_a_count_near_2_to_32_is_sent_in_time(muca, L, nch):
    """Chains that reject everything: all spins 0 (E_Delta = M = 0, every
    proposal is to E_Delta = 1) under a weight that holds them there."""
    N = L * L
    lnw = np.zeros(N + 1)
    lnw[0] = 1000.0
    nup = max(4096, 3 * N + 5)
    h, lat, _ = _sweep(muca, L, nch, lnw, np.zeros((nch, N), np.int8), muca.HOOK_AGED_RUN, 0, nup)
    assert not lat.any()
    assert int(h[0]) == nch * (nup + muca.AGED_RUN)
    assert not h[1:].any()


@pytest.mark.parametrize("L,nch", SHAPES)
def test_counts_sent_at_row_starts(muca, L, nch):
    N = L * L
    rng = np.random.default_rng(L)
    lnw = np.cumsum(rng.normal(0.0, 1.0, N + 1))
    lat = rng.integers(-1, 2, (nch, N)).astype(np.int8)
    nup = 2 * N + 3
    want, wl, _ = _sweep(muca, L, nch, lnw, lat, 0, 0, nup)
    ed, mag = (lat.astype(np.int64) ** 2).sum(1), lat.astype(np.int64).sum(1)
    assert int(want.sum()) == nch * nup
    got, gl, _ = _sweep(muca, L, nch, lnw, lat, muca.HOOK_FLUSH_ROWS, 0, nup)
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(gl, wl)
    aged, al, _ = _sweep(muca, L, nch, lnw, lat, muca.HOOK_AGED_RUN, 0, nup)
    np.add.at(want, _bin(ed, mag), np.uint64(muca.AGED_RUN))
    np.testing.assert_array_equal(aged, want)
    np.testing.assert_array_equal(al, wl)
