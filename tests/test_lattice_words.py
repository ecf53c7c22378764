"""Chain energies from whole packed words (k_lattice.cu) at every word
remainder, against the oracle: rows shorter and longer than a word, a last word
of 1 to 16 sites, row counts below and above the rows of a block, chain counts
that leave lanes empty."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("L", [2, 3, 7, 8, 15, 16, 17, 18, 31, 32, 33, 47, 49, 127, 128])
@pytest.mark.parametrize("nch", [1, 33, 70])
def test_energies(muca, orc, L, nch):
    rng = np.random.default_rng(100 * L + nch)
    lat = rng.choice(np.array([-1, 0, 1], np.int8), (nch, L * L), p=[0.4, 0.2, 0.4])
    lat[0] = rng.integers(0, 2) * 2 - 1  # all of one sign: the largest energies
    with muca.Engine(L, nchains=nch) as e:
        e.set_lattice(lat)
        got = e.chain_state()
        np.testing.assert_array_equal(e.get_lattice(), lat)
    for g, o in zip(got, orc.energies(L, lat)):
        np.testing.assert_array_equal(g, o)
