"""The windowed weight sweep's shared u32 histogram bins are flushed into
the u64 device histogram between rows whenever a launch could otherwise put
2^32 entries into one bin.  MUCA_HOOK_FLUSH_ROWS makes every recorded row
take that path; lattices, energies and histograms must still equal the
oracle's (the reference kernel mcs, muca_delta_multigpu.cu:737-829) bit for
bit, with the lattice in shared memory and behind the row ring, and with
therm and nup not multiples of a row so that the step-by-step tail runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nch", [(24, 256), (72, 128), (128, 64)])
def test_flushing_shared_bins_between_rows_changes_nothing(muca, orc, L, nch):
    N = L * L
    rng = np.random.default_rng(L)
    lnw = np.cumsum(rng.normal(0.0, 1.2, N + 1)) * 0.5
    therm, nup = N + 37, 3 * N + 11
    with muca.Engine(L, nchains=nch, kernel=muca.KERNEL_WINDOWED) as e:
        assert e.info.kernel == muca.KERNEL_WINDOWED
        e.set_weights(lnw)
        e.init_chains(muca.INIT_WEIGHT, 0)
        lat0 = e.get_lattice()
        ej0, ed0, _ = e.chain_state()
        e.set_test_hooks(muca.HOOK_FLUSH_ROWS)
        e.sweep(2, 100, 1000, therm, nup)
        lat1 = e.get_lattice()
        ej1, ed1, _ = e.chain_state()
        h = e.histogram()
        e.set_test_hooks(0)
    ej, ed = (np.ascontiguousarray(x, np.int32).copy() for x in (ej0, ed0))
    olat, oh = orc.weight_sweep(L, lat0.copy(), ej, ed, lnw.astype(np.float32), 2, 100, therm, nup, nthreads=8)
    np.testing.assert_array_equal(lat1, olat.reshape(nch, N))
    np.testing.assert_array_equal(ej1, ej)
    np.testing.assert_array_equal(ed1, ed)
    np.testing.assert_array_equal(h, oh)
    assert int(h.sum()) == nch * nup


# two warps of chains per SM with drawing warps (rows in whole groups and not),
# three and four warps, blocks of up to 512 chains (in shared memory, behind the
# row ring), a block's last warp with lanes without a chain
@pytest.mark.parametrize("L,nch", [(16, 9728), (10, 9000), (16, 14500), (14, 19000), (8, 60000), (72, 40000)])
def test_flushing_the_bins_of_several_warps_changes_nothing(muca, L, nch):
    N = L * L
    lnw = np.cumsum(np.random.default_rng(L).normal(0.0, 0.6, N + 1))
    nup = N + 11
    out = []
    for hooks in (0, muca.HOOK_FLUSH_ROWS):
        with muca.Engine(L, nchains=nch) as e:
            assert e.info.kernel == muca.KERNEL_WINDOWED
            e.set_weights(lnw)
            e.init_chains(muca.INIT_WEIGHT, 0)
            e.set_test_hooks(hooks)
            e.sweep(2, 100, 1000, 5, nup)
            out.append((e.get_lattice(), e.histogram()) + e.chain_state()[:2])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert int(out[0][1].sum()) == nch * nup


# lattices in shared memory (one warp and several) and in global memory; what
# is left after the last flush 0..3 attempts, and less than one segment
@pytest.mark.parametrize("L,nch,nup", [(8, 300, 64), (8, 300, 67), (9, 6000, 41), (16, 40000, 30), (128, 300, 25), (8, 40, 7)])
def test_flushing_random_site_bins_changes_nothing(muca, L, nch, nup):
    N = L * L
    lnw = np.cumsum(np.random.default_rng(nch).normal(0.0, 0.6, N + 1))
    out = []
    for hooks in (0, muca.HOOK_FLUSH_ROWS):
        with muca.Engine(L, nchains=nch, algorithm=muca.ALGO_RANDOM_SITE) as e:
            e.set_weights(lnw)
            e.init_chains(muca.INIT_MUCA_MAG, 1)
            e.set_test_hooks(hooks)
            e.sweep(3, 1, 0, 6, nup)
            out.append((e.get_lattice(), e.histogram()) + e.chain_state()[:2])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert int(out[0][1].sum()) == nch * nup
