"""The lean window of the sweep (window.cuh): the error bound of production's
fast test (CPU); chain counts that leave lanes without a chain, over several
launches, sizes that are not a multiple of 8, and more chains than one warp
per SM sub-partition, against the oracle (GPU).

The production window stages u[E] = fl32(w[E+1] - w[E]) and decides with
g = fma(-dDel, u, h), h = fl32(l - f2), where the reference decides
logf(u) < diff, diff = fl64(fl64(f2 + w[E+dDel]) - w[E])
(produce2_multigpu.cu:474).  stage_differences takes

    tol = 2 (2^-24 (2 m + 66) + 2^-53 (max|w| + 32 + 2 m))   (times 1.0001)

with m = max|u| and claims |g - (l - diff)| <= tol / 2 for |l| < 17.
"""
import numpy as np
import pytest

F2 = np.arange(-16, 17, 2, dtype=np.float32)  # -2 dE for dE in [-8, 8]


def _weights():
    rng = np.random.default_rng(23)
    N = 4096
    walk = np.cumsum(rng.normal(0.0, 1.5, N + 1)) * 0.5
    return {
        "zero": np.zeros(N + 1),
        "walk": walk,
        "walk_offset_1e4": walk + 1.0e4,
        "steep": np.cumsum(rng.normal(0.0, 40.0, N + 1)),
        "near_f2": np.cumsum(rng.choice([-16.0, -8.0, 8.0, 16.0], N + 1) + rng.normal(0.0, 1e-6, N + 1)),
        "large": rng.uniform(-1e5, 1e5, N + 1),
    }


@pytest.mark.parametrize("name", list(_weights().keys()))
def test_fast_difference_within_half_tol(name):
    w = _weights()[name]
    u = np.append(np.diff(w).astype(np.float32), np.float32(0))
    m = float(np.max(np.abs(u))) * 1.0001
    tol = np.float32((2.0 * 2.0 ** -24 * (2.0 * m + 66.0) +
                      2.0 * 2.0 ** -53 * (float(np.max(np.abs(w))) + 32.0 + 2.0 * m)) * 1.0001)
    rng = np.random.default_rng(3)
    E = np.arange(w.size)
    worst = 0.0
    for dd in (-1, 0, 1):
        e = E[(E + dd >= 0) & (E + dd < w.size)]
        ue = u[e - 1] if dd < 0 else u[e]
        for f2 in F2:
            diff = (np.float64(f2) + w[e + dd]) - w[e]
            l = np.log(((2 * rng.integers(0, 1 << 23, e.size) + 1) * 2.0 ** -24)).astype(np.float32)
            # half of them right at the threshold
            l = np.where(rng.random(e.size) < 0.5, np.clip(diff, -16.7, -2.0 ** -24).astype(np.float32), l)
            h = (l - f2).astype(np.float32)
            g = (np.float64(-dd) * ue.astype(np.float64) + h.astype(np.float64)).astype(np.float32)  # one rounding
            worst = max(worst, float(np.max(np.abs(g.astype(np.float64) - (l.astype(np.float64) - diff)))))
    assert worst <= tol / 2, (name, worst, float(tol))


# 1000 chains: 32 blocks of 32 lanes, 24 lanes of the last block without a
# chain; 33 chains: a warp with one chain; 300: the last warps partly filled
@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [0, 1, 2, 3])
@pytest.mark.parametrize("L,nch", [(40, 1000), (8, 33), (16, 300)])
@pytest.mark.parametrize("produce", [False, True])
def test_lanes_without_a_chain(muca, orc, L, nch, produce, kernel):
    """Several launches in a row: the lattices of lanes without a chain stay
    as they were made, and every chain follows the oracle."""
    N = L * L
    rng = np.random.default_rng(L + nch)
    lnw = np.cumsum(rng.normal(-0.6, 0.3, N + 1))
    with muca.Engine(L, nchains=nch, kernel=kernel, mode=muca.MODE_PRODUCE if produce else muca.MODE_WEIGHT) as e:
        e.set_weights(lnw)
        e.init_chains(muca.INIT_GRADED, 0)
        lat = e.get_lattice()
        state = [np.ascontiguousarray(x, np.int32).copy() for x in e.chain_state()]
        for it in range(3):
            therm, nup = N // 2, N // 2 + 5
            e.sweep(it, 100, 1000, therm, nup)
            if produce:
                lat, h = orc.produce_sweep(L, lat, *state, lnw, it, 100, therm, nup, nthreads=8)
            else:
                lat, h = orc.weight_sweep(L, lat, *state[:2], lnw.astype(np.float32), it, 100, therm, nup, nthreads=8)
            np.testing.assert_array_equal(e.get_lattice(), lat)
            ej, ed, mg = e.chain_state()
            np.testing.assert_array_equal(ej, state[0])
            np.testing.assert_array_equal(ed, state[1])
            if produce:
                np.testing.assert_array_equal(mg, state[2])
            assert np.array_equal(e.histogram(), h)


# sizes that are not a multiple of 8: every remainder of L mod 16, row-halves
# that leave the Philox groups at every offset, one word per row and several
@pytest.mark.gpu
@pytest.mark.parametrize("L", [10, 12, 14, 18, 20, 22, 26, 28, 30, 34, 36, 50, 100, 126])
@pytest.mark.parametrize("produce,rounds", [(False, 7), (True, 7), (False, 10)])
def test_even_sizes(muca, orc, L, produce, rounds):
    N, nch = L * L, 40
    rng = np.random.default_rng(L)
    lnw = np.cumsum(rng.normal(0.0, 1.2, N + 1)) * 0.5
    with muca.Engine(L, nchains=nch, rounds=rounds, mode=muca.MODE_PRODUCE if produce else muca.MODE_WEIGHT) as e:
        assert e.info.kernel == muca.KERNEL_WINDOWED
        e.set_weights(lnw)
        e.init_chains(muca.INIT_GRADED, 0)
        lat = e.get_lattice()
        state = [np.ascontiguousarray(x, np.int32).copy() for x in e.chain_state()]
        for it, (therm, nup) in enumerate([(N, N), (L // 2 + 3, 2 * L + 1), (0, 7), (5, 0)]):
            e.sweep(it, 100, 1000, therm, nup)
            if produce:
                lat, h = orc.produce_sweep(L, lat, *state, lnw, it, 100, therm, nup, rounds=rounds, nthreads=8)
            else:
                lat, h = orc.weight_sweep(L, lat, *state[:2], lnw.astype(np.float32), it, 100, therm, nup,
                                          rounds=rounds, nthreads=8)
            np.testing.assert_array_equal(e.get_lattice(), lat)
            ej, ed, mg = e.chain_state()
            np.testing.assert_array_equal(ej, state[0])
            np.testing.assert_array_equal(ed, state[1])
            if produce:
                np.testing.assert_array_equal(mg, state[2])
            assert np.array_equal(e.histogram(), h)
        e.set_log_bracket(1e30)  # every window on the exact path
        e.sweep(9, 100, 1000, L, L + 1)
        if produce:
            lat, h = orc.produce_sweep(L, lat, *state, lnw, 9, 100, L, L + 1, rounds=rounds, nthreads=8)
        else:
            lat, h = orc.weight_sweep(L, lat, *state[:2], lnw.astype(np.float32), 9, 100, L, L + 1, rounds=rounds,
                                      nthreads=8)
        np.testing.assert_array_equal(e.get_lattice(), lat)
        assert np.array_equal(e.histogram(), h)


# more chains than one warp per SM sub-partition: blocks of up to 512 chains,
# lattices in shared memory (L = 16, 40) and behind the row ring (64, 128)
@pytest.mark.gpu
@pytest.mark.parametrize("L,nch,smem", [(16, 20011, 1), (40, 60000, 1), (64, 80000, 0), (128, 30000, 0)])
@pytest.mark.parametrize("produce", [False, True])
def test_many_chains(muca, orc, L, nch, smem, produce):
    N = L * L
    rng = np.random.default_rng(L)
    lnw = np.cumsum(rng.normal(-0.6, 0.3, N + 1))
    therm, nup = 3 * L + 1, 5 * L + 2
    with muca.Engine(L, nchains=nch, mode=muca.MODE_PRODUCE if produce else muca.MODE_WEIGHT) as e:
        assert e.info.chains_per_block > 128 and e.info.lattice_in_smem == smem
        cpb = e.info.chains_per_block
        e.set_weights(lnw)
        e.init_chains(muca.INIT_GRADED, 0)
        lat0 = e.get_lattice()
        s0 = e.chain_state()
        e.sweep(2, 100, 1000, therm, nup)
        lat1 = e.get_lattice()
        s1 = e.chain_state()
        h = e.histogram()
    assert int(h.sum()) == nch * nup
    mid = (nch // cpb // 2) * cpb
    for lo, hi in ((0, 40), (mid - 20, mid + 20), (nch - 40, nch)):
        a = lat0[lo:hi].copy()
        st = [np.ascontiguousarray(x[lo:hi], np.int32).copy() for x in s0]
        if produce:
            orc.produce_sweep(L, a, *st, lnw, 2, 100, therm, nup, chain0=lo, nthreads=8)
            np.testing.assert_array_equal(s1[2][lo:hi], st[2])
        else:
            orc.weight_sweep(L, a, *st[:2], lnw.astype(np.float32), 2, 100, therm, nup, chain0=lo, nthreads=8)
        np.testing.assert_array_equal(lat1[lo:hi], a.reshape(hi - lo, N))
        np.testing.assert_array_equal(s1[0][lo:hi], st[0])
        np.testing.assert_array_equal(s1[1][lo:hi], st[1])


# the update of one cluster (L <= 90) and of three launches (above), one and
# two bins per thread, and bins at the edges of the cluster's strides
@pytest.mark.gpu
@pytest.mark.parametrize("L", [2, 8, 16, 30, 64, 66, 90, 92, 128])
@pytest.mark.parametrize("rule", [0, 1])
def test_update_over_a_cluster(muca, orc, L, rule):
    N = L * L
    rng = np.random.default_rng(L + rule)
    h = rng.integers(0, 4, N + 1).astype(np.uint64) * rng.integers(0, 5000, N + 1).astype(np.uint64)
    lnw = rng.normal(0.0, 50.0, N + 1)
    with muca.Engine(L, nchains=32) as e:
        e.set_weights(lnw)
        e.set_histogram(h)
        s = e.update_weights(rule)
        w = e.get_weights()
        assert np.array_equal(e.histogram(), h)
    with np.errstate(divide="ignore"):
        ln = np.log(h.astype(np.float64))
    upd = h > (1 if rule == 0 else 0)
    x = np.where(upd, lnw - ln, lnw)
    x = x - x[0] if rule == 0 else np.where(h > 0, x - x[0], x)
    np.testing.assert_allclose(w, x, rtol=1e-13, atol=1e-10)
    assert (s.start, s.end) == orc.hist_range(h)
    assert s.events == int(h.sum()) and s.visited == int((h > 0).sum()) and s.min_count == int(h.min())
    np.testing.assert_allclose(s.d_kl, orc.kull_leibler(h), rtol=1e-11)


# one and two walking warps per SM with warps that draw for them, and the first
# chain count past that; launches that end at, before and after a half of the
# ring (64 attempts), one half, several, none in one of the phases
@pytest.mark.gpu
@pytest.mark.parametrize("nch", [31, 5000, 9728, 9729])
@pytest.mark.parametrize("L", [8, 10])
@pytest.mark.parametrize("produce", [False, True])
def test_draws_from_other_warps(muca, orc, L, nch, produce):
    N = L * L
    lnw = np.cumsum(np.random.default_rng(L + nch).normal(-0.3, 0.6, N + 1))
    with muca.Engine(L, nchains=nch, mode=muca.MODE_PRODUCE if produce else muca.MODE_WEIGHT) as e:
        e.set_weights(lnw)
        e.init_chains(muca.INIT_GRADED, 0)
        lat = e.get_lattice()
        state = [np.ascontiguousarray(x, np.int32).copy() for x in e.chain_state()]
        for it, (therm, nup) in enumerate([(0, 1), (52, 1), (56, 0), (53, 4), (64, 57), (N, 3 * N), (127, 65), (0, 121)]):
            e.sweep(it, 100, 1000, therm, nup)
            if produce:
                lat, h = orc.produce_sweep(L, lat, *state, lnw, it, 100, therm, nup, nthreads=8)
            else:
                lat, h = orc.weight_sweep(L, lat, *state[:2], lnw.astype(np.float32), it, 100, therm, nup, nthreads=8)
            np.testing.assert_array_equal(e.get_lattice(), lat)
            ej, ed, mg = e.chain_state()
            np.testing.assert_array_equal(ej, state[0])
            np.testing.assert_array_equal(ed, state[1])
            if produce:
                np.testing.assert_array_equal(mg, state[2])
            assert np.array_equal(e.histogram(), h)
