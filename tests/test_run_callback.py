"""What a callback of muca_weight_run_stream finds in the context: the counts
of the iteration it is called for (one entry per chain and update,
muca_delta_multigpu.cu:404-439 logs from the same histogram), and whatever it
leaves there is gone before the next sweep."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _opts(muca, rule, starting_M, max_iter):
    return muca.RunOpts(starting_M=starting_M, rule=rule, max_iter=max_iter, reinit_chains=1,
                        init_scheme=muca.INIT_WEIGHT, d_kl_max=1e-30)


def _stream(muca, e, rule, starting_M, max_iter, seen):
    res = muca.RunResult()
    errors = []

    def cb(rec, _user):
        try:
            seen(rec.contents)
        except Exception as ex:  # noqa: BLE001
            errors.append(ex)

    o = _opts(muca, rule, starting_M, max_iter)
    st = e._lib.muca_weight_run_stream(e._h, C.byref(o), C.byref(res), muca.ITER_CB(cb), None)
    assert st in (0, 4)  # 4: not converged
    if errors:
        raise errors[0]
    return res


# every form of the update: one cluster (L = 16, 63, 64), several launches
# (L = 96), the recursion; and the random-site algorithm's sweep
@pytest.mark.parametrize("L,rule,algo", [(16, 0, 0), (16, 1, 0), (16, 2, 0), (63, 0, 0), (64, 0, 0), (96, 0, 0),
                                         (96, 2, 0), (12, 1, 1)])
def test_callback_sees_the_iterations_counts(muca, L, rule, algo):
    nch, iters = 64, 5
    with muca.Engine(L, nchains=nch, algorithm=algo) as e:
        sums, stats = [], []

        def seen(rec):
            sums.append((int(e.histogram().sum()), nch * rec.nupdates))
            st = e.hist_stats()
            stats.append((int(st.events), int(st.width) == rec.width_temp))

        _stream(muca, e, rule, 200, iters, seen)
        last = int(e.histogram().sum())
    assert len(sums) == iters
    for (got, want), (events, same_width) in zip(sums, stats):
        assert got == want and events == want and same_width
    assert last == sums[-1][1]


@pytest.mark.parametrize("L,rule", [(16, 0), (64, 0), (16, 2)])
def test_what_a_callback_leaves_is_cleared(muca, L, rule):
    """A callback that overwrites the histogram changes nothing of the run."""
    nch, iters = 64, 5
    N = L * L
    junk = np.arange(N + 1, dtype=np.uint64) + 7
    with muca.Engine(L, nchains=nch) as e:
        _, recs = e.weight_run(starting_M=200, rule=rule, max_iter=iters, d_kl_max=1e-30)
        want, want_h = e.get_weights(), e.histogram()
    widths = []
    with muca.Engine(L, nchains=nch) as e:
        def seen(rec):
            widths.append(rec.width_temp)
            if rec.k + 1 < iters:
                e.set_histogram(junk)
        _stream(muca, e, rule, 200, iters, seen)
        got, got_h = e.get_weights(), e.histogram()
    assert widths == [r.width_temp for r in recs]
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(got_h, want_h)
