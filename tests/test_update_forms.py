"""The trivial weight update has two forms, one cluster launch and three launches
over more blocks; the statistics and the updated weights do not depend on which
one serves a size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [8, 16, 63, 72, 90])
@pytest.mark.parametrize("graph", [0, 4])
def test_update_without_a_cluster(muca, L, graph):
    """Where no cluster can be placed the three launches serve every size: the
    same runs, records and host iterations."""
    N = L * L
    out = []
    for hooks in (0, muca.HOOK_NO_CLUSTER):
        with muca.Engine(L, nchains=96) as e:
            e.set_test_hooks(hooks)
            res, recs = e.weight_run(starting_M=3 * N, max_iter=8, graph_iters=graph, d_kl_max=1e-30)
            w, h = e.get_weights(), e.histogram()
            w2, h2 = np.zeros(N + 1), np.zeros(N + 1, np.uint64)
            e.iterate_host(w, 9, 100, 1000, N, 4 * N, muca.UPDATE_TRIVIAL_CPU, lnw_out=w2, hist_out=h2)
            s = e.hist_stats()
        out.append((w, h, w2, h2, [(r.width, r.nupdates, r.total_run) for r in recs], (s.start, s.end, s.events),
                    np.array([r.d_kl for r in recs] + [s.d_kl])))
    for a, b in zip(out[0][:4], out[1][:4]):
        np.testing.assert_array_equal(a, b)
    assert out[0][4:6] == out[1][4:6]
    # up to N + 1 terms P ln(P/Q) in another order; sum P = 1 and |ln(P/Q)| <= ln of
    # the entries (at most 4 N 96 < 3.2e6) < 15
    np.testing.assert_allclose(out[0][6], out[1][6], rtol=0, atol=15 * (N + 1) * 2.0 ** -53)
