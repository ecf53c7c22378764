"""The trivial weight update has two forms, one cluster launch and three launches
over more blocks; the statistics and the updated weights do not depend on which
one serves a size, and neither does the time by much."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph_time(muca, L):
    """Microseconds of one update in a graph of 32, every bin visited."""
    import torch
    s = torch.cuda.Stream()
    rng = np.random.default_rng(L)
    with muca.Engine(L, nchains=32, stream=s.cuda_stream) as e:
        e.set_histogram(rng.integers(50, 5000, L * L + 1).astype(np.uint64))
        e.update_weights(muca.UPDATE_TRIVIAL)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
            for _ in range(32):
                e.update_weights(muca.UPDATE_TRIVIAL, wait=False)
        best = float("inf")
        for _ in range(20):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            with torch.cuda.stream(s):
                a.record()
                for _ in range(4):
                    g.replay()
                b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3 / 128)
    return best


@pytest.mark.parametrize("L", [63, 64, 66, 72, 90])
def test_update_time_grows_with_the_size(muca, L):
    """No size may cost more than a larger one (L = 96, 9217 bins) by more than
    the clock's noise: there the other form would have been the better one."""
    t, larger = _graph_time(muca, L), _graph_time(muca, 96)
    assert t <= 1.1 * larger, (t, larger)


@pytest.mark.parametrize("L", [8, 16, 63])
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
    # up to 3970 terms P ln(P/Q) in another order; sum P = 1 and |ln(P/Q)| <= ln of
    # the entries (fewer than 2^21) < 15
    np.testing.assert_allclose(out[0][6], out[1][6], rtol=0, atol=15 * 3970 * 2.0 ** -53)
