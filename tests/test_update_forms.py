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
