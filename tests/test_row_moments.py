"""The reweighting sums' exact row moments (k_observables.cu) at the edges of
their split: rows of every remainder of a warp's chunk, bins at and beyond
2^29 (128-bit products) beside rows of small ones, empty rows, the largest
counts.  The reference is exact integer arithmetic per row; the device then
rounds each row's four sums, a Boltzmann factor, their product and a sum of up
to N + 1 positive terms in FP64 along a tree: below 40 roundings of 1.1e-16."""
import numpy as np
import pytest


def _moments(h, N, lnw, bd):
    s = [0.0] * 4
    for i in range(N + 1):
        row = [int(x) for x in h[i * (i + 1) // 2:(i + 1) * (i + 2) // 2]]
        m = [abs(2 * j - i) for j in range(i + 1)]
        bz = np.exp(np.float64(-bd * i - lnw[i]))
        for q, p in enumerate((0, 1, 2, 4)):
            s[q] += np.longdouble(sum(a * b ** p for a, b in zip(row, m))) * np.longdouble(bz)
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("L", [2, 3, 8, 17, 23])
@pytest.mark.parametrize("top", [1 << 10, (1 << 29) - 1, 1 << 29, 1 << 32, (1 << 63) - 1])
def test_row_moments(muca, L, top):
    import torch
    N = L * L
    rng = np.random.default_rng(L)
    n = (N + 1) * (N + 2) // 2
    h = rng.integers(0, 1 << 20, n).astype(np.int64)
    h[rng.random(n) < 0.3] = 0
    h[rng.random(n) < 0.02] = top
    h[0] = top  # the one bin of row 0
    e = N // 2
    h[e * (e + 1) // 2:(e + 1) * (e + 2) // 2] = 0
    lnw = rng.normal(0.0, 2.0, N + 1) - 0.3 * np.arange(N + 1)
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    hd, wd = torch.from_numpy(h).cuda(), torch.from_numpy(lnw).cuda()
    muca.observables_noalloc(0, hd.data_ptr(), wd.data_ptr(), L, 2.0, 0.15, out.data_ptr(),
                             torch.cuda.current_stream().cuda_stream)
    np.testing.assert_allclose(out.cpu().numpy(), np.array(_moments(h, N, lnw, 0.3), dtype=np.float64), rtol=1e-14)


def _large(torch, rows):
    """A histogram at L = 128 whose row i holds rows[i] in every bin, and its
    exact sums of |m|^p per row: S_p(i) = S_p(i - 2) + 2 i^p."""
    N = 128 * 128
    counts = torch.arange(1, N + 2, device="cuda")
    h = torch.repeat_interleave(torch.from_numpy(np.asarray(rows, np.int64)).cuda(), counts)
    S = {p: [0 ** p, 2] for p in (0, 1, 2, 4)}
    for p in S:
        for i in range(2, N + 1):
            S[p].append(S[p][i - 2] + 2 * i ** p)
    return h, S


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["all", "alternating", "first_rows", "middle"])
def test_rows_of_large_counts_at_the_largest_size(muca, name):
    """The longest rows (257 terms per lane), rows with and without bins of 2^29
    and more in turn, counts up to the last bit of the low part and above."""
    import torch
    N = 128 * 128
    i = np.arange(N + 1)
    big = np.array([(1 << 29) - 1, 1 << 29, (1 << 30) + 5, (1 << 35) - 1, (1 << 45) + 3], dtype=np.int64)[i % 5]
    small = 1000 + i % 77
    on = {"all": i >= 0, "alternating": i // 3 % 2 == 0, "first_rows": i < 1000, "middle": (i > 5000) & (i < 12000)}[name]
    rows = np.where(on, big, small)
    h, S = _large(torch, rows)
    lnw = 1e-4 * i
    w, out = torch.from_numpy(lnw).cuda(), torch.zeros(4, dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream()
    muca.observables_noalloc(0, h.data_ptr(), w.data_ptr(), 128, 2.0, 0.0, out.data_ptr(), s.cuda_stream)
    bz = np.exp(-lnw).astype(np.longdouble)
    want = [float(sum(np.longdouble(int(rows[k]) * S[p][k]) * bz[k] for k in range(N + 1))) for p in (0, 1, 2, 4)]
    np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-14)


@pytest.mark.gpu
def test_large_counts_cost_at_most_another_pass(muca):
    """Bins of 2^29 and more: the histogram is read at most twice, so the time is
    at most twice that of small counts (and a quarter for the longer additions)."""
    import torch
    N = 128 * 128
    n = (N + 1) * (N + 2) // 2
    w, out = torch.zeros(N + 1, dtype=torch.float64, device="cuda"), torch.zeros(4, dtype=torch.float64, device="cuda")
    best = []
    for v in (1000, 1 << 30):
        h = torch.full((n,), v, dtype=torch.int64, device="cuda")
        t = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            muca.observables_noalloc(0, h.data_ptr(), w.data_ptr(), 128, 2.0, 0.0, out.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        best.append(min(t))
    assert best[1] <= 2.25 * best[0], best
