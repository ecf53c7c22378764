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
