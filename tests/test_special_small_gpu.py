"""GPU tests of the special FFT's column passes on vectors of fewer columns than a
CTA has lanes (2^5 .. 2^10 points), whose CTAs take several vectors each: ragged
batches against the oracle, and lanes that are not idle."""
import numpy as np
import pytest
import torch

from test_special_gpu import TOL, random_table, rel_l2, run_ours

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [np.complex128, np.complex64])
@pytest.mark.parametrize("n_power,batch", [(5, 1), (5, 8 * 148 * 6 + 5), (6, 9), (7, 131), (8, 2003), (9, 4 * 148 + 3),
                                           (9, 1), (10, 2), (10, 1025), (11, 3)])
def test_special_small_vectors(gf, O, dev, C, n_power, batch):
    rng = np.random.default_rng(70 + n_power)
    M = 1 << n_power
    x = (rng.standard_normal(batch * M) + 1j * rng.standard_normal(batch * M)).astype(C)
    table = random_table(rng, M, C)
    for fft_type, mi in ((0, 1.0 + 0j), (1, complex(1.0 / M, 0.25 / M))):
        got = run_ours(gf, dev, x, table, n_power, fft_type, mi, batch)
        want = O.gpu_special_fft(x, table, n_power, fft_type, mi, batch)
        assert rel_l2(got, want) < TOL[C]


def test_special_small_vectors_fill_their_lanes(gf, dev):
    # 20000 vectors of 2^8 points, FP64: the passes of spans 1 .. 8 and 16 .. 128 move
    # the same bytes through the same number of threads, so they take the same time
    # (1.0); with a vector's 16 columns to a CTA of 128 threads the second took 1.4
    n, batch = 8, 20000
    x = torch.randn(batch, 1 << n, dtype=torch.complex128, device=dev)
    tab = torch.polar(torch.ones(1 << n, dtype=torch.float64, device=dev),
                      torch.rand(1 << n, dtype=torch.float64, device=dev))
    L, best = gf.lib(), {}
    for _ in range(12):
        x.normal_()
        gf.trace_enable(True)
        try:
            gf.check(L.gpufft_special_fft_f64(x.data_ptr(), tab.data_ptr(), n, 1, 0.5, 0.0, batch, None), "special")
            torch.cuda.synchronize()
        finally:
            gf.trace_enable(False)
        for r in gf.trace_collect():
            key = r["kernel"].split("<")[0]
            best[key] = min(r["ms"], best.get(key, r["ms"]))
    assert best["special_col"] <= 1.2 * best["special_first"]
