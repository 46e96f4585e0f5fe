"""GPU tests of the exact product on FP64 transforms (gf_split_tile.cuh): the same
integers as the limb plan's chain and as the exact negacyclic product, over ring
sizes (one-kernel and three-kernel forms), signs, widths that take one, two or three
limbs, ragged batches and waves, and rows that are not uniform."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def exact(a, b):
    """c mod 2^64 from 8-bit digits: every digit product's coefficients stay below
    2^34, where FP64 convolutions are exact to 2^-14."""
    n = a.shape[1]
    w = torch.polar(torch.ones(n, dtype=torch.float64, device=a.device),
                    torch.arange(n, dtype=torch.float64, device=a.device) * (np.pi / n))

    def digits(x):
        x = x.long()
        return [torch.fft.fft(((x >> s) & 255 if s < 24 else x >> s).double() * w) for s in (0, 8, 16, 24)]

    A, B = digits(a), digits(b)
    c = torch.zeros(a.shape, dtype=torch.int64, device=a.device)
    for i in range(4):
        for j in range(4):
            c += torch.round((torch.fft.ifft(A[i] * B[j]) * w.conj()).real).long() << (8 * (i + j))
    return c


def rows(gf, dev, n, batch, bits, nonneg, seed):
    g = torch.Generator(device=dev).manual_seed(seed)
    lo = 0 if nonneg else 1 - (1 << bits)
    return torch.randint(lo, 1 << bits, (2, batch, n), dtype=torch.int32, device=dev, generator=g)


@pytest.mark.parametrize("n_power,batch,bits,nonneg", [
    (5, 63, 24, True), (5, 65, 16, False), (6, 1, 8, True), (8, 17, 24, False), (9, 8, 20, True), (10, 3, 16, True),
    (11, 5, 24, True), (12, 1, 24, False), (12, 3, 16, True), (13, 17, 24, True), (13, 9, 16, False),
    (13, 20, 27, False), (14, 37, 24, True), (14, 38, 10, False), (15, 19, 24, True), (16, 10, 24, True),
    (16, 11, 16, False), (16, 10, 28, True), (17, 5, 20, True), (17, 6, 24, False)])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_exact_matches_chain_and_integers(gf, dev, n_power, batch, bits, nonneg, precision):
    n = 1 << n_power
    a, b = rows(gf, dev, n, batch, bits, nonneg, 100 * n_power + bits)
    a[0, : n // 2] = a[0, 0]  # a row that is not uniform
    try:
        plan = gf.split_plan(n_power, bits, nonneg, precision)
    except gf.GpufftError:
        pytest.skip("no limb plan for this width")
    kw = dict(input_bits=bits, non_negative=nonneg, limbs=plan, precision=precision, return_error=True)
    want = exact(a, b)
    prev = gf.set_split_tile(1)
    try:
        c, e = gf.negacyclic_mul_split(a, b, **kw)
        gf.set_split_tile(0)
        c0, e0 = gf.negacyclic_mul_split(a, b, **kw)
    finally:
        gf.set_split_tile(prev)
    if float(e0.item()) >= 0.5 and torch.equal(c, c0) and float(e.item()) == float(e0.item()):
        return  # the call runs the chain (28 bits, FP32), which reports that it does not hold the constant half row
    assert float(e.item()) < 0.5
    assert torch.equal(c, want)
    if float(e0.item()) < 0.25:
        assert torch.equal(c0, want)


@pytest.mark.parametrize("n_power,batch,ws_products", [(16, 30, 12), (14, 100, 41), (17, 11, 6)])
def test_exact_waves(gf, dev, n_power, batch, ws_products):
    # a workspace of fewer products than the batch: several waves, the last one ragged
    n = 1 << n_power
    a, b = rows(gf, dev, n, batch, 24, True, n_power)
    k = gf.split_plan(n_power, 24, True)[1]
    per = int(gf.lib().gpufft_negacyclic_mul_split_workspace_bytes(n_power, 1, k))
    ws = torch.empty(per * ws_products, dtype=torch.uint8, device=dev)
    c = gf.negacyclic_mul_split(a, b, input_bits=24, non_negative=True, workspace=ws)
    assert torch.equal(c, exact(a, b))


@pytest.mark.parametrize("n_power,batch,bits,nonneg", [
    (10, 40, 24, True), (12, 200, 20, True), (12, 30, 24, False), (13, 40, 24, False), (14, 40, 24, True),
    (15, 20, 16, True), (16, 12, 16, True), (16, 12, 20, True)])
@pytest.mark.parametrize("kind", ["zero", "half", "one", "max", "few"])
def test_exact_coherent_rows(gf, dev, n_power, batch, bits, nonneg, kind):
    # rows whose products add up instead of averaging out: zero, zero-padded,
    # monomial, constant and small operands
    n = 1 << n_power
    a, b = rows(gf, dev, n, batch, bits, nonneg, 31 * n_power + bits)
    if kind == "zero":
        a.zero_()
    elif kind == "half":
        a[:, n // 2:] = 0
        b[:, n // 2:] = 0
    elif kind == "one":
        a.zero_()
        a[:, 5] = 1
    elif kind == "max":
        a.fill_((1 << bits) - 1)
        b.fill_((1 << bits) - 1)
    else:
        a.remainder_(3)
    c, e = gf.negacyclic_mul_split(a, b, input_bits=bits, non_negative=nonneg, return_error=True)
    assert float(e.item()) <= 0.5
    assert torch.equal(c, exact(a, b))
