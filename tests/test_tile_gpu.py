"""GPU tests of the 2048-point tile kernels (gf_tile.cuh) and of the two-lane
column passes around them: rows computed in a batch that takes them have the
bits of the same rows computed in a batch too small for them (the 4096-point
passes run the same butterflies), and integer products are exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(gf, dev, n, batch, dtype, seed):
    g = torch.Generator(device=dev).manual_seed(seed)
    hi = 1 << (12 if dtype in (torch.float64, torch.complex128) else 4)
    re = torch.randint(-hi, hi, (2, 2 * batch, n), device=dev, generator=g, dtype=torch.int32)
    if dtype.is_complex:
        x = torch.complex(re[0].double(), re[1].double()).to(dtype)
    else:
        x = re[0].to(dtype)
    return x[:batch], x[batch:]


# 296 tiles (two per SM of a 148-SM B200) is the smallest wave of the tile
# kernel: 74 products of N = 2^14 (four tiles each), 10 of 2^17, 19 of 2^16
@pytest.mark.parametrize("n_power,batch,dtype", [
    (14, 73, torch.float64), (14, 74, torch.float64), (14, 75, torch.float32), (15, 41, torch.float32),
    (16, 19, torch.float64), (16, 85, torch.float64), (17, 10, torch.float64), (17, 11, torch.float32)])
def test_negacyclic_tile_rows(gf, O, dev, n_power, batch, dtype):
    n = 1 << n_power
    a, b = operands(gf, dev, n, batch, dtype, n_power + batch)
    c = gf.negacyclic_mul(a, b)
    few = gf.negacyclic_mul(a[-2:].contiguous(), b[-2:].contiguous())
    assert torch.equal(c[-2:], few)
    idx = np.sort(np.random.default_rng(batch).choice(n, 64, replace=False)).astype(np.int32)
    got = c[0].double().cpu().numpy()[idx]
    want = O.wrap64(O.negacyclic_coeffs(a[0].cpu().numpy().astype(np.int64), b[0].cpu().numpy().astype(np.int64), idx))
    if dtype == torch.float64:
        assert np.array_equal(np.rint(got).astype(np.int64), want)
    else:  # 2^-24 per operation through log2(N) stages of three transforms, against the row's scale
        scale = 16.0 ** 2 / 3 * np.sqrt(n)
        assert np.abs(got - want).max() <= 3 * n_power * 2.0 ** -24 * 8 * scale


@pytest.mark.parametrize("n_power,batch,dtype", [
    (13, 74, torch.complex128), (13, 75, torch.complex64), (15, 19, torch.complex128), (16, 10, torch.complex128),
    (16, 10, torch.complex64)])
def test_cyclic_tile_rows(gf, dev, n_power, batch, dtype):
    a, b = operands(gf, dev, 1 << n_power, batch, dtype, 7 * n_power + batch)
    c = gf.cyclic_mul(a, b)
    few = gf.cyclic_mul(a[-2:].contiguous(), b[-2:].contiguous())
    assert torch.equal(c[-2:], few)
    want = torch.fft.ifft(torch.fft.fft(a[:3].to(torch.complex128)) * torch.fft.fft(b[:3].to(torch.complex128)))
    err = torch.linalg.norm(c[:3].to(torch.complex128) - want) / torch.linalg.norm(want)
    assert err.item() < (1e-14 if dtype == torch.complex128 else 2e-6) * n_power


@pytest.mark.parametrize("n_power,batch", [(13, 74), (14, 37), (15, 19), (16, 10), (16, 9)])
def test_vjp_tile_rows(gf, dev, n_power, batch):
    n = 1 << n_power
    g = torch.Generator(device=dev).manual_seed(n_power * 100 + batch)
    up = torch.randn(batch, 2 * n, device=dev, generator=g)
    a, b = torch.randn(2, batch, n, device=dev, generator=g)
    ga, gb = gf.linear_mul_vjp(up, a, b)
    fa, fb = gf.linear_mul_vjp(up[-2:].contiguous(), a[-2:].contiguous(), b[-2:].contiguous())
    assert torch.equal(ga[-2:], fa) and torch.equal(gb[-2:], fb)
    G = torch.fft.rfft(up[:2].double(), 4 * n)
    for got, x in ((ga, b), (gb, a)):
        want = torch.fft.irfft(G * torch.fft.rfft(x[:2].double(), 4 * n).conj(), 4 * n)[:, :n]
        assert (torch.linalg.norm(got[:2] - want) / torch.linalg.norm(want)).item() < 2e-5
