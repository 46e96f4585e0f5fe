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


def reference_table(gf, n, dtype, dev):
    r, ri, _ = gf.host_fft_tables(n // 2, dtype)
    return torch.from_numpy(r).to(dev), torch.from_numpy(ri).to(dev)


# one-pass rows of 2048 and 4096 points from one tile per SM on (148), two passes
# (L, 11) from 296 tiles on, (L, 12) from 222 for FP64 FFNT; zero-padded and plain rows
@pytest.mark.parametrize("n_power,batch,dtype", [
    (12, 149, "f64"), (12, 200, "f32"), (13, 74, "f64"), (13, 75, "f32"), (13, 149, "f64"), (14, 75, "f32"),
    (15, 28, "f64"), (16, 15, "f64"), (16, 19, "f32"), (17, 7, "f64"), (17, 10, "f32"), (18, 5, "f64")])
def test_ffnt_tile_passes(gf, O, dev, n_power, batch, dtype):
    n = 1 << n_power
    T = torch.float64 if dtype == "f64" else torch.float32
    C = torch.complex128 if dtype == "f64" else torch.complex64
    g = torch.Generator(device=dev).manual_seed(n_power * 1000 + batch)
    x = torch.randint(-(1 << 10), 1 << 10, (2 * batch, n), device=dev, generator=g, dtype=torch.int32).to(T)
    roots, inv, twist, untwist = (torch.from_numpy(t).to(dev) for t in gf.host_ffnt_tables(n, dtype))
    fwd = gf.fft_configuration(n_power=n_power, fft_type=gf.FORWARD)
    bwd = gf.fft_configuration(n_power=n_power, fft_type=gf.INVERSE, mod_inverse=complex(2.0 / n))

    def product(rows, b):
        temp = torch.empty(2 * b * n // 2, dtype=C, device=dev)
        out = torch.empty(b, n, dtype=T, device=dev)
        gf.GPU_FFNT(rows, temp, twist, roots, fwd, 2 * b, False)
        gf.GPU_FFNT(out, temp, untwist, inv, bwd, b, True)
        return out

    c = product(x, batch)
    few = product(torch.cat([x[batch - 1: batch], x[-1:]]), 1)  # too few rows for the tiles
    assert torch.equal(c[-1:], few)
    idx = np.sort(np.random.default_rng(batch).choice(n, 64, replace=False)).astype(np.int32)
    want = O.wrap64(O.negacyclic_coeffs(x[0].cpu().numpy().astype(np.int64), x[batch].cpu().numpy().astype(np.int64),
                                        idx))
    got = c[0].double().cpu().numpy()[idx]
    if dtype == "f64":
        assert np.array_equal(np.rint(got).astype(np.int64), want)
    else:
        scale = 1024.0 ** 2 / 3 * np.sqrt(n)
        assert np.abs(got - want).max() <= 3 * n_power * 2.0 ** -24 * 8 * scale


@pytest.mark.parametrize("zero_pad", [False, True])
@pytest.mark.parametrize("neg", [False, True])
@pytest.mark.parametrize("n_power,batch,dtype,real", [
    (12, 149, "f64", False), (12, 150, "f32", True), (12, 75, "f64", True), (13, 75, "f64", True),
    (14, 38, "f32", False), (16, 10, "f64", False), (17, 5, "f32", False), (17, 5, "f64", True),
    (18, 3, "f64", False), (19, 2, "f32", False), (20, 2, "f32", True)])
def test_fft_tile_passes(gf, dev, n_power, batch, dtype, real, neg, zero_pad):
    n = 1 << n_power
    T = torch.float64 if dtype == "f64" else torch.float32
    C = torch.complex128 if dtype == "f64" else torch.complex64
    g = torch.Generator(device=dev).manual_seed(n_power * 1000 + batch)
    if neg:  # X^N + 1: n entries e^(i pi (2 br(k) + 1) / 2^(s+1)) at [2^s, 2^(s+1))
        import oracle
        r, ri, _ = oracle.fft_tables(n, dtype)
        roots, inv = torch.from_numpy(r).to(dev), torch.from_numpy(ri).to(dev)
    else:
        roots, inv = reference_table(gf, n, dtype, dev)
    poly = gf.X_N_plus if neg else gf.X_N_minus
    fwd = gf.fft_configuration(n_power=n_power, fft_type=gf.FORWARD, reduction_poly=poly, zero_padding=zero_pad)
    bwd = gf.fft_configuration(n_power=n_power, fft_type=gf.INVERSE, reduction_poly=poly, mod_inverse=complex(1.0 / n))
    x = torch.randn(2 * batch, n, device=dev, generator=g, dtype=T if real else C)

    def product(rows, b):
        if real:
            temp = torch.empty(2 * b * n, dtype=C, device=dev)
            out = torch.empty(b, n, dtype=T, device=dev)
            gf.GPU_FFT(rows, temp, roots, fwd, 2 * b, False)
            gf.GPU_FFT(out, temp, inv, bwd, b, True)
            return out
        buf = rows.clone()
        gf.GPU_FFT(buf, roots, fwd, 2 * b, False)
        gf.GPU_FFT(buf, inv, bwd, b, True)
        return buf[:b]

    c = product(x, batch)
    few = product(torch.cat([x[batch - 1: batch], x[-1:]]), 1)
    assert torch.equal(c[-1:], few)
    u, v = x[:2].to(torch.complex128), x[batch:batch + 2].to(torch.complex128)
    if zero_pad:
        u[:, n // 2:] = 0
        v[:, n // 2:] = 0
    w = torch.exp(1j * np.pi / n * torch.arange(n, device=dev, dtype=torch.float64)) if neg else 1.0
    want = torch.fft.ifft(torch.fft.fft(u * w) * torch.fft.fft(v * w)) / w
    want = want.real if real else want
    err = (torch.linalg.norm(c[:2].to(want.dtype) - want) / torch.linalg.norm(want)).item()
    assert err < (1e-12 if dtype == "f64" else 2e-5)


# one-kernel products (gf_single.cuh): 2^(11-m) to a tile, ragged last tiles, fewer
# tiles than CTAs, several tiles per CTA
@pytest.mark.parametrize("n_power,batch", [
    (5, 1), (5, 127), (5, 129), (6, 33), (8, 5000), (9, 7), (10, 3), (10, 2501), (11, 65), (12, 67), (12, 601),
    (13, 66), (13, 300)])
@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_single_products(gf, dev, n_power, batch, dtype):
    n = 1 << n_power
    T, C = (torch.float64, torch.complex128) if dtype == "f64" else (torch.float32, torch.complex64)
    tol = (1e-14 if dtype == "f64" else 2e-6) * (n_power + 1)
    g = torch.Generator(device=dev).manual_seed(n_power * 1000 + batch)

    def err(got, want):
        return (torch.linalg.norm(got.to(want.dtype) - want) / torch.linalg.norm(want)).item()

    a, b = torch.randn(2, batch, n, device=dev, generator=g, dtype=T)
    w = torch.exp(1j * np.pi / n * torch.arange(n, device=dev, dtype=torch.float64))
    want = (torch.fft.ifft(torch.fft.fft(a.double() * w) * torch.fft.fft(b.double() * w)) / w).real
    c = gf.negacyclic_mul(a, b)
    assert err(c, want) < tol
    inplace = a.clone()
    assert torch.equal(gf.negacyclic_mul(inplace, b, out=inplace), c)
    A, B = torch.fft.rfft(a.double(), 2 * n), torch.fft.rfft(b.double(), 2 * n)
    if n_power <= 12:
        assert err(gf.linear_mul(a, b), torch.fft.irfft(A * B, 2 * n)) < tol
        x, y = torch.complex(a, b), torch.complex(b, a)
        want = torch.fft.ifft(torch.fft.fft(x.to(torch.complex128)) * torch.fft.fft(y.to(torch.complex128)))
        assert err(gf.cyclic_mul(x, y), want) < tol
    if n_power <= 12 and dtype == "f32":
        up = torch.randn(batch, 2 * n, device=dev, generator=g)
        ga, gb = gf.linear_mul_vjp(up, a, b)
        G = torch.fft.rfft(up.double(), 4 * n)
        for got, z in ((ga, b), (gb, a)):
            w4 = torch.fft.irfft(G * torch.fft.rfft(z.double(), 4 * n).conj(), 4 * n)[:, :n]
            assert err(got, w4) < tol
        a2, b2 = a.clone(), b.clone()  # results over the operands
        gf.linear_mul_vjp(up, a2, b2, grad_a=a2, grad_b=b2)
        assert torch.equal(a2, ga) and torch.equal(b2, gb)


# the tile pass of the smallest spans: from 148 2048-point tiles on
@pytest.mark.parametrize("n_power,batch", [(11, 148), (11, 149), (12, 75), (13, 38), (14, 19), (15, 10), (16, 5), (17, 9),
                                           (20, 2)])
@pytest.mark.parametrize("C", [torch.complex128, torch.complex64])
def test_special_tile_rows(gf, O, dev, n_power, batch, C):
    n = 1 << n_power
    g = torch.Generator(device=dev).manual_seed(n_power * 100 + batch)
    x = torch.randn(batch, n, device=dev, generator=g, dtype=C)
    tab = torch.polar(torch.ones(n, device=dev, dtype=torch.float64),
                      torch.rand(n, device=dev, generator=g, dtype=torch.float64) * 6.283185307179586).to(C)
    mi = complex(1.0 / n, 0.5 / n)
    for kind in (gf.FORWARD, gf.INVERSE):
        cfg = gf.fft_configuration(n_power=n_power, fft_type=kind, mod_inverse=mi)
        y, few = x.clone(), x[-1:].clone()
        gf.GPU_Special_FFT(y, tab, cfg, batch)
        gf.GPU_Special_FFT(few, tab, cfg, 1)
        assert torch.equal(y[-1:], few)
        if n_power <= 16:
            np_c = np.complex128 if C == torch.complex128 else np.complex64
            want = O.gpu_special_fft(x[0].cpu().numpy().astype(np_c), tab.cpu().numpy(), n_power, kind, mi, 1)
            err = np.linalg.norm(y[0].cpu().numpy() - want.ravel()) / np.linalg.norm(want)
            assert err < (1e-12 if C == torch.complex128 else 2e-5)
