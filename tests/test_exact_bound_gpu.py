"""GPU tests of what the exact product holds on rows whose coefficients add up
(constant, half-range, zero and zero-padded operands): the number of limbs has to
follow the largest magnitude such rows give a limb's product,
    N 2^top 2^B,  three times that for centred (non-negative) inputs,
whatever the ring, the width and the sign. Sets whose one-limb or two-limb product
would pass 2^48, where an FP64 transform's error nears 0.5. And what calls with FP64
tables report."""
import pytest
import torch

from test_exact_gpu import exact, rows

pytestmark = pytest.mark.gpu


def operands(kind, n, batch, bits, nonneg, dev):
    top = (1 << bits) - 1
    half = 1 << (bits - 1)
    a = torch.zeros(batch, n, dtype=torch.int32, device=dev)
    b = torch.zeros(batch, n, dtype=torch.int32, device=dev)
    if kind == "max":
        a.fill_(top)
        b.fill_(top)
    elif kind == "halfrange":
        a.fill_(half)
        b.fill_(half)
    elif kind == "padded":
        a[:, : n // 2] = top
        b[:, : n // 2] = top
    elif kind == "padded60":
        a[:, : n // 2] = int(0.6 * top)
        b[:, : n // 2] = int(0.6 * top)
    elif kind == "low":
        a.fill_(0 if nonneg else -top)
        b.fill_(top)
    elif kind == "steps":  # a linear ramp against its reverse
        r = torch.linspace(0 if nonneg else -top, top, n, device=dev, dtype=torch.float64).round().to(torch.int32)
        a[:] = r
        b[:] = r.flip(0)
    return a, b


@pytest.mark.parametrize("n_power,batch,bits,nonneg", [
    (16, 10, 17, True), (16, 10, 18, False), (14, 38, 19, False), (13, 9, 19, True), (12, 40, 20, True),
    (10, 64, 20, False), (16, 10, 24, True), (15, 19, 24, True), (17, 5, 24, True), (17, 5, 24, False),
    (14, 38, 26, True), (13, 40, 27, False), (12, 40, 28, True), (9, 64, 30, True)])
@pytest.mark.parametrize("kind", ["max", "halfrange", "padded", "padded60", "low", "steps"])
def test_exact_holds_coherent_rows(gf, dev, n_power, batch, bits, nonneg, kind):
    a, b = operands(kind, 1 << n_power, batch, bits, nonneg, dev)
    c, e = gf.negacyclic_mul_split(a, b, input_bits=bits, non_negative=nonneg, return_error=True)
    assert torch.equal(c, exact(a, b))
    assert float(e.item()) < 0.5


@pytest.mark.parametrize("n_power,batch,bits,nonneg", [
    (16, 10, 24, True), (14, 38, 22, True), (13, 40, 24, False), (10, 64, 24, True),  # two limbs
    (16, 10, 16, False), (13, 40, 16, False), (11, 64, 18, True)])                    # one limb
def test_f64_plan_keeps_its_error(gf, dev, n_power, batch, bits, nonneg):
    # calls with FP64 tables report what their own limb plan leaves: the plan's passes
    # and the form with b whole differ at most by the order of roundings (a maximum
    # over batch N values moves by less than a factor of two)
    a, b = rows(gf, dev, 1 << n_power, batch, bits, nonneg, n_power + bits)
    kw = dict(input_bits=bits, non_negative=nonneg, precision="f64", return_error=True)
    prev = gf.set_split_tile(0)
    try:
        c0, e0 = gf.negacyclic_mul_split(a, b, **kw)
        gf.set_split_tile(1)
        c1, e1 = gf.negacyclic_mul_split(a, b, **kw)
    finally:
        gf.set_split_tile(prev)
    assert torch.equal(c0, c1) and torch.equal(c1, exact(a, b))
    assert float(e1.item()) <= 2 * float(e0.item())


@pytest.mark.parametrize("batch,bits", [(1, 24), (296, 24), (592, 24), (593, 24), (1201, 24), (2, 26), (701, 26), (889, 26), (3, 28)])
def test_exact_2e11_ctas_per_sm(gf, dev, batch, bits):
    # two or three CTAs per SM by the number of limbs and CTAs (two products each)
    a, b = rows(gf, dev, 1 << 11, batch, bits, True, batch + bits)
    a[0, 1024:] = 0
    c, e = gf.negacyclic_mul_split(a, b, input_bits=bits, non_negative=True, return_error=True)
    assert float(e.item()) < 0.5 and torch.equal(c, exact(a, b))


def test_exact_2e11_few_products_not_slower_than_the_chain(gf, dev):
    # two products of N = 2^11, 24 bits: 19 us against the limb chain's 21.6 (27 where
    # the one-kernel form spills for a third CTA per SM); sides in turn, best of many
    a, b = rows(gf, dev, 1 << 11, 2, 24, True, 5)
    tables = gf.ffnt_tables(11, "f32")
    out = torch.empty(a.shape, dtype=torch.int64, device=dev)
    ws = torch.empty(1 << 22, dtype=torch.uint8, device=dev)
    best = {}
    try:
        for _ in range(15):
            for on in (1, 0):
                gf.set_split_tile(on)
                t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                for k in range(40):
                    if k == 10:
                        t0.record()
                    gf.negacyclic_mul_split(a, b, out=out, input_bits=24, non_negative=True, tables=tables, workspace=ws)
                t1.record()
                torch.cuda.synchronize()
                t = t0.elapsed_time(t1)
                best[on] = min(t, best.get(on, t))
    finally:
        gf.set_split_tile(1)
    assert best[1] <= 1.05 * best[0]
