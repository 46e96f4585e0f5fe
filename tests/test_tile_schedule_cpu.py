"""CPU checks of the index schedule of the 2^LT-point tiles (gf_tile.cuh,
gf_tile_pass.cuh, the tile pass of gf_special.cu, exact_tile's order of U), restated
in Python: every thread's register points, the padded transpose buffer, and for every
butterfly the table entry that the staged twiddles give it against the entry of the
plain stage loop."""
import numpy as np
import pytest

R = 16


def shape(LT):
    P = 1 << LT
    HT = P // R
    HI0 = LT - 8
    N0 = 8 if HI0 == 4 else 7
    return P, HT, LT - 4, LT - 8, HI0, N0, HT + 1, 9  # P, threads, W1, W2, HI0, N0, S0, S2


def point(t, r, W):
    return ((t & ((1 << W) - 1)) | ((t >> W) << (W + 4))) + (r << W)


@pytest.mark.parametrize("LT", [11, 12])
def test_windows_and_buffer(LT):
    P, HT, W1, W2, *_ = shape(LT)
    for W in (W1, W2, 0):
        e = np.array([[point(t, r, W) for r in range(R)] for t in range(HT)])
        assert sorted(e.ravel()) == list(range(P))
        pos = e + (e >> 4)
        assert len(set(pos.ravel())) == P and pos.max() < P + P // 16
        base = pos[:, :1]
        off = np.array([(r << W) + ((r << W) >> 4) for r in range(R)])
        assert (pos == base + off).all()  # a base and immediates
        # 8-byte points: a warp's access touches every 8-byte column of 32 banks twice, 16-byte ones in quarters
        for r in range(R):
            for w0 in range(0, HT, 32):
                assert max(np.bincount(pos[w0:w0 + 16, r] % 16)) == 1
                for q in range(0, 32, 8):
                    assert max(np.bincount(pos[w0 + q:w0 + q + 8, r] % 8)) == 1


def staged_even(LT, T, m):
    """stage_twiddles: position -> table entry; short transforms (m < 11) have 2^(m-1) entries."""
    P, HT, W1, W2, HI0, N0, S0, S2 = shape(LT)
    entries = (1 << (m - 1)) if m < 11 else 1 << 60
    tw = {}

    def put(at, e):
        if e < entries:
            assert at not in tw and 0 <= at < N0 * S0 + 16 * S2 + 8
            tw[at] = e

    inner, middle, outer = (N0 - 8) * S0, N0 * S0, N0 * S0 + 16 * S2
    for t in range(HT):
        if HI0 == 4:
            put(inner + t, (T << 8) + t)
        for k in range(7):
            p = (0 if k == 0 else (k - 1) * HT if k < 3 else (k - 3) * HT) + t
            lg = 0 if k == 0 else 1 if k < 3 else 2
            put(inner + (p >> lg) + ((1 << lg) + (p & ((1 << lg) - 1))) * S0, (T << (LT - 3 + lg)) + 2 * p)
        if t < 128:
            i, pos = t >> 3, t & 7
            lg = pos.bit_length()
            put(middle + i * S2 + pos, (T << (4 + lg)) + (i << lg) + (0 if pos == 0 else 2 * (pos - (1 << (lg - 1)))))
        if t < 8:
            lg = t.bit_length()
            put(outer + t, (T << lg) + (0 if t == 0 else 2 * (t - (1 << (lg - 1)))))
    return tw, inner, middle, outer


@pytest.mark.parametrize("LT,m,T", [(11, 11, 0), (11, 11, 5), (11, 11, 511), (12, 12, 0)] +
                         [(11, m, 0) for m in range(4, 11)])
def test_even_twiddles(LT, m, T):
    P, HT, W1, W2, HI0, N0, S0, S2 = shape(LT)
    tw, inner, middle, outer = staged_even(LT, T, m)
    seen = set()
    for W, HI in ((W1, 4), (W2, 4), (0, HI0)):
        for t in range(HT):
            if m >= W + 4:
                mask = (1 << (m - 4 - W)) - 1
                at, st = ((outer, 1) if W == W1 else (middle + ((t >> W2) & mask) * S2, 1) if W == W2
                          else (inner + (t & mask), S0))
                bits = range(HI)
            elif m > W:
                at, st, bits = outer + 4, 1, range(m - W)
            else:
                continue
            for pb in bits:
                for r in range(R):
                    if r & (1 << pb):
                        continue
                    if m >= W + 4:
                        h, nt = r >> (pb + 1), 1 << (3 - pb)
                        got = tw[at + ((nt >> 1) + (h >> 1)) * st]
                    else:
                        nt = 1 << (m - W - 1 - pb)
                        h = (r >> (pb + 1)) & (nt - 1)
                        got = tw[at + (h >> 1)]
                    e, q = point(t, r, W), W + pb  # bit of the tile's points, of the transform's in a tile of several
                    u = m - 1 - q
                    want = (T << u) + ((e & ((1 << m) - 1)) >> (q + 1))
                    # an odd entry is i times the even one before it; a stage with one
                    # twiddle per thread stages the entry itself
                    assert got == want if (m >= W + 4 and nt == 1) else got + (h & 1) == want and got % 2 == 0
                    seen.add((W, pb, e))
    assert len(seen) == m * P // 2  # every butterfly of every stage once


@pytest.mark.parametrize("LT,T,s0,neg", [(11, 0, 0, 0), (11, 3, 2, 0), (11, 3, 2, 1), (12, 0, 0, 1), (12, 9, 4, 0)])
def test_pass_twiddles(LT, T, s0, neg):
    # the drop-in's passes stage every twiddle of the caller's table
    P, HT, W1, W2, HI0, *_ = shape(LT)
    N0, S0, S2 = (15 if HI0 == 4 else 14), HT + 1, 17
    inner, middle, outer = (N0 - 16) * S0, N0 * S0, N0 * S0 + 16 * S2

    def base(u):
        return (T << u) + ((1 << (s0 + u)) if neg else 0)

    tw = {}

    def put(at, e):
        assert at not in tw and 0 <= at < N0 * S0 + 16 * S2 + 16
        tw[at] = e

    for t in range(HT):
        for k in range(N0):
            q = k + 16 - N0
            lg = q.bit_length() - 1
            p = (q - (1 << lg)) * HT + t
            put(inner + (p >> lg) + ((1 << lg) + (p & ((1 << lg) - 1))) * S0, base(LT - 4 + lg) + p)
        for k in range(256 // HT):
            p = k * HT + t
            i, pos = p >> 4, p & 15
            if pos:
                lg = pos.bit_length() - 1
                put(middle + i * S2 + pos, base(4 + lg) + (i << lg) + pos - (1 << lg))
        if 0 < t < 16:
            lg = t.bit_length() - 1
            put(outer + t, base(lg) + t - (1 << lg))
    for W, HI in ((W1, 4), (W2, 4), (0, HI0)):
        for t in range(HT):
            at, st = (outer, 1) if W == W1 else (middle + (t >> W2) * S2, 1) if W == W2 else (inner + t, S0)
            for pb in range(HI):
                for r in range(R):
                    if not r & (1 << pb):
                        q = W + pb
                        assert tw[at + ((1 << (3 - pb)) + (r >> (pb + 1))) * st] == base(LT - 1 - q) + (point(t, r, W) >> (q + 1))


@pytest.mark.parametrize("LT", [11, 12])
def test_special_twiddles(LT):
    P, HT, W1, W2, HI0, *_ = shape(LT)
    for W, HI in ((0, HI0), (W2, 4), (W1, 4)):
        for t in range(HT):
            lo = 0 if W == 0 else t & ((1 << W2) - 1) if W == W2 else t
            for i in range(HI):
                for r in range(R):
                    if not r & (1 << i):
                        got = (1 << (W + i)) + lo + ((r & ((1 << i) - 1)) << W)
                        assert got == (1 << (W + i)) + (point(t, r, W) & ((1 << (W + i)) - 1))


def test_exact_tile_order_of_u():
    # U of point j in the tables' order: each 4096-point tile permuted e -> (e >> 4) + 256 (e & 15)
    for g in (0, 1, 2, 7):
        for t in range(128):
            for r in range(R):
                j = 2048 * g + 16 * t + r
                assert ((g >> 1) << 12) + ((g & 1) << 7) + t + 256 * r == (j & ~4095) | ((j & 4095) >> 4) | ((j & 15) << 8)
