"""The tile compositor's rules against the sequential ones, on the CPU: the segments an edge is
binned under hold every cell its walk touches (slopes and positions of every size, wrapped ones
included), and the packed pixel arithmetic is pix's, channel by channel."""
import numpy as np
import pytest

ONE = 1 << 16


def i32(v):
    return (v + 2**31) % 2**32 - 2**31


def fxmul(a, b):
    return i32((a * b) >> 16)


def fxdiv(a, b):  # low half of the quotient, truncated
    q = (abs(a) << 16) // abs(b)
    return i32(-q if (a < 0) != (b < 0) else q)


def edge(ax, ay, bx, by):
    (ux, uy), (lx, ly) = ((ax, ay), (bx, by)) if by > ay else ((bx, by), (ax, ay))
    dx, dy = i32(lx - ux), i32(ly - uy)
    step = min(abs(fxdiv(dy, dx)), ONE) if dx else 0
    inv = fxdiv(dx, dy)
    ybot = i32(((uy + ONE) >> 16 << 16) - uy)
    return dict(uy=uy, ly=ly, x0=i32(ux + fxmul(inv, ybot)), inv=inv, step=step, start=uy >> 16, end=ly >> 16)


def cells(e, y, W):
    """First and last cell of the walk in row y (None: none)."""
    fu, fl = e["uy"] & 0xFFFF, e["ly"] & 0xFFFF
    st, en = y == e["start"], y == e["end"]
    cov = ((fl + 128) >> 8 if en else 256) - ((fu + 128) >> 8 if st else 0)
    xb = i32(e["x0"] + i32((y - e["start"]) * e["inv"]))
    x0 = i32(xb - fxmul(e["inv"], ONE - fu)) if st else i32(xb - e["inv"])
    x1 = i32(xb - fxmul(e["inv"], ONE - fl)) if en and fl else xb
    mn, mx = min(x0, x1), max(x0, x1)
    minp = mn >> 16
    if cov <= 0 or minp >= W:
        return None
    step = e["step"] if e["step"] > 0 else ONE
    if minp == mx >> 16:
        r = ((ONE - (i32(mx + mn) // 2 & 0xFFFF)) * cov) >> 8
    else:
        r = (ONE - (mn & 0xFFFF)) >> 1
    first = (r * step >> 16) + 128
    last = minp + max(0, -(-(cov * 256 - first) // step))  # the cell whose sum reaches cov
    return max(minp, 0), min(max(last, 0), W - 1)


def edge_segs(e, segs, w):
    fu, fl = e["uy"] & 0xFFFF, e["ly"] & 0xFFFF
    end = (e["end"] - e["start"]) * e["inv"] + e["x0"] - fxmul(e["inv"], ONE - fl)
    far = 1 << 29
    if abs(end) >= far or abs(e["x0"]) >= far or abs(e["inv"]) >= far:
        return 0, segs - 1
    a = e["x0"] - fxmul(e["inv"], ONE - fu)
    n = int(np.float32(66191.36) / np.float32(e["step"]) * np.float32(0.99999)) + 3 if e["step"] > 0 else 4
    lo, hi = (min(a, end) >> 16) - 2, (max(a, end) >> 16) + 2 + n
    return sum(lo >= k * w for k in range(1, segs)), sum(hi >= k * w for k in range(1, segs))


@pytest.mark.parametrize("segs,w", [(2, 1024), (2, 256), (3, 512), (4, 128), (4, 1024)])
def test_edges_stay_in_their_segments(segs, w):
    rng = np.random.default_rng(segs * w)
    W = segs * w - 37
    for k in range(3000):
        spread = float(rng.choice([2, 40, 600, 30000]))
        x = rng.uniform(-0.3, 1.3) * W
        pts = np.rint(65536 * np.clip([x, rng.uniform(-20, 60), x + rng.normal() * spread,
                                       rng.uniform(-20, 60) if k % 3 else rng.uniform(-2e4, 2e4)], -32767, 32767))
        ax, ay, bx, by = (int(v) for v in pts)
        if k % 5 == 0:
            by = ay + int(rng.integers(1, 400))  # nearly flat
        if ay == by:
            continue
        e = edge(ax, ay, bx, by)
        g = edge_segs(e, segs, w)
        for y in range(max(e["start"], -20), min(e["end"], 60) + 1):
            c = cells(e, y, W)
            if c:
                assert g[0] <= c[0] // w and c[1] // w <= g[1], (e, y, c, g)


def mul(a, b):  # pix's Ch8 product
    return (((a << 4) | (a >> 4)) * ((b << 4) | (b >> 4))) >> 16


def test_alpha0_powers():
    """k composites of alpha 0, one after the other, and as one packed step."""
    d = np.arange(256, dtype=np.uint64)
    steps = d.copy()
    for k in range(16):
        for lanes in (1, 0x01010101):
            v = d * lanes
            hi = (((v & 0x70707070) + 0x70707070) | v) & 0x80808080
            low = ~((hi >> 7) * 255) & 0xFFFFFFFF
            t = ((v & low) | 0x10101010) - k * 0x01010101
            got = (v & ~low & 0xFFFFFFFF) | (t & 0x0F0F0F0F & ((t >> 4 & 0x01010101) * 15) & low)
            assert (got == steps * lanes).all(), k
        steps = mul(steps, 255)
    assert (steps[1:16] == 0).all() and (mul(d, 255)[16:] == d[16:]).all()


def test_packed_source_over():
    rng = np.random.default_rng(1)
    d, clr = rng.integers(0, 2**32, (2, 200000), dtype=np.uint64)
    alpha = rng.integers(0, 256, 200000).astype(np.uint64)
    ch = lambda v, c: (v >> np.uint64(8 * c)) & np.uint64(255)
    inv = 255 - mul(ch(clr, 3), alpha)
    want = sum(np.minimum(mul(ch(clr, c), alpha) + mul(ch(d, c), inv), 255) << np.uint64(8 * c) for c in range(4))
    wide = lambda v: (v << 4) | (v >> 4)
    ra, ri = wide(alpha), wide(inv)
    pair = lambda a, b: (a >> 16) | ((b >> 16) << 16)
    e, o = d & 0x00FF00FF, (d >> 8) & 0x00FF00FF
    le, lo = (e << 4) | (e >> 4 & 0x000F000F), (o << 4) | (o >> 4 & 0x000F000F)
    half = lambda l: pair((l & 0xFFFF) * ri, (l >> 16) * ri)
    cap = lambda v: np.minimum(v & 0xFFFF, 255) | (np.minimum(v >> 16, 255) << 16)
    src = [wide(ch(clr, c)) * ra for c in range(4)]
    got = cap(pair(src[0], src[2]) + half(le)) | (cap(pair(src[1], src[3]) + half(lo)) << 8)
    assert (got == want).all()
