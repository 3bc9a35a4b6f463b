"""The quantised box test's float form (csrc/quantised.cuh SetUp and
csrc/quantise.cu Cells), restated in numpy: for any ray its near plane is at
most, and its far plane at least, what the slab test computes in floats."""
import numpy as np
import pytest

F = np.float32


def fma(a, b, c):
    """Float32 fused multiply-add: the product is exact in float64, and the
    float64 sum's rounding is 2^-29 of the float32 result's."""
    with np.errstate(all="ignore"):
        return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def planes(lo, hi, glo, cell, o, d):
    """(near, far) of both forms for boxes [lo, hi] on one axis."""
    with np.errstate(all="ignore"):
        inv = F(1.0) / d
        neg = np.signbit(inv)
        nb, fb = np.where(neg, hi, lo), np.where(neg, lo, hi)
        exact = (nb - o) * inv, (fb - o) * inv
        ql = np.floor((lo.astype(np.float64) - glo) / cell) - 1
        qh = np.ceil((hi.astype(np.float64) - glo) / cell) + 1
        assert (ql >= 0).all() and (qh <= 65535).all()
        s = cell * inv
        b0 = (glo - o) * inv
        big = ~(np.abs(s) <= F(1e30))
        s = np.where(big, np.copysign(F(1e30), inv), s)
        b0 = np.where(big, (glo - o) / cell * s, b0).astype(F)
        e = np.abs(b0) * F(6.0e-7)
        ok = (np.abs(s) >= F(1e-30)) & (np.abs(b0) <= F(1e37))
        base = np.full_like(s, -8388608.0)
        bn, bf = fma(base, s, b0 - e), fma(base, s, b0 + e)
        qn, qf = np.where(neg, qh, ql), np.where(neg, ql, qh)
        near = fma((8388608.0 + qn).astype(F), s, bn)
        far = fma((8388608.0 + qf).astype(F), s, bf)
    return exact, (near, far), ok, big


@pytest.mark.parametrize("extent", [1e-3, 1.0, 100.0, 1e6])
@pytest.mark.parametrize("away", [0.0, 1.0, 30.0, 1e3, 1e6])
def test_box_test_is_conservative(extent, away):
    rng = np.random.default_rng(int(away) + 7)
    n = 200_000
    cell = F(extent) / F(65500.0)
    glo = F(F(extent) * F(rng.uniform(-2, 2)))
    base = glo + F(8.0) * cell
    a, b = (base + F(extent) * rng.uniform(0, 1, n).astype(F) for _ in range(2))
    lo, hi = np.minimum(a, b), np.maximum(a, b)
    thin = rng.random(n) < 0.3
    hi = np.where(thin, lo, hi)
    o = (glo + F(extent) * ((away + rng.uniform(0, 1, n)) * rng.choice([-1, 1], n))).astype(F)
    on = rng.random(n) < 0.2
    o = np.where(on, lo, o)  # on a plane
    d = (rng.choice([-1, 1], n) * 10.0 ** rng.uniform(-12, 1, n)).astype(F)
    (en, ef), (qn, qf), ok, big = planes(lo, hi, glo, cell, o, d)
    use = ok & ~big & ~np.isnan(en) & ~np.isnan(ef)
    assert use.mean() > 0.9
    assert (qn[use] <= en[use]).all() and (qf[use] >= ef[use]).all()
    # A zero component: inside the box's planes, the axis must not reject any
    # t of a ray whose largest component is at least 1e-10.
    for zero in (F(0.0), F(-0.0)):
        _, (qn, qf), ok, _ = planes(lo, hi, glo, cell, o, np.full(n, zero))
        inside = ok & (o >= lo) & (o <= hi)
        assert (qn[inside] <= -1e29).all() and (qf[inside] >= 1e29).all()
