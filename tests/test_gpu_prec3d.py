"""Precision mode's FP64 tet update: every rounding is written out, so a host evaluation
with correctly rounded operations (multiply-adds through exact fractions) gives the same
bits.  The inputs take two corner times a few units in the last place apart, where the
inner discriminant cancels and its sign hangs on the last rounding."""
import math
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LARGE = 1e7


def _fma(a, b, c):
    if not all(map(math.isfinite, (a, b, c))):
        return a * b + c
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _ms(swap, x, y, z, w):  # x*y - z*w, the second product fused if swap
    return _fma(-z, w, x * y) if swap else _fma(x, y, -(z * w))


def _sqrt32(x):
    return float(np.sqrt(np.float32(x))) if x >= 0 else math.nan


def _roots(p, q, r):
    delta = _ms(False, q, q, 4 * p, r)
    if not delta >= 0 or p == 0:
        return []
    sd, i = math.sqrt(delta), 1.0 / (2 * p)
    return [(-q + sd) * i, (-q - sd) * i]


def _edge(TX, TC, XX, XC, CC):
    T = TC - TX
    out = [TX + _sqrt32((XX + XC) + (XC + CC)), TC + _sqrt32(CC)]
    for l in _roots(_ms(False, XX * T, T, XX, XX), _ms(False, (XC + XC) * T, T, 2 * XX, XC), _ms(False, T * T, CC, XC, XC)):
        if 0 <= l <= 1:
            out.append(_fma(TX, l, TC * (1 - l)) + _sqrt32(_fma(_fma(l, XX, XC), l, _fma(l, XC, CC))))
    return out


def _update(k, TA, TB, TC, aa, ab, ac, bb, bc, cc):
    """aa = AC.AC, ab = AC.BC, ac = AC.CD, bb = BC.BC, bc = BC.CD, cc = CD.CD"""
    out = [LARGE] + _edge(TB, TC, bb, bc, cc) + _edge(TA, TC, aa, ac, cc)
    T = TB - TA
    gx, gy, gz = aa - ab, ab - bb, ac - bc
    u2 = _ms(False, bb * T, T, gy, gy)
    u3 = _ms(False, (ab + ab) * T, T, 2 * gx, gy)
    u5 = _ms(False, (bc + bc) * T, T, 2 * gy, gz)
    p = (_ms(False, T * T, aa, gx, gx) + u2) - u3
    q = ((-u2 * 2 + u3) + _ms(False, (ac + ac) * T, T, 2 * gx, gz)) - u5
    r = (_ms(False, T * T, bb, gy, gy) + u5) + _ms(False, T * T, cc, gz, gz)
    for l in _roots(p, q, r):
        m = 1 - l
        if 0 <= l <= 1:
            x, y, z = _fma(l, aa, m * ab) + ac, _fma(l, ab, m * bb) + bc, _fma(l, ac, m * bc) + cc
            out.append(_fma(TA, l, TB * m) + _sqrt32((x * l + y * m) + z))
    A, B = TC - TA, TC - TB
    s, t, h = _ms(False, A, ab, B, aa), _ms(k < 3, A, bc, B, ac), -_ms(True, A, bb, B, ab)
    p1, p2 = _ms(False, A * A, aa, aa, aa), _ms(False, bb * A, A, ab, ab)
    p3, p4 = _ms(False, (ab + ab) * A, A, 2 * aa, ab), _ms(False, (ac + ac) * A, A, 2 * aa, ac)
    p5 = _ms(k == 2, (bc + bc) * A, A, 2 * ab, ac)
    p = _fma(p3 * s, h, _fma(p2 * s, s, p1 * h * h))
    q = _fma(p5 * s, h, _fma(p4 * h, h, _fma(p2 * 2 * s, t, p3 * t * h)))
    r = _fma(_ms(False, A * A, cc, ac, ac) * h, h, _fma(_ms(False, A * A, bb, ab, ab) * t, t, p5 * t * h))
    for a in _roots(p, q, r):
        b = _fma(s, a, t) * (1.0 / (h + 0.00000001))
        c = 1 - a - b
        if 0 <= a <= 1 and 0 <= b <= 1 and 0 <= c <= 1:
            x, y = _fma(a, aa, _fma(b, ab, ac)), _fma(a, ab, _fma(b, bb, bc))
            out.append(_fma(TC, c, _fma(TA, a, TB * b)) +
                       _sqrt32(_fma(x, a, _fma(y, b, _fma(a, ac, _fma(b, bc, cc))))))
    return min(v for v in out if not math.isnan(v))


def _apexes(row):
    A, B, C, D, acbc, bccd, accd, adbd, acad, bcbd = map(float, row)
    adbc, acbd = acbc + bccd, acbc + accd
    cdbd, adcd = adbd - acbd, adbd - adbc
    cdcd, adad, acac = adcd - accd, adcd + acad, acad - accd
    bdbd, bcbc = bcbd + cdbd, bcbd - bccd
    return [_update(0, B, D, C, bcbc, -bccd, -acbc, cdcd, accd, acac),
            _update(1, A, D, C, acac, -accd, -acbc, cdcd, bccd, bcbc),
            _update(2, A, B, D, adad, adbd, -adcd, bdbd, -cdbd, cdcd),
            _update(3, A, B, C, acac, acbc, accd, bcbc, bccd, cdcd)]


@pytest.mark.parametrize("flat", [1.0, 0.03])
def test_update_has_the_stated_roundings(eik, flat):
    rng = np.random.default_rng(int(1000 * flat))
    n = 600
    p = rng.normal(size=(n, 4, 3)) * [0.05, 0.05, 0.05 * flat]
    m = rng.normal(size=(n, 3, 3))
    m = np.einsum("nij,nkj->nik", m, m) + 0.2 * np.eye(3)
    v = lambda i, j: p[:, j] - p[:, i]  # noqa: E731
    dot = lambda a, b: np.einsum("ni,nij,nj->n", a, m, b)  # noqa: E731
    AC, AD, BC, BD, CD = v(0, 2), v(0, 3), v(1, 2), v(1, 3), v(2, 3)
    g = np.stack([dot(AC, BC), dot(BC, CD), dot(AC, CD), dot(AD, BD), dot(AC, AD), dot(BC, BD)], 1).astype(np.float32)
    w = rng.normal(size=(n, 3))
    w = np.einsum("nij,nj->ni", np.linalg.cholesky(m), w / np.linalg.norm(w, axis=1, keepdims=True))
    t = (1.0 + np.einsum("nki,ni->nk", p, w)).astype(np.float32)
    near, a, b = rng.random(n) < 0.7, rng.integers(0, 4, n), rng.integers(0, 4, n)
    i = np.arange(n)[near]
    t[i, a[near]] = (t[i, b[near]].view(np.int32) + rng.integers(-30, 31, i.size).astype(np.int32)).view(np.float32)
    k = rng.integers(0, 4, n)
    t[np.arange(n), k] = 5.0
    rows = np.concatenate([t, g], 1)
    got = eik.selftest_local_update(7, rows)[np.arange(n), k]
    want = np.array([min(np.float32(_apexes(r)[k[j]]), np.float32(5.0)) for j, r in enumerate(rows)], np.float32)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert (got < 5.0).mean() > 0.9
