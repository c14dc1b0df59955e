"""The fused epilogue's logarithm and rounding check (rnj_device.cuh,
neg_quarter_ln, undecided_at) restated in numpy: whenever the check accepts,
the float must be the reference's float (KimuraDistance.cpp:322-349,
JCdistance.cpp:171-183).  Fused multiply-adds are done in extended precision and
rounded to double once more, within the error terms the bound allows for.
"""
import os
import re

import numpy as np
import pytest

HERE = os.path.dirname(__file__)
LD = np.longdouble


def _table():
    text = open(os.path.join(HERE, "..", "rapidnj_b200", "csrc", "rnj_logtab_q.h")).read()
    rows = re.findall(r"\{(-?0x[0-9a-fp.+-]+), (0x[0-9a-fp.+-]+)\}", text)
    tab = np.array([[float.fromhex(a), float.fromhex(b)] for a, b in rows])
    assert tab.shape == (128, 2)
    off = int(re.search(r"kLnOff = (0x[0-9A-F]+)u", text).group(1), 16)
    ln2 = float.fromhex(re.search(r"kNegQuarterLn2 = (\S+);", text).group(1))
    return tab, off, ln2


TAB, OFF, NQLN2 = _table()


def fma(a, b, c):
    return (LD(1) * a * b + c).astype(np.float64)


def neg_quarter_ln(x):
    bits = np.ascontiguousarray(x).view(np.uint64)
    t2 = ((bits >> np.uint64(32)).astype(np.int64) - (OFF - 0x20000000)).astype(np.int64)
    # arguments of valid pairs: up to 1, and at least 2^-126 (a and b are multiples of 2^-41)
    assert (t2 >= 0x18000000).all() and (t2 <= 0x20096000).all()
    e = TAB[(t2 >> 13) & 127]
    hz = (t2 & 0xFFFFF) + OFF
    z = ((hz.astype(np.uint64) << np.uint64(32)) | (bits & np.uint64(0xFFFFFFFF))).view(np.float64)
    r = fma(z, e[:, 1], -1.0)
    assert np.abs(r).max(initial=0) < 2.0 ** -7
    dk = (t2 >> 20).astype(np.float64) - 512.0
    s = fma(dk, NQLN2, e[:, 0])
    q = np.full_like(r, -1.0 / 20.0)
    for c in (1.0 / 16.0, -1.0 / 12.0, 0.125, -0.25):
        q = fma(q, r, c)
    return fma(q, r, s)


def undecided(dd, m):
    lo = dd.view(np.uint64) & np.uint64(0xFFFFFFFF)
    k1 = (8 * m - (1 << 31)) % (1 << 32)
    return ((lo.astype(np.int64) * 8 + k1) % (1 << 32)) < 16 * m


def check(dd, ref, m, most):
    und = undecided(dd, m)
    got = dd.astype(np.float32)
    assert np.array_equal(got[~und].view(np.int32), ref[~und].view(np.int32))
    assert und.mean() <= most
    return und


def k2p(P, Q, n, L):
    ts = (P.astype(np.float64) / n).astype(np.float32).astype(np.float64)
    tv = (Q.astype(np.float64) / n).astype(np.float32).astype(np.float64)
    a, b = 1.0 - 2.0 * ts - tv, 1.0 - 2.0 * tv
    ok = (a > 0) & (b > 0)
    a, b = a[ok], b[ok]
    d = -0.5 * np.log(a) - 0.25 * np.log(b)
    dd = neg_quarter_ln((a * a) * b)
    m = 4096 + L
    # half of the margin covers the difference (in units of 2^-53, relative)
    rel = np.abs(dd - d) / np.where(d > 0, d, 1.0) * 2.0 ** 53
    assert (rel <= m / 2 + 4).all()
    check(dd, d.astype(np.float32), m, 4.0 * m / 2.0 ** 29 + 1e-4)


@pytest.mark.parametrize("n", [1, 2, 3, 7, 100, 997, 1000, 2048])
def test_k2p_exhaustive(n):
    P, Q = np.meshgrid(np.arange(n + 1), np.arange(n + 1), indexing="ij")
    keep = P + Q <= n
    k2p(P[keep], Q[keep], float(n), n)


def test_k2p_large_counts():
    rng = np.random.default_rng(0)
    n = rng.integers(2048, 65536, size=1_500_000)
    P = (rng.random(n.size) ** 3 * 0.4 * n).astype(np.int64)  # near identity and beyond
    Q = (rng.random(n.size) ** 3 * 0.45 * n).astype(np.int64)
    k2p(P, Q, n.astype(np.float64), 65535)
    # next to the saturation boundary 2 P + Q = n
    Q = (rng.random(n.size) * 0.5 * n).astype(np.int64)
    P = np.maximum(0, (n - Q) // 2 - rng.integers(0, 4, size=n.size))
    k2p(P, Q, n.astype(np.float64), 65535)


def test_identical_pairs_give_minus_zero():
    dd = neg_quarter_ln(np.ones(1))
    assert dd[0] == 0.0 and np.signbit(dd[0])


@pytest.mark.parametrize("n", [1, 2, 7, 100, 997, 10000, 65535])
@pytest.mark.parametrize("alpha", [4, 20])
def test_jc_exhaustive(n, alpha):
    b = (alpha - 1.0) / alpha
    p = (np.arange(n + 1).astype(np.float32) / np.float32(n)).astype(np.float32)
    q = p.astype(np.float64) / b
    # the float comparison that decides saturation
    top = np.float32(0.75) if alpha == 4 else np.float32(0.95) + np.float32(2.0 ** -24)
    assert np.array_equal(q >= 1.0, p >= top)
    p, q = p[q < 1.0], q[q < 1.0]
    d = -b * np.log(1.0 - q)
    # the device's q is the correctly rounded quotient too (div_by_b), so 1 - q is the same
    dd = (4.0 * b) * neg_quarter_ln(1.0 - q)
    check(dd, d.astype(np.float32), 4096, 1e-3)


def test_protein_kimura():
    rng = np.random.default_rng(3)
    v = rng.integers(1, 65536, size=2_000_000)
    mism = (rng.random(v.size) ** 2 * 0.75 * v).astype(np.int64)
    p = (mism.astype(np.float32) / v.astype(np.float32)).astype(np.float32)
    p = p[p < np.float32(0.75)]
    sq = (p * p).astype(np.float32).astype(np.float64)
    p = p.astype(np.float64)
    ref = np.abs((-np.log((1.0 - p) - sq * 0.2)).astype(np.float32))
    dd = neg_quarter_ln(fma(sq, -0.2, 1.0 - p))
    und = undecided(dd, 4096 + 2 * 65535)
    got = np.abs(np.float32(4.0) * dd.astype(np.float32))
    assert np.array_equal(got[~und].view(np.int32), ref[~und].view(np.int32))
    assert und.mean() < 2e-3
    # the float comparison of the band's upper end
    edge = np.float32(0.93)
    for f in (np.nextafter(edge, np.float32(0)), edge, np.nextafter(edge, np.float32(1))):
        assert (float(f) > 0.930) == (f >= edge)
