"""The ratio pass's logarithm (log_pair, xpass.cuh), its constants read from
the source: every float of one period of its argument reduction, and the ends
of the range it is given, against float64 (CPU)."""
import os
import re

import numpy as np

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deconwolf_b200", "csrc", "xpass.cuh")
F = np.float32


def _constants():
    text = open(SRC).read()
    body = text[text.index("float2 log_pair(float2 q)"):]
    body = body[: body.index("\n}")]
    poly = [F(c) for c in re.findall(r"both\((-?0\.\d+)f\)\)?;", body)]
    lo, hi = re.search(r"both\((\S+?)f \* kScale\), t\)", body), re.search(r"both\((\S+?)f \* kScale\), __fadd2", body)
    return poly, F(lo.group(1)), F(hi.group(1)), int(re.search(r"i0 - (0x[0-9a-f]+)\)", body).group(1), 16)


def _fma(a, b, c):
    # the product of two floats is exact in float64
    return (a.astype(np.float64) * np.asarray(b, np.float64) + c).astype(F)


def _log(q):
    poly, ln2_lo, ln2_hi, mid = _constants()
    assert len(poly) == 10 and float(ln2_hi) == 355 / 512
    i = q.view(np.int32)
    k = (i - np.int32(mid)) & np.int32(np.uint32(0xff800000).view(np.int32))
    e = k.astype(F)
    f = (i - k).view(F) - F(1)
    p = np.full_like(f, poly[0])
    for c in poly[1:]:
        p = _fma(p, f, c)
    t = (f * f) * p
    lo = _fma(e, ln2_lo / F(8388608), t)
    return _fma(e, ln2_hi / F(8388608), f + lo)


def _ulps(q):
    exact = np.log(q.astype(np.float64))
    unit = np.spacing(np.abs(exact).astype(F)).astype(np.float64)
    return np.abs(_log(q) - exact) / unit


def test_every_float_of_one_period():
    mid = _constants()[3]
    worst = total = n = 0.0
    for a in range(mid, mid + (1 << 23), 1 << 20):
        q = np.arange(a, min(a + (1 << 20), mid + (1 << 23)), dtype=np.int32).view(F)
        q = q[q != 1]
        u = _ulps(q)
        worst, total, n = max(worst, u.max()), total + u.sum(), n + u.size
    assert _log(np.array([1.0], F))[0] == 0
    assert worst < 0.86 and total / n < 0.26


def test_ends_of_the_range():
    rng = np.random.default_rng(3)
    tiny, big = np.finfo(F).tiny, np.finfo(F).max
    q = np.concatenate([[tiny, big], np.exp(rng.uniform(np.log(tiny), np.log(big), 200000))]).astype(F)
    assert _ulps(q[(q >= tiny) & (q <= big)]).max() < 0.86
