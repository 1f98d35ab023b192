"""The certificate constants of the tensor-core iteration (ckm_tc.cu) as the
centroid kernels compute them, in FP32 with directed rounding: |c|^2 as a pair of
floats, the rounding errors' norms, t1, te and t2.  They are no smaller than the
same formulas in FP64, and with them the reference's label stays among the
candidates at scales down to where squares underflow."""
import os
import re

import numpy as np
import pytest

from test_tc_certificate_cpu import near_tie_set, reference_labels, scale_exponent

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = open(os.path.join(ROOT, "cl-kmeans_gb300", "csrc", "ckm_tc.cu")).read()
F = np.float32
LD = np.longdouble


def up(x):
    """x rounded up to a float."""
    r = F(x)
    return r if LD(r) >= LD(x) else np.nextafter(r, F(np.inf))


def mul_up(a, b):
    return up(LD(a) * LD(b))


def add_up(a, b):
    return up(LD(a) + LD(b))


def sqrt_up(a):
    return up(np.sqrt(LD(a)))


def two_sum(hi, lo, v):
    s = F(hi + v)
    b = F(s - hi)
    return s, F(lo + F(F(hi - F(s - b)) + F(v - b)))


def norm2(row):
    """|c|^2 of a centroid: 32 lanes, then a butterfly, as a pair of floats."""
    hi, lo = np.zeros(32, F), np.zeros(32, F)
    for f in range(0, len(row), 32):
        v = np.zeros(32, F)
        v[: len(row[f:f + 32])] = row[f:f + 32]
        sq = F(v * v)
        hi, lo = two_sum(hi, lo, sq)
        lo = F(lo + F(LD(v) * v - sq))
    for o in (16, 8, 4, 2, 1):
        at = np.arange(32) ^ o
        h, low = hi[at], lo[at]
        hi, lo = two_sum(hi, lo, h)
        lo = F(lo + low)
    return F(hi[0] + lo[0])


def constants(C, d_pad):
    d = C.shape[1]
    cn = np.array([norm2(c) for c in C], F)
    ec = scale_exponent(float(np.abs(C).max()))
    b = F(C * F(2.0 ** ec))
    e = F(b.astype(np.float16).astype(F) - b)
    ee = F((e * e).sum(1, dtype=F) * F(1 + 2.0 ** -14)).max()
    grow = F(1 + 2.0 ** -20)
    cm, fe = mul_up(sqrt_up(cn.max()), grow), mul_up(sqrt_up(ee), grow)
    fm = mul_up(add_up(fe, F(F(d) * F(2.0 ** -74))), F(2.0 ** -ec))
    gam, safety, cf = F(2 * F(d_pad) * F(2.0 ** -23)), F(1 + 2.0 ** -9), add_up(cm, fm)
    acc = mul_up(F(4 * gam), cf)
    t1 = mul_up(up(LD(4) * fm + acc), safety)
    te = mul_up(up(LD(4) * cf + acc), safety)
    t2 = mul_up(F(F(F(2 * F(2.0 ** -23)) * F(1.01)) + F(F(F(2) * F(F(d) + F(2))) * F(2.0 ** -24)) * F(1.01)), safety)
    return cn, ec, dict(cm=cm, t1=t1, te=te, t2=t2, t0=F(F(F(d) + F(8)) * F(2.0 ** -146)))


def test_lines_are_the_kernels():
    code = re.sub(r"\s+", " ", SOURCE)
    for line in (
        "cm = __fmul_ru(__fsqrt_ru(__uint_as_float(__ldcg(&it->cmax_bits))), 1.0f + 0x1p-20f);",
        "fe = __fmul_ru(__fsqrt_ru(__uint_as_float(__ldcg(&it->fmax_bits))), 1.0f + 0x1p-20f);",
        "fm = __fmul_ru(__fadd_ru(fe, (float)d * 0x1p-74f), ldexpf(1.0f, -ec));",
        "gam = 2.0f * (float)d_pad * 0x1p-23f, safety = 1.0f + 0x1p-9f, cf = __fadd_ru(cm, fm);",
        "acc = __fmul_ru(4.0f * gam, cf);",
        "it->t1 = __fmul_ru(__fmaf_ru(4.0f, fm, acc), safety);",
        "it->te = __fmul_ru(__fmaf_ru(4.0f, cf, acc), safety);",
        "it->t2 = __fmul_ru(2.0f * 0x1p-23f * 1.01f + 2.0f * ((float)d + 2.0f) * 0x1p-24f * 1.01f, safety);",
        "it->t0 = ((float)d + 8.0f) * 0x1p-146f;",
        "__uint_as_float(ee * (1.0f + 0x1p-14f))".replace("__uint_as_float(", "__float_as_uint("),
    ):
        assert line in code, line


@pytest.mark.parametrize("scale", [1e-15, 1e-3, 1.0, 30.0, 1e12])
@pytest.mark.parametrize("d,k", [(33, 40), (64, 100), (100, 30), (256, 20)])
def test_no_smaller_than_in_64_bits(d, k, scale):
    rng = np.random.default_rng(d + k)
    C = F(rng.standard_normal((k, d)) * scale * 10.0 ** rng.uniform(-3, 0, (k, 1)))
    d_pad = (d + 63) // 64 * 64
    cn, ec, c = constants(C, d_pad)
    c64 = LD(C)
    n2 = (c64 * c64).sum(1)
    # the pair's sum rounds once (and a little)
    assert np.all(np.abs(LD(cn) - n2) <= n2 * 2.0 ** -24 * (1 + 2.0 ** -10))
    sc = LD(2.0 ** ec)
    err = LD(F(C * F(2.0 ** ec)).astype(np.float16)) / sc - c64
    cm, fm = np.sqrt(n2).max(), np.sqrt((err * err).sum(1)).max()
    g, s = 2.0 * d_pad * 2.0 ** -23, 1 + 2.0 ** -10
    assert LD(c["cm"]) >= cm
    assert LD(c["t1"]) >= (4 * fm + 4 * g * (cm + fm)) * s
    assert LD(c["te"]) >= (4 * (cm + fm) + 4 * g * (cm + fm)) * s
    assert LD(c["t2"]) >= (2 * 2.0 ** -23 * 1.01 + 2 * (d + 2) * 2.0 ** -24 * 1.01) * s


@pytest.mark.parametrize("scale", [1e-21, 1e-19, 1e-4, 1.0, 1e13])
@pytest.mark.parametrize("d,k", [(128, 60), (100, 33)])
def test_reference_label_is_a_candidate(d, k, scale):
    rng = np.random.default_rng(d * 1000 + k)
    X, C = near_tie_set(600, d, k, rng, 2.0)
    X, C = F(X * F(scale)), F(C * F(scale))
    ref = reference_labels(X, C)
    d_pad = (d + 63) // 64 * 64
    cn, ec, c = constants(C, d_pad)
    ex = scale_exponent(float(np.abs(X).max()))
    xs, cs = F(X * F(2.0 ** ex)), F(C * F(2.0 ** ec))
    xq, cq = xs.astype(np.float16).astype(F), cs.astype(np.float16).astype(F)
    e = F(xq - xs)
    near, over = F(1 + 2.0 ** -14), F(1 + 2.0 ** -20)
    xn = F(np.sqrt(F((X * X).sum(1, dtype=F) * near)) * over)
    xe = F(F(F(np.sqrt(F((e * e).sum(1, dtype=F) * near)) * over) + F(F(d) * F(2.0 ** -149))) / F(2.0 ** ex))
    for order in (np.arange(d), np.arange(d)[::-1], rng.permutation(d)):
        dot = np.zeros((len(X), k), F)
        for f in order:
            dot = F(dot + np.outer(xq[:, f], cq[:, f]))
        s = F(-2.0 ** (1 - ex - ec) * dot.astype(np.float64) + cn)
        r = F(xn + c["cm"])
        T = (LD(c["t2"]) * r * r + LD(c["te"]) * xe + LD(c["t1"]) * xn + LD(c["t0"])) * (1 + 2.0 ** -10)
        cand = LD(s) <= (LD(s.min(1)) + T)[:, None]
        assert cand[np.arange(len(ref)), ref].all()
        single = cand.sum(1) == 1
        assert np.array_equal(cand[single].argmax(1), ref[single])
