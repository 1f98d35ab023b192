"""The certificate of the tensor-core labels of any shape (ckm_wide.cu), redone on
the CPU: the shift and scale, the fp16 halves, the FP32 accumulation in several
orders, |c|^2 less each cluster's part of the bound, the scores and the bound T.

- The scores bound the exact ones as the kernel's comment derives it.
- A label that the certificate proves is the reference's, on sets with near ties,
  far centroids, an offset, tiny and huge values; with T / 64 labels are lost.
"""
import os
import re

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = open(os.path.join(ROOT, "cl-kmeans_gb300", "csrc", "ckm_wide.cu")).read()
F = np.float32
LD = np.longdouble


def f32(x):
    return np.asarray(x).astype(F)


def fma(a, b, c):  # one rounding (the products of floats are exact in FP64, the sums nearly)
    return f32(LD(1) * a * b + c)


def test_constants_are_the_kernels():
    """The lines that the emulation below restates."""
    code = re.sub(r"\s+", " ", SOURCE)
    for line in (
        "t2 = (3.001f * 0x1p-22f + 1.01f * 2.0f * fd * 0x1p-23f * 1.005f + (0.25f * fk + (sizeof(T) == 4 ? 18.0f : 26.0f)) * 0x1p-24f) * 1.002f;",
        "origin = sizeof(T) == 4 ? 0.0f : fmaf(__uint_as_float(s_omax), 0x1p-43f, 0x1p-120f) * scale;",
        "t1 = (4.1f * 0x1p-25f + 8.2f * origin) * sqrtf(fk) * 1.001f;",
        "w = (2.0f * t2 + t1 * 0x1p-7f) * 1.001f;",
        "s_cn[c] * (1.0f - (0.5f * w + 0x1p-24f))",
        "t00 = t1 * 32.0f + 0x1p-40f, wc = 2.0f * (w * 1.001f + 0x1p-22f) * 1.003f;",
        "ta = 2.0f * t2 + wc;",
        "rho = sizeof(T) == 4 ? 2.02f * (fd + 4.0f) * 0x1p-24f * 1.001f : 0x1p-40f;",
        "t0 = 2.0f * (fd + 8.0f) * 0x1p-149f * scale * scale;",
        "S = fmaf(ta * aa, aa, fmaf(t1, aa, fmaf(wc, h, t00)));",
        "T_ = (S + fmaf(rho, h + S, t0)) * (1.0f + 0x1p-10f);",
    ):
        assert line in code, line


def medians(C):
    """The origin: medians of three of 27 centroids, three times."""
    k = len(C)
    m = C[[lane * k // 27 for lane in range(27)]]
    for _ in range(3):
        m = np.median(m.reshape(-1, 3, m.shape[1]), axis=1)
    return m[0]


def split64(x):
    h = f32(x)
    return h, f32(x - h.astype(np.float64))


def shift(V, mu, scale, f64):
    if not f64:
        return fma(V, F(scale), f32(-LD(mu) * scale))
    (h, l), (mh, ml) = split64(V), split64(mu)
    return f32(f32(f32(h - mh) + f32(l - ml)) * F(scale))


def halves(x):
    hi = x.astype(np.float16)
    return hi, f32(x - f32(hi)).astype(np.float16)


def toward_zero(s):
    r = f32(s)
    over = np.abs(r.astype(np.float64)) > np.abs(s)
    return np.where(over, np.nextafter(r, F(0)), r)


def dot(x, c, order):
    """x.c of the halves: the cross products, then the high ones, in FP32."""
    (xh, xl), (ch, cl) = halves(x), halves(c)
    acc = np.zeros((len(x), len(c)), F)
    for a, b in ((xh, cl), (xl, ch), (xh, ch)):
        a, b = a.astype(np.float64), b.astype(np.float64)
        if order == "blocks":  # 16 products exactly, one addition cut off
            for f in range(0, a.shape[1], 16):
                acc = toward_zero(a[:, f:f + 16] @ b[:, f:f + 16].T + acc)
        else:
            fs = range(a.shape[1]) if order == "ascending" else range(a.shape[1] - 1, -1, -1)
            for f in fs:
                acc = toward_zero(np.outer(a[:, f], b[:, f]) + acc)
    return acc


def norms(x):
    """Sums of squares in pairs, eight features at a time."""
    x = np.pad(x, ((0, 0), (0, -x.shape[1] % 8)))
    total = np.zeros(len(x), F)
    for f in range(0, x.shape[1], 8):
        even, odd = np.zeros(len(x), F), np.zeros(len(x), F)
        for e in range(0, 8, 2):
            even, odd = fma(x[:, f + e], x[:, f + e], even), fma(x[:, f + e + 1], x[:, f + e + 1], odd)
        total = f32(total + f32(even + odd))
    return total


def screen(X, C, f64, order):
    d = X.shape[1]
    fd, fk = d, (d + 15) // 16 * 16
    mu = medians(C)
    if not f64:
        mu = f32(mu)
    cmax = np.abs(f32(C - mu)).max()
    e = np.frexp(cmax)[1] if cmax > 0 else 8
    scale = 2.0 ** min(60, max(-60, 8 - int(e)))
    x, c = shift(X, mu, scale, f64), shift(C, mu, scale, f64)
    t2 = (3.001 * 2.0 ** -22 + 1.01 * 2 * fd * 2.0 ** -23 * 1.005 + (0.25 * fk + (26 if f64 else 18)) * 2.0 ** -24) * 1.002
    origin = (np.abs(mu).max() * 2.0 ** -43 + 2.0 ** -120) * scale if f64 else 0.0
    t1 = (4.1 * 2.0 ** -25 + 8.2 * origin) * np.sqrt(fk) * 1.001
    w = (2 * t2 + t1 * 2.0 ** -7) * 1.001
    cn = f32(norms(c) * F(1 - (0.5 * w + 2.0 ** -24)))
    s = f32(-2.0 * dot(x, c, order).astype(np.float64) + cn.astype(np.float64))
    nx = norms(x).astype(np.float64) * (1 + 2.0 ** -15)
    a = np.sqrt(nx) * (1 + 2.0 ** -16)
    t00, wc = t1 * 32 + 2.0 ** -40, 2 * (w * 1.001 + 2.0 ** -22) * 1.003
    m1 = s.min(1).astype(np.float64)
    h = np.maximum(m1 + nx, 0)
    S = (2 * t2 + wc) * a * a + t1 * a + wc * h + t00
    rho = 2.0 ** -40 if f64 else 2.02 * (fd + 4) * 2.0 ** -24 * 1.001
    T = (S + rho * (h + S) + 2 * (fd + 8) * 2.0 ** -149 * scale * scale) * (1 + 2.0 ** -10)
    A = 2 * t2 * a * a + t1 * a + t00
    return dict(s=s, T=T, A=A, S=S, mu=mu, scale=scale, x=x)


def reference(X, C):
    """The reference's distances and labels (FP32, or FP64 for FP64 points)."""
    acc = np.zeros((len(X), len(C)), X.dtype)
    for f in range(X.shape[1]):
        t = (X[:, f][:, None] - C[:, f][None, :]).astype(X.dtype)
        acc = (LD(1) * t * t + acc).astype(X.dtype)
    return acc.argmin(1)


def sets(kind, n, d, k, f64, seed):
    rng = np.random.default_rng(seed)
    C = rng.uniform(-10, 10, (k, d))
    X = C[rng.integers(0, k, n)] + rng.standard_normal((n, d))
    if kind == "near":  # about the bisectors of pairs of centroids
        i, j = rng.integers(0, k, n), rng.integers(0, k, n)
        C = C[:1] + 0.05 * rng.standard_normal((k, d))
        step = 10.0 ** rng.uniform(-9, -2, (n, 1))
        X = (C[i] + C[j]) / 2 + step * (C[i] - C[j]) + 10 * rng.standard_normal((n, d)) * (rng.random((n, 1)) < 0.3)
    elif kind == "far":
        C[::7] *= 10.0 ** rng.uniform(1, 4, (len(C[::7]), 1))
    elif kind == "offset":
        X, C = X + 1000.0, C + 1000.0
    elif kind == "tiny":
        X, C = X * 1e-18, C * 1e-18
    elif kind == "huge":
        X, C = X * 1e15, C * 1e15
    t = np.float64 if f64 else F
    return X.astype(t), C.astype(t)


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("kind", ["plain", "near", "far", "offset", "tiny", "huge"])
@pytest.mark.parametrize("d,k", [(3, 40), (16, 64), (37, 20), (64, 33), (128, 16)])
def test_bound_and_proved_labels(d, k, kind, f64):
    X, C = sets(kind, 300, d, k, f64, d + k)
    ref = reference(X, C)
    proved = 0
    for order in ("ascending", "descending", "blocks"):
        r = screen(X, C, f64, order)
        xs, cs = (LD(X) - LD(r["mu"])) * LD(r["scale"]), (LD(C) - LD(r["mu"])) * LD(r["scale"])
        exact = (cs * cs).sum(1)[None, :] - 2 * (xs @ cs.T)
        s = LD(r["s"])
        lab = r["s"].argmin(1)
        at = np.arange(len(X))
        usable = (np.abs(r["x"]).max(1) < 2.0 ** 15)  # larger ones are not screened (fp16)
        low = exact - s
        assert np.all(low[usable] >= -LD(r["A"])[usable, None] / 2), (order, float((-low / r["A"][:, None]).max()))
        assert np.all((exact - s)[at, lab][usable] <= (r["S"] - r["A"] / 2)[usable])
        gap = np.partition(r["s"], 1, axis=1)
        gap = gap[:, 1].astype(np.float64) - gap[:, 0]
        sure = usable & (gap > r["T"])
        assert np.array_equal(lab[sure], ref[sure]), order
        proved += int(sure.sum())
    if kind != "near":
        assert proved >= 0.9 * 3 * len(X)


def test_a_smaller_bound_loses_labels():
    lost = 0
    for seed in range(6):
        X, C = sets("near", 2000, 64, 33, False, seed)
        ref = reference(X, C)
        r = screen(X, C, False, "blocks")
        gap = np.partition(r["s"], 1, axis=1)
        sure = (gap[:, 1].astype(np.float64) - gap[:, 0]) > r["T"] / 64
        lost += int((r["s"].argmin(1)[sure] != ref[sure]).sum())
    assert lost > 0
