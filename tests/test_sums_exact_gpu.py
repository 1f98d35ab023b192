"""Accuracy of the FP32 feature sums where one cluster holds most of many
points: as far from the FP64 sums as the rounding of the result, whatever the
length of the ranges that the tables take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROUND = 2.0 ** -24 * (1 + 2.0 ** -10)  # half an ulp of the result; pairs of floats add nothing to it


def skewed(torch, cuda, n, k, seed):
    g = torch.Generator(device=cuda).manual_seed(seed)
    lab = torch.randint(0, k, (n,), generator=g, device=cuda, dtype=torch.int32)
    lab[torch.rand(n, generator=g, device=cuda) < 0.9] = 0
    return lab


# shapes whose sums the generic kernel adds in FP64, at the ends of the table
# sizes; the last has fewer tables than the generic kernel has CTAs
@pytest.mark.parametrize("n,d,k", [(1 << 22, 128, 128), (1 << 22, 8, 1366), (1 << 21, 64, 190), (1 << 22, 5, 2100),
                                   (1 << 22, 12, 3000), (1 << 19, 240, 52), (1 << 19, 400, 30)])
@pytest.mark.parametrize("kind", ["equal", "normal"])
def test_centroid_update_of_a_dominant_cluster(ckm, cuda, n, d, k, kind):
    import torch
    g = torch.Generator(device=cuda).manual_seed(d)
    P = (torch.full((n * d,), 0.1, device=cuda) if kind == "equal"
         else torch.randn(n * d, generator=g, device=cuda) + 5)
    L = skewed(torch, cuda, n, k, n + k)
    C, M = torch.zeros(k * d, device=cuda), torch.zeros(k, dtype=torch.int32, device=cuda)
    S = ckm.new_scratch(d, k, cuda)
    ckm.centroid_update(P, C, L, M, S, n, d, k)
    for f in range(0, d, max(1, d // 16)):
        x = P[f * n:(f + 1) * n].double()
        want = torch.zeros(k, dtype=torch.float64, device=cuda).index_add_(0, L.long(), x)
        got = C[f * k:(f + 1) * k].double()
        assert bool(((got - want).abs() <= ROUND * want.abs()).all()), (f, float(((got - want) / want).abs().max()))
    assert not torch.any(S != 0)


@pytest.mark.parametrize("n,d,k", [(1 << 20, 128, 128), (1 << 21, 40, 256)])
def test_fused_of_a_dominant_cluster(ckm, cuda, n, d, k):
    import torch
    P = torch.full((n * d,), 0.1, device=cuda)
    C = 10.0 + torch.arange(k * d, device=cuda).float().reshape(d, k)
    C[:, 3] = 0.25
    N, L = torch.zeros(k * d, device=cuda), torch.zeros(n, dtype=torch.int32, device=cuda)
    M, S = torch.zeros(k, dtype=torch.int32, device=cuda), ckm.new_scratch(d, k, cuda)
    ckm.fused(P, C.reshape(-1).contiguous(), N, L, M, S, n, d, k)
    assert bool((L == 3).all()) and int(M[3]) == n and int(M.sum()) == n
    want = float(np.float32(0.1))
    assert float((N.reshape(d, k)[:, 3].double() - want).abs().max()) <= ROUND * want


@pytest.mark.parametrize("n,d,k", [(20011, 10, 4), (20011, 128, 128), (30001, 8, 1300), (3001, 4, 6000)])
def test_sums_beyond_the_float_range(ckm, cuda, n, d, k):
    """Partial sums beyond FP32's range whose FP64 sums, and means, are not:
    multiples of 2^120, with whole numbers (exact in any order) beside them, and
    clusters with an infinite and a NaN point."""
    import torch
    rng = np.random.default_rng(n + k)
    X = rng.integers(-8, 9, (n, d)).astype(np.float64)
    X[:, ::3] = rng.integers(1, 9, X[:, ::3].shape) * 2.0 ** 120
    lab = rng.integers(0, k, n)
    lab[: n // 2] = 1  # long sums
    lab[n - 1], lab[n - 2] = 2, 3
    X[lab == 2, 1] = 5.0
    where = np.nonzero(lab == 2)[0]
    X[where[0], 1] = np.inf
    X[np.nonzero(lab == 3)[0][-1], d - 1] = np.nan
    P = np.ascontiguousarray(X.astype(np.float32).T).reshape(-1)
    dP = torch.from_numpy(P).to(cuda)
    dL = torch.from_numpy(lab.astype(np.int32)).to(cuda)
    C, M, S = torch.zeros(k * d, device=cuda), torch.zeros(k, dtype=torch.int32, device=cuda), ckm.new_scratch(d, k, cuda)
    ckm.centroid_update(dP, C, dL, M, S, n, d, k, mode=ckm.MODE_DEFER)
    ckm.finalize(C, M, S, d, k)
    mass = np.bincount(lab, minlength=k)
    got = C.cpu().numpy().reshape(d, k)
    with np.errstate(all="ignore"):
        for f in range(d):
            want = (np.bincount(lab, weights=X[:, f], minlength=k) / mass).astype(np.float32)
            assert np.array_equal(got[f], want, equal_nan=True), (f, np.nonzero(got[f] != want)[0][:5])
    assert np.isinf(got[1, 2]) and np.isnan(got[d - 1, 3])
    assert not torch.any(S != 0)


# m, q: the FP64 product of q m and the rounded reciprocal of m rounds to another
# float than q does, q being the midpoint of two floats
MIDPOINTS = [
    (49, 27228575), (75, 29327761), (77, 30237505), (91, 24366061), (93, 27066901), (98, 26454107), (99, 21930277),
    (103, 26067659), (105, 22320305), (107, 29451291), (117, 20817589), (123, 31892409), (150, 29915121),
    (154, 30440621), (161, 27951659), (167, 32838917), (182, 31181453), (186, 27366901), (187, 32418583),
    (191, 31270513), (196, 28632851), (197, 28231067), (198, 24992261), (206, 30796555), (210, 27534425),
    (211, 33302149), (214, 25047515), (221, 27058693), (227, 24038417), (234, 19458689), (237, 30637779),
    (239, 26562607), (243, 22114497), (245, 26043025), (246, 23777441), (249, 23492523), (253, 31761835),
]


def test_means_are_rounded_quotients(ckm, cuda):
    """The mean is the FP64 quotient rounded to FP32, as ckm_finalize has it."""
    import torch
    n, d, k = 200000, 10, len(MIDPOINTS) + 1
    X = np.zeros((n, d))
    lab = np.full(n, k - 1)
    at = k
    for c, (m, q) in enumerate(MIDPOINTS):
        # q m as two floats far apart, so that no FP32 table adds both
        s = q * m
        high = s >> 20 << 20
        assert np.float32(high) == high and np.float32(s - high) == s - high
        lab[c] = lab[n - 1 - c] = c
        X[c, :], X[n - 1 - c, :] = high, s - high
        lab[at:at + m - 2] = c
        at += m - 2
    assert at < n // 2
    P = torch.from_numpy(np.ascontiguousarray(X.astype(np.float32).T).reshape(-1)).to(cuda)
    mass = np.bincount(lab, minlength=k)
    want = np.array([s / m for s, m in zip([q * m for m, q in MIDPOINTS], mass)]).astype(np.float32)
    assert all(np.float32(np.float64(q * m) * (1.0 / m)) != w for (m, q), w in zip(MIDPOINTS, want))
    # labels of a fused call: the centroids are far apart in a feature of its own
    X2 = np.concatenate([X, 1000.0 * lab[:, None] * 2.0 ** 20], axis=1)
    C = np.zeros((d + 1, k))
    C[d] = 1000.0 * np.arange(k) * 2.0 ** 20
    P2 = torch.from_numpy(np.ascontiguousarray(X2.astype(np.float32).T).reshape(-1)).to(cuda)
    dC = torch.from_numpy(C.astype(np.float32).reshape(-1)).to(cuda)
    N, L = torch.zeros((d + 1) * k, device=cuda), torch.full((n,), -1, dtype=torch.int32, device=cuda)
    M, S = torch.zeros(k, dtype=torch.int32, device=cuda), ckm.new_scratch(d + 1, k, cuda)
    ckm.fused(P2, dC, N, L, M, S, n, d + 1, k)
    assert np.array_equal(L.cpu().numpy(), lab) and np.array_equal(M.cpu().numpy(), mass)
    got = N.cpu().numpy().reshape(d + 1, k)
    for f in range(d):
        assert np.array_equal(got[f, : k - 1], want), (f, np.nonzero(got[f, : k - 1] != want)[0])
    # and of a deferred centroid update with ckm_finalize
    C1, M1, S1 = torch.zeros(d * k, device=cuda), torch.zeros_like(M), ckm.new_scratch(d, k, cuda)
    ckm.centroid_update(P, C1, L, M1, S1, n, d, k, mode=ckm.MODE_DEFER)
    ckm.finalize(C1, M1, S1, d, k)
    for f in range(d):
        assert np.array_equal(C1.cpu().numpy().reshape(d, k)[f, : k - 1], want), f
