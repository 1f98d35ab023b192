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
