"""The tensor-core labels (ckm_wide.cu) where they are given up or prove little:
waits that run out, and sets with points far outside, centroids far outside,
equal centroids or many ties.  The labels are the oracle's either way, and the
counts and sums are theirs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [  # n, d, k: four and two epilogue groups, one and two point stages, the last with FP64 centroids beyond shared memory
    (1, 9, 2), (129, 9, 17), (45001, 10, 30), (20000, 16, 64), (60007, 33, 40), (9001, 100, 100), (5003, 128, 256),
]


def check(ckm, oracle, cuda, X, Cr, dtype):
    import torch
    ft = np.float32 if dtype == "f32" else np.float64
    n, d = X.shape
    k = Cr.shape[0]
    P, C = (np.ascontiguousarray(a.astype(ft).T).reshape(-1) for a in (X, Cr))
    ref = (oracle.label_f32 if dtype == "f32" else oracle.label_f64)(P, n, d, k, C).astype(np.int64)
    dP, dC = torch.from_numpy(P).to(cuda), torch.from_numpy(C).to(cuda)
    dL = torch.full((n,), -1, dtype=torch.int32 if dtype == "f32" else torch.int64, device=cuda)
    dL2, dM = torch.full_like(dL, -1), torch.full((k,), -1, dtype=dL.dtype, device=cuda)
    dN, S = torch.zeros_like(dC), ckm.new_scratch(d, k, cuda)
    ckm.labeling(dP, dC, dL2, n, d, k)
    ckm.fused(dP, dC, dN, dL, dM, S, n, d, k)
    for got in (dL2, dL):
        lab = got.cpu().numpy()
        assert np.array_equal(lab, ref), (n, d, k, int((lab != ref).sum()))
    mass = np.bincount(ref, minlength=k)
    assert np.array_equal(dM.cpu().numpy(), mass), (n, d, k)
    assert not torch.any(S != 0), (n, d, k)
    # FP32 or FP64 partial sums of at most a cluster's points, and the division
    u = 2.0 ** -24 if dtype == "f32" else 2.0 ** -52
    P2, N = P.reshape(d, n).astype(np.float64), dN.cpu().numpy().reshape(d, k)
    has = mass > 0
    for f in range(0, d, 7):
        want, size = (np.bincount(ref, weights=w, minlength=k) for w in (P2[f], np.abs(P2[f])))
        assert np.all(np.abs(N[f] * mass - want)[has] <= u * ((mass + 4) * size)[has]), (n, d, k, f)
    assert np.all(np.isnan(N[:, ~has]))


def mixture(n, d, k):
    rng = np.random.default_rng(n + 31 * d + k)
    centres = rng.uniform(-10, 10, (k, d))
    X = centres[rng.integers(0, k, n)] + rng.standard_normal((n, d))
    return rng, X, centres + 0.1 * rng.standard_normal((k, d))


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("limit_ns", ["0", "700", "4000"])
def test_waits_that_run_out(ckm, oracle, cuda, monkeypatch, dtype, limit_ns):
    """At 0 every wait for points, scores or a free stage that is not over when
    it begins runs out; the CTA then labels its points without the tensor cores."""
    monkeypatch.setenv("CKM_FUSED_UMMA", "1")
    monkeypatch.setenv("CKM_WIDE_TEST_WAIT_NS", limit_ns)
    for n, d, k in SHAPES:
        _, X, C = mixture(n, d, k)
        check(ckm, oracle, cuda, X, C, dtype)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("kind", ["far_points", "far_centroid", "far_centroids", "equal_centroids", "pairs", "lattice",
                                  "few_far", "nan_points"])
def test_sets_that_prove_little(ckm, oracle, cuda, monkeypatch, dtype, kind):
    monkeypatch.setenv("CKM_FUSED_UMMA", "1")
    for n, d, k in SHAPES:
        rng, X, C = mixture(n, d, k)
        if kind == "far_points":
            X[::3] *= 1e5
        elif kind == "few_far":
            X[::100] *= 1e4
        elif kind == "nan_points":
            X[::50, d - 1] = np.nan
        elif kind == "far_centroid":
            C[k // 2] *= 1e3
        elif kind == "far_centroids":
            C[: k // 2] *= 10.0 ** rng.uniform(0, 6, (k // 2, 1))
        elif kind == "equal_centroids":
            C[:] = C[0]
        elif kind == "pairs":
            C[k // 2:] = C[: k - k // 2]
        else:
            X, C = np.round(X / 4), np.round(C / 4)
        check(ckm, oracle, cuda, X, C, dtype)
