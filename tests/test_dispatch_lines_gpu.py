"""Both sides of the lines between the kernels of a call, on whole-number
coordinates: FP32 sums of these are exact in any order, so the sums have to be
equal, and a partial sum that is lost or added twice shows whatever the number
of points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def whole(n, d, k, dtype, cuda, seed):
    import torch
    g = torch.Generator(device=cuda).manual_seed(seed)
    X = torch.randint(-7, 8, (d, n), generator=g, device=cuda)
    L = torch.randint(0, k, (n,), generator=g, device=cuda)
    return X.to(dtype).reshape(-1).contiguous(), L


def exact_sums(P, L, n, d, k):
    import torch
    return torch.stack([torch.zeros(k, dtype=torch.float64, device=P.device).index_add_(0, L, P[f * n:(f + 1) * n].double())
                        for f in range(d)]).reshape(-1)


F32_SUMS = [  # n, d, k
    (100000, 1, 600), (1 << 19, 3, 600), (1 << 19, 3, 601), ((1 << 19) - 1, 5, 400), (65536, 10, 600), (65536, 11, 601),
    (49151, 10, 300), (49152, 10, 300), (20000, 12, 12), (20000, 12, 13), (20000, 13, 257), (20000, 13, 258), (70001, 9, 33),
    (20000, 20, 512), (20000, 20, 513), (65536, 20, 1024), (65535, 21, 1024),
    (65537, 20, 1025), (9001, 40, 1024), (9001, 40, 1025), (9001, 70, 1300), (9001, 70, 1301), (13001, 200, 3072),
]
F64_SUMS = [
    (20000, 16, 1300), (20000, 16, 1301), (20000, 5, 16), (20000, 5, 17), (1 << 19, 5, 64), (1 << 19, 5, 65),
    (65535, 9, 24), (65535, 9, 25), (65536, 9, 32), (65536, 9, 33), (65535, 8, 16), (65535, 8, 17), (65536, 8, 722), (65536, 8, 723), (65535, 8, 723),
    (65536, 8, 1024), (65536, 8, 1025),
]


@pytest.mark.parametrize("n,d,k,f64", [s + (False,) for s in F32_SUMS] + [s + (True,) for s in F64_SUMS])
def test_centroid_update_lines(ckm, cuda, n, d, k, f64):
    import torch
    P, L = whole(n, d, k, torch.float64 if f64 else torch.float32, cuda, n + d + k)
    lab = L if f64 else L.int()
    S = ckm.new_scratch(d, k, cuda)
    C, M = torch.zeros(k * d, dtype=P.dtype, device=cuda), torch.zeros(k, dtype=lab.dtype, device=cuda)
    want = exact_sums(P, L, n, d, k)
    ckm.centroid_update(P, C, lab, M, S, n, d, k)
    assert torch.equal(C.double(), want)
    assert not torch.any(S != 0)
    ckm.centroid_update(P, None, lab, M, S, n, d, k, mode=ckm.MODE_DEFER)
    ckm.finalize(C, M, S, d, k)
    mass = torch.bincount(L, minlength=k)
    assert torch.equal(M.long(), mass)
    mean = (want.reshape(d, k) / mass).to(P.dtype).reshape(-1)
    assert torch.equal(torch.nan_to_num(C, nan=-99.0), torch.nan_to_num(mean, nan=-99.0))


FUSED = [  # n, d, k, type: the tensor-core labels against the low-d and the generic kernel,
    # and the low-d kernel's clusters (two and four tiles of 2048 points for each of two CTAs per SM)
    (70000, 10, 29, "f32"), (70000, 10, 30, "f32"), (1 << 18, 10, 5, "f32"), ((1 << 18) - 1, 10, 5, "f32"),
    (20000, 15, 4, "f32"), (20000, 15, 5, "f32"), (65535, 8, 64, "f32"), (65536, 8, 64, "f32"), (65536, 8, 80, "f32"),
    (2 * 304 * 2048 - 2048, 4, 49, "f32"), (2 * 304 * 2048 + 1, 4, 49, "f32"), (2 * 304 * 2048 + 1, 4, 48, "f32"),
    (4 * 304 * 2048 - 2047, 4, 48, "f32"), (4 * 304 * 2048 + 5, 4, 48, "f32"), (1 << 20, 4, 180, "f32"),
    (65535, 8, 2, "f64"), (65536, 8, 2, "f64"), (20000, 7, 2, "f64"), (20000, 16, 3, "f64"),
]


@pytest.mark.parametrize("n,d,k,kind", FUSED)
def test_fused_and_labeling_lines(ckm, oracle, cuda, n, d, k, kind):
    import torch
    f64 = kind == "f64"
    P, _ = whole(n, d, k, torch.float64 if f64 else torch.float32, cuda, n + d + k)
    rng = np.random.default_rng(n)
    C = (rng.integers(-14, 15, (d, k)) / 2).astype(np.float64 if f64 else np.float32).reshape(-1)
    ref = (oracle.label_f64 if f64 else oracle.label_f32)(P.cpu().numpy(), n, d, k, C).astype(np.int64)
    L = torch.from_numpy(ref).to(cuda)
    dC, N = torch.from_numpy(C).to(cuda), torch.zeros(k * d, dtype=P.dtype, device=cuda)
    lab = torch.full((n,), -1, dtype=torch.int64 if f64 else torch.int32, device=cuda)
    M, S = torch.zeros(k, dtype=lab.dtype, device=cuda), ckm.new_scratch(d, k, cuda)
    ckm.labeling(P, dC, lab, n, d, k)
    assert torch.equal(lab.long(), L)
    lab.fill_(-1)
    ckm.fused(P, dC, N, lab, M, S, n, d, k, mode=ckm.MODE_ACCUMULATE)
    assert torch.equal(lab.long(), L)
    assert torch.equal(M.long(), torch.bincount(L, minlength=k))
    assert torch.equal(N.double(), exact_sums(P, L, n, d, k))
    assert not torch.any(S != 0)


@pytest.mark.parametrize("n,d,k", [(260097, 4, 10), (200001, 8, 16), (1 << 19, 2, 32)])
def test_sorted_fused_sums(ckm, oracle, cuda, n, d, k):
    import torch
    P, _ = whole(n, d, k, torch.float32, cuda, n)
    rng = np.random.default_rng(n)
    C = (rng.integers(-14, 15, (d, k)) / 2).astype(np.float32).reshape(-1)
    o, _ = ckm.spatial_sort(P, n, d)
    L = torch.from_numpy(oracle.label_f32(o.cpu().numpy(), n, d, k, C).astype(np.int64)).to(cuda)
    lab = torch.full((n,), -1, dtype=torch.int32, device=cuda)
    N, M, S = torch.zeros(k * d, device=cuda), torch.zeros(k, dtype=torch.int32, device=cuda), ckm.new_scratch(d, k, cuda)
    ckm.fused_sorted(o, torch.from_numpy(C).to(cuda), N, lab, M, S, n, d, k, mode=ckm.MODE_ACCUMULATE)
    assert torch.equal(lab.long(), L) and torch.equal(M.long(), torch.bincount(L, minlength=k))
    assert torch.equal(N.double(), exact_sums(o, L, n, d, k))
    assert not torch.any(S != 0)
