"""Multi-vector products on split tensor-core operands (FP32 and mixed storage, 2 to 32
vectors a pass): accuracy against 64 bits at the edges of the kernels' tiles, and the
values that the split does not take.  No reference counterpart (the reference
multiplies one vector per apply_h_matrix_mvp call, hmglib.cu:271-286)."""
import numpy as np
import pytest

from helpers import engine, fp64_rows, make_points, rel_err

pytestmark = pytest.mark.gpu

GAUSS, MATERN = 3, 4


def _build(hmg, gen, n, dim, leaf, prec, eps=1e-8, kmax=96, rule=1):
    p = make_points(gen, n, dim, 5)
    H = engine(hmg, p, p, 1.5, leaf, rule=rule)
    H.set_kernel(MATERN if dim == 3 else GAUSS, 0.2 if dim == 3 else 0.05, 0.0)
    H.precompute_aca(kmax, eps, prec)
    H.precompute_dense(hmg.PREC_FP32)
    return H, n


# Tolerance: FP32 entries, vectors and sums (2^-24 each, sums over up to 16384 columns in
# steps of 16 per FP32 addition) and the ACA's and the short tiers' own error at eps 1e-8,
# 1e-7 each: below 1e-6 together, the bound the engine states for these products.
@pytest.mark.parametrize("case", [
    ("uniform", 700, 2, 16),      # tiles of at most 16 rows, ranks below one K step
    ("uniform", 6001, 3, 64),     # odd sizes: ragged rows, columns and terms
    ("gmm", 20000, 2, 64),        # blocks above and below the column split
    ("uniform", 12000, 3, 130),   # two tiles a leaf: four row groups
], ids=["tiny-tiles", "odd", "clustered", "wide-leaves"])
@pytest.mark.parametrize("storage", ["fp32", "mixed"])
@pytest.mark.parametrize("nrhs", [2, 9, 17, 32])
def test_accuracy_against_64_bits(hmg, cuda, case, storage, nrhs):
    torch = cuda
    gen, n, dim, leaf = case
    H, n = _build(hmg, gen, n, dim, leaf, hmg.PREC_MIXED if storage == "mixed" else hmg.PREC_FP32)
    X = torch.from_numpy(np.random.default_rng(nrhs).uniform(-1, 1, (nrhs, n))).cuda()
    Y = torch.full_like(X, float("nan"))
    H.matvec_multi(X, Y)
    torch.cuda.synchronize()
    rows = np.arange(n) if n <= 6001 else np.random.default_rng(1).choice(n, 4096, replace=False)
    Yh = Y.cpu().numpy()
    assert np.isfinite(Yh).all()
    for j in {0, nrhs // 2, nrhs - 1}:
        e = rel_err(Yh[j][rows], fp64_rows(torch, H, X[j].contiguous(), rows))
        assert e < 1e-6, (j, e)
    H.close()


# (3.4e38 in FP32 storage only: the stored FP8 terms reach 448 before their scale is
# applied, so that entry overflows in the single-vector product of mixed storage too)
@pytest.mark.parametrize("storage,bad", [("fp32", float("inf")), ("mixed", float("inf")), ("fp32", float("nan")),
                                         ("mixed", float("nan")), ("fp32", 3.4e38)])
def test_values_that_do_not_split(hmg, cuda, storage, bad):
    """One such entry in one vector: the other vectors are those of the product without it
    (FP32 multiply-adds instead of split ones: 1e-6), and the vector itself has the
    single-vector product's finite, infinite and undefined entries."""
    torch = cuda
    H, n = _build(hmg, "uniform", 9000, 2, 64, hmg.PREC_MIXED if storage == "mixed" else hmg.PREC_FP32)
    X = torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, (12, n))).cuda()
    Y0 = torch.empty_like(X)
    H.matvec_multi(X, Y0)
    X[5, 1234] = bad
    Y = torch.empty_like(X)
    H.matvec_multi(X, Y)
    y1 = torch.empty(n, dtype=torch.float64, device="cuda")
    H.matvec(X[5].contiguous(), y1)
    torch.cuda.synchronize()
    a, b, one = Y.cpu().numpy(), Y0.cpu().numpy(), y1.cpu().numpy()
    for j in range(12):
        if j != 5:
            assert rel_err(a[j], b[j]) < 1e-6
    fin = np.isfinite(one)
    if bad == 3.4e38:
        assert fin.all() and np.isfinite(a[5]).all()
        assert rel_err(a[5], one) < 1e-6
    else:
        np.testing.assert_array_equal(np.isfinite(a[5]), fin)
        np.testing.assert_array_equal(a[5][np.isinf(one)], one[np.isinf(one)])
    H.close()


def test_zero_vectors_and_a_later_finite_product(hmg, cuda):
    """Zero vectors give exact zeros, and a product with infinities leaves nothing behind."""
    torch = cuda
    H, n = _build(hmg, "uniform", 5000, 3, 64, hmg.PREC_MIXED)
    X = torch.zeros(7, n, dtype=torch.float64, device="cuda")
    Y = torch.full_like(X, float("nan"))
    H.matvec_multi(X, Y)
    assert float(Y.abs().max()) == 0.0
    Z = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, (7, n))).cuda()
    A, B = torch.empty_like(Z), torch.empty_like(Z)
    H.matvec_multi(Z, A)
    W = Z.clone()
    W[0, 0] = float("inf")
    H.matvec_multi(W, Y)
    H.matvec_multi(Z, B)
    torch.cuda.synchronize()
    assert torch.equal(A, B)
    H.close()


@pytest.mark.parametrize("storage", ["fp32", "mixed"])
def test_sums_that_overflow_on_the_way(hmg, cuda, storage):
    """Vectors near the FP32 limit whose V^T x overflows in some blocks while others are still
    being multiplied: every product of the same vectors is the same, bit for bit, and its other
    vectors keep their values."""
    torch = cuda
    H, n = _build(hmg, "uniform", 9000, 2, 64, hmg.PREC_MIXED if storage == "mixed" else hmg.PREC_FP32)
    X = torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, (9, n))).cuda()
    Y0 = torch.empty_like(X)
    H.matvec_multi(X, Y0)
    X[4] = 2e36  # finite; sums of 200 of them are not
    Y, Z = torch.empty_like(X), torch.empty_like(X)
    H.matvec_multi(X, Y)
    for _ in range(20):
        H.matvec_multi(X, Z)
        torch.cuda.synchronize()
        assert torch.equal(Y.nan_to_num(nan=7.0), Z.nan_to_num(nan=7.0)) and torch.equal(Y.isnan(), Z.isnan())
    assert not bool(torch.isfinite(Y[4]).all())
    for j in (0, 8):
        assert rel_err(Y[j].cpu().numpy(), Y0[j].cpu().numpy()) < 1e-6
    H.close()
