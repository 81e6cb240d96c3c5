"""What FP32 multiply-adds give and operands of fewer bits would not: multi-vector products of
FP32 and mixed storage with vectors of single entries, with sums of one sign, and of vectors at
both ends of the FP32 range.  No reference counterpart (the reference multiplies one vector per
apply_h_matrix_mvp call, hmglib.cu:271-286)."""
import numpy as np
import pytest

from helpers import engine, make_points, rel_err

pytestmark = pytest.mark.gpu

GAUSS, MATERN = 3, 4


def _dense(hmg, n, dim, param, scale=1.0):
    p = make_points("uniform", n, dim, 11, scale)
    H = engine(hmg, p, p, 1.5, n, rule=1)
    H.set_kernel(MATERN, param, 0.0)
    H.precompute_aca(8, 1e-6, hmg.PREC_FP32)
    H.precompute_dense(hmg.PREC_FP32)
    assert H.info()["aca_count"] == 0
    return H


@pytest.mark.parametrize("n,nrhs", [(130, 2), (700, 8), (700, 19), (1025, 32)])
def test_unit_vectors_give_the_stored_entries(hmg, cuda, n, nrhs):
    """Dense blocks only: a unit vector returns the stored FP32 entries, as the single-vector
    product does, bit for bit; a power of two of it likewise."""
    torch = cuda
    H = _dense(hmg, n, 3, 0.2)
    cols = np.random.default_rng(n).choice(n, nrhs, replace=False)
    X = torch.zeros(nrhs, n, dtype=torch.float64, device="cuda")
    for j, c in enumerate(cols):
        X[j, int(c)] = 2.0 ** (j % 5 - 2) * (-1) ** j
    Y, y = torch.full_like(X, float("nan")), torch.empty(n, dtype=torch.float64, device="cuda")
    H.matvec_multi(X, Y)
    for j in range(nrhs):
        H.matvec(X[j], y)
        torch.cuda.synchronize()
        assert torch.equal(Y[j], y)
    H.close()


@pytest.mark.parametrize("nrhs", [3, 16, 24, 32])
def test_sums_of_one_sign_have_no_mean_error(hmg, cuda, nrhs):
    """Entries between 0.3 and 1, vectors between 0.5 and 1.5 (FP32 values): against the
    FP64-arithmetic product of the same storage, the mean relative error over all rows is below
    1e-8, a sixth of half a unit in the last place (2^-24): rounding to nearest leaves some 1e-7
    / sqrt(rows), a truncated sum half a unit."""
    torch = cuda
    n = 1500
    H = _dense(hmg, n, 3, 1.5)
    X = torch.from_numpy(np.random.default_rng(3).uniform(0.5, 1.5, (nrhs, n)).astype(np.float32).astype(np.float64)).cuda()
    Y, y = torch.empty_like(X), torch.empty(n, dtype=torch.float64, device="cuda")
    H.matvec_multi(X, Y)
    H.set_product_precision(hmg.PREC_FP64)
    mean, worst = [], 0.0
    for j in range(nrhs):
        H.matvec(X[j], y)
        torch.cuda.synchronize()
        e = (Y[j] - y) / y
        mean.append(float(e.mean()))
        worst = max(worst, float(e.abs().max()))
    assert abs(np.mean(mean)) < 1e-8, np.mean(mean)
    assert worst < 1e-6
    H.close()


@pytest.mark.parametrize("storage", ["fp32", "mixed"])
@pytest.mark.parametrize("log2", [-120, -75, -60, 50, 62, 100])
def test_both_ends_of_the_range(hmg, cuda, storage, log2):
    """The same vectors times a power of two: the same product times it, as precise (FP32 sums
    in two orders, 1e-6: outside 2^-70 .. 2^59 they are FP32 multiply-adds)."""
    torch = cuda
    n = 5000
    p = make_points("uniform", n, 2, 5)
    H = engine(hmg, p, p, 1.5, 64, rule=1)
    H.set_kernel(GAUSS, 0.05, 0.0)
    H.precompute_aca(64, 1e-8, hmg.PREC_MIXED if storage == "mixed" else hmg.PREC_FP32)
    H.precompute_dense(hmg.PREC_FP32)
    X = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, (5, n))).cuda()
    A, B = torch.empty_like(X), torch.empty_like(X)
    H.matvec_multi(X, A)
    H.matvec_multi(X * 2.0**log2, B)
    torch.cuda.synchronize()
    B *= 2.0**-log2
    for j in range(5):
        assert rel_err(B[j].cpu().numpy(), A[j].cpu().numpy()) < 1e-6
    H.close()


@pytest.mark.parametrize("reg", [3.39e38, 1e39, -1e39, 1e13])
@pytest.mark.parametrize("storage", ["fp32", "mixed"])
def test_stored_values_that_do_not_split(hmg, cuda, tmp_path, storage, reg):
    """A regularization near, beyond and far below the FP32 limit: the stored diagonal is huge or
    infinite, and the multi-vector products have the single-vector product's finite, infinite
    and undefined entries (one vector is zero at some points) and its values to 1e-6."""
    torch = cuda
    n = 3000
    p = make_points("uniform", n, 2, 5)
    H = engine(hmg, p, p, 1.5, 64, rule=1)
    H.set_kernel(GAUSS, 0.05, reg)
    H.precompute_aca(64, 1e-8, hmg.PREC_MIXED if storage == "mixed" else hmg.PREC_FP32)
    H.precompute_dense(hmg.PREC_FP32)
    X = torch.from_numpy(np.random.default_rng(1).uniform(0.1, 0.9, (3, n))).cuda()
    X[1, ::7] = 0.0
    X[2] *= -1.0
    Y, y = torch.empty_like(X), torch.empty(n, dtype=torch.float64, device="cuda")
    H.matvec_multi(X, Y)
    for j in range(3):
        H.matvec(X[j], y)
        torch.cuda.synchronize()
        a, one = Y[j].cpu().numpy(), y.cpu().numpy()
        np.testing.assert_array_equal(np.isfinite(a), np.isfinite(one))
        np.testing.assert_array_equal(a[np.isinf(one)], one[np.isinf(one)])
        fin = np.isfinite(one)
        if fin.any():
            assert rel_err(a[fin], one[fin]) < 1e-6
    # the same through a file
    H.save(str(tmp_path / "h"))
    L = hmg.load(str(tmp_path / "h"))
    Z = torch.empty_like(Y)
    L.matvec_multi(X, Z)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(Z.cpu().numpy(), Y.cpu().numpy())
    L.close()
    # another regularization, the same handle: back to finite products
    H.set_kernel(GAUSS, 0.05, 0.5)
    H.precompute_aca(64, 1e-8, hmg.PREC_MIXED if storage == "mixed" else hmg.PREC_FP32)
    H.precompute_dense(hmg.PREC_FP32)
    H.matvec_multi(X, Y)
    H.matvec(X[0], y)
    torch.cuda.synchronize()
    assert rel_err(Y[0].cpu().numpy(), y.cpu().numpy()) < 1e-6
    H.close()
