"""Dense blocks of very many columns in the tile kernels, one vector and several, stored
and on the fly (the reference multiplies such blocks in one dgemv of its batch,
linear_algebra.cu:2817-3137)."""
import numpy as np
import pytest

from helpers import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["fp64", "fp32", "mixed", "onthefly"])
def test_long_dense_pairs(hmg, cuda, storage):
    """Points of which a few lie far from a dense cluster: leaves of a handful of points
    meet dense blocks of thousands of columns, which the tile kernels cut into runs of 256
    columns.  Against FP64 direct sums: FP64 storage 1e-9 (ACA eps 1e-11), FP32 arithmetic
    1e-6, one vector and several, relative to the sums of magnitudes |K| |x| (nearly all
    entries are close to 1 here, so the sums themselves cancel a thousandfold)."""
    torch = cuda
    rng = np.random.default_rng(8)
    n = 6007
    p = 0.5 + 1e-3 * rng.standard_normal((2, n))
    p[:, :9] = rng.random((2, 9))
    H = engine(hmg, p, p, 1.5, 64, rule=1)
    s1l, s1u, s2l, s2u, typ = H.blocks()
    assert int((s2u - s2l + 1)[typ == 2].max()) > 1024  # the long pairs are there
    H.set_kernel(3, 0.05, 0.0)
    f64 = storage == "fp64"
    H.precompute_aca(64, 1e-11 if f64 else 1e-8, hmg.PREC_FP64 if f64 else hmg.PREC_MIXED if storage == "mixed" else hmg.PREC_FP32)
    if storage != "onthefly":
        H.precompute_dense(hmg.PREC_FP64 if f64 else hmg.PREC_FP32)
    X = torch.from_numpy(rng.uniform(-1, 1, (5, n))).cuda()
    Y, y, ref, mag = torch.empty_like(X), torch.empty_like(X[0]), torch.empty_like(X[0]), torch.empty_like(X[0])
    H.matvec_multi(X, Y)
    for j in (0, 4):
        H.matvec(X[j].contiguous(), y)
        H.full_matvec(X[j].contiguous(), ref)
        H.full_matvec(X[j].abs().contiguous(), mag)  # every entry of K is positive
        torch.cuda.synchronize()
        for got in (y, Y[j]):
            err = float(torch.linalg.norm(got - ref) / torch.linalg.norm(mag))
            assert err < (1e-9 if f64 else 1e-6), err
    H.close()
