"""The ACA of single blocks at the edges of its size classes (warp per block up to 128
rows and columns, CTAs above 128, 256 and 512): two point sets far enough apart that the
whole matrix is one admissible block.  Against the kernel matrix in FP64, and in the
fixed-rank mode against the oracle's restatement (linear_algebra.cu:3684-4012)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(5, 33), (1, 7), (128, 128), (128, 129), (129, 40), (256, 255), (257, 256), (512, 300), (300, 513), (1100, 90),
         (700, 2049)]
MATERN = 4


def _block(hmg, m1, m2, dim, k, eps, prec, seed=3):
    rng = np.random.default_rng(seed)
    p1 = rng.random((dim, m1))
    p2 = rng.random((dim, m2))
    p2[0] += 3.0
    H = hmg.HMatrix(m1, m2, dim)
    H.set_points(0, p1)
    H.set_points(1, p2)
    H.setup(1.5, 16, rule=hmg.ADMISSIBLE_MAX)
    H.set_kernel(MATERN, 0.9, 0.0)
    H.precompute_aca(k, eps, prec)
    i = H.info()
    assert i["block_count"] == 1 and i["aca_count"] == 1
    z1, z2 = H.points(0), H.points(1)
    r = np.sqrt(((z1[:, :, None] - z2[:, None, :]) ** 2).sum(0)) * np.sqrt(3.0) / 0.9
    return H, (1.0 + r) * np.exp(-r), int(H.ranks()[0])


# Adaptive: the last term is below eps |S|_F and the terms fall by a factor of 2 or more on
# average here, so what is left out is below 10 eps |K|_F.
@pytest.mark.parametrize("m1,m2", SIZES)
@pytest.mark.parametrize("eps,k", [(1e-4, 64), (1e-9, 200)])
def test_adaptive_accuracy(hmg, cuda, m1, m2, eps, k):
    H, K, r = _block(hmg, m1, m2, 3, k, eps, hmg.PREC_FP64)
    U, V = H.factors(0, m1, m2, r)
    assert 1 <= r <= min(k, m1, m2)
    err = np.linalg.norm(U.T @ V - K) / np.linalg.norm(K)
    assert err < 10 * eps, (err, r)
    # one term fewer does not reach it: the test stops where it holds, not later
    if 1 < r < min(m1, m2):
        last = np.linalg.norm(U[r - 2]) * np.linalg.norm(V[r - 2])
        assert last > eps * np.linalg.norm(U[: r - 1].T @ V[: r - 1])
    H.close()


@pytest.mark.parametrize("m1,m2", SIZES)
def test_mixed_storage_of_the_terms(hmg, cuda, m1, m2):
    """Tiers and scales from the terms' norms: the stored block is within 3e-7 of the FP64
    one (FP16 terms hold 1e-4 of the norm to 2^-11, FP8 terms 1.5e-6 to 2^-4, FP32 2^-24)."""
    H, K, r = _block(hmg, m1, m2, 2, 96, 1e-8, hmg.PREC_MIXED)
    U, V = H.factors(0, m1, m2, r)
    assert np.linalg.norm(U.T @ V - K) / np.linalg.norm(K) < 3e-7
    H.close()


@pytest.mark.parametrize("m1,m2", SIZES)
@pytest.mark.parametrize("k", [1, 13, 40])
def test_fixed_rank_equals_the_oracle(hmg, cuda, oracle, m1, m2, k):
    H, K, r = _block(hmg, m1, m2, 3, k, 0.0, hmg.PREC_FP64)
    U, V = H.factors(0, m1, m2, r)
    O = oracle
    z1, z2 = H.points(0), H.points(1)
    s1l, s1u, s2l, s2u, typ = H.blocks()
    # the oracle's own factors of the same block, as products (the terms below 1e-13 of the
    # residual are rounding noise): equal to 1e-10 of the matrix
    s, o, z = O.order_points(z1, 20)
    t, q, w = O.order_points(z2, 20)
    blocks = O.tree(z, s, w, t, 1.5, 16)
    par = O.kernel_param(MATERN, 0.9)
    fac = O.aca(MATERN, par, 0.0, z, w, blocks.subset(blocks.type == 1), k)
    x = np.random.default_rng(k).uniform(-1, 1, m2)
    y = O.hmatvec(MATERN, par, 0.0, z, w, blocks, fac, x)
    assert np.linalg.norm(U.T @ (V @ x) - y) < 1e-10 * np.linalg.norm(K) * np.linalg.norm(x)
    H.close()
