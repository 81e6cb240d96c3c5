"""A block whose V^T passes 4 GiB: 64 rows against 2^25 columns, one admissible block of rank
40 in FP32 storage, so that the rows of V^T from the 33rd on start beyond a 32-bit offset."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_rows_beyond_4_gib(hmg, cuda):
    """Two vectors a pass against one (the kernel of which uses 64-bit offsets), 64 entries of
    each vector set: about a hundred FP32 roundings a row and product (1e-6), times the
    cancellation among the 40 terms, at most 10: 1e-5.  A row of V^T taken from elsewhere
    changes the product by its own size: rows pivot in Z order, so late terms are no smaller."""
    torch = cuda
    free, _ = torch.cuda.mem_get_info()
    if free < 60 << 30:
        pytest.skip("needs 60 GB of device memory")
    m1, m2, k = 64, 1 << 25, 40
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    p1 = torch.rand(2, m1, dtype=torch.float64, device="cuda", generator=g)
    p2 = torch.rand(2, m2, dtype=torch.float64, device="cuda", generator=g)
    p1[0] *= 0.01
    p2[0] += 0.02
    H = hmg.HMatrix(m1, m2, 2)
    H.set_points(0, p1)
    H.set_points(1, p2)
    H.setup(1e4, 64, rule=hmg.ADMISSIBLE_MAX)
    i = H.info()
    assert i["block_count"] == 1 and i["aca_count"] == 1
    H.set_kernel(4, 0.1, 0.0)
    H.precompute_aca(k, 0.0, hmg.PREC_FP32)
    H.precompute_dense(hmg.PREC_FP32)
    assert int(H.ranks()[0]) == k and k * 4 * m2 > 1 << 32
    X = torch.zeros(2, m2, dtype=torch.float64, device="cuda")
    near = torch.nonzero(p2[0] < 0.12)[:64, 0]
    X[:, near] = torch.rand(2, 64, dtype=torch.float64, device="cuda", generator=g) * 2.0 - 1.0
    Y = torch.empty(2, m1, dtype=torch.float64, device="cuda")
    y = torch.empty(m1, dtype=torch.float64, device="cuda")
    H.matvec_multi(X, Y)
    for j in range(2):
        H.matvec(X[j], y)
        torch.cuda.synchronize()
        assert float(torch.linalg.norm(Y[j] - y) / torch.linalg.norm(y)) < 1e-5
    H.close()
