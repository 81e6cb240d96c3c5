"""Calls that fail half way: an allocation or a copy answers with an error (made on the host,
by fakes of the runtime's calls in a copy of the library, tests/fault_shim.c).  The call
reports it, and later calls neither use what it left behind nor miss what it kept.  The
reference exits on any error (hmglib.cu:46-66)."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from helpers import engine, fp64_rows, make_points, rel_err

pytestmark = pytest.mark.gpu

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
WRAPPED = ["cudaMalloc", "cudaMallocFromPoolAsync", "cudaMemcpyAsync"]
MALLOC, POOL, COPY = range(3)


@pytest.fixture(scope="module")
def faulty(hmg, cuda, tmp_path_factory):
    """hmglib_b200 on a copy of the library whose runtime calls can be made to fail:
    faulty(which, after) arms one failure."""
    from hmglib_b200 import _lib, build
    objs = [os.path.join(ROOT, "hmglib_b200", "_build", os.path.basename(s) + ".o") for s in build.sources()]
    if not all(os.path.exists(o) for o in objs):
        build.build(force=True)
    d = tmp_path_factory.mktemp("faulty")
    shim, so = str(d / "shim.o"), str(d / "libhmg_faulty.so")
    subprocess.run([NVCC, "-Xcompiler", "-fPIC", "-c", os.path.join(ROOT, "tests", "fault_shim.c"), "-o", shim], check=True)
    wrap = [a for w in WRAPPED for a in ("-Xlinker", f"--wrap={w}")]
    subprocess.run([NVCC, *build.ARCH, "-shared", "-cudart", "static", "-o", so, *objs, shim, *wrap, "-lpthread", "-ldl",
                    "-lrt"], check=True)
    saved = _lib._lib, _lib.LIB_PATH
    _lib._lib, _lib.LIB_PATH = None, so
    lib = _lib.lib()
    yield lib.hmg_test_fail
    _lib._lib, _lib.LIB_PATH = saved


def test_descriptors_after_a_failed_rebuild(hmg, cuda, faulty):
    """BF16 factors with the near field at FP32 accuracy, long dense pairs: a product in FP64
    arithmetic that cannot allocate its pair lists fails, and the next multi-vector product
    builds its own instead of following the missing ones."""
    torch = cuda
    rng = np.random.default_rng(8)
    n = 6007
    p = 0.5 + 1e-3 * rng.standard_normal((2, n))
    p[:, :9] = rng.random((2, 9))
    H = engine(hmg, p, p, 1.5, 64, rule=1)
    H.set_kernel(3, 0.05, 0.0)
    H.precompute_aca(64, 1e-6, hmg.PREC_FP32)
    H.precompute_dense(hmg.PREC_FP32)
    H.build_bf16_factors(near=hmg.PREC_FP32)
    X = torch.from_numpy(rng.uniform(-1, 1, (3, n))).cuda()
    A, B, y = torch.empty_like(X), torch.empty_like(X), torch.empty_like(X[0])
    H.matvec_multi(X, A)
    for after in (0, 1):
        H.set_product_precision(hmg.PREC_FP64)
        faulty(POOL, after)
        with pytest.raises(hmg.HmgError):
            H.matvec(X[0].contiguous(), y)
        faulty(POOL, -1)
        H.set_product_precision(hmg.PREC_FP32)
        B.fill_(float("nan"))
        H.matvec_multi(X, B)
        torch.cuda.synchronize()
        assert torch.equal(A, B)
    H.close()


def test_near_mode_changed_between_products(hmg, cuda):
    """The same operands: a single-vector product with the near field on the fly in between
    leaves descriptors that the multi-vector product must not take for its own.  Against FP64
    direct sums; BF16 factors of X, V and U (5e-3, test_gpu_tc.py)."""
    torch = cuda
    n = 6000
    p = make_points("uniform", n, 3, 5)
    H = engine(hmg, p, p, 1.5, 64, rule=1)
    H.set_kernel(4, 0.2, 0.0)
    H.precompute_aca(64, 1e-6, hmg.PREC_FP32)
    H.precompute_dense(hmg.PREC_FP32)
    H.build_bf16_factors(near=hmg.PREC_FP32)
    X = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, (4, n))).cuda()
    A, B, y = torch.empty_like(X), torch.empty_like(X), torch.empty_like(X[0])
    H.matvec_multi(X, A)
    H.set_near_mode(hmg.NEAR_ONTHEFLY)
    H.matvec(X[0].contiguous(), y)
    H.set_near_mode(hmg.NEAR_STORED)
    H.matvec_multi(X, B)
    torch.cuda.synchronize()
    assert rel_err(B[0].cpu().numpy(), fp64_rows(torch, H, X[0].contiguous(), np.arange(n))) < 5e-3
    assert torch.equal(A, B)
    H.close()


def test_tasks_after_a_failed_copy(hmg, cuda, faulty):
    """The first multi-vector product cannot copy its task list to the device: it fails, and the
    next one builds the list instead of using the uninitialised one."""
    torch = cuda
    n = 6000
    p = make_points("uniform", n, 2, 5)
    out = []
    for fail in (False, True):
        H = engine(hmg, p, p, 1.5, 64, rule=1)
        H.set_kernel(3, 0.05, 0.0)
        H.precompute_aca(64, 1e-8, hmg.PREC_FP32)
        H.precompute_dense(hmg.PREC_FP32)
        X = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, (3, n))).cuda()
        Y = torch.full_like(X, float("nan"))
        H.matvec(X[0], Y[0])  # the descriptors are there
        if fail:
            faulty(COPY, 0)
            with pytest.raises(hmg.HmgError):
                H.matvec_multi(X, Y)
            faulty(COPY, -1)
        H.matvec_multi(X, Y)
        torch.cuda.synchronize()
        out.append(Y)
        H.close()
    assert torch.equal(*out)


@pytest.mark.parametrize("which", [MALLOC, POOL, COPY], ids=["malloc", "pool", "copy"])
def test_construction_that_fails_gives_its_memory_back(hmg, cuda, faulty, which):
    """hmg_precompute_aca with each of its allocations or copies failing in turn: it reports the
    error, a retry on the same handle gives the factors of an undisturbed call, and with the
    handle closed the device has all the memory that it had."""
    torch = cuda
    n = 20000
    p = make_points("uniform", n, 3, 5)
    x = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, n)).cuda()
    y, ref = torch.empty_like(x), torch.empty_like(x)

    def handle():
        H = engine(hmg, p, p, 1.5, 64, rule=1)
        H.set_kernel(4, 0.2, 0.0)
        return H

    def finish(H, out):
        H.precompute_aca(96, 1e-6, hmg.PREC_MIXED)
        H.precompute_dense(hmg.PREC_MIXED)
        H.matvec(x, out)
        torch.cuda.synchronize()
        H.close()

    finish(handle(), ref)
    free, _ = torch.cuda.mem_get_info()
    failed, after = 0, 0
    while True:
        H = handle()
        faulty(which, after)
        try:
            H.precompute_aca(96, 1e-6, hmg.PREC_MIXED)
            done = True
        except hmg.HmgError as e:
            done = False
            failed += 1
            assert which == COPY or e.status == 3, e  # HMG_ERR_NOMEM
        faulty(which, -1)
        if done:
            H.close()
            break
        if after % 4 == 0:
            finish(H, y)
            assert torch.equal(y, ref)
        else:
            H.close()
        assert torch.cuda.mem_get_info()[0] == free, after
        after += 1
    assert failed >= {MALLOC: 2, POOL: 10, COPY: 8}[which]
