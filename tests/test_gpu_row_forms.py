"""Row kernels at the edges of their forms: row lengths 0 .. 16 (short-row
HLL and ELL, FP32 row pairs) and 0 .. 35 (groups of 8 entries, tails of 1 to 7
in groups of 4), odd row counts, a row permutation, alpha and beta; FP64
products bit for bit the CPU csmv's, FP32 ones the FP64 row sum rounded once."""
import numpy as np
import pytest

import oracle as O
from psblas3_b200 import gen

pytestmark = pytest.mark.gpu


def _rows(n, longest, seed):
    rng = np.random.default_rng(seed)
    k = np.minimum(rng.integers(0, longest + 1, n), n)
    k[-1] = min(longest, n)  # the longest row there is
    irp = np.concatenate([[1], 1 + np.cumsum(k)]).astype(np.int32)
    ja = np.concatenate([np.sort(rng.choice(n, size=c, replace=False)) + 1 for c in k]).astype(np.int32)
    return irp, ja, rng.standard_normal(len(ja))


def _hll(psb, irp, ja, va, perm=None):
    import torch
    n = len(irp) - 1
    d = [torch.from_numpy(a).cuda() for a in (irp, ja, va)]
    p = None if perm is None else torch.from_numpy(perm).cuda()
    torch.cuda.synchronize()
    return psb.HllMat.from_csr_device(n, n, len(ja), *(t.data_ptr() for t in d), 32, None if p is None else p.data_ptr())


@pytest.mark.parametrize("n", [1, 31, 33, 1001])
@pytest.mark.parametrize("longest", [16, 17, 35])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.5, 2.0)])
def test_row_forms(psb, n, longest, alpha, beta):
    irp, ja, va = _rows(n, longest, n + longest)
    rng = np.random.default_rng(1)
    x, y0 = rng.uniform(-1, 1, (2, n))
    ref = O.csr_csmv(irp, ja, va, alpha, x, beta, y0.copy())
    ia, _, _ = gen.csr_to_coo(irp, ja, va)
    perm = rng.permutation(n).astype(np.int32)
    mats = [_hll(psb, irp, ja, va), _hll(psb, irp, ja, va, perm), psb.EllMat.from_coo_gpu(n, ia, ja, va)]
    for A in mats:
        X, Y = psb.DVect.bld(x), psb.DVect.bld(y0)
        psb.psb_spmm(alpha, A, X, beta, Y)
        assert np.array_equal(Y.get_vect(), ref)
    # FP32: exact products added in FP64 in stored order, rounded once, then
    # alpha * sum + beta * y in FP32
    v32, x32, y32 = va.astype(np.float32), x.astype(np.float32), y0.astype(np.float32)
    s = O.csr_csmv(irp, ja, v32.astype(np.float64), 1.0, x32.astype(np.float64), 0.0, np.zeros(n)).astype(np.float32)
    ref32 = np.float32(alpha) * s
    if beta != 0.0:
        ref32 = ref32 + np.float32(beta) * y32
    for A in mats[:2]:
        A.make_single()
        X, Y = psb.DVect.bld(x32), psb.DVect.bld(y32)
        A.spmv(alpha, X, beta, Y)
        assert np.array_equal(Y.get_vect(), ref32)


def _bands(n, longest, seed):
    """Rows of 0 .. longest neighbouring columns, the longest row among them."""
    rng = np.random.default_rng(seed)
    k = rng.integers(0, longest + 1, n)
    k[n // 2] = longest
    irp = np.concatenate([[1], 1 + np.cumsum(k)]).astype(np.int32)
    first = rng.integers(1, n - longest + 2, n)
    ja = (np.repeat(first, k) + np.arange(irp[-1] - 1) - np.repeat(irp[:-1] - 1, k)).astype(np.int32)
    return irp, ja, rng.standard_normal(len(ja))


@pytest.mark.parametrize("longest", [1, 3, 4, 6, 7, 8, 9, 13, 16, 21])
@pytest.mark.parametrize("blocks", [4, 5, 6, 10, 12])
def test_forms_at_grid_lines(psb, blocks, longest):
    """The forms of the row products change with the row length and the grid
    (4, 5, 6, 10 and 12 blocks of 256 rows per SM): one row past each line,
    hack sizes 32 and 16, ELL, FP64 and FP32."""
    from psblas3_b200._lib import lib
    n = 256 * blocks * lib.getGPUMultiProcessors() + 1
    irp, ja, va = _bands(n, longest, 7)
    rng = np.random.default_rng(5)
    x, y0 = rng.uniform(-1, 1, (2, n))
    ref = O.csr_csmv(irp, ja, va, -0.5, x, 2.0, y0.copy())
    v32, x32, y32 = va.astype(np.float32), x.astype(np.float32), y0.astype(np.float32)
    s = O.csr_csmv(irp, ja, v32.astype(np.float64), 1.0, x32.astype(np.float64), 0.0, np.zeros(n)).astype(np.float32)
    ref32 = np.float32(-0.5) * s + np.float32(2.0) * y32
    ia, _, _ = gen.csr_to_coo(irp, ja, va)
    import torch
    d = [torch.from_numpy(a).cuda() for a in (irp, ja, va)]
    torch.cuda.synchronize()
    mats = [psb.HllMat.from_csr_device(n, n, len(ja), *(t.data_ptr() for t in d), hk) for hk in (32, 16)]
    mats.append(psb.EllMat.from_coo_gpu(n, ia, ja, va))
    for A in mats:
        X, Y = psb.DVect.bld(x), psb.DVect.bld(y0)
        psb.psb_spmm(-0.5, A, X, 2.0, Y)
        assert np.array_equal(Y.get_vect(), ref)
    for A in mats[:2]:
        A.make_single()
        X, Y = psb.DVect.bld(x32), psb.DVect.bld(y32)
        A.spmv(-0.5, X, 2.0, Y)
        assert np.array_equal(Y.get_vect(), ref32)


@pytest.mark.parametrize("longest", [1, 3, 8, 17, 23, 24, 29])
@pytest.mark.parametrize("n", [33, 160_001])
def test_ell_float_forms(psb, n, longest):
    """FP32 ELL rows on either side of the line at 24 entries: the FP64 row sum
    rounded once."""
    import ctypes as C
    from psblas3_b200._lib import lib
    irp, ja, va = _bands(n, longest, 3)
    irn = np.diff(irp).astype(np.int32)
    h = C.c_void_p()
    assert lib.FallocEllDevice(C.byref(h), n, longest, len(ja), n, 1, 1) == 0
    pitch = lib.getEllDevicePitch(h)
    rows = np.repeat(np.arange(n), irn)
    at = (np.arange(len(ja)) - np.repeat(irp[:-1] - 1, irn)) * pitch + rows
    eja, eva = np.ones(pitch * longest, np.int32), np.zeros(pitch * longest, np.float32)
    eja[at], eva[at] = ja, va
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert lib.writeEllDeviceFloat(h, ptr(eva), ptr(eja), pitch, ptr(irn), ptr(np.zeros(n, np.int32))) == 0
    x, y0 = np.random.default_rng(4).uniform(-1, 1, (2, n)).astype(np.float32)
    s = O.csr_csmv(irp, ja, va.astype(np.float32).astype(np.float64), 1.0, x.astype(np.float64), 0.0,
                   np.zeros(n)).astype(np.float32)
    for alpha, beta in ((1.0, 0.0), (-0.5, 2.0)):
        X, Y = psb.DVect.bld(x), psb.DVect.bld(y0)
        assert lib.spmvEllDeviceFloat(h, np.float32(alpha), X.h, np.float32(beta), Y.h) == 0
        ref = np.float32(alpha) * s
        assert np.array_equal(Y.get_vect(), ref if beta == 0.0 else ref + np.float32(beta) * y0)
    lib.freeEllDevice(h)
