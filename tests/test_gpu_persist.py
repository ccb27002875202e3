"""The one-kernel CG / BiCGSTAB of small systems against the
kernel-per-step drivers of the same library, which take the same solves when
itmax is above the one-kernel solver's bound (100,000): the same operations
in the same order except for the order in which a dot's partial sums meet,
and those are compensated, so iterations and solutions agree."""
import numpy as np
import pytest

import oracle as O
from psblas3_b200 import gen

pytestmark = pytest.mark.gpu

GENERAL = 200_000  # itmax that goes to the kernel-per-step drivers


def _dominant(n, seed, long_row=0):
    """Random diagonally dominant CSR (1-based); row 0 holds long_row entries."""
    rng = np.random.default_rng(seed)
    k = rng.integers(0, 9, n)
    if long_row:
        k[0] = long_row
    k = np.minimum(k, n - 1)
    irp, ja, va = [1], [], []
    for i in range(n):
        c = rng.choice(n - 1, size=k[i], replace=False) if k[i] else np.zeros(0, np.int64)
        c = c + (c >= i)
        v = rng.standard_normal(k[i])
        c, v = np.append(c, i), np.append(v, np.abs(v).sum() + 1.0)
        o = np.argsort(c)
        ja.append(c[o] + 1)
        va.append(v[o])
        irp.append(irp[-1] + len(c))
    return np.array(irp, np.int32), np.concatenate(ja).astype(np.int32), np.concatenate(va)


def _matrix(psb, fmt, irp, ja, va, perm=False):
    import torch
    n = len(irp) - 1
    if fmt == "CSR":
        return psb.CsrMat(n, irp, ja, va)
    ia, _, _ = gen.csr_to_coo(irp, ja, va)
    if fmt == "ELL":
        return psb.EllMat.from_coo_gpu(n, ia, ja, va)
    if fmt == "HLL16":
        return psb.HllMat.from_coo_gpu(n, ia, ja, va, 16)
    d = [torch.from_numpy(a).cuda() for a in (irp, ja, va)]
    p = None
    if perm:
        p = torch.from_numpy(np.random.default_rng(0).permutation(n).astype(np.int32)).cuda()
    torch.cuda.synchronize()
    return psb.HllMat.from_csr_device(n, n, len(ja), *(t.data_ptr() for t in d), 32, None if p is None else p.data_ptr())


def _solve(psb, A, method, b, itmax, istop=2, prec=True, x0=None, eps=1e-10):
    P = psb.DiagPrec("DIAG").build(A) if prec else None
    B, X = psb.DVect.bld(b), psb.DVect.bld(np.zeros_like(b) if x0 is None else x0)
    l0 = psb.kernel_launches()
    it, err = psb.psb_krylov(method, A, P, B, X, eps=eps, istop=istop, itmax=itmax)
    return it, err, X.get_vect(), psb.kernel_launches() - l0


def _agree(psb, A, method, b, **kw):
    it1, err1, x1, l1 = _solve(psb, A, method, b, 5000, **kw)
    it2, err2, x2, l2 = _solve(psb, A, method, b, GENERAL, **kw)
    assert l1 == 1 and l2 > 1  # one kernel, and the general path
    assert it1 == it2
    # a dot that rounds differently moves the iterates by about the unit roundoff times the
    # iterations of a well conditioned system
    np.testing.assert_allclose(err1, err2, rtol=1e-6)
    assert np.max(np.abs(x1 - x2)) <= 1e-12 * max(1.0, np.max(np.abs(x2)))


@pytest.mark.parametrize("method", ["CG", "BICGSTAB"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 256, 257, 4100, 10240, 10241, 20001, 75777])
def test_sizes(psb, method, n):
    """One row to more rows than threads: partial slices, one and many blocks
    (both ways of publishing a reduction, with 40 and 41 blocks at the line),
    several slices per warp.  (On one or two rows BiCGSTAB breaks down before
    its first update of x, in every restart.)"""
    if method == "BICGSTAB" and n < 3:
        n = 3
    irp, ja, va = gen.powerlaw(n, kmax=min(6, n - 1), seed=n) if n > 2 else _dominant(n, n)
    if method == "CG" and n > 2:
        irp, ja, va = gen.powerlaw_spd(n, kmax=min(6, n - 1), seed=n)
    b = np.random.default_rng(n).uniform(-1, 1, n)
    _agree(psb, _matrix(psb, "HLL", irp, ja, va), method, b)


@pytest.mark.parametrize("fmt,perm", [("HLL", False), ("HLL", True), ("HLL16", False), ("ELL", False), ("CSR", False)])
@pytest.mark.parametrize("istop", [1, 2, 3])
@pytest.mark.parametrize("prec", [True, False])
def test_forms(psb, fmt, perm, istop, prec):
    """Formats, a row permutation, stop tests, with and without the
    preconditioner, from a nonzero x0; one row is longer than the rest."""
    irp, ja, va = _dominant(1999, 5, long_row=60)
    b, x0 = np.random.default_rng(1).uniform(-1, 1, (2, 1999))
    _agree(psb, _matrix(psb, fmt, irp, ja, va, perm), "BICGSTAB", b, istop=istop, prec=prec, x0=x0)


def test_rows_beyond_shared_memory(psb):
    """Blocks whose rows do not all fit: a CSR row of every column (its slice
    stays in global memory), beside slices that are staged."""
    irp, ja, va = _dominant(9000, 6, long_row=8999)
    b = np.random.default_rng(2).uniform(-1, 1, 9000)
    _agree(psb, _matrix(psb, "CSR", irp, ja, va), "BICGSTAB", b)


def test_upper_end(psb):
    """The largest systems of the range, and the first beyond it."""
    for side, one in ((86, True), (96, False)):
        irp, ja, va = gen.poisson7(side)
        A = _matrix(psb, "HLL", irp, ja, va)
        b = np.random.default_rng(3).uniform(-1, 1, side ** 3)
        it, err, x, launches = _solve(psb, A, "CG", b, 3000, eps=1e-8)
        assert (launches == 1) == one and err <= 1e-8
        r = b - gen.csr_matvec(irp, ja, va, x)
        assert np.linalg.norm(r) <= 2e-8 * np.linalg.norm(b)


@pytest.mark.parametrize("fmt", ["CSR", "HLL16", "ELL"])
def test_uneven_rows_go_to_the_drivers(psb, fmt):
    """Rows in order of length: the first blocks would hold most of the entries
    and read them alone, so the kernel declines and x is the drivers'; the same
    rows shuffled, and a grid with as many unstaged entries, stay in it."""
    n = 300_000
    irp, ja, va = gen.powerlaw_spd(n, kmax=40, seed=4)
    b = np.random.default_rng(8).uniform(-1, 1, n)
    sirp, sja, sva = gen.sort_rows_by_length(irp, ja, va)[:3]
    A = _matrix(psb, fmt, sirp, sja, sva)
    it1, err1, x1, l1 = _solve(psb, A, "CG", b, 5000)
    it2, err2, x2, l2 = _solve(psb, A, "CG", b, GENERAL)
    assert l1 == l2 + 1  # the kernel that declined, then the same launches
    assert (it1, err1) == (it2, err2) and np.array_equal(x1, x2)
    if fmt != "ELL":  # (padded to the longest row everywhere)
        assert _solve(psb, _matrix(psb, fmt, irp, ja, va), "CG", b, 5000)[3] == 1
    irp, ja, va = gen.poisson7(66)
    assert _solve(psb, _matrix(psb, fmt, irp, ja, va), "CG", b[:66 ** 3], 5000)[3] == 1


# 3 x 3 blocks whose solves break down exactly (small integers and powers of
# two up to there) in the second iteration, x moved by the first, and converge
# after the restart: matrix, right-hand side, x0
_BREAKING = {
    "CG": [([[2, 3, 0], [3, 3, 1], [0, 1, -1]], [0, -3, 2], [1, -1, -2]),
           ([[-3, 1, 2], [1, -2, 0], [2, 0, -1]], [-3, 2, 1], [-1, -1, -2])],
    "BICGSTAB": [([[2, 1, 3], [1, 2, 0], [-1, 1, 1]], [3, 3, 1], [-1, 2, -2]),
                 ([[-3, -1, 1], [0, -2, 0], [3, 0, 0]], [3, 2, -2], [-2, 1, -2])],
}


@pytest.mark.parametrize("method", ["CG", "BICGSTAB"])
@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("copies", [1, 1500, 7000])
def test_restart_after_breakdown(psb, method, which, copies):
    """A breakdown with x past x0: each block stores its rows of x, and the
    restart's product reads the rows of other blocks (the three rows of a
    system are `copies` apart).  One block, blocks up to 64 and beyond; as the
    oracle and the kernel-per-step drivers."""
    import scipy.sparse as sp
    a, b, x0 = _BREAKING[method][which]
    m = sp.kron(sp.csr_matrix(np.array(a, float)), sp.identity(copies)).tocsr()
    m.eliminate_zeros()
    m.sort_indices()
    irp, ja, va = (m.indptr + 1).astype(np.int32), (m.indices + 1).astype(np.int32), m.data
    b, x0 = (np.repeat(np.array(v, float), copies) for v in (b, x0))
    xo, ito, _ = O.krylov(method, irp, ja, va, b, x0=x0, eps=1e-10, itmax=40)
    assert ito == 5  # two iterations, the restart, three more
    A = _matrix(psb, "CSR", irp, ja, va)
    for itmax in (40, GENERAL):
        it, err, x, launches = _solve(psb, A, method, b, itmax, prec=False, x0=x0)
        assert (launches == 1) == (itmax == 40)
        assert it == ito and err <= 1e-10
        assert np.max(np.abs(x - xo)) <= 1e-9 * max(1.0, np.max(np.abs(xo)))


@pytest.mark.parametrize("method", ["CG", "BICGSTAB"])
def test_breakdown_and_itmax(psb, method):
    """A breakdown at every restart ends at itmax with x untouched, as in the
    oracle; a solve that does not converge ends there too, and b = 0 at once
    or by breakdowns."""
    irp, ja, va = np.array([1, 2, 3], np.int32), np.array([2, 1], np.int32), np.array([1.0, 1.0])
    A = _matrix(psb, "CSR", irp, ja, va)
    b = np.array([1.0, 0.0])
    xo, ito, _ = O.krylov(method, irp, ja, va, b, itmax=7)
    it, _, x, launches = _solve(psb, A, method, b, 7, prec=False)
    assert launches == 1 and it == ito == 7 and np.array_equal(x, xo)
    irp, ja, va = gen.poisson7(12)
    A = _matrix(psb, "HLL", irp, ja, va)
    it, err, _, launches = _solve(psb, A, method, np.random.default_rng(0).uniform(-1, 1, 1728), 5)
    assert it == 5 and err > 1e-10 and launches == 1
    _, ito, _ = O.krylov(method, irp, ja, va, np.zeros(1728), itmax=9)
    it, err, x, _ = _solve(psb, A, method, np.zeros(1728), 9)
    assert it == ito and not x.any()
