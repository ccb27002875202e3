"""HLL arrays of a caller whose hacks start at odd entries: the kernels that
read two adjacent rows in one load cannot take them, the row-per-thread ones
can.  Products equal the CPU csmv's (FP64 bit for bit, FP32 the FP64 row sum
rounded once); the mixed CG, which has no other product, refuses them."""
import numpy as np
import pytest

import oracle as O
from psblas3_b200 import gen
from psblas3_b200._lib import PsbxError

pytestmark = pytest.mark.gpu


def _odd(psb, irp, ja, va):
    """The matrix as host HLL arrays with one unused entry in front."""
    n = len(irp) - 1
    ia, _, _ = gen.csr_to_coo(irp, ja, va)
    h = O.hll_from_coo(n, ia, ja, va, 32)
    return psb.HllMat.from_host_hll(n, 32, h["irn"], np.asarray(h["hkoffs"]) + 1, np.concatenate([[1], h["ja"]]),
                                    np.concatenate([[0.0], h["val"]]), h["idiag"])


@pytest.mark.parametrize("tpr", [0, -2])
@pytest.mark.parametrize("case", ["short", "wide"])
def test_products(psb, case, tpr):
    if case == "short":
        irp, ja, va = gen.poisson7(11)
    else:  # hacks wider than 64 entries: two rows per thread by default
        irp, ja, va, _ = gen.sort_rows_by_length(*gen.powerlaw_spd(3000, kmax=900, seed=2))
    n = len(irp) - 1
    A = _odd(psb, irp, ja, va)
    A.set_threads_per_row(tpr)
    A.set_wide_split(False)  # stored-order sums
    x = np.random.default_rng(3).uniform(-1, 1, n)
    X, Y = psb.DVect.bld(x), psb.DVect(n)
    psb.psb_spmm(1.0, A, X, 0.0, Y)
    assert np.array_equal(Y.get_vect(), O.csr_csmv(irp, ja, va, 1.0, x, 0.0, np.zeros(n)))
    A.make_single()
    v32, x32 = va.astype(np.float32), x.astype(np.float32)
    X, Y = psb.DVect.bld(x32), psb.DVect.bld(np.zeros(n, np.float32))
    A.spmv(1.0, X, 0.0, Y)
    ref = O.csr_csmv(irp, ja, v32.astype(np.float64), 1.0, x32.astype(np.float64), 0.0, np.zeros(n))
    assert np.array_equal(Y.get_vect(), ref.astype(np.float32))


def test_mixed_refuses(psb):
    A = _odd(psb, *gen.poisson7(8))
    B, X = psb.DVect.bld(np.ones(512)), psb.DVect(512)
    with pytest.raises(PsbxError):
        psb.psb_mixed_cg(A, None, B, X)
