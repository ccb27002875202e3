"""The batch engine at the edges of its tiles and passes: row counts around
one pass of a block (128 rows with eight right-hand sides, 256 with one) and
around a tile (1,024 rows), rows long enough for the long-row tiles, one and
eight right-hand sides, FP32 and FP64 inner iterations; all systems together,
each solution checked against the FP64 residual, and one of them against
the same system alone (same bits)."""
import numpy as np
import pytest
import scipy.sparse as sp

from psblas3_b200 import gen

pytestmark = pytest.mark.gpu


def _hll(psb, irp, ja, va):
    import torch
    n = len(irp) - 1
    d = [torch.from_numpy(a).cuda() for a in (irp, ja, va)]
    torch.cuda.synchronize()
    A = psb.HllMat.from_csr_device(n, n, len(ja), *(t.data_ptr() for t in d), 32)
    return A, psb.DiagPrec("DIAG").build(A)


@pytest.mark.parametrize("nrhs", [1, 8])
@pytest.mark.parametrize("fp64", [False, True])
def test_tile_edges(psb, nrhs, fp64):
    import torch
    systems = []
    for n in (2, 31, 127, 128, 129, 255, 257, 1023, 1024, 1025, 2049):
        systems.append(gen.powerlaw_spd(n, kmax=min(7, n - 1), seed=n))
    # rows beyond 64 entries: long-row tiles among the others, and at the front
    systems.append(gen.powerlaw_spd(1500, kmax=300, seed=3))
    irp, ja, va, _ = gen.sort_rows_by_length(*gen.powerlaw_spd(1200, kmax=400, seed=4))
    systems.append((irp, ja, va))
    total = sum(len(s[0]) - 1 for s in systems)

    def solve(idx):
        eng = psb.BatchSolver(len(idx), total, nrhs, inner_fp64=fp64)
        out, slots = {}, {}
        for i in idx:
            A, P, b = mats[i]
            x = torch.zeros_like(b)
            slots[i] = eng.add(A, b, x, P.dv.data_ptr, eps=1e-10)
            out[i] = x
        torch.cuda.synchronize()
        eng.run(replays_per_step=2)
        for i in idx:
            assert eng.poll(slots[i])[0] == 1
        res = {i: out[i].cpu().numpy() for i in idx}
        eng.free()
        return res

    mats = []
    for i, (irp, ja, va) in enumerate(systems):
        n = len(irp) - 1
        b = np.random.default_rng(i).uniform(-1, 1, (n, nrhs))
        mats.append((*_hll(psb, irp, ja, va), torch.from_numpy(b.reshape(-1)).cuda()))
    torch.cuda.synchronize()
    res = solve(range(len(systems)))
    for i, (irp, ja, va) in enumerate(systems):
        n = len(irp) - 1
        a = sp.csr_matrix((va, ja - 1, irp - 1), shape=(n, n))
        b, x = mats[i][2].cpu().numpy().reshape(n, nrhs), res[i].reshape(n, nrhs)
        rel = np.linalg.norm(b - a @ x, axis=0) / np.linalg.norm(b, axis=0)
        assert rel.max() <= 1.01e-10  # the engine's own residual, summed in another order
    for i in (8, 9, 11, 12):
        assert np.array_equal(solve([i])[i], res[i])


def test_one_plan_for_both_engines(psb):
    """A matrix that engines of one and of eight right-hand sides add in turn
    (one tile plan, built once): the same bits every time, and each column of
    eight equals the solve of that column alone."""
    import torch
    irp, ja, va = gen.powerlaw_spd(2300, kmax=40, seed=6)
    n = len(irp) - 1
    assert np.diff(irp).max() <= 64  # longer rows are summed in another way for eight
    A, P = _hll(psb, irp, ja, va)
    b = np.random.default_rng(2).uniform(-1, 1, (n, 8))

    def solve(nrhs, cols):
        eng = psb.BatchSolver(1, n, nrhs)
        d = torch.from_numpy(np.ascontiguousarray(cols).reshape(-1)).cuda()
        x = torch.zeros_like(d)
        torch.cuda.synchronize()
        slot = eng.add(A, d, x, P.dv.data_ptr, eps=1e-10)
        eng.run(replays_per_step=2)
        assert eng.poll(slot)[0] == 1
        res = x.cpu().numpy().reshape(n, nrhs)
        eng.free()
        return res

    one = solve(1, b[:, :1])
    eight = solve(8, b)
    assert np.array_equal(solve(1, b[:, :1]), one)
    assert np.array_equal(solve(8, b), eight)
    assert np.array_equal(solve(1, b[:, 5:6])[:, 0], eight[:, 5]) and np.array_equal(one[:, 0], eight[:, 0])
