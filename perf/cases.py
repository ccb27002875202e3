"""The work users of this library have it do, as timed cases.

Each case goes through the public entry points (psblas3_b200.psb, and
psbx_wrapMultiVecDevice for vectors that live in torch tensors).  Kinds:

* ``spmv``   -- y = A x, the product behind psb_spmm: formats HLL / ELL / CSR,
                FP64 and (HLL) FP32, stencil operators and row-sorted power-law
                matrices, from a few thousand rows to the 27-point 200^3 grid.
* ``step``   -- the vector part of a Krylov step as host code writes it with
                psb_geaxpby / psb_gedot / psb_genrm2 / the DIAG apply.
* ``solve``  -- psb_krylov('CG' | 'BICGSTAB') with the DIAG preconditioner.
* ``mixed``  -- psb_mixed_cg, one large SPD system.
* ``batch``  -- the batch engine: many systems of uneven size, each with 1 or 8
                right-hand sides, from admission to removal.

Matrices are made on the GPU from the seed; stencils of the product cases have
varying coefficients (a heterogeneous medium), those of the solves are the
constant-coefficient operators of the benchmark configurations.  Right-hand
sides of the solves are b = A u* with u* random, so u* is the exact answer.
"""
import ctypes
import math
import random

import numpy as np
import torch

from psblas3_b200 import psb
from psblas3_b200._lib import check, lib

POWER_ALPHA = 2.1


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the roofline operator of the benchmark: the largest product
        {"name": "spmv_hll_27pt_200", "kind": "spmv", "fmt": "hll", "op": "27pt", "side": 200, "bits": 64},
        # one product of the convection-diffusion test problem, 64,000 rows: launch and latency
        {"name": "spmv_hll_pde_40", "kind": "spmv", "fmt": "hll", "op": "pde", "side": 40, "bits": 64},
        # the single-precision product (the s types, and the inner products of mixed solvers)
        {"name": "spmv_hll_f32_27pt_100", "kind": "spmv", "fmt": "hll", "op": "27pt", "side": 100, "bits": 32},
        # host code that keeps its matrices in CSR
        {"name": "spmv_csr_27pt_128", "kind": "spmv", "fmt": "csr", "op": "27pt", "side": 128, "bits": 64},
        # ELL, an odd grid side: 1.0M rows, not a multiple of the warp size
        {"name": "spmv_ell_27pt_101", "kind": "spmv", "fmt": "ell", "op": "27pt", "side": 101, "bits": 64},
        # an unstructured matrix with power-law rows (1 to 4,096 entries), rows held in length order
        {"name": "spmv_hll_power_4m", "kind": "spmv", "fmt": "hll", "op": "power", "rows": 4_000_000, "bits": 64},
        # the vector operations of one iteration of hand-written Krylov code on the 64,000-row problem
        {"name": "step_64000", "kind": "step", "rows": 64_000},
        # the test problem of the reference's drivers: BiCGSTAB + DIAG, 64,000 rows, to 1e-9
        {"name": "bicgstab_pde_40", "kind": "solve", "method": "BICGSTAB", "side": 40, "eps": 1e-9},
        # an ordinary FP64 solve whose data no longer fits the L2 cache
        {"name": "cg_poisson7_128", "kind": "solve", "method": "CG", "side": 128, "eps": 1e-10},
        # the large mixed-precision solve: 16.8M rows
        {"name": "mixed_poisson7_256", "kind": "mixed", "side": 256},
        # a batch of small anisotropic 2-D systems, 8 right-hand sides each
        {"name": "batch_aniso_128x8", "kind": "batch", "mix": "aniso", "systems": 128, "nrhs": 8, "lot": 1},
        # the mix a solve server has in flight: 3-D grids and power-law systems, one right-hand side each
        {"name": "batch_mix_32x1", "kind": "batch", "mix": "serve", "systems": 32, "nrhs": 1, "lot": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv", "step", "solve", "solve", "mixed", "batch"])
    if kind == "spmv":
        op = rng.choice(["27pt", "pde", "power"])
        if op == "power":  # held as row-sorted HLL, or as CSR
            return {"kind": kind, "fmt": rng.choice(["hll", "csr"]), "op": op, "rows": _log(rng, 20_000, 4_000_000),
                    "bits": 64}
        fmt = rng.choice(["hll", "hll", "ell", "csr"])
        bits = rng.choice([64, 32]) if fmt == "hll" else 64
        # up to the rows of the largest listed case of the format
        top = {"hll": 200, "ell": 101, "csr": 128}[fmt]
        return {"kind": kind, "fmt": fmt, "op": op, "side": int(round(_log(rng, 12 ** 3, top ** 3) ** (1 / 3))),
                "bits": bits}
    if kind == "step":
        return {"kind": kind, "rows": _log(rng, 1_000, 16_000_000)}
    if kind == "solve":
        method = rng.choice(["CG", "BICGSTAB"])
        top = 128 if method == "CG" else 112
        return {"kind": kind, "method": method, "side": int(round(_log(rng, 12 ** 3, top ** 3) ** (1 / 3))),
                "eps": rng.choice([1e-9, 1e-10])}
    if kind == "mixed":
        return {"kind": kind, "side": int(round(_log(rng, 24 ** 3, 256 ** 3) ** (1 / 3)))}
    nrhs = rng.choice([1, 8])
    return {"kind": kind, "mix": "aniso" if nrhs == 8 else "serve", "systems": _log(rng, 4, 128 if nrhs == 8 else 32),
            "nrhs": nrhs, "lot": rng.randrange(1 << 20)}


def _systems(case):
    """The systems of a batch: (kind, size, coefficient), a function of the case alone."""
    r = random.Random(case["lot"])
    if case["mix"] == "aniso":  # grids of side 32..256, anisotropy log-uniform in [1e-2, 1]
        return [("aniso", r.randint(32, 256), math.exp(r.uniform(math.log(1e-2), 0.0))) for _ in range(case["systems"])]
    return [("poisson", r.randint(10, 96), 0.0) if k % 2 == 0 else ("power", _log(r, 1_000, 500_000), 0.0)
            for k in range(case["systems"])]


# ---------------------------------------------------------------- matrices, made on the GPU
def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + salt) % (1 << 62))
    return g


def _uniform(n, g, lo=0.0, hi=1.0):
    return torch.empty(n, dtype=torch.float64, device="cuda").uniform_(lo, hi, generator=g)


def _stencil(side, dims, points, g=None):
    """CSR (1-based, int32) of a stencil on a side^dims grid, x fastest.
    points: (dx, dy, dz, value) in ascending column order; g: vary each entry
    by up to 25 % either way."""
    n = side ** dims
    i = torch.arange(n, dtype=torch.int32, device="cuda")
    c = [i % side, i // side % side, i // (side * side)]
    ja = torch.empty((n, len(points)), dtype=torch.int32, device="cuda")
    ok = torch.empty((n, len(points)), dtype=torch.bool, device="cuda")
    for k, (dx, dy, dz, _) in enumerate(points):
        m = torch.ones(n, dtype=torch.bool, device="cuda")
        for d, x in zip((dx, dy, dz), c):
            if d:
                m &= (x + d >= 0) & (x + d < side)
        ok[:, k] = m
        ja[:, k] = i + (1 + dx + dy * side + dz * side * side)
    irp = torch.ones(n + 1, dtype=torch.int32, device="cuda")
    irp[1:] += torch.cumsum(ok.sum(1), 0).to(torch.int32)
    va = torch.tensor([p[3] for p in points], dtype=torch.float64, device="cuda").expand(n, -1)[ok]
    if g is not None:
        va *= _uniform(va.numel(), g, 0.75, 1.25)
    return irp, ja[ok], va


def _pde_points(side):
    """The 7-point convection-diffusion operator, b = (1,1,1)/sqrt(3)."""
    h = 1.0 / (side + 1)
    d, v = 1.0 / (h * h), 1.0 / math.sqrt(3.0) / (2.0 * h)
    return [(0, 0, -1, -d - v), (0, -1, 0, -d - v), (-1, 0, 0, -d - v), (0, 0, 0, 6.0 * d),
            (1, 0, 0, -d + v), (0, 1, 0, -d + v), (0, 0, 1, -d + v)]


_POISSON = [(0, 0, -1, -1.0), (0, -1, 0, -1.0), (-1, 0, 0, -1.0), (0, 0, 0, 6.0),
            (1, 0, 0, -1.0), (0, 1, 0, -1.0), (0, 0, 1, -1.0)]


def _points27():
    return [(x, y, z, 26.0 if x == y == z == 0 else -1.0) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)]


def _aniso_points(eps):
    return [(0, -1, 0, -1.0), (-1, 0, 0, -eps), (0, 0, 0, 2.0 * eps + 2.0), (1, 0, 0, -eps), (0, 1, 0, -1.0)]


def _power_law(n):
    k = np.arange(1, min(4096, n - 1) + 1, dtype=np.float64)
    p = k ** -POWER_ALPHA
    return k, p / p.sum()


def _row_sums(vals, lens):
    """Sums of consecutive runs, each in order (the same bits every time)."""
    return torch.segment_reduce(vals, "sum", lengths=lens, unsafe=True, initial=0.0)


def _with_diag(key, vals, n):
    """CSR of the sorted, distinct off-diagonal entries key = row*n + column
    plus the dominant diagonal."""
    diag = _row_sums(vals.abs(), torch.bincount(key // n, minlength=n)) + 1.0
    i = torch.arange(n, device="cuda")
    key, at = torch.sort(torch.cat([key, i * n + i]))
    irp = torch.ones(n + 1, dtype=torch.int32, device="cuda")
    irp[1:] += torch.cumsum(torch.bincount(key // n, minlength=n), 0).to(torch.int32)
    return irp, (key % n + 1).to(torch.int32), torch.cat([vals, diag])[at]


def _power_entries(n, g):
    k, p = _power_law(n)
    cdf = torch.from_numpy(np.cumsum(p)).cuda()
    lens = (torch.searchsorted(cdf, _uniform(n, g)) + 1).clamp_(max=len(k))
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    cols = torch.randint(0, n - 1, (rows.numel(),), device="cuda", generator=g)
    cols += cols >= rows  # not the diagonal
    key = torch.unique(rows * n + cols)  # sorted, without repeats
    return key, torch.randn(key.numel(), dtype=torch.float64, device="cuda", generator=g)


def _power(n, g):
    return _with_diag(*_power_entries(n, g), n)


def _power_spd(n, g):
    """Symmetric, diagonally dominant, rows and columns in decreasing-length order."""
    key, v = _power_entries(n, g)
    r, c = key // n, key % n
    key, inv = torch.unique(torch.cat([r * n + c, c * n + r]), return_inverse=True)
    order = torch.argsort(inv, stable=True)  # each key's values are added in a fixed order
    ends = torch.cumsum(torch.bincount(inv), 0) - 1
    vv = torch.cat([v, v])[order]
    two = torch.zeros_like(ends, dtype=torch.bool)
    two[1:] = ends[1:] - ends[:-1] == 2
    two[0] = ends[0] == 1
    vals = vv[ends] + torch.where(two, vv[(ends - 1).clamp(min=0)], torch.zeros((), dtype=torch.float64, device="cuda"))
    r, c = key // n, key % n
    place = torch.empty(n, dtype=torch.int64, device="cuda")
    place[torch.argsort(torch.bincount(r, minlength=n), descending=True, stable=True)] = torch.arange(n, device="cuda")
    key, at = torch.sort(place[r] * n + place[c])
    return _with_diag(key, vals[at], n)


def _times(csr, x):
    """A x in 64 bits by torch."""
    irp, ja, va = csr
    return _row_sums(va * x[ja - 1], (irp[1:] - irp[:-1]).to(torch.int64))


# ---------------------------------------------------------------- library objects
def _vect(t):
    """A torch tensor as a library vector (its memory, no copy)."""
    v = psb.DVect.__new__(psb.DVect)
    v.n = v.pitch = t.numel()
    v.count = 1
    double = t.dtype == torch.float64
    v.dtype, v.tname = (np.dtype(np.float64), "Double") if double else (np.dtype(np.float32), "Float")
    v.h = ctypes.c_void_p()
    check(lib.psbx_wrapMultiVecDevice(ctypes.byref(v.h), ctypes.c_void_p(t.data_ptr()), v.n, 2 if double else 1),
          "wrap")
    v.tensor = t
    return v


def _hll(csr, perm=None):
    irp, ja, va = csr
    torch.cuda.synchronize()
    n = irp.numel() - 1
    return psb.HllMat.from_csr_device(n, n, ja.numel(), irp.data_ptr(), ja.data_ptr(), va.data_ptr(), 32,
                                      None if perm is None else perm.data_ptr())


def _ell(csr):
    irp, ja, va = csr
    n = irp.numel() - 1
    lens = (irp[1:] - irp[:-1]).to(torch.int64)
    nzm = int(lens.max())
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    j = torch.arange(ja.numel(), device="cuda") - (irp[:-1] - 1).to(torch.int64)[rows]
    eja = torch.ones((nzm, n), dtype=torch.int32, device="cuda")
    eva = torch.zeros((nzm, n), dtype=torch.float64, device="cuda")
    eja[j, rows], eva[j, rows] = ja, va
    idiag = torch.zeros(n, dtype=torch.int32, device="cuda")
    d = ja == rows + 1
    idiag[rows[d]] = (j[d] + 1).to(torch.int32)
    return psb.EllMat.from_host_ell(n, nzm, lens.to(torch.int32).cpu().numpy(), eja.cpu().numpy(), eva.cpu().numpy(),
                                    idiag.cpu().numpy(), n, nnz=ja.numel())


def _matrix(case, seed):
    g = _gen(seed)
    if case["op"] == "power":
        return _power(case["rows"], g)
    return _stencil(case["side"], 3, _points27() if case["op"] == "27pt" else _pde_points(case["side"]), g)


def _solve_csr(case):
    return _stencil(case["side"], 3, _pde_points(case["side"]) if case.get("method") == "BICGSTAB" else _POISSON)


def _batch_csr(spec, seed, k):
    kind, size, eps = spec
    if kind == "aniso":
        return _stencil(size, 2, _aniso_points(eps))
    return _stencil(size, 3, _POISSON) if kind == "poisson" else _power_spd(size, _gen(seed, 2 * k + 1))


# ---------------------------------------------------------------- prepare, run
def prepare(case, seed):
    psb.init(0)
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "spmv":
        csr = _matrix(case, seed)
        n = csr[0].numel() - 1
        if case["fmt"] == "hll":
            lens = csr[0][1:] - csr[0][:-1]
            perm = torch.argsort(lens, descending=True, stable=True).to(torch.int32) if case["op"] == "power" else None
            s["a"] = _hll(csr, perm)
            if case["bits"] == 32:
                s["a"].make_single()
        elif case["fmt"] == "ell":
            s["a"] = _ell(csr)
        else:
            s["a"] = psb.CsrMat(n, *(t.cpu().numpy() for t in csr))
        x = _uniform(n, _gen(seed, 7), -1.0, 1.0)
        x = x if case["bits"] == 64 else x.float()
        s["x"], s["y"] = _vect(x), _vect(torch.zeros_like(x))
    elif kind == "step":
        r, v = (_uniform(case["rows"], _gen(seed, k), -1.0, 1.0) for k in (1, 2))
        d = _uniform(case["rows"], _gen(seed, 3), 0.1, 0.5)
        s.update(r=_vect(r), v=_vect(v), d=_vect(d), w=_vect(torch.zeros_like(r)), z=_vect(torch.zeros_like(r)))
    elif kind in ("solve", "mixed"):
        csr = _solve_csr(case)
        s["a"] = _hll(csr)
        if kind == "mixed":
            s["a"].make_single()
        s["prec"] = psb.DiagPrec("DIAG").build(s["a"])
        b = _times(csr, _uniform(csr[0].numel() - 1, _gen(seed, 5)))
        s.update(b=_vect(b), x=_vect(torch.zeros_like(b)), method=case.get("method"), eps=case.get("eps", 1e-10))
    else:
        specs, k = _systems(case), case["nrhs"]
        s["sys"], total = [], 0
        us, bs = [], []
        for i, spec in enumerate(specs):
            csr = _batch_csr(spec, seed, i)
            n = csr[0].numel() - 1
            u = _uniform(n * k, _gen(seed, 2 * i + 2), -1.0, 1.0).view(n, k)
            bs.append(torch.stack([_times(csr, u[:, j].contiguous()) for j in range(k)], 1).contiguous())
            a = _hll(csr)
            a.make_single()
            s["sys"].append((a, psb.DiagPrec("DIAG").build(a)))
            total += n
        s["b"] = bs
        # the solutions, end to end in one buffer
        s["all"] = _vect(torch.zeros(total * k, dtype=torch.float64, device="cuda"))
        s["x"] = list(s["all"].tensor.split([b.numel() for b in bs]))
        s["eng"] = psb.BatchSolver(len(specs), total, k)
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "spmv":
        psb.psb_spmm(1.0, s["a"], s["x"], 0.0, s["y"])
        return s["y"].tensor
    if kind == "step":  # w = r - alpha v ; z = M^-1 w ; (w, z) ; ||w||
        psb.psb_geaxpby(1.0, s["r"], 0.0, s["w"])
        psb.psb_geaxpby(-0.37, s["v"], 1.0, s["w"])
        psb.psb_gemlt(1.0, s["d"], s["w"], 0.0, s["z"])
        return s["w"].tensor, s["z"].tensor, float(psb.psb_gedot(s["w"], s["z"])), float(psb.psb_genrm2(s["w"]))
    if kind == "solve":
        s["x"].zero()
        psb.psb_krylov(s["method"], s["a"], s["prec"], s["b"], s["x"], eps=s["eps"], itmax=5000)
        return s["x"].tensor
    if kind == "mixed":
        s["x"].zero()
        psb.psb_mixed_cg(s["a"], s["prec"], s["b"], s["x"], eps=1e-10, itmax=20000, delta=0.1)
        return s["x"].tensor
    eng = s["eng"]
    s["all"].zero()
    slots = [eng.add(a, b, x, p.dv.data_ptr, eps=1e-10) for (a, p), b, x in zip(s["sys"], s["b"], s["x"])]
    eng.run(replays_per_step=4)
    for slot in slots:
        if eng.poll(slot)[0] != 1:
            raise RuntimeError("a system of the batch did not converge")
        eng.remove(slot)
    return s["all"].tensor


# ---------------------------------------------------------------- work, tolerance, exact
def _nnz(op, side):
    return {"27pt": (3 * side - 2) ** 3, "pde": 7 * side ** 3 - 6 * side ** 2}[op]


def work(case):
    """A product reads its matrix (values, 4-byte indices, row lengths) and x
    and writes y.  An iteration of a solve cannot do without its products
    and five vectors read or written (two in a mixed solve's or the batch
    engine's FP32); the iterations are the method's own on the operator, from
    its convergence on grids of several sizes."""
    kind = case["kind"]
    if kind == "spmv":
        w = case["bits"] // 8
        if case["op"] == "power":
            n = case["rows"]
            k, p = _power_law(n)
            nnz = n * (1.0 + float((k * p).sum()))
        else:
            n, nnz = case["side"] ** 3, _nnz(case["op"], case["side"])
        return {"bytes": nnz * (w + 4) + n * (2 * w + 4), "flops": 2 * nnz}
    if kind == "step":  # r, v, d read, w, z written
        return {"bytes": 40 * case["rows"], "flops": 8 * case["rows"]}
    if kind in ("solve", "mixed"):
        n, nnz = case["side"] ** 3, _nnz("pde", case["side"])
        if kind == "mixed":
            it, w, products = 3.2 * case["side"], 4, 1
        elif case["method"] == "CG":
            it, w, products = 3.2 * case["side"], 8, 1
        else:
            it, w, products = 2.7 * case["side"], 8, 2
        return {"bytes": it * (products * (nnz * (w + 4) + 4 * n) + 5 * w * n),
                "flops": it * (products * 2 * nnz + 12 * n)}
    total = flops = 0.0
    k = case["nrhs"]
    for sys_kind, size, _ in _systems(case):
        if sys_kind == "aniso":
            n, nnz, it = size ** 2, 5 * size ** 2 - 4 * size, 5.0 * size
        elif sys_kind == "poisson":
            n, nnz, it = size ** 3, _nnz("pde", size), 3.2 * size
        else:
            d, p = _power_law(size)
            n, nnz, it = size, size * (1.0 + 2.0 * float((d * p).sum())), 30.0
        total += it * (nnz * 8 + 4 * n + 5 * 4 * k * n)
        flops += it * k * (2 * nnz + 12 * n)
    return {"bytes": total, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("spmv", "step"):
        # sums of a row in another order: 2.7e-16 measured against exact(); FP32 2.5e-8 with the
        # sums in 64 bits, about 2e-7 with them in 32
        return {"rel": 2e-15, "max": 1e-12} if case.get("bits", 64) == 64 else {"rel": 1e-6, "max": 1e-5}
    # a solve stops where its residual meets the tolerance; the error against the exact answer that
    # the stop test leaves is 3e-9 to 1e-7 on these operators, and two solves differ by as much
    return {"rel": 1e-6, "max": 4e-5}


def exact(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        irp, ja, va = _matrix(case, seed)
        x = _uniform(irp.numel() - 1, _gen(seed, 7), -1.0, 1.0)
        if case["bits"] == 32:
            x, va = x.float().double(), va.float().double()
        return _times((irp, ja, va), x)
    if kind == "step":
        r, v = (_uniform(case["rows"], _gen(seed, k), -1.0, 1.0) for k in (1, 2))
        w = r - 0.37 * v
        z = w * _uniform(case["rows"], _gen(seed, 3), 0.1, 0.5)
        return w, z, float(torch.dot(w, z)), float(torch.linalg.vector_norm(w))
    if kind in ("solve", "mixed"):
        return _uniform(case["side"] ** 3, _gen(seed, 5))
    us = [_uniform((size if kind == "power" else size ** (2 if kind == "aniso" else 3)) * case["nrhs"],
                   _gen(seed, 2 * i + 2), -1.0, 1.0) for i, (kind, size, _) in enumerate(_systems(case))]
    return torch.cat(us)
