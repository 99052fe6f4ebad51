"""Performance cases: the calls that a program built on this library spends its time in.

A case names one call (or the few calls that belong together) of the Python binding over the C ABI,
with its sizes, element type and options.  Three levels are covered:

* MatrixSwitch and pspBLAS operations on device matrices: dense products, dense x CSC, CSC x dense,
  transposed adds with the trace that follows them;
* the derivative calls: the gradient of the Kim functional at given coefficients, and the adjoint of
  the converged energy with respect to the parameters of H;
* whole minimisations (omm), in FP64 and in the mixed-precision mode.

Sizes are those of the test-suite's products, of the generator's workloads (dense m = 832 with
n = 128; 24-orbital atoms on a periodic cubic lattice with two-spacing neighbour shells; dense
complex m = 4,096 with n = 512 and 16 sparse perturbations) and generic odd ones between them.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "omm-bundle_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ommgpu as G  # noqa: E402
from ommgpu import synth  # noqa: E402

_DEV = "cuda"
_STEPS = 32  # CG steps of a minimisation to the default tolerance, for work() only


# ------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest products: a k-point example's or a unit test's size, where a call's latency counts
        dict(name="mm_small_real", kind="mm", M=37, N=53, K=61, opA="n", opB="t", cplx=False),
        # an ordinary dense product of odd size with a transposed left operand
        dict(name="mm_odd_real", kind="mm", M=1001, N=515, K=2003, opA="t", opB="n", cplx=False),
        # the Gram product of complex coefficients (n = 512, m = 4,096): C H C^H
        dict(name="mm_gram_complex", kind="mm", M=512, N=512, K=4096, opA="n", opB="c", cplx=True),
        # pspBLAS dense x CSC: coefficients times an atom-block Hamiltonian
        dict(name="gemspm_blocks_real", kind="gemspm", Lx=8, Ly=8, Lz=8, norb=24, M=1536, pattern="blocks", opA="n", opB="n",
             cplx=False),
        # pspBLAS dense x CSC with an irregular complex matrix (2 % fill), odd sizes
        dict(name="gemspm_scatter_complex", kind="gemspm", K=2501, N=2501, M=333, fill=0.02, pattern="scatter",
             opA="n", opB="n", cplx=True),
        # pspBLAS CSC x dense with an atom-block matrix
        dict(name="gespmm_blocks_real", kind="gespmm", Lx=5, Ly=5, Lz=5, norb=24, N=375, pattern="blocks", opA="n", opB="n",
             cplx=False),
        # B + alpha A^H and its overlap with B, on odd complex matrices
        dict(name="add_trace_complex", kind="add", rows=2049, cols=1537, op="c", cplx=True),
        # gradient of the functional for a lattice of 343 atoms (n = 1,029, m = 8,232)
        dict(name="grad_lattice_real", kind="grad", Lx=7, Ly=7, Lz=7, norb=24, nocc=3),
        # derivative of the converged energy for 16 sparse perturbations of a dense complex problem
        dict(name="adjoint_complex", kind="adjoint", m=4096, n=512, nv=16, fill=0.02, cplx=True),
        # a whole minimisation of a small dense problem: many short steps
        dict(name="omm_dense_real", kind="omm", problem="dense", m=832, n=128, cplx=False, flavour=0, label="gpu"),
        # a whole minimisation of the 512-atom lattice in FP64, and of the 216-atom one (n = 648) in mixed precision
        dict(name="omm_lattice_fp64", kind="omm", problem="lattice", Lx=8, Ly=8, Lz=8, norb=24, nocc=3, label="gpu"),
        dict(name="omm_lattice_mixed", kind="omm", problem="lattice", Lx=6, Ly=6, Lz=6, norb=24, nocc=3, label="gmx"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _atoms(rng):
    """Lattice sides, orbitals per atom and occupied states per atom (one state in eight)."""
    norb, nocc = rng.choice([(8, 1), (13, 2), (16, 2), (24, 3)])
    return dict(Lx=rng.randint(5, 8), Ly=rng.randint(5, 8), Lz=rng.randint(5, 8), norb=norb, nocc=nocc)


def draw(rng):
    kind = rng.choice(["mm", "gemspm", "gespmm", "add", "grad", "adjoint", "omm_dense", "omm_lattice"])
    cplx = rng.random() < 0.5
    if kind == "mm":
        return dict(kind="mm", M=_log_int(rng, 16, 3000), N=_log_int(rng, 16, 3000), K=_log_int(rng, 16, 6000),
                    opA=rng.choice("ntc"), opB=rng.choice("ntc"), cplx=cplx)
    if kind in ("gemspm", "gespmm"):
        rows = _log_int(rng, 17, 1600)
        dense = "M" if kind == "gemspm" else "N"
        ops = dict(opA=rng.choice("nt"), opB=rng.choice("nt"), cplx=cplx)
        if rng.random() < 0.5:
            a = _atoms(rng)
            del a["nocc"]
            if cplx:
                a["Lx"] = 5
            return {"kind": kind, "pattern": "blocks", dense: rows, **a, **ops}
        other = "N" if kind == "gemspm" else "M"
        return {"kind": kind, "pattern": "scatter", "K": _log_int(rng, 60, 4000), other: _log_int(rng, 60, 4000),
                dense: rows, "fill": round(rng.uniform(0.005, 0.1), 4), **ops}
    if kind == "add":
        return dict(kind="add", rows=_log_int(rng, 20, 6000), cols=_log_int(rng, 20, 6000), op=rng.choice("ntc"),
                    cplx=cplx)
    if kind == "grad":
        return dict(kind="grad", **_atoms(rng))
    if kind == "adjoint":
        m = _log_int(rng, 300, 4096)
        return dict(kind="adjoint", m=m, n=max(4, int(m * rng.uniform(0.05, 0.2))), nv=rng.randint(1, 16),
                    fill=round(rng.uniform(0.002, 0.02), 4), cplx=cplx)
    if kind == "omm_dense":
        m = _log_int(rng, 60, 1200)
        return dict(kind="omm", problem="dense", m=m, n=max(4, int(m * rng.uniform(0.08, 0.35))), cplx=cplx,
                    flavour=rng.choice([0, 0, 3]), label="gpu")
    return dict(kind="omm", problem="lattice", label=rng.choice(["gpu", "gpu", "gmx"]), **_atoms(rng))


# ------------------------------------------------------------------------------------ the inputs
def _dtype(cplx):
    return torch.complex128 if cplx else torch.float64


def _randn(gen, *shape, cplx=False):
    return torch.randn(*shape, dtype=_dtype(cplx), device=_DEV, generator=gen)


class _Dense:
    """A column-major matrix in torch memory with its library handle; .t is the rows x cols tensor."""

    def __init__(self, t):
        self.buf = t.t().contiguous()
        self.t = self.buf.t()
        self.h = G.Matrix.register_gden(self.buf.data_ptr(), t.shape[0], t.shape[1], t.is_complex(), keep=self.buf)


def _shell():
    r = range(-2, 3)
    return [(x, y, z) for x in r for y in r for z in r if x * x + y * y + z * z <= 4]


def _atom_count(c):
    return c["Lx"] * c["Ly"] * c["Lz"]


def _lattice_pattern(c):
    """Neighbour lists of a periodic lattice: (sorted neighbours, shell index of each, unsorted neighbours, shell)."""
    Lx, Ly, Lz = c["Lx"], c["Ly"], c["Lz"]
    sh = np.array(_shell())
    a = np.arange(Lx * Ly * Lz)
    x, y, z = a // (Ly * Lz), (a // Lz) % Ly, a % Lz
    b = (((x[:, None] + sh[:, 0]) % Lx) * Ly + (y[:, None] + sh[:, 1]) % Ly) * Lz + (z[:, None] + sh[:, 2]) % Lz
    order = np.argsort(b, axis=1, kind="stable")
    return np.take_along_axis(b, order, 1), order, b, sh


def _lattice_csc(norb, pattern, blocks):
    """CSC of the block matrix whose block (neighbour d of atom j, j) is blocks[j, d]."""
    nb, order, _, sh = pattern
    na, ns = nb.shape
    v = torch.gather(blocks, 1, torch.from_numpy(order).to(_DEV)[:, :, None, None].expand(-1, -1, norb, norb))
    val = v.permute(0, 3, 1, 2).reshape(-1).cpu().numpy()  # atom, column, neighbour, row
    rows = (nb[:, :, None] * norb + np.arange(norb)).reshape(na, 1, ns * norb)
    rowind = np.broadcast_to(rows, (na, norb, ns * norb)).reshape(-1).astype(np.int32)
    m = na * norb
    colptr = (np.arange(m + 1) * (ns * norb)).astype(np.int32)
    return synth.CSCMatrix(m, m, colptr, rowind, val)


def _hermitian_blocks(gen, pattern, norb, scale, onsite, cplx):
    """Random blocks with block(i, j) = block(j, i)^H, offsite ones scaled by distance, and a given onsite block."""
    _, _, b, sh = pattern
    na, ns = b.shape
    R = _randn(gen, na, ns, norb, norb, cplx=cplx)
    at = {tuple(d): k for k, d in enumerate(sh.tolist())}
    back = torch.tensor([at[tuple((-d).tolist())] for d in sh], device=_DEV)  # index of -d
    other = R[torch.from_numpy(b).to(_DEV), back[None, :].expand(na, -1)]
    R = (R + other.transpose(2, 3).conj()) / math.sqrt(2.0)
    r = torch.from_numpy(np.sqrt((sh * sh).sum(1))).to(_DEV)
    out = scale(r)[None, :, None, None] * R
    k0 = at[(0, 0, 0)]
    out[:, k0] = onsite(R[:, k0])
    return out


def _lattice_HS(gen, c, cplx=False):
    """H and S of norb orbitals per atom, nocc of them occupied, with a gap around zero."""
    norb, nocc = c["norb"], c["nocc"]
    pat = _lattice_pattern(c)
    w = math.sqrt(24.0 / norb)  # the same band width for every basis size
    levels = torch.ones(norb, dtype=_dtype(cplx), device=_DEV)
    levels[:nocc] = -1.0
    eye = torch.eye(norb, dtype=_dtype(cplx), device=_DEV)
    S = _hermitian_blocks(gen, pat, norb, lambda r: 0.04 * w * torch.exp(-r * r), lambda R: eye, cplx)
    H = _hermitian_blocks(gen, pat, norb, lambda r: 0.06 * w * torch.exp(-r),
                          lambda R: torch.diag(levels) + 0.07 * R, cplx)
    H = H + 0.345 * S  # the middle of the gap at zero
    return _lattice_csc(norb, pat, H), _lattice_csc(norb, pat, S)


def _scatter_csc(gen, rows, cols, fill, cplx, hermitian=False, scale=1.0):
    mask = torch.rand(cols, rows, device=_DEV, generator=gen) < (0.5 * fill if hermitian else fill)
    v = _randn(gen, cols, rows, cplx=cplx) * scale * mask
    if hermitian:
        v = v + v.t().conj()
    at = v.nonzero()  # column-major order: column, then row
    colptr = np.zeros(cols + 1, dtype=np.int32)
    colptr[1:] = torch.bincount(at[:, 0], minlength=cols).cumsum(0).cpu().numpy()
    return synth.CSCMatrix(rows, cols, colptr, at[:, 1].to(torch.int32).cpu().numpy(),
                           v[at[:, 0], at[:, 1]].cpu().numpy())


def _dense_HS(gen, m, n, cplx):
    """S = L L^H and H = L Q diag(lam) Q^H L^H with n negative eigenvalues and a gap."""
    eye = torch.eye(m, dtype=_dtype(cplx), device=_DEV)
    Lf = eye + (0.1 / math.sqrt(m)) * _randn(gen, m, m, cplx=cplx).tril()
    Q, _ = torch.linalg.qr(_randn(gen, m, m, cplx=cplx))
    u = torch.rand(m, dtype=torch.float64, device=_DEV, generator=gen)
    lam = torch.where(torch.arange(m, device=_DEV) < n, -2.0 + 1.5 * u, 0.1 + 2.9 * u)
    W = Lf @ Q
    H = (W * lam) @ W.mH
    S = Lf @ Lf.mH
    return 0.5 * (H + H.mH), 0.5 * (S + S.mH), Lf, Q, lam


def _coefficients(gen, m, n, cplx=False):
    return _randn(gen, n, m, cplx=cplx) / math.sqrt(m)


def _op(t, op):
    return t if op == "n" else t.t() if op == "t" else t.mH


def _inputs(c, seed):
    """The case's host and torch inputs, before any handle is made."""
    gen = torch.Generator(device=_DEV)
    gen.manual_seed(int(seed))
    k = c["kind"]
    if k == "mm":
        a = (c["M"], c["K"]) if c["opA"] == "n" else (c["K"], c["M"])
        b = (c["K"], c["N"]) if c["opB"] == "n" else (c["N"], c["K"])
        return dict(A=_randn(gen, *a, cplx=c["cplx"]), B=_randn(gen, *b, cplx=c["cplx"]))
    if k in ("gemspm", "gespmm"):
        sop, dop = ("opB", "opA") if k == "gemspm" else ("opA", "opB")
        if c["pattern"] == "blocks":
            pat = _lattice_pattern(c)
            S = _lattice_csc(c["norb"], pat,
                             _hermitian_blocks(gen, pat, c["norb"], lambda r: torch.exp(-r), lambda R: R, c["cplx"]))
            r, s = S.dim1, S.dim2
        else:
            r, s = (c["K"], c["N"]) if k == "gemspm" else (c["M"], c["K"])
            shape = (r, s) if c[sop] == "n" else (s, r)
            S = _scatter_csc(gen, *shape, c["fill"], c["cplx"])
        M, N, K = (c["M"], s, r) if k == "gemspm" else (r, c["N"], s)
        d = (M, K) if k == "gemspm" else (K, N)
        return dict(S=S, X=_randn(gen, *(d if c[dop] == "n" else d[::-1]), cplx=c["cplx"]), M=M, N=N, K=K)
    if k == "add":
        a = (c["rows"], c["cols"]) if c["op"] == "n" else (c["cols"], c["rows"])
        return dict(A=_randn(gen, *a, cplx=c["cplx"]), B=_randn(gen, c["rows"], c["cols"], cplx=c["cplx"]))
    if k == "grad":
        H, S = _lattice_HS(gen, c)
        return dict(H=H, S=S, C=_coefficients(gen, H.dim1, _atom_count(c) * c["nocc"]))
    if k == "adjoint":
        m, n = c["m"], c["n"]
        Lf = torch.eye(m, dtype=_dtype(c["cplx"]), device=_DEV)
        Lf = Lf + (0.1 / math.sqrt(m)) * _randn(gen, m, m, cplx=c["cplx"]).tril()
        return dict(S=Lf @ Lf.mH, C=_coefficients(gen, m, n, c["cplx"]),
                    V=[_scatter_csc(gen, m, m, c["fill"], c["cplx"], hermitian=True, scale=0.1)
                       for _ in range(c["nv"])])
    if c["problem"] == "dense":
        H, S, Lf, Q, lam = _dense_HS(gen, c["m"], c["n"], c["cplx"])
        return dict(H=H, S=S, Lf=Lf, Q=Q, lam=lam, m=c["m"], n=c["n"])
    H, S = _lattice_HS(gen, c)
    return dict(H=H, S=S, m=H.dim1, n=_atom_count(c) * c["nocc"])


def prepare(case, seed):
    """Registered matrices and result buffers, as a program holds them between calls."""
    G.set_log(None)
    c, x = case, _inputs(case, seed)
    k = c["kind"]
    s = {"case": c}
    zeros = lambda r, q, cplx: _Dense(torch.zeros(r, q, dtype=_dtype(cplx), device=_DEV))  # noqa: E731
    if k == "mm":
        s.update(A=_Dense(x["A"]), B=_Dense(x["B"]), C=zeros(c["M"], c["N"], c["cplx"]))
    elif k in ("gemspm", "gespmm"):
        s.update(S=G.Matrix.from_csc(x["S"]), X=_Dense(x["X"]), C=zeros(x["M"], x["N"], c["cplx"]),
                 dims=(x["M"], x["N"], x["K"]))
    elif k == "add":
        s.update(A=_Dense(x["A"]), B=_Dense(x["B"]), C=zeros(c["rows"], c["cols"], c["cplx"]))
    elif k == "grad":
        n, m = x["C"].shape
        s.update(H=G.Matrix.from_csc(x["H"]), S=G.Matrix.from_csc(x["S"]), C=_Dense(x["C"]), G=zeros(n, m, False))
    elif k == "adjoint":
        s.update(S=_Dense(x["S"]), C=_Dense(x["C"]), V=[G.Matrix.from_csc(v) for v in x["V"]])
    else:
        cplx = bool(c.get("cplx"))
        reg = G.Matrix.from_csc if c["problem"] == "lattice" else _Dense
        s.update(H=reg(x["H"]), S=reg(x["S"]), m=x["m"], n=x["n"], C=zeros(x["n"], x["m"], cplx),
                 D=zeros(x["m"], x["m"], cplx))
    torch.cuda.synchronize()
    return s


# -------------------------------------------------------------------------------------- the call
def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "mm":
        G.mm_multiply(s["A"].h, c["opA"], s["B"].h, c["opB"], s["C"].h)
        return s["C"].t
    if k == "gemspm":
        G.psp_gemspm(*s["dims"], s["X"].h, c["opA"], s["S"], c["opB"], s["C"].h)
        return s["C"].t
    if k == "gespmm":
        G.psp_gespmm(*s["dims"], s["S"], c["opA"], s["X"].h, c["opB"], s["C"].h)
        return s["C"].t
    if k == "add":
        G.m_add(s["B"].h, "n", s["C"].h, 1.0, 0.0)
        G.m_add(s["A"].h, c["op"], s["C"].h, 0.75, 0.5)
        t = complex(G.mm_trace(s["B"].h, s["C"].h))
        return {"C": s["C"].t, "trace": np.array([t.real, t.imag])}
    if k == "grad":
        omega = G.functional_grad(s["C"].t.shape[1], s["C"].t.shape[0], s["H"], s["S"], s["C"].h, s["G"].h)
        return {"G": s["G"].t, "omega": np.array(omega)}
    if k == "adjoint":
        return G.energy_adjoint(s["C"].t.shape[1], s["C"].t.shape[0], s["S"].h, s["C"].h, s["V"])
    H, S = (s["H"].h, s["S"].h) if c["problem"] == "dense" else (s["H"], s["S"])
    e, _ = G.omm(s["m"], s["n"], H, S, True, s["D"].h, False, 0.0, s["C"].h, False, flavour=c.get("flavour", 0),
                 dealloc=True, m_operation=c["label"])
    return {"e": np.array(e), "C": s["C"].t, "D": s["D"].t}


# ------------------------------------------------------------------------------ the work of a pass
def _block_nnz(c):
    return _atom_count(c) * len(_shell()) * c["norb"] ** 2


def work(case):
    c, k = case, case["kind"]
    z = 4 if c.get("cplx") else 1  # flops of a complex product over a real one's
    w = 16 if c.get("cplx") else 8  # bytes of an element
    if k == "mm":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": w * (M * K + K * N + M * N), "flops": 2 * z * M * N * K}
    if k in ("gemspm", "gespmm"):
        if c["pattern"] == "blocks":
            r = q = _atom_count(c) * c["norb"]
            nnz = _block_nnz(c)
        else:
            r, q = (c["K"], c["N"]) if k == "gemspm" else (c["M"], c["K"])
            nnz = int(c["fill"] * r * q)
        d = c["M"] if k == "gemspm" else c["N"]
        return {"bytes": nnz * (w + 4) + 4 * (q + 1) + w * d * (r + q), "flops": 2 * z * nnz * d}
    if k == "add":
        e = c["rows"] * c["cols"]
        return {"bytes": 3 * w * e, "flops": 6 * z * e}
    if k == "grad":
        m, n, nnz = _atom_count(c) * c["norb"], _atom_count(c) * c["nocc"], _block_nnz(c)
        return {"bytes": 2 * nnz * 12 + 8 * (m + 1) + 16 * n * m, "flops": 4 * nnz * n + 8 * n * n * m}
    if k == "adjoint":
        m, n = c["m"], c["n"]
        nnz = c["nv"] * c["fill"] * m * m
        return {"bytes": nnz * (w + 4) + w * (m * m + n * m), "flops": z * (2 * n * m * m + 4 * n * n * m + 2 * nnz * n)}
    if c["problem"] == "dense":
        m, n = c["m"], c["n"]
        op, opb = 2 * m * m * n, w * m * m
    else:
        m, n = _atom_count(c) * c["norb"], _atom_count(c) * c["nocc"]
        nnz = _block_nnz(c)
        op, opb = 2 * nnz * n, 12 * nnz
    return {"bytes": 2 * opb + w * (n * m + m * m), "flops": z * (_STEPS * (2 * op + 12 * n * n * m) + 2 * n * m * m)}


# ------------------------------------------------------------------------- the results in 64 bits
def _dense_of(S):
    cols = torch.repeat_interleave(torch.arange(S.dim2, device=_DEV),
                                   torch.from_numpy(np.diff(S.colptr).astype(np.int64)).to(_DEV))
    out = torch.zeros(S.dim1, S.dim2, dtype=_dtype(np.iscomplexobj(S.val)), device=_DEV)
    out[torch.from_numpy(S.rowind.astype(np.int64)).to(_DEV), cols] = torch.from_numpy(S.val).to(_DEV)
    return out


def exact(case, seed):
    c, x = case, _inputs(case, seed)
    k = c["kind"]
    if k == "mm":
        return _op(x["A"], c["opA"]) @ _op(x["B"], c["opB"])
    if k == "gemspm":
        return _op(x["X"], c["opA"]) @ _op(_dense_of(x["S"]), c["opB"])
    if k == "gespmm":
        return _op(_dense_of(x["S"]), c["opA"]) @ _op(x["X"], c["opB"])
    if k == "add":
        C = 0.75 * _op(x["A"], c["op"]) + 0.5 * x["B"]
        t = complex((x["B"].conj() * C).sum())
        return {"C": C, "trace": np.array([t.real, t.imag])}
    if k == "grad":
        HC, SC = x["C"] @ _dense_of(x["H"]), x["C"] @ _dense_of(x["S"])
        HW, SW = HC @ x["C"].t(), SC @ x["C"].t()
        omega = 2.0 * HW.diagonal().sum() - (HW * SW).sum()
        return {"G": 4.0 * HC - 2.0 * SW @ HC - 2.0 * HW @ SC, "omega": np.array(float(omega))}
    if k == "adjoint":
        C = x["C"]
        SW = C @ x["S"] @ C.mH
        D = C.mH @ (2.0 * C - SW @ C)
        return np.array([float((D.conj() * _dense_of(v)).sum().real) for v in x["V"]])
    if c["problem"] == "dense":  # the spectrum is constructed
        n = x["n"]
        U = torch.linalg.solve_triangular(x["Lf"].mH, x["Q"][:, :n], upper=True)
        return {"e": np.array(float(x["lam"][:n].sum())), "C": None, "D": U @ U.mH}
    if x["m"] > 4000:  # the eigensolver takes too long
        return None
    H, S = _dense_of(x["H"]), _dense_of(x["S"])
    Lf = torch.linalg.cholesky(S)
    A = torch.linalg.solve_triangular(Lf, H, upper=False)
    A = torch.linalg.solve_triangular(Lf, A.mH, upper=False)
    lam, Q = torch.linalg.eigh(0.5 * (A + A.mH))
    U = torch.linalg.solve_triangular(Lf.mH, Q[:, :x["n"]], upper=True)
    return {"e": np.array(float(lam[:x["n"]].sum())), "C": None, "D": U @ U.mH}
