"""The FP64 column-group kernel at the edges of its tiles: rows around the 32, 64 and 128 row blocks,
group widths with and without zero cells, complex matrices as two value sets, transposed output
(psp_gespmm) and odd leading dimensions, against dense products in numpy."""
import numpy as np
import pytest

import ommgpu as G
from ommgpu import synth

pytestmark = pytest.mark.gpu


def _case(norb, cplx, seed):
    p = synth.lattice((5, 5, 5), seed=seed, norb=norb, nocc=1, compute_mu=False)
    H = p.H
    if cplx:
        rng = np.random.default_rng(seed)
        H = synth.CSCMatrix(H.dim1, H.dim2, H.colptr, H.rowind, H.val * np.exp(1j * rng.uniform(0, 6, H.nnz)))
    return H


def _rnd(rng, shape, cplx):
    a = rng.standard_normal(shape)
    return np.asfortranarray(a + 1j * rng.standard_normal(shape) if cplx else a)


def _op(a, op):
    return a if op == "n" else a.T if op == "t" else a.conj().T


def _check(got, ref, mag):
    # a sum of at most 33 * norb products in FP64, in any order: n eps sum|a||b|, with a margin of 4
    bound = 4 * (33 * 32 + 8) * np.finfo(float).eps * (mag + np.abs(ref))
    assert np.all(np.abs(got - ref) <= bound), float(np.max(np.abs(got - ref) / np.maximum(bound, 1e-300)))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("norb", [8, 13, 16, 24, 32])
@pytest.mark.parametrize("n", [1, 31, 33, 65, 129, 300])
def test_gemspm_rows_and_widths(norb, n, cplx):
    H = _case(norb, cplx, 50 + norb)
    rng = np.random.default_rng(n)
    m, Hd = H.dim1, H.to_dense()
    A, C0 = _rnd(rng, (n, m), cplx), _rnd(rng, (n, m), cplx)
    al, be = (0.7 - 0.2j, 0.3 + 0.1j) if cplx else (0.7, 0.3)
    C = G.Matrix.from_numpy(C0)
    G.psp_gemspm(n, m, m, G.Matrix.from_numpy(A), "n", G.Matrix.from_csc(H), "n", C, al, be)
    _check(C.numpy(), al * (A @ Hd) + be * C0, np.abs(A) @ np.abs(Hd) + np.abs(C0))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("opA", ["n", "t", "c"])
@pytest.mark.parametrize("opB", ["n", "t", "c"])
@pytest.mark.parametrize("norb,n", [(8, 65), (13, 33), (24, 130)])
def test_gespmm_ops_and_widths(norb, n, opA, opB, cplx):
    H = _case(norb, cplx, 70 + norb)
    rng = np.random.default_rng(n)
    m, Hd = H.dim1, H.to_dense()
    B = _rnd(rng, (m, n) if opB == "n" else (n, m), cplx)
    C0 = _rnd(rng, (m, n), cplx)
    al, be = (0.7 - 0.2j, 0.3 + 0.1j) if cplx else (0.7, 0.3)
    C = G.Matrix.from_numpy(C0)
    G.psp_gespmm(m, n, m, G.Matrix.from_csc(H), opA, G.Matrix.from_numpy(B), opB, C, al, be)
    a, b = _op(Hd, opA), _op(B, opB)
    _check(C.numpy(), al * (a @ b) + be * C0, np.abs(a) @ np.abs(b) + np.abs(C0))


@pytest.mark.parametrize("norb", [13, 24])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_gespmm_nonfinite_stays_in_its_rows(norb, bad):
    """A row of the dense operand that holds an Inf or NaN reaches the rows of the product whose sparse
    rows hold that column, and no others."""
    H = _case(norb, False, 90)
    rng = np.random.default_rng(4)
    m, n, k = H.dim1, 40, 77
    B = _rnd(rng, (m, n), False)
    B[k, 3] = bad
    C = G.Matrix.allocate(m, n)
    G.psp_gespmm(m, n, m, G.Matrix.from_csc(H), "n", G.Matrix.from_numpy(B), "n", C, 1.0, 0.0)
    got = C.numpy()
    touched = np.zeros((m, n), bool)
    touched[:, 3] = H.to_dense()[:, k] != 0.0
    assert np.array_equal(~np.isfinite(got), touched)


@pytest.mark.parametrize("opA", ["n", "t"])
@pytest.mark.parametrize("cplx", [False, True])
def test_gespmm_with_a_long_row_union(opA, cplx):
    """A filled CSC whose column groups span more rows than the group kernel's plan can hold (51,200): the
    product takes the gather kernel.  psp_gemspm, which has no other kernel for it, refuses it."""
    rng = np.random.default_rng(8)
    long, short, n = 52000, 40, 5
    v = rng.standard_normal((long, short)) + (1j * rng.standard_normal((long, short)) if cplx else 0)
    # 't': a long x short matrix; 'n': a short x long one, whose transpose is planned
    d = v if opA == "t" else v.T
    A = synth.CSCMatrix(d.shape[0], d.shape[1], (np.arange(d.shape[1] + 1) * d.shape[0]).astype(np.int32),
                        np.tile(np.arange(d.shape[0], dtype=np.int32), d.shape[1]), d.T.reshape(-1).copy())
    B, C0 = _rnd(rng, (long, n), cplx), _rnd(rng, (short, n), cplx)
    h, C = G.Matrix.from_csc(A), G.Matrix.from_numpy(C0)
    for _ in range(2):
        C.upload(C0)
        G.psp_gespmm(short, n, long, h, opA, G.Matrix.from_numpy(B), "n", C, 0.7, 0.3)
        bar = 4 * long * np.finfo(float).eps * (np.abs(v.T) @ np.abs(B) + np.abs(C0))
        assert np.all(np.abs(C.numpy() - (0.7 * (v.T @ B) + 0.3 * C0)) <= bar)
    wide = G.Matrix.from_numpy(_rnd(rng, (n, long), cplx))
    with pytest.raises(G.OmmError):
        G.psp_gemspm(n, short, long, wide, "n", h, "n" if opA == "t" else "t", G.Matrix.from_numpy(_rnd(rng, (n, short), cplx)))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("norb", [0, 13, 24])
def test_gespmm_beta_zero_multiplies(norb, cplx):
    """beta = 0 multiplies C: a NaN that C holds stays where it is, whatever kernel the pattern takes (column
    groups with and without zero cells, norb = 0: no groups)."""
    if norb:
        H = _case(norb, cplx, 90)
    else:
        rng = np.random.default_rng(1)
        d = np.where(rng.random((300, 300)) < 0.02, rng.standard_normal((300, 300)), 0.0) * (1j if cplx else 1.0)
        at = np.nonzero(d.T)
        colptr = np.concatenate([[0], np.cumsum(np.bincount(at[0], minlength=300))]).astype(np.int32)
        H = synth.CSCMatrix(300, 300, colptr, at[1].astype(np.int32), d.T[at])
    rng = np.random.default_rng(2)
    m, n = H.dim1, 33
    C0 = _rnd(rng, (m, n), cplx)
    C0[5, 7] = np.nan
    C = G.Matrix.from_numpy(C0)
    G.psp_gespmm(m, n, m, G.Matrix.from_csc(H), "n", G.Matrix.from_numpy(_rnd(rng, (m, n), cplx)), "n", C, 1.0, 0.0)
    held = np.zeros((m, n), bool)
    held[5, 7] = True
    assert np.array_equal(np.isnan(C.numpy()), held)


@pytest.mark.parametrize("shuffled", [False, True])
def test_gespmm_duplicates_do_not_hide_a_zero_cell(shuffled):
    """An atom-block matrix with one entry of a column given twice (the two add up) and another one missing:
    as many entries as cells, but an Inf of the dense operand at the missing entry's row does not reach that
    column's result."""
    H = _case(24, False, 33)
    rng = np.random.default_rng(33)
    j, m = 100, H.dim2
    lo, hi = int(H.colptr[j]), int(H.colptr[j + 1])
    rowind, val = H.rowind.copy(), H.val.copy()
    hole = int(rowind[lo + 30])
    rowind[lo + 30] = rowind[lo + 29]
    if shuffled:
        p = lo + rng.permutation(hi - lo)
        rowind[lo:hi], val[lo:hi] = rowind[p], val[p]
    A = synth.CSCMatrix(H.dim1, m, H.colptr, rowind, val)
    dense = np.zeros((H.dim1, m))
    np.add.at(dense, (rowind, np.repeat(np.arange(m), np.diff(H.colptr))), val)
    B = _rnd(rng, (H.dim1, 40), False)
    C = G.Matrix.allocate(m, 40)
    G.psp_gespmm(m, 40, H.dim1, G.Matrix.from_csc(A), "t", G.Matrix.from_numpy(B), "n", C, 1.0, 0.0)
    _check(C.numpy(), dense.T @ B, np.abs(dense).T @ np.abs(B))
    B[hole, 3] = np.inf
    C = G.Matrix.allocate(m, 40)
    G.psp_gespmm(m, 40, H.dim1, G.Matrix.from_csc(A), "t", G.Matrix.from_numpy(B), "n", C, 1.0, 0.0)
    touched = np.zeros((m, 40), bool)
    touched[:, 3] = dense[hole] != 0.0
    assert not touched[j, 3] and np.array_equal(~np.isfinite(C.numpy()), touched)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("identity", [False, True])
def test_solve_with_operators_without_groups(identity, cplx):
    """A small solve (its steps run as graphs) with CSC H and S of no column groups: the gather kernel's products
    inside the graph give the energy and the density of the same operators held dense."""
    m, n = 150, 30
    rng = np.random.default_rng(6)

    def hermitian(scale, diag):
        x = np.where(rng.random((m, m)) < 0.01, _rnd(rng, (m, m), cplx), 0.0) * scale
        x = x + x.conj().T
        np.fill_diagonal(x, diag)
        return np.asfortranarray(x)

    H = hermitian(0.03, np.where(np.arange(m) < n, -1.0, 1.0))
    S = None if identity else hermitian(0.01, 1.0)
    lbl = "gzden" if cplx else "gdden"
    got = []
    G.set_log(None)
    for sparse in (True, False):
        def reg(x):
            if x is None or not sparse:
                return x if x is None else G.Matrix.from_numpy(x)
            at = np.nonzero(x.T)
            colptr = np.concatenate([[0], np.cumsum(np.bincount(at[0], minlength=m))]).astype(np.int32)
            return G.Matrix.from_csc(synth.CSCMatrix(m, m, colptr, at[1].astype(np.int32), x.T[at]))

        C, D = G.Matrix.allocate(n, m, lbl), G.Matrix.allocate(m, m, lbl)
        e, rc = G.omm(m, n, reg(H), reg(S), True, D, False, 0.0, C, False, cg_tol=1e-12, dealloc=True)
        assert rc == 0
        got.append((e, D.numpy()))
    lam, U = np.linalg.eigh(H if S is None else np.linalg.solve(np.linalg.cholesky(S), np.linalg.solve(
        np.linalg.cholesky(S), H).conj().T))
    want = float(lam[:n].sum())
    for e, _ in got:  # the energies' relative steps fell to 1e-12: within 1e-9 of the eigenvalues' sum
        assert abs(e - want) <= 1e-9 * abs(want)
    assert np.abs(got[0][1] - got[1][1]).max() <= 1e-4  # the density's error is the energy's square root
