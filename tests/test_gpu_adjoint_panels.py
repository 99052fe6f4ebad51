"""The energy adjoint on both sides of its rule (density panels or one dot product per nonzero) and at the
panels' edges, against the dense density in numpy."""
import numpy as np
import pytest

import ommgpu as G
from ommgpu import synth

pytestmark = pytest.mark.gpu


def _sparse(rng, m, nnz, cplx):
    cols = np.sort(rng.integers(0, m, nnz))
    colptr = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=m))]).astype(np.int32)
    rows = rng.integers(0, m, nnz).astype(np.int32)
    v = rng.standard_normal(nnz)
    return synth.CSCMatrix(m, m, colptr, rows, v + 1j * rng.standard_normal(nnz) if cplx else v)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n,nnz,nv", [(300, 40, 900, 3), (1000, 129, 900, 1), (1025, 130, 400000, 2),
                                        (1300, 257, 250000, 33)])
def test_adjoint_matches_dense_density(m, n, nnz, nv, cplx):
    rng = np.random.default_rng(m + n)
    C = rng.standard_normal((n, m)) + (1j * rng.standard_normal((n, m)) if cplx else 0)
    C = np.asfortranarray(C / np.sqrt(m))
    V = [_sparse(rng, m, nnz, cplx) for _ in range(nv)]
    got = G.energy_adjoint(m, n, None, G.Matrix.from_numpy(C), [G.Matrix.from_csc(v) for v in V])
    D = C.conj().T @ (2.0 * C - (C @ C.conj().T) @ C)
    aD = np.abs(C).T @ (2.0 * np.abs(C) + (np.abs(C) @ np.abs(C).T) @ np.abs(C))
    for k, v in enumerate(V):
        cols = np.repeat(np.arange(m), np.diff(v.colptr))
        ref = float(np.sum((np.conj(D[v.rowind, cols]) * v.val).real))
        # every element of D within (m + 2n) eps of its sum of magnitudes
        tol = 4 * (m + 2 * n) * np.finfo(float).eps * float(np.sum(aD[v.rowind, cols] * np.abs(v.val)))
        assert abs(got[k] - ref) <= tol, (k, got[k], ref, tol)
