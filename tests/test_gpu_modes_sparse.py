"""The sparse eigensolve's cooperative kernels at sizes around their CTAs and
past what the chip holds at once, with none, one and two null vectors:
eigenvalues against the separable problem's, residuals and orthonormality."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(n, rng, dirichlet):
    """Symmetric graded second difference; with ``dirichlet`` no null vector."""
    w = rng.uniform(0.8, 1.2, n)
    g = 1.0 / (0.5 * (w[:-1] + w[1:]))
    L = np.diag(np.concatenate([g, [0.0]]) + np.concatenate([[0.0], g])) - np.diag(g, 1) - np.diag(g, -1)
    if dirichlet:
        L[0, 0] += 2.0 / w[0]
    r = 1.0 / np.sqrt(w)
    return (L * r[:, None]) * r[None, :], np.sqrt(w / w.sum())


@pytest.mark.parametrize("nu,nv,n_modes,null,copies", [
    (3, 2, 1, 1, 1),        # the block is every vector beside the null one
    (73, 7, 3, 1, 1),       # 511 rows: one short of a filter CTA
    (32, 16, 2, 0, 1),      # 512
    (27, 19, 16, 1, 1),     # 513, the most modes
    (21, 13, 2, 2, 2),      # two regions, each with its null vector
    (300, 230, 2, 1, 1),    # 69000 rows: more than the CTAs of one launch take at once
])
def test_lowest_modes_of_a_graded_plane(nu, nv, n_modes, null, copies):
    import scipy.sparse as sp

    from magnelio_b200.engine import sparse_eigs

    rng = np.random.default_rng(9)
    (A, za), (B, zb) = _chain(nu, rng, null == 0), _chain(nv, rng, False)
    L = sp.kron(sp.csr_matrix(A), sp.identity(nv)) + sp.kron(sp.identity(nu), sp.csr_matrix(B))
    z = np.kron(za, zb)
    want = np.sort(np.add.outer(np.linalg.eigvalsh(A), np.linalg.eigvalsh(B)).ravel())
    want = want[1:] if null else want
    if copies == 2:
        L = sp.block_diag([L, L])
        want = np.repeat(want, 2)
        Z = np.zeros((2, 2 * z.size))
        Z[0, : z.size] = Z[1, z.size:] = z
    else:
        Z = z[None] if null else None
    L = sp.csr_matrix(L)
    lam, vec, info = sparse_eigs(L, n_modes, Z)
    b = float(np.max(np.abs(L).sum(axis=1)))
    assert info["residual"] <= 1e-12
    assert np.max(np.abs(lam - want[:n_modes])) <= 1e-11 * b
    assert np.max(np.abs(vec.T @ vec - np.eye(n_modes))) <= 1e-12
    assert np.max(np.abs(L @ vec - vec * lam)) <= 1e-11 * b
    if Z is not None:
        assert np.max(np.abs(Z @ vec)) <= 1e-11
