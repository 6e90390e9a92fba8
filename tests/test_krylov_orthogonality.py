"""The Gram-Schmidt of the device's restart cycles (csrc/topo_krylov.cuh): one classical pass, repeated
where less than kReorthogonalise of |w|^2 is left.  Restated here with the source's threshold on the
fluid's operator with a diagonal preconditioner, where some 15 % of |w|^2 are left at every step:
over a whole restart the basis has to stay orthogonal to roundings.

A vector that keeps the share t of |w|^2 is orthogonal to 1 / sqrt(t) roundings of a sum of n
products; 60 vectors and n = 1,000 give at most 60 sqrt(2) 1e-15 = 1e-13.
"""
import os
import re

import numpy as np
import scipy.sparse as sp

from tests.test_fluid_rows import _oracle

SOURCE = os.path.join(os.path.dirname(__file__), "..", "topomax_gb300", "csrc", "topo_krylov.cuh")
RESTART = 60


def test_a_restart_cycle_keeps_its_basis_orthogonal():
    threshold = float(re.search(r"kReorthogonalise = ([\d.]+);", open(SOURCE).read())[1])
    o = _oracle(10, 10)
    rng = np.random.default_rng(1)
    A = sp.csr_matrix(o.assemble(rng.uniform(0.0, 1.0, o.nv)))
    free = np.ones(o.n, bool)
    free[o.bc_dofs] = False
    A = A[free][:, free]
    nu = int(free[:o.nuv].sum())
    A = sp.vstack([A[:nu], -A[nu:]]).tocsr()  # symmetric form
    scale = np.concatenate([1.0 / A.diagonal()[:nu], 1.0 / o.vertex_weights])
    V = np.zeros((RESTART + 1, A.shape[0]))
    V[0] = rng.standard_normal(A.shape[0])
    V[0] /= np.linalg.norm(V[0])
    for j in range(RESTART):
        w = A @ (scale * V[j])
        for _ in range(2):
            before, h = w @ w, V[:j + 1] @ w
            w = w - V[:j + 1].T @ h
            if before - h @ h >= threshold * before:
                break
        V[j + 1] = w / np.linalg.norm(w)
    assert np.abs(V @ V.T - np.eye(RESTART + 1)).max() <= 1e-13
