"""Paired Cholesky steps (trailing updates with 64 and 128 panel columns) at
orders around the rule's bound and with odd numbers of steps in the interior
and in the b set, through the displacements of a solve.

Bound: as tests/test_gpu_ksolve.py: PCPG at eps 1e-11 leaves about 1e-10
relative against a direct solve of the whole mesh; the bar is 1e-8.  A wrong
or missing panel product would leave an error of the size of u.
"""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from oracle.htfeti_oracle import hex8_element

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [
    ([6, 5], [7], [6]),                 # about 1 000 DOFs each, around the bound
    ([8, 7], [8], [7]),                 # above it, both interiors long
    ([3, 11], [9], [8]),                # one subdomain below, one above
    ([9, 10], [2], [13]),               # thin: few interior rows, many b rows
])
def test_displacements_against_direct_solve(w):
    import hfls_b200 as hb

    spec = hb.mesh_spec(subs=(2, 1, 1), widths=w, jitter=0.1, seed=7, E=2.0, nu=0.3, body_force=(0.3, -0.2, -1.0))
    m = hb.generate_mesh(spec)
    s = hb.Solver({"typeBc": "cor", "eps_iter": "1e-11", "max_iter": "2000"})
    s.set_mesh(m)
    s.setup()
    u, _ = s.pcpg()
    n = 3 * m.n_nodes
    Ke, fe = hex8_element(m.coords[m.elems], m.sub_E[m.elem_sub], m.sub_nu[m.elem_sub], m.body_force)
    dof = np.concatenate([3 * m.elems + c for c in range(3)], axis=1)
    rows, cols = np.repeat(dof, 24, axis=1), np.tile(dof, (1, 24))
    K = sp.csr_matrix((Ke.reshape(len(Ke), -1).ravel(), (rows.ravel(), cols.ravel())), shape=(n, n))
    b = np.bincount(dof.ravel(), fe.ravel(), minlength=n)
    free = np.setdiff1d(np.arange(n), m.dirichlet)
    ref = np.zeros(n)
    ref[free] = spl.spsolve(K[free][:, free].tocsc(), b[free])
    assert np.linalg.norm(u[0] - ref) < 1e-8 * np.linalg.norm(ref)
    s.close()
