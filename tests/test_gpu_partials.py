"""The SYMV's partial sums: few units per row block (one subdomain pair of 5^3
elements) and more than one pass of 128 of them (two plates whose common face
has 5 292 DOFs, 166 tile rows: the first row block is in some 140 units), the
explicit S_i blocks against L_bb of the same factor.

Bound: both come from one factorisation of order N <= 10 584; the sums differ
by N rounding errors at most, 2.2e-16 N = 2.4e-12 of the operator's norm, on a
random vector; ten times that and the elimination's own constant: 1e-10.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elems", [(5, 5, 5), (1, 41, 41)])
def test_explicit_and_implicit_preconditioner(elems):
    import hfls_b200 as hb

    m = hb.generate_mesh(hb.mesh_spec(subs=(2, 1, 1), elems=elems, jitter=0.1, seed=9))
    out = {}
    for pre in ("Dirichlet_explicit", "Dirichlet_implicit"):
        s = hb.Solver({"typeBc": "cor", "preconditioner": pre})
        s.set_mesh(m)
        s.setup()
        w = np.random.default_rng(3).standard_normal((1, s.n_lambda()))
        out[pre] = s.preconditioning(w)[0]
        s.close()
    a, b = out.values()
    assert np.linalg.norm(a - b) < 1e-10 * np.linalg.norm(a)
