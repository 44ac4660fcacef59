"""The projector of a batch: more coefficients than one pass of 64 (twelve
clusters) and more chunks of dual rows in a cluster than one pass of 32 (216
subdomains in one), every load case against its solve alone.

Bound: the two forms sum in different orders and stop by the same rule at
eps 1e-10, so the stop may move by a step and u by about 1e-10 relative; the
bars are 2 iterations and 1e-8, the repository's displacement bar.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [3, 17])
@pytest.mark.parametrize("clusters,subs,elems", [((4, 3, 1), (2, 1, 1), (3, 2, 3)), ((1, 1, 1), (6, 6, 6), (4, 4, 4))])
def test_projector_passes(clusters, subs, elems, nrhs):
    import hfls_b200 as hb

    spec = hb.mesh_spec(clusters=clusters, subs=subs, elems=elems, jitter=0.1, seed=5, body_force=(0.0, 0.1, -1.0))
    f = hb.traction(spec, seed=2, n_rhs=nrhs, scale=1e-2)
    s = hb.Solver({"typeBc": "cor", "eps_iter": "1e-10", "max_iter": "1000"})
    s.set_mesh(hb.generate_mesh(spec))
    s.setup()
    u, st = s.solve(f)
    its = list(st.iterations[:nrhs])
    for j in range(0, nrhs, 8):
        u1, st1 = s.solve(f[j:j + 1])
        assert abs(st1.iterations[0] - its[j]) <= 2
        assert np.linalg.norm(u[j] - u1[0]) < 1e-8 * np.linalg.norm(u1[0])
    s.close()
