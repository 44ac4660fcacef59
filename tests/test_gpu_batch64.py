"""Several FP64 load cases in one htf_solve: solved together (16 or 32 columns
at once, the last one or two alone), each with the result it has alone.

Bound: both stop at eps 1e-10 with the same rule; the two forms sum in
different orders, so the iterates differ by round-off amplified over the
iterations and the stop can move by a step, which moves u by the size of the
residual left, about 1e-10 relative (E contrast 10).  The bar is 1e-8, the
repository's displacement bar, and 2 iterations.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pre", ["Dirichlet_explicit", "lumped"])
@pytest.mark.parametrize("nrhs", [2, 3, 16, 17, 33])
def test_load_cases_together_and_alone(nrhs, pre):
    import hfls_b200 as hb

    spec = hb.mesh_spec(clusters=(2, 1, 1), subs=(2, 2, 1), widths=([3, 5, 2, 4], [4, 6], [3]), jitter=0.1, seed=5,
                        material=hb.HTF_MAT_LOGUNIFORM, E=1.0, E_hi=10.0, body_force=(0.0, 0.1, -1.0))
    m = hb.generate_mesh(spec)
    f = hb.traction(spec, seed=2, n_rhs=nrhs, scale=1e-2)
    s = hb.Solver({"typeBc": "cor", "eps_iter": "1e-10", "max_iter": "1000", "preconditioner": pre})
    s.set_mesh(m)
    s.setup()
    u, st = s.solve(f)
    its = list(st.iterations[:nrhs])
    hist = [s.residual_history(j) for j in range(nrhs)]
    for j in range(nrhs):
        u1, st1 = s.solve(f[j:j + 1])
        assert abs(st1.iterations[0] - its[j]) <= 2
        assert np.linalg.norm(u[j] - u1[0]) < 1e-8 * np.linalg.norm(u1[0])
        h1 = s.residual_history(0)
        assert len(hist[j]) == its[j] + 1 and hist[j][0] == 1.0 and hist[j][-1] < 1e-10 <= hist[j][-2]
        assert np.allclose(hist[j][:8], h1[:8], rtol=1e-6)
    s.close()


def test_failing_load_case_keeps_its_code():
    import hfls_b200 as hb

    spec = hb.mesh_spec(subs=(2, 2, 1), elems=(4, 3, 3), jitter=0.1, seed=5)
    s = hb.Solver({"typeBc": "cor", "eps_iter": "1e-10", "max_iter": "3"})
    s.set_mesh(hb.generate_mesh(spec))
    s.setup()
    with pytest.raises(hb.HTFError) as e:
        s.solve(hb.traction(spec, seed=2, n_rhs=5))
    assert e.value.code == hb.HTF_ENOCONV
    s.close()
