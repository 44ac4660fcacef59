"""htf_profile runs more iterations than max_iter (its state has no limit):
the residual history ends at its own end, and nothing beside it changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_timed_iterations_stay_inside_the_history():
    import hfls_b200 as hb

    spec = hb.mesh_spec(clusters=(2, 1, 1), subs=(2, 2, 1), elems=(3, 3, 3), jitter=0.1, seed=5, E=1.0,
                        body_force=(0.0, 0.1, -1.0))
    f = hb.traction(spec, seed=2, n_rhs=1, scale=1e-2)

    def solver(max_iter):
        s = hb.Solver({"typeBc": "cor", "eps_iter": "1e-10", "max_iter": str(max_iter)})
        s.set_mesh(hb.generate_mesh(spec))
        s.setup()
        return s

    s = solver(2)
    x = np.random.default_rng(0).standard_normal((1, s.n_lambda()))
    for _ in range(2):
        with pytest.raises(hb.HTFError) as e:
            s.solve(f)
        assert e.value.code == hb.HTF_ENOCONV
        h = s.residual_history(0)
        ops = [s.mult_Ff(x), s.projection(x), s.preconditioning(x)]
        assert len(h) == 3
        if _ == 0:
            first = h, ops
            s.profile(500)
    assert np.array_equal(h, first[0])
    assert all(np.array_equal(a, b) for a, b in zip(ops, first[1]))
    s.close()


def test_history_of_a_solve_that_reaches_max_iter():
    import hfls_b200 as hb

    spec = hb.mesh_spec(subs=(2, 2, 1), elems=(3, 3, 3), jitter=0.1, seed=5, E=1.0, body_force=(0.0, 0.1, -1.0))
    hist = []
    for max_iter in (5, 200):
        s = hb.Solver({"typeBc": "cor", "eps_iter": "1e-10", "max_iter": str(max_iter)})
        s.set_mesh(hb.generate_mesh(spec))
        s.setup()
        try:
            s.pcpg()
        except hb.HTFError as e:
            assert e.code == hb.HTF_ENOCONV
        hist.append(s.residual_history(0))
        s.close()
    assert len(hist[0]) == 6 and np.array_equal(hist[0], hist[1][:6])
