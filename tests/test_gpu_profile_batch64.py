"""htf_profile reports the iteration of one load case after any FP64 solve,
also when all its load cases were solved together, and changes no later solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_profile_after_load_cases_solved_together():
    import hfls_b200 as hb

    spec = hb.mesh_spec(subs=(2, 2, 2), elems=(4, 3, 4), jitter=0.1, seed=5, E=1.0, body_force=(0.0, 0.1, -1.0))
    f = hb.traction(spec, seed=2, n_rhs=4, scale=1e-2)

    def solver():
        s = hb.Solver({"typeBc": "cor", "eps_iter": "1e-10", "max_iter": "1000"})
        s.set_mesh(hb.generate_mesh(spec))
        s.setup()
        return s

    s = solver()
    assert s.profile(3).iteration_ms == 0.0          # nothing solved yet
    four, _ = s.solve(f)
    p = s.profile(3)
    assert p.iteration_ms > 0.0 and p.kernels_per_iteration > 0
    again, _ = s.solve(f)
    one, _ = s.solve(f[:1])
    assert s.profile(3).kernels_per_iteration == p.kernels_per_iteration
    s.close()
    t = solver()
    one_new, _ = t.solve(f[:1])
    four_new, _ = t.solve(f)
    assert np.array_equal(four, again) and np.array_equal(four, four_new) and np.array_equal(one, one_new)
    t.close()
