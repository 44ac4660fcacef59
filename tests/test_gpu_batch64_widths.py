"""Width of FP64 load cases solved together: it follows from the call alone.

A call of 3 to 16 load cases runs in 16 columns, a larger one in 32, whatever
calls came before, so a repeated call gives the same bits; where 32 columns do
not apply (here: (c + 6) 32 > 2048 for c Bc rows of a subdomain) 16 are used."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solver(spec, mesh=None):
    import hfls_b200 as hb

    s = hb.Solver({"typeBc": "cor", "eps_iter": "1e-10", "max_iter": "1000"})
    s.set_mesh(mesh if mesh is not None else hb.generate_mesh(spec))
    s.setup()
    return s


@pytest.mark.parametrize("small", [3, 8, 16])
def test_a_call_does_not_depend_on_the_calls_before(small):
    import hfls_b200 as hb

    spec = hb.mesh_spec(clusters=(2, 1, 1), subs=(2, 2, 1), widths=([3, 5, 2, 4], [4, 6], [3]), jitter=0.1, seed=5,
                        material=hb.HTF_MAT_LOGUNIFORM, E=1.0, E_hi=10.0, body_force=(0.0, 0.1, -1.0))
    f = hb.traction(spec, seed=2, n_rhs=20, scale=1e-2)
    s = solver(spec)
    u0, st0 = s.solve(f[:small])
    h0 = [s.residual_history(j) for j in range(small)]
    u20, _ = s.solve(f)
    u1, st1 = s.solve(f[:small])
    assert np.array_equal(u0, u1)
    assert list(st0.iterations[:small]) == list(st1.iterations[:small])
    assert all(np.array_equal(h0[j], s.residual_history(j)) for j in range(small))
    again, _ = s.solve(f)
    assert np.array_equal(u20, again)
    s.close()
    # and 20 first, on a new solver
    t = solver(spec)
    v20, _ = t.solve(f)
    v1, _ = t.solve(f[:small])
    assert np.array_equal(u20, v20) and np.array_equal(u0, v1)
    t.close()


def test_sixteen_columns_where_32_do_not_apply():
    import hfls_b200 as hb

    spec = hb.mesh_spec(subs=(2, 1, 1), elems=(4, 4, 4), jitter=0.1, seed=7, E=1.0, body_force=(0.0, 0.1, -1.0))
    m = hb.generate_mesh(spec)
    # 22 of the interface's 25 nodes are corners: 66 Bc rows, 72 columns of V
    face = np.flatnonzero(np.arange(m.n_nodes) % 9 == 4)
    assert len(face) == 25
    m.corner = (3 * face[:22, None] + np.arange(3)).ravel().astype(np.int32)
    f = hb.traction(spec, seed=2, n_rhs=20, scale=1e-2)
    s = solver(spec, m)
    u16, _ = s.solve(f[:16])
    u4, _ = s.solve(f[16:])
    s.close()
    t = solver(spec, m)
    u, st = t.solve(f)                               # 16 and 4
    assert np.array_equal(u[:16], u16) and np.array_equal(u[16:], u4)
    again, _ = t.solve(f[:16])
    assert np.array_equal(again, u16)
    one, st1 = t.solve(f[:1])
    assert abs(st1.iterations[0] - st.iterations[0]) <= 2
    assert np.linalg.norm(one[0] - u[0]) < 1e-8 * np.linalg.norm(one[0])
    t.close()
