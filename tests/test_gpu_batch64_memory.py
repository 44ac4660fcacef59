"""FP64 load cases together take at most a quarter of the free device memory
for their vectors, as counted before anything is allocated; with less room
they are solved one at a time, and together again once there is room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def leave_free(free):
    """Blocks that leave about `free` bytes of device memory (to 4 MiB)."""
    import torch

    blocks = []
    for _ in range(4):
        over = torch.cuda.mem_get_info()[0] - int(free)
        if over < 4 << 20:
            break
        blocks.append(torch.empty(over // (2 << 20) * (2 << 20), dtype=torch.uint8, device="cuda"))
    got = torch.cuda.mem_get_info()[0]
    assert abs(got - free) < 6 << 20
    return blocks


def give_back(blocks):
    import torch

    blocks.clear()
    torch.cuda.empty_cache()


def test_a_quarter_of_the_free_memory_bounds_the_batch():
    import hfls_b200 as hb

    spec = hb.mesh_spec(clusters=(2, 2, 2), subs=(2, 2, 2), elems=(5, 5, 5), jitter=0.1, seed=5, E=1.0,
                        body_force=(0.0, 0.1, -1.0))
    f = hb.traction(spec, seed=2, n_rhs=4, scale=1e-2)

    def solver():
        s = hb.Solver({"typeBc": "cor", "eps_iter": "1e-10", "max_iter": "1000"})
        s.set_mesh(hb.generate_mesh(spec))
        s.setup()
        return s

    held = lambda s: s.profile(1).device_bytes
    s = solver()
    s.solve(f[:2])
    before = held(s)
    together, _ = s.solve(f)
    about = held(s) - before                         # the vectors and the loads of two more cases
    s.close()
    s = solver()
    s.solve(f[:1])
    blocks = leave_free(1.5 * about)
    alone, _ = s.solve(f)
    before = held(s)
    give_back(blocks)
    again, _ = s.solve(f)                            # there is room now
    size = held(s) - before
    assert size > 32 << 20 and np.array_equal(again, together)
    s.close()

    s = solver()
    s.solve(f[:1])
    blocks = leave_free(1.5 * about)
    s.solve(f)                                       # the loads of four cases are allocated
    give_back(blocks)
    before = held(s)
    blocks = leave_free(4 * 0.92 * size)             # the vectors would take a little over a quarter
    one, _ = s.solve(f)
    assert held(s) == before and np.array_equal(one, alone)
    give_back(blocks)
    blocks = leave_free(4 * 1.08 * size)
    four, _ = s.solve(f)
    assert held(s) == before + size and np.array_equal(four, together)
    give_back(blocks)
    assert np.allclose(alone, together, rtol=0, atol=1e-8 * np.abs(alone).max())
    s.close()
