"""The limiter's status spreading (sweeps from one status buffer to the other,
the last two in one launch) at more helper layers than the default, which
take more sweeps, at periodic and walled domains where a neighbour's neighbour
is the cell itself or lies outside, in 2D and 3D: statuses equal to the
oracle's after every step, fields to 1e-11 (test_gpu_limiter's bound)."""
import numpy as np
import pytest

import pyoracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eb():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import exahype_b200
    exahype_b200.load()
    return exahype_b200


@pytest.mark.parametrize("dim,cells,bc,layers,steps", [
    (2, (13, 11), 0, 2, 6), (2, (9, 7), -1, 3, 5), (2, (12, 3), 0, 1, 6), (3, (7, 6, 5), 0, 2, 3)])
def test_statuses_vs_oracle(eb, dim, cells, bc, layers, steps):
    from exahype_b200 import problems
    u, fv, _ = problems.explosion(dim, 3, cells, seed=4)
    size = (1.0,) * dim
    g = eb.LimitingMesh(eb.Solver(dim, 3), cells, (0.0,) * dim, size, bc, helper_layers=layers)
    o = pyoracle.LimitingMesh(dim, 3, cells, size, bc, helper_layers=layers)
    for m in (g, o):
        m.set_solution(u)
        m.set_fv_initial(fv)
        m.init(0.0)
    for _ in range(steps):
        g.step(1)
        o.step(1)
        assert np.array_equal(g.status(), o.status())
    assert np.linalg.norm(g.get_solution() - o.get_solution()) <= 1e-11 * np.linalg.norm(o.get_solution())


def test_priority_between_steps(eb):
    """a new stream, and new side streams, between steps change no result"""
    from exahype_b200 import problems
    u, fv, _ = problems.explosion(2, 3, (12, 11), seed=4)
    out = []
    for levels in ((), (1, 3, 0)):
        m = eb.LimitingMesh(eb.Solver(2, 3), (12, 11), (0.0, 0.0), (1.0, 1.0), 0)
        m.set_solution(u)
        m.set_fv_initial(fv)
        m.init(0.0)
        for k in range(3):
            m.step(1)
            if levels:
                m.set_priority(levels[k])
            m.run_until(1.0, 2)
        out.append((m.get_solution(), m.status(), m.state()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1]) and out[0][2] == out[1][2]
