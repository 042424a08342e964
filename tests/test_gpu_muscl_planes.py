"""The plane-by-plane 3D MUSCL-Hancock update at the orders the limiter-kernel
tests do not reach (4 and 7: other plane sizes, other remainders of the block),
with the check and the bound of test_gpu_limiter_kernels (1e-12 relative
max-norm); for lists of any length, which the kernel-level call gives a block per
cell; and on limiting meshes with more FV-active cells than the device holds
blocks, where a block takes several."""
import numpy as np
import pytest

import pyoracle
import test_gpu_limiter as lim
import test_gpu_limiter_kernels as lk
from test_gpu_limiter_kernels import eb  # noqa: F401  (fixture)

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_muscl_2d_edges_in_two_rounds(eb):  # noqa: F811
    """2D order 7, where a block has fewer threads than a patch has edges"""
    lk.test_musclhancock_update_vs_oracle(eb, 2, 7, 19)


@pytest.mark.parametrize("order,n", [(4, 5), (7, 2)])
def test_muscl_planes_vs_oracle(eb, order, n):  # noqa: F811
    lk.test_musclhancock_update_vs_oracle(eb, 3, order, n)


def test_many_cells_equal_single_calls(eb):  # noqa: F811
    """a long list gives each cell what a call of its own gives, bit for bit"""
    rng = np.random.default_rng(3)
    order, n = 3, 1200
    lim = lk.states(rng, (n, (2 * order + 5) ** 3))
    s, dx, dt = eb.Solver(3, order), [0.05, 0.04, 0.045], lk.dev(np.array([2e-4]))
    scratch = torch.empty(s.fv_musclhancock_scratch_bytes(n) // 8, dtype=torch.float64, device="cuda")
    got, old = lk.dev(lim), lk.dev(np.zeros_like(lim))
    s.fv_musclhancock_update(got, old, None, dt, dx, n, None, scratch, scratch.numel() * 8)
    assert np.array_equal(lk.host(old), lim)
    for c in (0, 599, n - 1):
        one, prev = lk.dev(lim[c:c + 1]), lk.dev(np.zeros_like(lim[:1]))
        s.fv_musclhancock_update(one, prev, None, dt, dx, 1, None, scratch, scratch.numel() * 8)
        assert np.array_equal(lk.host(one)[0], lk.host(got)[c])


def test_blocks_take_several_cells(eb):  # noqa: F811
    """3D order 7 (one block an SM): a rough state under a maximum principle without
    slack makes every cell FV-active, so that blocks walk their patches one after
    the other; first in the recomputation, then in the update"""
    order, cells = 7, (6, 6, 6)
    rng = np.random.default_rng(11)
    n = int(np.prod(cells))
    luh = np.zeros((n, 8 ** 3, 5))
    luh[..., 0] = 1.0 + 0.01 * rng.random(luh.shape[:2])
    luh[..., 1:4] = 0.01 * (rng.random(luh.shape[:2] + (3,)) - 0.5)
    luh[..., 4] = 2.5 + 0.01 * rng.random(luh.shape[:2])
    g = eb.LimitingMesh(eb.Solver(3, order), cells, [0.0] * 3, [1.0] * 3, 0, relax=0.0, scale=0.0)
    o = pyoracle.LimitingMesh(3, order, cells, [1.0] * 3, 0, relax=0.0, scale=0.0, nthreads=8)
    for m in (g, o):
        m.set_solution(luh)
        m.init(0.0)
    for k in range(2):
        g.step(1)
        o.step(1)
        status = lim.compare(g, o, 3, order, "step %d" % (k + 1))
        assert np.sum(status >= 2) > torch.cuda.get_device_properties(0).multi_processor_count
    assert o.state()["irregular_steps"] >= 1
