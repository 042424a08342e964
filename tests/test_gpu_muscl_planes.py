"""The plane-by-plane 3D MUSCL-Hancock update at the orders the limiter-kernel
tests do not reach (4 and 7: other plane sizes, other remainders of the block)
and for one cell and more cells than the device holds blocks, with the check
and the bound of test_gpu_limiter_kernels (1e-12 relative max-norm)."""
import numpy as np
import pytest

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
