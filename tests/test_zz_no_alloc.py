"""exa_fv_musclhancock_update_noalloc (no caller scratch, no device allocation):
two calls in a row, each fed the previous call's output. Its result agrees with
the oracle's on some of the cells (1e-12 relative max-norm, as in
test_gpu_limiter_kernels) and bit for bit with exa_fv_musclhancock_update, the
same kernel behind the call that asks for scratch, on all."""
import numpy as np
import pytest

import pyoracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

RTOL = 1e-12


@pytest.fixture(scope="module")
def eb():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import exahype_b200
    exahype_b200.load()
    return exahype_b200


def states(rng, shape):
    q = np.zeros(shape + (5,))
    q[..., 0] = 1.0 + 0.3 * rng.random(shape)
    q[..., 1:4] = 0.2 * (rng.random(shape + (3,)) - 0.5)
    q[..., 4] = 2.5 + 0.5 * rng.random(shape)
    return q


def rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.parametrize("dim,order,n", [(3, 3, 200), (3, 5, 60), (2, 5, 150), (3, 5, 200), (3, 3, 800), (2, 7, 400)])
def test_noalloc_two_calls_vs_oracle_and_caller_scratch(eb, dim, order, n):
    rng = np.random.default_rng(7 * dim + order)
    E = 2 * order + 5
    lim0 = torch.as_tensor(states(rng, (n, E ** dim))).cuda()
    dx = [0.05, 0.04, 0.045][:dim]
    dt = torch.tensor([2e-4], dtype=torch.float64, device="cuda")
    cells = torch.as_tensor(rng.permutation(n)[: (3 * n) // 4].astype(np.int32)).cuda()
    m = int(cells.numel())
    s, k = eb.Solver(dim, order), pyoracle.Kernels(dim, order)
    nb = s.fv_musclhancock_scratch_bytes(m)
    scratch = torch.empty(max(nb, 8) // 8, dtype=torch.float64, device="cuda")

    a_lim, a_old = lim0.clone(), torch.zeros_like(lim0)
    b_lim, b_old = lim0.clone(), torch.zeros_like(lim0)
    a_luh = torch.zeros((n, (order + 1) ** dim, 5), dtype=torch.float64, device="cuda")
    b_luh = torch.zeros_like(a_luh)
    listed = cells.cpu().numpy()
    for call in range(2):
        before = b_lim.cpu().numpy()
        s.fv_musclhancock_update(a_lim, a_old, a_luh, dt, dx, m, cells, scratch, nb)
        s.fv_musclhancock_update_noalloc(b_lim, b_old, b_luh, dt, dx, m, cells)
        torch.cuda.synchronize()
        assert torch.equal(a_lim, b_lim), "call %d: patches differ" % call
        assert torch.equal(a_old, b_old), "call %d: previous patches differ" % call
        assert torch.equal(a_luh, b_luh), "call %d: DG projections differ" % call
        after, luh = b_lim.cpu().numpy(), b_luh.cpu().numpy()
        for c in [listed[0], listed[m // 2], listed[m - 1]]:
            assert rel(after[c], k.musclhancock(before[c], dx, 2e-4).reshape(E ** dim, 5)) < RTOL
            assert rel(luh[c], k.project_dg(after[c]).reshape(-1, 5)) < RTOL
        rest = np.setdiff1d(np.arange(n), listed)
        assert np.array_equal(after[rest], before[rest])
    assert not torch.equal(a_lim, lim0)  # the patches did change
