"""The tensor-memory predictor (variants 0 and 8 of the Euler solvers) where
cells of one block, or of one warp, need different numbers of sweeps: constant
states (one sweep) beside smooth ones, a cell whose state is not a number (all
sweeps, and none of its neighbours' results may change), one cell alone, blocks
that are not full, a permuted list, counts on either side of the line between
the blocks for few cells and the others (296). Sweep counts equal to the oracle's, arrays
to 1e-12 of their largest entry (test_gpu_aderdg's FP64 bound)."""
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


@pytest.mark.parametrize("variant", [0, 8])
@pytest.mark.parametrize("n", [1, 7, 296, 331])
@pytest.mark.parametrize("dim,order", [(2, 3), (2, 4), (2, 5), (2, 7), (3, 3), (3, 4), (3, 5), (3, 7)])
def test_mixed_sweep_counts_vs_oracle(eb, dim, order, n, variant):
    rng = np.random.default_rng(100 * dim + 10 * order + n)
    b = order + 1
    P, F = b ** dim, b ** (dim - 1)
    u = np.zeros((n, P, 5))
    u[..., 0], u[..., 4] = 1.2, 2.6
    for c in range(0, n, 3):  # cells 1, 2, 4, 5, ... stay constant
        u[c, :, 0] += 0.2 * rng.random(P)
        u[c, :, 1:4] += 0.3 * (rng.random((P, 3)) - 0.5)
    bad = 5 if n > 5 else -1
    if bad >= 0:
        u[bad, P // 2, 4] = np.nan
    lst = rng.permutation(n).astype(np.int32)
    dx, dt = [0.05, 0.04, 0.03][:dim], 4e-4
    out = [torch.zeros(n, 2 * dim * F * 5, device="cuda", dtype=torch.float64) for _ in range(2)]
    du = torch.zeros(n, P * 5, device="cuda", dtype=torch.float64)
    it = torch.zeros(n, device="cuda", dtype=torch.int32)
    s = eb.Solver(dim, order, eb.PDE_EULER)
    s.variant = variant
    s.space_time_predictor(torch.as_tensor(u).cuda(), *out, du, torch.tensor([dt], device="cuda", dtype=torch.float64),
                           dx, n, iterations=it, cell_list=torch.as_tensor(lst).cuda())
    torch.cuda.synchronize()
    qb, fb, du, it = (t.cpu().numpy() for t in (*out, du, it))
    k = pyoracle.Kernels(dim, order, pde=0)
    for c in range(n) if n < 20 else [0, 1, 2, 3, 4, 5, 6, 7, n // 2, n - 3, n - 2, n - 1]:
        if c == bad:
            assert np.isnan(du[c]).any()
            continue
        o = k.predictor(u[c], dx, dt)
        assert it[c] == o["iterations"]
        # volume term and fluxes of a constant state cancel: their scale is the flux's
        scale = max(np.max(np.abs(o["lFhbnd"])), 1.0) / min(dx)
        assert np.max(np.abs(qb[c] - o["lQhbnd"])) <= 1e-12 * np.max(np.abs(o["lQhbnd"]))
        assert np.max(np.abs(fb[c] - o["lFhbnd"])) <= 1e-12 * np.max(np.abs(o["lFhbnd"]))
        assert np.max(np.abs(du[c] - o["lduh"])) <= 1e-12 * max(np.max(np.abs(o["lduh"])), scale)


@pytest.mark.parametrize("pde,twin", [(0, 8), (2, 1)])
def test_autotune_times_one_kernel_once(eb, pde, twin):
    """variants 0 and 8 of the Euler predictor are one kernel, 0 and 1 of the linear one"""
    for _ in range(3):
        s = eb.Solver(2, 3, pde)
        chosen, ms = s.autotune(64)
        assert ms[twin] == ms[0] > 0 and chosen != twin and s.variant == chosen
