"""AMR transfers and the vertex projection at the shapes around the line where an
axis has more lines than a block has threads (3D order 7: 320 lines, one round;
the elastic state at order 5: 432, two) and at 2D order 7, with the checks and the bound of test_gpu_amr
(1e-12 of the largest value: the same sums in another order)."""
import pytest

import test_gpu_amr as amr
from test_gpu_amr import eb  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

ROUNDS = [(3, 7, 0), (3, 5, 2), (2, 7, 0)]  # (dim, N, pde)


@pytest.mark.parametrize("dim,N,pde", ROUNDS)
def test_transfers_in_rounds(eb, dim, N, pde):  # noqa: F811
    amr.test_volume_transfers_vs_oracle(eb, dim, N, pde)
    amr.test_face_transfers_vs_oracle(eb, dim, N, pde)
    amr.test_plot_vertices_vs_oracle(eb, dim, N, pde)
