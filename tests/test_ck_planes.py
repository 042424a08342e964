"""The plane table of the linear predictor (CKPlanes in csrc/linear.cuh) against the
bank model it comes from (csrc/gen_planes.py)."""
import os
import sys

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "exahype_b200", "csrc")
sys.path.insert(0, CSRC)
import gen_planes as gp  # noqa: E402

sys.path.pop(0)


def test_wavefronts_of_the_table():
    res = gp.table()
    assert len(res) == gp.PLANES == 30 and all(0 <= r < 16 for r in res)
    assert gp.per_level(gp.placed_at(res)) == 966
    assert gp.per_level(gp.in_a_row(), placed=False) == 1188
    # the planes hold a cell each and do not overlap
    at = gp.placed_at(res)
    assert all(b - a >= gp.P for a, b in zip(at, at[1:]))


def test_components_meet_nowhere():
    assert gp.components() == gp.table()[gp.ND:]
    at = gp.placed_at(gp.table())
    least = gp.B * -(-gp.P // 16)  # every store of 216 threads in 14 wavefronts
    assert all(gp.stores(at, rounds=(d,)) == least for d in range(3))
