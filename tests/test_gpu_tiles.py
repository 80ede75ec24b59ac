"""Work lists of the sweeps at the sizes where they can go wrong: the rows per 2-D tile
follow the grid size (tile_rows_2d, mdg_sweep2d.cu), so the results must not depend on where
the tiles are cut.  Bars as in test_gpu_parity.py: <= 1e-12 per step."""
import numpy as np
import pytest

from medusa_b200 import problems as P
from medusa_b200.solver import Solver
from oracle import pyoracle
from tests._cases import field_rel_err, pointwise_rel_err

pytestmark = pytest.mark.gpu


# one-row tiles; a last tile of one row; columns at the 126- and 128-column edges; a size
# whose tiles are cut to a few rows; one that keeps the longest tiles of direction 1
@pytest.mark.parametrize("n1,n2", [(5, 4), (33, 127), (64, 126), (67, 129), (130, 253), (515, 260), (1030, 300)])
@pytest.mark.parametrize("kind", ["kh", "blast"])
def test_2d_tile_edges_match_the_oracle(kind, n1, n2):
    pb = P.kelvin_helmholtz(n1, n2) if kind == "kh" else P.blast_2d(n1, n2, bc=P.REFLECT)
    steps = 2
    with Solver(pb) as s:
        s.step(steps)
        s.synchronize()
        got = s.update_cpu(0)
    o = pyoracle.Oracle(pb)
    o.advance(steps)
    ref, _ = o.state()
    assert np.all(np.isfinite(got))
    assert field_rel_err(got, ref) <= 1.0e-12 * steps
    assert pointwise_rel_err(got, ref, pb) <= 1.0e-12 * steps
