"""Work lists of the sweeps at the sizes where they can go wrong: the rows per 2-D tile
follow the grid size (tile_rows_2d, mdg_sweep2d.cu), and the dendritic sweeps pack rows of 1 to 256 phi zones
into CTAs and cut their runs by the grid size, so the results must not depend on where the
cuts fall.  Bars as in test_gpu_parity.py: <= 1e-12 per step; run lengths bit for bit."""
import numpy as np
import pytest

from medusa_b200 import problems as P
from medusa_b200.solver import PREC_FP64, PREC_MIXED, Solver
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


# 2-D rows of one phi zone (a last CTA with idle lanes), small 3-D rows several to a CTA, rows
# of 128 phi zones (cut segments) on a grid whose runs the size rule leaves at 1, 8 and more
@pytest.mark.parametrize("dims", [(71, 64, 1), (33, 16, 32), (60, 64, 128), (220, 64, 128)])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_dendritic_work_lists_do_not_change_the_results(dims, prec):
    n1, n2, n3 = dims
    pb = P.sedov_2d_spherical(n1, n2, noise=0.01) if n3 == 1 else P.sedov_3d(n1, n2, n3, noise=0.01)
    out = []
    for run in (1, 3, 64):
        with Solver(pb, precision=prec) as s:
            s.set_launch_config(run_length=run)
            s.step(2)
            s.synchronize()
            out.append(s.update_cpu(0))
    assert np.all(np.isfinite(out[0]))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
