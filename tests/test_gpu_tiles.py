"""Work lists of the sweeps at the sizes where they can go wrong: the rows per 2-D tile
follow the grid size (tile_rows_2d, mdg_sweep2d.cu), and the dendritic sweeps pack rows of 1 to 256 phi zones
into CTAs and cut their runs by the grid size, so the results must not depend on where the
cuts fall.  Bars as in test_gpu_parity.py: <= 1e-12 per step; run lengths bit for bit."""
import numpy as np
import pytest

from medusa_b200 import problems as P
from medusa_b200.solver import PREC_FP64, PREC_MIXED, MdgError, Solver
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


# The mixed sweep on the same edges, against the plain FP64 oracle: FP32 face states and star-state
# increments carry 6e-8 of rho v^2 + p (mdg_mixed.cuh), a few of them a zone and stage, and the blast's
# declined faces are solved again in FP64 from the tables.
@pytest.mark.parametrize("n1,n2", [(5, 4), (33, 127), (64, 126), (67, 129), (130, 253), (515, 260), (1030, 300)])
@pytest.mark.parametrize("kind", ["kh", "blast"])
def test_2d_tile_edges_mixed(kind, n1, n2):
    pb = P.kelvin_helmholtz(n1, n2) if kind == "kh" else P.blast_2d(n1, n2, bc=P.REFLECT)
    steps = 2
    with Solver(pb, precision=PREC_MIXED) as s:
        s.step(steps)
        s.synchronize()
        got = s.update_cpu(0)
    o = pyoracle.Oracle(pb)
    o.advance(steps)
    ref, _ = o.state()
    assert np.all(np.isfinite(got))
    assert field_rel_err(got[:, :2], ref[:, :2]) <= 1.0e-6 * steps
    vscale = max(np.abs(ref[:, 2:4]).max(), np.sqrt(pb.gam * (pb.gam - 1.0) * ref[:, 1] / ref[:, 0]).max())
    assert np.abs(got[:, 2:5] - ref[:, 2:5]).max() <= 1.0e-6 * steps * vscale


# 2-D rows of one phi zone (a last CTA with idle lanes), small 3-D rows several to a CTA, rows
# of 128 phi zones (cut segments)
@pytest.mark.parametrize("dims", [(71, 64, 1), (33, 16, 32), (60, 64, 128)])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_dendritic_work_lists_do_not_change_the_results(dims, prec):
    n1, n2, n3 = dims
    pb = P.sedov_2d_spherical(n1, n2, noise=0.01) if n3 == 1 else P.sedov_3d(n1, n2, n3, noise=0.01)
    out = {}
    for run, small in ((1, 1), (1, 0), (3, 1), (16, 0), (64, 1), (64, 0)):
        with Solver(pb, precision=prec) as s:
            s.set_run_shape(run, small)
            assert s.run_shape() == (run, 7 * small)
            s.step(2)
            s.synchronize()
            out[run, small] = s.update_cpu(0)
    assert np.all(np.isfinite(out[1, 1]))
    for run, small in out:   # (the mixed kernels' two variants contract differently)
        assert np.array_equal(out[run, small], out[1, small if prec == PREC_MIXED else 1])
    assert field_rel_err(out[1, 0], out[1, 1]) <= 1.0e-6


# the lengths and kernels that the size rules give, the largest grid's those of full-size ones,
# against one-face runs by the kernels that the reference's fixtures (all small grids) are run with
@pytest.mark.parametrize("dims,run,small", [((71, 64, 1), 1, 7), ((60, 64, 128), 2, 0), ((220, 64, 128), 8, 0),
                                            ((400, 64, 128), 16, 0)])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_dendritic_size_rules_give_the_same_bits(dims, run, small, prec):
    n1, n2, n3 = dims
    pb = P.sedov_2d_spherical(n1, n2, noise=0.01) if n3 == 1 else P.sedov_3d(n1, n2, n3, noise=0.01)
    out = []
    with Solver(pb, precision=prec) as s:
        assert s.run_shape() == (run, small)
        for shape in ((0, -1), (1, -1 if prec == PREC_MIXED else 1)):
            s.set_run_shape(*shape)
            assert shape[1] == 1 or s.run_shape()[1] == small
            s.upload(0, pb.ic)
            s.step(2)
            out.append(s.update_cpu(0))
    assert np.all(np.isfinite(out[0]))
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_dendritic_autotune_tries_lengths_as_they_are(prec):
    """On a mid-size grid the tuned run length may lie above the size rule's; the state stays."""
    pb = P.sedov_3d(60, 64, 128, noise=0.01)
    with Solver(pb, precision=prec) as s:
        cfg, ms = s.autotune(trial_steps=2)
        by_size, used = 2, s.run_shape()[0]
        assert ms > 0 and (used == cfg["run_length"] or (cfg["run_length"] == 16 and used == by_size))
        s.step(2)
        got = s.update_cpu(0)
        s.set_launch_config(run_length=3)       # by the size rule again
        assert s.run_shape()[0] == 3
    with Solver(pb, precision=prec) as s:
        s.step(2)
        assert np.array_equal(s.update_cpu(0), got)
        with pytest.raises(MdgError):
            s.set_run_shape(65)
        with pytest.raises(MdgError):
            s.set_run_shape(4, 2)
    with Solver(P.sod(64)) as s:
        with pytest.raises(MdgError):
            s.set_run_shape(4)
