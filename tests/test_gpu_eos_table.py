"""Tabulated EOS on the GPU (mdg_eos_table.cu) against the reference's own zone update
(the committed fixture of eos/burrows/eos_stuff.c:768-902 on the synthetic table at the
reference's table sizes) and against the oracle's restatement on a small table with inputs
inside and outside its range.

Bar: 1e-11 relative per value.  The kernel keeps the reference's operation order; its
log10, exp and pow are CUDA's, whose last-place differences from the host's are amplified
by the interpolation (1/d(log rho) ~ 20 on the reference grid) and by T = 10^(log T)
(ln 10)."""
import os

import numpy as np
import pytest

from medusa_b200 import eos_table as ET
from oracle import pyoracle
from tests._cases import record

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
TOL = 1.0e-11


def _rel(a, b):
    return float(np.max(np.abs(a - b) / np.maximum(np.abs(b), 1e-300)))


def test_gpu_eos_matches_reference_fixture():
    g = ET.REFERENCE_GRID
    f = np.load(os.path.join(HERE, "golden", "eos_table_ref.npz"))
    with ET.EosTable(ET.synthetic_table(g), g) as t:
        temp, press, cs, ent, gam1 = t.given_rex(f["rho"], f["u"], f["ye"], f["temp_guess"])
    got = np.stack([press, cs, temp, ent, gam1], axis=1)
    err = _rel(got, f["out"])
    record("eos_table_reference_fixture", rel_err=err, bit_identical=float(np.mean(got == f["out"])))
    assert err <= TOL


def test_gpu_eos_small_table_and_clamped_inputs_match_oracle():
    g = ET.EosGrid(nrec=12, ny=7, nr=20, nt=30, r1=2.0, r2=12.0, t1=-1.5, t2=1.5, y1=0.05, y2=0.5,
                   const_hack=0.25)
    tab = ET.synthetic_table(g)
    rho, u, ye, tg = ET.synthetic_zones(g, 3000, seed=3, table=tab)
    # outside the table: densities and Ye beyond both ends, guesses far off
    rho = np.concatenate([rho, [10.0 ** 1.0, 10.0 ** 13.5, 10.0 ** 7.0, 10.0 ** 7.0]])
    u = np.concatenate([u, [u[0], u[1], u[2], u[3]]])
    ye = np.concatenate([ye, [0.3, 0.3, 0.01, 0.7]])
    tg = np.concatenate([tg, [1.0e3, 1.0e-5, 0.0, 1.0]])
    ref = pyoracle.eos_given_rex(tab, pyoracle.EosGrid(g.nrec, g.ny, g.nr, g.nt, g.r1, g.r2, g.t1, g.t2, g.y1, g.y2,
                                                        g.const_hack), rho, u, ye, tg)
    with ET.EosTable(tab, g) as t:
        temp, press, cs, ent, gam1 = t.given_rex(rho, u, ye, tg)
    got = np.stack([press, cs, temp, ent, gam1], axis=1)
    err = _rel(got, ref)
    record("eos_table_small_oracle", rel_err=err)
    assert err <= TOL


def test_gpu_eos_device_path_equals_host_path():
    import torch
    g = ET.EosGrid(nrec=12, ny=9, nr=40, nt=50)
    tab = ET.synthetic_table(g)
    rho, u, ye, tg = ET.synthetic_zones(g, 20000, seed=8, table=tab)
    with ET.EosTable(tab, g) as t:
        host = t.given_rex(rho, u, ye, tg)
        dev = [torch.tensor(a, dtype=torch.float64, device="cuda:0") for a in (rho, u, ye, tg)]
        outs = [torch.empty(rho.size, dtype=torch.float64, device="cuda:0") for _ in range(4)]
        t.given_rex_device(rho.size, *[x.data_ptr() for x in dev], *[o.data_ptr() for o in outs],
                           stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    assert np.array_equal(dev[3].cpu().numpy(), host[0])
    for k in range(4):
        assert np.array_equal(outs[k].cpu().numpy(), host[k + 1])


def test_gpu_eos_results_do_not_depend_on_the_guess():
    """Guesses in the right row, one and two rows off either way and at both ends of the table
    bracket the same rows: the same bits."""
    g = ET.EosGrid(nrec=12, ny=9, nr=40, nt=50)
    tab = ET.synthetic_table(g)
    rho, u, ye, tg = ET.synthetic_zones(g, 4000, seed=5, table=tab)
    row = 10.0 ** ((g.t2 - g.t1) / (g.nt - 1))
    with ET.EosTable(tab, g) as t:
        want = t.given_rex(rho, u, ye, tg)
        for guess in [want[0] * row ** k for k in (-2, -1, 0, 1, 2)] + [np.full_like(tg, 10.0 ** x) for x in (g.t1, g.t2)]:
            got = t.given_rex(rho, u, ye, guess)
            assert all(np.array_equal(a, b) for a, b in zip(got, want))
