"""The reconstruction that the FP64 sweeps run (para_recon_fast, mdg_recon.h) against the
reference's dividing form, on the host: equal bits wherever its guards accept, and the
guards decline rarely on the grids that the solvers build."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("recon") / "recon_forms")
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-std=c++17",
                           "-I", os.path.join(ROOT, "medusa_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                           os.path.join(HERE, "recon_forms.cpp"), "-o", out])
    return out


@pytest.mark.parametrize("seed", [1, 2])
def test_forms_agree_bit_for_bit(exe, seed):
    rows = [l.split() for l in subprocess.check_output([exe, str(seed), "200000"], text=True).splitlines()]
    assert len(rows) == 11
    for name, count, flat, declined, differ in rows:
        assert int(differ) == 0, name
        if name.endswith("e-110/0"):
            # volumes below the guarded range: every zone that is not flat is declined
            assert int(declined) > 0.9 * (int(count) - int(flat))
        else:
            assert int(declined) < 0.02 * int(count), name
