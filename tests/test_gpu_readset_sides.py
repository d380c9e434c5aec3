"""Read-set check (test_gpu_readset.py) of the FP32 kernel's other copy widths:
sides that are odd (single words) and 2 mod 4 (pairs), isothermal and Euler, both
FP32 precisions.  A mesh of odd side has a zone at the origin, where the model's
Keplerian speed has no bound: the gas rotates rigidly inside a core, and the Euler
gas, coarse as it is, has a pressure floor."""
import numpy as np
import pytest

import test_gpu_readset as readset

pytestmark = pytest.mark.gpu

CASES = {"%s_%s_%dx%d" % (hydro, precision, nb, bs): (hydro, nb, bs, precision, None, rows)
         for hydro in ("iso", "euler") for precision in ("fp32_comp", "fp32_state64")
         for nb, bs, rows in ((5, 25, 0), (5, 25, 9), (5, 50, 17))}


def test_poisoned_build_reproduces_the_states(tmp_path, monkeypatch):
    monkeypatch.setattr(readset, "CASES", CASES)
    before = "    cons = b2.initial_state("
    assert readset.RUNNER.count(before) == 1
    monkeypatch.setattr(readset, "RUNNER", readset.RUNNER.replace(
        before, "    model = dataclasses.replace(model, core_radius=1.0)\n"
                "    if hyd == 'euler':\n        hydro = dataclasses.replace(hydro, pressure_floor=1e-6)\n" + before))
    readset.test_poisoned_build_reproduces_the_states(tmp_path)
    assert len(list((tmp_path / "p").iterdir())) == len(CASES)
    for f in (tmp_path / "p").iterdir():
        assert np.isfinite(np.load(f)).all()
