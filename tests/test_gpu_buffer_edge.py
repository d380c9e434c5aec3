"""A buffer of scale 0: full rate beyond the domain radius, none inside, as
tanh(+-inf) gives in the reference's formula (physics.rs:440-446)."""
import dataclasses

import numpy as np
import pytest

from helpers import rel_err, run_pair
from test_gpu_strips import BUFFER, L1_TOL, TOL, case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["plain", "euler"])
@pytest.mark.parametrize("precision", ["fp64", "fp32_comp", "fp32_state64"])
def test_sharp_edge(variant, precision):
    mesh, hydro, physics, model = case(4, 16, variant)
    # no zone centre is within rounding of the edge: r^2 = (a^2 + b^2) (dx / 2)^2 with a and b odd
    n = mesh.num_blocks * mesh.block_size
    x = (2 * np.arange(n) + 1 - n).astype(int)
    assert np.abs((x[:, None] ** 2 + x[None, :] ** 2) - n * n).min() >= 1
    physics = dataclasses.replace(physics, buffer_scale=0.0)
    r = run_pair(mesh, hydro, physics, model, fold=2, advances=2, precision=precision)
    assert np.isfinite(r["ref"]).all()
    assert np.isfinite(r["gpu"]).all() and np.isfinite(r["led"]).all()
    for led in (r["led_ref"], r["led"]):
        assert np.all(led[1:3, 1:3, BUFFER] == 0.0)      # the blocks inside the edge
        assert np.all(led[::3, ::3, BUFFER, 0] != 0.0)   # the corners
    assert rel_err(r["gpu"], r["ref"]) <= (1e-12 if precision == "fp64" else TOL)
    assert np.abs(r["gpu"][..., 0] - r["ref"][..., 0]).sum() <= L1_TOL * np.abs(r["ref"][..., 0]).sum()
