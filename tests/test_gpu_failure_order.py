"""Several zones fail in one stage: the zone that is reported is the one that the
reference meets first (error_key, csrc/stage.cuh), whichever CTA runs first."""
import dataclasses

import numpy as np
import pytest

import binary2d as b2
from helpers import make_case
from oracle import binding

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32_state64", "fp32_comp"])
@pytest.mark.parametrize("where", [[(2, 3), (7, 3)], [(1, 1), (1, 7)], [(6, 6), (0, 0), (3, 3)]])
def test_the_first_failing_zone_is_reported(precision, where):
    """Zones in block rows and columns far apart on a mesh of many waves of
    CTAs.  The last block row and column are neighbours of the first, so that
    zones there come first although their CTAs run last."""
    mesh, hydro, physics, model = b2.presets.iso_disk(8, 128, seed=61)
    physics = dataclasses.replace(physics, rk_order="RK1")
    cons, cfg = make_case(mesh, hydro, physics, model)
    bad = cons.copy()
    for k, (i, j) in enumerate(where):
        bad[i, j, 100, 60 + k, 0] = -1e-3
    with pytest.raises(binding.OracleHydroError) as eo:
        binding.OracleState(cfg, bad, background=cons).advance(1)
    err = eo.value.err
    with b2.Runtime([b2.Run(mesh, hydro, physics)], precision=precision) as rt:
        if precision != "fp64":
            rt.set_tile(0, 1)
        rt.upload(0, bad, background=cons)
        for _ in range(5):
            with pytest.raises(b2.HydroError) as e:
                rt.advance(1)
            assert e.value.block == (err.block_i, err.block_j) and e.value.zone == (err.zone_i, err.zone_j)
