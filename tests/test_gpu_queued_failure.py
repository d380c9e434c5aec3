"""A failing advance with another one queued behind it leaves the context as it
was before the failing advance: state, time, ledger, orbital elements and tracers.
The slots of the advances alternate, so the queued one's output slots are those
that the failing one began from."""
import dataclasses

import numpy as np
import pytest

import binary2d as b2
from helpers import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32_state64", "fp32_comp"])
@pytest.mark.parametrize("rk", ["RK1", "RK2", "RK3"])
@pytest.mark.parametrize("fold", [1, 2])
@pytest.mark.parametrize("queued", [1, 2])
def test_queued_advances_leave_the_kept_state(precision, rk, fold, queued):
    mesh, hydro, physics, model = b2.presets.iso_disk(3, 32, seed=51)
    physics = dataclasses.replace(physics, rk_order=rk, sink_radius=0.3)
    cons, _ = make_case(mesh, hydro, physics, model)
    xy = np.random.default_rng(7).uniform(-7.0, 7.0, (500, 2))
    with b2.Runtime([b2.Run(mesh, hydro, physics)], precision=precision) as rt:
        rt.upload(0, cons)
        rt.set_tracers(0, xy)
        for _ in range(2):
            rt.advance(fold)
        bad = rt.download(0)[0]
        bad[2, 1, 5, 7, 0] = -1e-3
        rt.upload_conserved(0, bad)
        kept = (rt.download(0)[0], rt.ledger(0), rt.elements(0), rt.tracers(0)), rt.time(0)
        assert np.any(kept[0][1]) and np.any(kept[0][2])
        for _ in range(1 + queued):
            rt.advance_async(fold)
        with pytest.raises(b2.HydroError) as e:
            rt.synchronize()
        assert e.value.kind == "NegativeDensity" and e.value.block == (2, 1) and e.value.zone == (5, 7)
        got = (rt.download(0)[0], rt.ledger(0), rt.elements(0), rt.tracers(0)), rt.time(0)
        for a, b in zip(got[0], kept[0]):
            assert np.array_equal(a, b)
        assert got[1] == kept[1]
