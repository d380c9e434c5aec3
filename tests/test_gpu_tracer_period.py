"""FP32 tracers that cross the domain's edge within a step of which the half-width
is no FP32 number: the average with the base is taken on the image a whole period
away, not an FP32 rounding of it."""
import dataclasses

import numpy as np
import pytest

import binary2d as b2
from helpers import make_case
from oracle import binding

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32_comp", "fp32_state64"])
@pytest.mark.parametrize("rk", ["RK2", "RK3"])
@pytest.mark.parametrize("R", [8.1, 12.3])
def test_crossing(precision, rk, R):
    mesh, hydro, physics, model = b2.presets.iso_disk(4, 64, seed=97)
    mesh = dataclasses.replace(mesh, domain_radius=R)
    physics = dataclasses.replace(physics, buffer_rate=10.0, rk_order=rk)
    cons, cfg = make_case(mesh, hydro, physics, model)
    dx = 2.0 * R / 256
    off = np.array([1e-6, 1e-5, 1e-4, 1e-3, 3e-3])
    edge = np.concatenate([R - off, -R + off])
    along = np.linspace(-0.9 * R, 0.9 * R, 40)
    e, a = (g.reshape(-1) for g in np.meshgrid(edge, along))
    xy = np.concatenate([np.stack([e, a], 1), np.stack([a, e], 1), np.stack([e, np.roll(e, 3)], 1)])
    ref = binding.OracleState(cfg, cons)
    ref.set_tracers(xy)
    ref.advance(1)
    with b2.Runtime([b2.Run(mesh, hydro, physics)], precision=precision) as rt:
        rt.upload(0, cons)
        rt.set_tracers(0, xy)
        rt.advance(1)
        got = rt.tracers(0)
    assert (np.abs(ref.tracers - xy) > R).sum() > 50            # they do cross
    d = got - ref.tracers
    d -= 2.0 * R * np.round(d / (2.0 * R))
    # as in test_gpu_tracer_edges.py: a few tens of FP32 roundings of a displacement of at most cfl dx
    assert np.abs(d).max() <= 64 * 2.0 ** -24 * physics.cfl * dx
