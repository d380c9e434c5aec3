"""Tracers of the FP32 paths where their double-float arithmetic has edges: on
cell centres and faces, at zero and next to it, at and next to the domain's
edge (crossing it and not), on meshes of even, odd and non-binary spacing."""
import numpy as np
import pytest

import binary2d as b2
from helpers import make_case
from oracle import binding

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32_comp", "fp32_state64"])
@pytest.mark.parametrize("nb,bs,R", [(2, 32, 8.0), (3, 25, 8.0), (2, 31, 7.3)])
def test_tracers_on_edges(precision, nb, bs, R):
    """One RK2 step.  A tracer moves by dt v, |dt v| <= cfl dx.  Velocities,
    weights, dt and the products each carry a few FP32 roundings, as does the
    state between the stages: 64 of them bound the difference from the
    oracle's FP64 step."""
    import dataclasses
    mesh, hydro, physics, model = b2.presets.iso_disk(nb, bs, seed=97)
    mesh = dataclasses.replace(mesh, domain_radius=R)
    physics = dataclasses.replace(physics, buffer_rate=10.0)
    cons, cfg = make_case(mesh, hydro, physics, model)
    N = nb * bs
    dx = 2.0 * R / N
    line = np.concatenate([
        -R + dx * np.arange(N), -R + dx * (np.arange(N) + 0.5),          # faces, centres
        [0.0, -0.0, 1e-300, -1e-300, 1e-30, 2.0 ** -70, -(2.0 ** -71), 1.0, -1.0, 1.0 / 3.0],
        [-R, np.nextafter(-R, 0), np.nextafter(R, 0), R - 1e-9, -R + 1e-9, R - 0.25 * dx, -R + 0.25 * dx],
    ])
    line = line[(line >= -R) & (line < R)]
    rng = np.random.default_rng(5)
    xy = np.stack([np.concatenate([line, rng.permutation(line)]), np.concatenate([rng.permutation(line), line])], axis=1)
    ref = binding.OracleState(cfg, cons)
    ref.set_tracers(xy)
    ref.advance(1)
    with b2.Runtime([b2.Run(mesh, hydro, physics)], precision=precision) as rt:
        rt.upload(0, cons)
        rt.set_tracers(0, xy)
        rt.advance(1)
        got = rt.tracers(0)
    assert np.all((got >= -R) & (got < R))
    d = got - ref.tracers
    d -= 2.0 * R * np.round(d / (2.0 * R))
    assert np.abs(ref.tracers - xy).max() > 0
    assert np.abs(d).max() <= 64 * 2.0 ** -24 * physics.cfl * dx
