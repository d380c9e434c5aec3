"""The FP32 stage kernel copies rows by four columns, by two or by one, as the
sides of all runs of a context allow.  A run alone copies as wide as its own
side allows; beside a run whose side is even, or odd, it copies by two, or by
one: the states, steps and ledgers are the same bit for bit."""
import dataclasses

import numpy as np
import pytest

import binary2d as b2
from helpers import make_case

pytestmark = pytest.mark.gpu


def case(nb, bs, hydro):
    mesh, iso, physics, model = b2.presets.iso_disk(nb, bs, seed=87, q=0.4, e=0.3, domain_radius=4.0)
    physics = dataclasses.replace(physics, buffer_rate=10.0, cfl=0.2)
    if hydro == "iso":
        return mesh, b2.Isothermal(mach_number=10.0, density_floor=1e-8), physics, model
    physics = dataclasses.replace(physics, cfl=0.1, sink_radius=0.3, viscosity=("alpha", 0.1))
    return (mesh, b2.Euler(gamma_law_index=5.0 / 3.0, cooling_coefficient=1e-6, pressure_floor=1e-12), physics,
            b2.DiskModel(surface_density=1e-3, mach_number=5.0, noise=1e-3, seed=5, core_radius=1.0, edge_width=1.0))


def advance(runs, cons, precision):
    with b2.Runtime(runs, precision=precision) as rt:
        for k, c in enumerate(cons):
            rt.upload(k, c)
        dts = [rt.advance(3)[0] for _ in range(2)]
        return rt.download(0)[0], dts, rt.ledger(0)


# sides 60 (one strip), 68, 100 and 124 (a strip and 8, 40 and 64 columns)
@pytest.mark.parametrize("bs", [15, 17, 25, 31])
@pytest.mark.parametrize("hydro", ["iso", "euler"])
@pytest.mark.parametrize("precision", ["fp32_comp", "fp32_state64"])
def test_widths_agree(bs, hydro, precision):
    mesh, hy, physics, model = case(4, bs, hydro)
    run, cons = b2.Run(mesh, hy, physics), make_case(mesh, hy, physics, model)[0]
    want = advance([run], [cons], precision)
    assert np.all(np.isfinite(want[0]))
    for nb in (2, 3):
        m, h, p, md = case(nb, bs, hydro)
        got = advance([run, b2.Run(m, h, p)], [cons, make_case(m, h, p, md)[0]], precision)
        assert np.array_equal(got[0], want[0])
        assert got[1] == want[1]
        assert np.array_equal(got[2], want[2])
