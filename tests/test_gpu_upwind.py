"""HLLE fluxes of the FP32 stage kernel where the flow is supersonic: the downwind
state drops out exactly (csrc/stagew.cuh, faces2).

Stripes of 8 columns whose densities differ by 1e6 cross the mesh at Mach 50 along
y.  A downwind weight of one rounding (1e-7) instead of 0 puts a tenth of a light
zone's flux into the face between a light zone and the heavy stripe downwind."""
import dataclasses

import numpy as np
import pytest

import binary2d as b2
from helpers import make_case
from oracle import binding

pytestmark = pytest.mark.gpu


def stripes(hydro_kind, sign):
    """One uniform row after another; the second sign is the mirror image in y of the first."""
    mesh, hydro, physics, model = b2.presets.iso_disk(2, 32, seed=3)
    physics = dataclasses.replace(physics, rk_order="RK1", viscosity=("constant_nu", 0.0), buffer_rate=0.0, sink_rate=0.0)
    N = 64
    rho = np.where((np.arange(N) // 8) % 2 == 0, 1.0, 1e-6) * (1.0 + 0.1 * np.sin(0.7 * np.arange(N)))
    vy = 5.0 * (1.0 + 0.01 * np.cos(1.3 * np.arange(N)))
    if sign < 0:
        rho, vy = rho[::-1], -vy[::-1]
    planes = np.zeros((3 if hydro_kind == "iso" else 4, N, N))
    planes[0], planes[2] = rho, rho * vy
    if hydro_kind == "euler":
        hydro = b2.Euler(gamma_law_index=5.0 / 3.0, cooling_coefficient=0.0)
        planes[3] = 0.5 * rho * vy * vy + 1e-2 * rho / (5.0 / 3.0 - 1.0)
    nf = planes.shape[0]
    cons = planes.reshape(nf, 2, 32, 2, 32).transpose(1, 3, 2, 4, 0).copy()
    return mesh, hydro, physics, cons


def to_planes(cons):
    nf = cons.shape[-1]
    return cons.transpose(4, 0, 2, 1, 3).reshape(nf, 64, 64)


@pytest.mark.parametrize("precision", ["fp32_comp", "fp32_state64"])
@pytest.mark.parametrize("kind", ["iso", "euler"])
def test_downwind_state_drops_out(kind, precision):
    got = []
    for sign in (1, -1):
        mesh, hydro, physics, cons = stripes(kind, sign)
        with b2.Runtime([b2.Run(mesh, hydro, physics)], precision=precision) as rt:
            rt.upload(0, cons)
            dt = rt.advance(1)[0]
            got.append((to_planes(rt.download(0)[0]), dt))
        ref = binding.OracleState(b2.to_c(mesh, hydro, physics), cons)
        ref.advance(1)
        # The density of a zone is u - (F_out - F_in) dt / dx, with F_out and F_in products of upwind
        # densities of this zone's or the upwind zone's size: a few tens of FP32 roundings of terms no larger
        # than the largest, which the largest Courant number of 0.4 keeps below 3 times the result.
        a, b = got[-1][0][0], to_planes(ref.cons)[0]
        assert np.abs(a / b - 1.0).max() <= 64 * 2.0 ** -24
    # the mirror image in y, bit for bit
    (a, da), (b, db) = got
    assert da == db
    b = b[:, :, ::-1].copy()
    b[2] *= -1.0
    assert np.array_equal(a, b)
