"""The FP64 stage kernel's sub-tiles (csrc/stage64.cuh): blocks of any size,
split evenly into sub-tiles of at most 16 x 32 (Euler: 12 x 32) zones, against
the oracle at the parity tests' 1e-12; and several sub-tiles per CTA, which
the allocation-free stage takes where one ledger piece each would not fit.

The cell spacing is no power of two for most of these meshes, so that the
quotients by it go through their residual step."""
import dataclasses

import numpy as np
import pytest

import binary2d as b2
from helpers import ledger_err, rel_err, run_pair
from test_zz_no_alloc import compare_with_advance

pytestmark = pytest.mark.gpu

TOL = 1e-12
COOLING = b2.ITEMS.index("cooling")
# one zone per block; narrower than a warp; just over a sub-tile; a ragged split; several of them
SHAPES = [(16, 1), (3, 5), (2, 33), (3, 50), (2, 100)]


def light(model):
    """Light gas: a coarse block's pull must not unbind the binary."""
    return dataclasses.replace(model, surface_density=1e-3)


@pytest.mark.parametrize("nb,bs", SHAPES)
@pytest.mark.parametrize("variant", ["plain", "alpha_rk3", "euler"])
def test_block_sizes(nb, bs, variant):
    mesh, hydro, physics, model = b2.presets.iso_disk(nb, bs, seed=81, q=0.4, e=0.3)
    hydro = b2.Isothermal(mach_number=10.0, density_floor=1e-8)   # 16 zones a side go negative without one
    if variant == "alpha_rk3":
        physics = dataclasses.replace(physics, viscosity=("alpha", 0.1), rk_order="RK3", lambda_multiplier=0.7,
                                      sink_model="torque_free", sink_radius=0.3)
    elif variant == "euler":
        hydro = b2.Euler(gamma_law_index=5.0 / 3.0, cooling_coefficient=1e-9, pressure_floor=1e-12)
        physics = dataclasses.replace(physics, cfl=0.1)
        model = b2.DiskModel(surface_density=1.0, mach_number=5.0, noise=1e-3, seed=5, core_radius=1.0, edge_width=1.0)
    r = run_pair(mesh, hydro, physics, light(model), fold=2, advances=2)
    assert np.all(np.isfinite(r["gpu"]))
    assert rel_err(r["gpu"], r["ref"]) <= TOL
    assert np.allclose(r["dt"], r["dt_ref"], rtol=TOL, atol=0)
    led, ref = r["led"].copy(), r["led_ref"].copy()
    # the cooling item is the difference of two nearly equal states, a round trip through the primitives: it
    # agrees to the rounding of the state, not of itself (it does so to the last bit only where the states do)
    cool = np.abs(led[:, :, COOLING] - ref[:, :, COOLING]).sum(axis=(0, 1))
    assert (cool <= TOL * np.abs(r["ref"]).sum(axis=(0, 1, 2, 3))).all()
    led[:, :, COOLING] = ref[:, :, COOLING] = 0.0
    assert ledger_err(led, ref) <= TOL


def test_several_sub_tiles_per_cta():
    """110 x 110 blocks of 33^2 zones: at one ledger piece per sub-tile (six a
    block) the pieces alone would need 12 MB of the 4 MB scratch."""
    mesh, hydro, physics, model = b2.presets.iso_disk(110, 33, seed=82)
    compare_with_advance(mesh, hydro, physics, model)
