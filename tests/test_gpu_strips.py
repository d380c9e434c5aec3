"""The FP32 stage kernel's strips (csrc/stagew.cuh): 60 columns a warp over
meshes and blocks of any size — odd sides (single-word copies), sides under a
strip and just over one, blocks that strips cut anywhere — in chunks from one
row up, on both FP32 precisions.  Against the oracle at the FP32 parity tests'
tolerances, and bit for bit between tilings."""
import dataclasses

import numpy as np
import pytest

import binary2d as b2
from helpers import ledger_err, make_case, rel_err, run_pair

pytestmark = pytest.mark.gpu

TOL, L1_TOL, LED_TOL, BUFFER_TOL = 2e-4, 1e-5, 1e-4, 5e-3   # as in test_gpu_paired.py
BUFFER, COOLING = b2.ITEMS.index("buffer"), b2.ITEMS.index("cooling")


def case(nb, bs, variant):
    # a half-width and a buffer rate at which meshes of 15 zones a side are still stable
    mesh, hydro, physics, model = b2.presets.iso_disk(nb, bs, seed=85, q=0.4, e=0.3, domain_radius=4.0)
    physics = dataclasses.replace(physics, buffer_rate=10.0, cfl=0.2)
    model = dataclasses.replace(model, surface_density=1e-3)   # a coarse block's pull must not unbind the binary
    hydro = b2.Isothermal(mach_number=10.0, density_floor=1e-8)
    if variant == "alpha_rk3":
        physics = dataclasses.replace(physics, viscosity=("alpha", 0.1), rk_order="RK3", lambda_multiplier=0.7,
                                      sink_model="torque_free", sink_radius=0.3)
    elif variant == "euler":
        hydro = b2.Euler(gamma_law_index=5.0 / 3.0, cooling_coefficient=1e-9, pressure_floor=1e-12)
        physics = dataclasses.replace(physics, cfl=0.1, sink_radius=0.3)
        model = b2.DiskModel(surface_density=1e-3, mach_number=5.0, noise=1e-3, seed=5, core_radius=1.0, edge_width=1.0)
    return mesh, hydro, physics, model


# odd side under a strip; one zone per block; a strip and one column; ragged blocks; odd side of three strips
SHAPES = [(3, 5), (16, 1), (1, 61), (3, 50), (5, 25), (2, 100)]


@pytest.mark.parametrize("nb,bs", SHAPES)
@pytest.mark.parametrize("variant", ["plain", "alpha_rk3", "euler"])
@pytest.mark.parametrize("precision", ["fp32_comp", "fp32_state64"])
def test_sizes(nb, bs, variant, precision):
    r = run_pair(*case(nb, bs, variant), fold=2, advances=2, precision=precision)
    assert np.all(np.isfinite(r["gpu"]))
    assert rel_err(r["gpu"], r["ref"]) <= TOL
    assert np.abs(r["gpu"][..., 0] - r["ref"][..., 0]).sum() <= L1_TOL * np.abs(r["ref"][..., 0]).sum()
    items = [k for k in range(7) if k not in (BUFFER, COOLING)]
    led, ref = r["led"][:, :, items], r["led_ref"][:, :, items]
    if nb % 2:
        # the block around the binary: its net pull is the difference of opposite pulls that are
        # three orders larger, so its FP32 rounding is no measure of the items
        led[nb // 2, nb // 2] = ref[nb // 2, nb // 2] = 0.0
    assert ledger_err(led, ref) <= LED_TOL
    assert r["it"] == r["it_ref"]


@pytest.mark.parametrize("nb,bs,heights,rows", [(3, 50, (1, 2, 5, 10, 50), (8, 17, 50)), (5, 25, (1, 5, 25), (9, 25)),
                                                (2, 64, (1, 2, 64), (8, 50))])
@pytest.mark.parametrize("variant", ["plain", "euler"])
def test_tilings_agree(nb, bs, heights, rows, variant):
    """Chunks of any height, block-aligned or not, give the same states bit for
    bit and the same ledgers to FP32 summation order."""
    mesh, hydro, physics, model = case(nb, bs, variant)
    cons = make_case(mesh, hydro, physics, model)[0]
    out = []
    for th, strip in [(h, 0) for h in heights] + [(heights[-1], r) for r in rows]:
        with b2.Runtime([b2.Run(mesh, hydro, physics)], precision="fp32_comp") as rt:
            rt.set_tile(0, th)
            rt.set_strip_rows(strip)
            rt.upload(0, cons)
            dts = [rt.advance(3)[0] for _ in range(2)]
            out.append((rt.download(0)[0], dts, rt.ledger(0)))
    for s, dts, led in out[1:]:
        assert np.array_equal(s, out[0][0])
        assert dts == out[0][1]
        assert ledger_err(led, out[0][2]) <= 1e-5


def test_autotuned_batch_matches_runs_alone():
    """Runs of different sides in one launch, tuned, equal the same runs alone."""
    cases = [case(nb, bs, "plain") for nb, bs in ((2, 50), (5, 50), (3, 50))]
    runs = [b2.Run(m, h, p) for m, h, p, _ in cases]
    cons = [make_case(*c)[0] for c in cases]
    with b2.Runtime(runs, precision="fp32_comp") as rt:
        for k, c in enumerate(cons):
            rt.upload(k, c)
        rt.autotune()
        for _ in range(2):
            rt.advance(3)
        batch = [rt.download(k)[0] for k in range(3)]
    for k, (run, c) in enumerate(zip(runs, cons)):
        with b2.Runtime([run], precision="fp32_comp") as rt:
            rt.upload(0, c)
            for _ in range(2):
                rt.advance(3)
            assert np.array_equal(rt.download(0)[0], batch[k])
