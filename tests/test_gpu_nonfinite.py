"""Infinities and NaN in the FP64 stage: what a zone gets from them is what the
reference's formulas give, whatever its neighbours in the warp are.  One stage
(b2d_stage_noalloc, since an advance ends at the ledger's NaN) against the
oracle's: the same zones are NaN and the same are infinite, and away from the
planted zones the values are the parity tests'."""
import dataclasses

import numpy as np
import pytest

import binary2d as b2
from binary2d import _lib
from helpers import make_case
from oracle import binding
from test_zz_no_alloc import call, planes

pytestmark = pytest.mark.gpu


def supersonic(mesh, hydro):
    """Mach 50 along both axes, so that every face has an upwind side."""
    N = mesh.num_blocks * mesh.block_size
    k = np.arange(N)
    rho = (1.0 + 0.1 * np.sin(0.7 * k))[:, None] * (1.0 + 0.2 * np.cos(0.3 * k))[None, :]
    vx, vy = 5.0 + 0.1 * np.sin(k)[:, None], 5.0 + 0.1 * np.cos(k)[None, :]
    u = [rho, rho * vx, rho * vy]
    if b2.num_fields(hydro) == 4:
        u.append(0.5 * rho * (vx * vx + vy * vy) + 1e-2 * rho / (hydro.gamma_law_index - 1.0))
    nb, bs = mesh.num_blocks, mesh.block_size
    return np.stack(u).reshape(len(u), nb, bs, nb, bs).transpose(1, 3, 2, 4, 0).copy()


@pytest.mark.parametrize("flow", ["supersonic", "disk"])
@pytest.mark.parametrize("kind", ["iso", "euler"])
@pytest.mark.parametrize("sink", ["impartial", "torque_free"])
def test_one_stage(flow, kind, sink):
    torch = pytest.importorskip("torch")
    lib = _lib.load()
    mesh, hydro, physics, model = b2.presets.iso_disk(2, 48, seed=71)
    physics = dataclasses.replace(physics, sink_radius=0.3, sink_model=sink)
    if kind == "euler":
        hydro = b2.Euler(gamma_law_index=5.0 / 3.0, cooling_coefficient=0.0)
        model = b2.DiskModel(surface_density=1.0, mach_number=5.0, noise=1e-3, seed=5, core_radius=1.0)
    cons, cfg = make_case(mesh, hydro, physics, model)
    if flow == "supersonic":
        cons = supersonic(mesh, hydro)
    bg, nf = cons.copy(), cons.shape[-1]
    dev = torch.device("cuda:0")
    zeros = np.zeros((2, 2, 7, nf))
    # in the sub-tiles' interiors and at their corners, beside the binary and in the buffer
    spots = [(0, 0, 5, 9), (0, 1, 15, 16), (1, 0, 47, 0), (1, 1, 0, 0), (0, 0, 47, 40), (1, 1, 20, 47)]
    compared = 0
    for value in (np.nan, np.inf, -np.inf):
        for field in range(nf):
            if field in (0, 3) and value == -np.inf:
                continue            # a negative density or pressure is an error
            if kind == "euler" and flow == "disk" and field > 0 and np.isnan(value):
                continue            # the kernel's limiter passes over NaN, the oracle's is 0 there: in this flow
                                    # that decides whether a pressure two zones away comes out negative
            bad = cons.copy()
            hit = spots[field::2]
            for s in hit:
                bad[s + (field,)] = value
            want, led_want = np.empty_like(bad), np.empty_like(zeros)
            with np.errstate(invalid="ignore"):
                try:
                    binding.stage_rows(cfg, bad, want, bg, zeros, led_want, 0.0, 1e-3, 0, 2)
                except binding.OracleHydroError:
                    continue        # (an infinite momentum makes the pressure negative)
            a, g = torch.from_numpy(planes(bad)).to(dev), torch.from_numpy(planes(bg)).to(dev)
            out = torch.empty_like(a)
            z = torch.zeros(zeros.size, dtype=torch.float64, device=dev)
            led = torch.empty_like(z)
            torch.cuda.synchronize()
            call(lib, cfg, a, g, None, out, z, None, led, 0.0, 1e-3, 0.0)
            torch.cuda.synchronize()
            got, ref = out.cpu().numpy(), planes(want)
            assert np.array_equal(np.isnan(got), np.isnan(ref)), (value, field)
            assert np.array_equal(np.isinf(got), np.isinf(ref)), (value, field)
            wrong = np.argwhere(np.isnan(led.cpu().numpy().reshape(led_want.shape)) != np.isnan(led_want))
            assert len(wrong) == 0, (value, field, wrong[:4])
            fine = np.isfinite(ref)
            near = ~fine
            for axis in (1, 2):     # three zones around what is not finite: their slopes differ by the rule for NaN
                near = np.logical_or.reduce([np.roll(near, k, axis) for k in range(-3, 4)])
            far = ~near.any(axis=0)
            scale = np.abs(ref[:, far]).max(axis=1)
            assert (np.abs(got[:, far] - ref[:, far]).max(axis=1) <= 1e-12 * scale).all(), (value, field)
            compared += 1
    assert compared >= 3
