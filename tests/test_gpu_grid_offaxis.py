"""Rectangular screens beside the rays' axis, the field focused on a tile's corner.

There the mixed phase E of nearly every ray is the planner's bound, with one sign, and
nothing averages out of what the product leaves out of exp(iE).

Tolerance: the orders left out, a tenth of the requested 1e-4, and the coherent worst of
160 accumulation steps truncated at 2^-24 (6.4e-6).
"""
import numpy as np
import pytest

import cases
import xrt_rs
from test_gpu_grid import grid, grid_ctx  # noqa: F401

pytestmark = pytest.mark.gpu


# Offsets of the focus, distance [mm], energy; the screen is 512^2 points around the focus.
# 256, 128, .. 8 rows and columns of a tile all end there.
@pytest.mark.parametrize("fx,fy,dist,energy,half", [
    (5.9, 5.9, 1000.0, 10_000.0, 0.2), (-5.0, 4.0, 1000.0, 10_000.0, 0.2),
    (12.0, -3.0, 1500.0, 12_000.0, 0.2), (2.0, 2.0, 400.0, 9_000.0, 0.1),
    (40.0, 40.0, 4000.0, 8_000.0, 0.2), (3.0, 30.0, 2000.0, 20_000.0, 0.3)])
@pytest.mark.parametrize("polarizations", [1, 2])
def test_focus_on_a_tile_corner(grid_ctx, oracle, fx, fy, dist, energy, half, polarizations):
    rng = np.random.default_rng(3)
    n = 16384
    x, y = rng.uniform(-0.05, 0.05, n), rng.uniform(-0.05, 0.05, n)
    k = energy / 1973.2697177417986 * 1e7
    es = np.exp(-1j * k * np.sqrt((fx - x) ** 2 + (fy - y) ** 2 + dist ** 2))
    ep = 0.5 * es * (1.0 if polarizations == 1 else rng.choice([0.9, 1.1], n))
    rays = cases.rays_from(x, y, 0.0, es=es, ep=ep, energy=energy)
    v = np.linspace(-half, half, 512)
    pix = grid(fx + v, fy + v, dist, "xyz")
    out, st = xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=grid_ctx,
                                          return_stats=True)
    assert st["path"] == xrt_rs.XK_PATH_F32PR
    i, j = np.meshgrid(np.arange(236, 276), np.arange(236, 276), indexing="ij")
    idx = (i * 512 + j).ravel()
    sub = {c: np.ascontiguousarray(pix[c][idx]) for c in "xyz"}
    err = cases.rel_l2([o[idx] for o in out], oracle.kahan_ld(*cases.as_lists(rays, sub)))
    print(f"focus at ({fx}, {fy}, {dist}): {err:.2e} sweep {st['sweep']} tiles {st['n_tiles']}")
    assert err < 1e-5 + 6.4e-6
