"""Screens on which the mixed phase E of a whole tile is past first order: the product with
the second order, -E^2 / 2, on 256 x 256 tiles in stages of 16 rays.

Tolerance as in test_gpu_grid.py, 1e-5 of the field's norm: 160 accumulation steps
truncated at 2^-24, E^3 / 6 within a tenth of the requested 1e-4 at the worst corner, and
the operands' roundings, 3.5e-4 of E <= 0.03 at random over the pairs.
"""
import numpy as np
import pytest

import cases
import xrt_rs
from test_gpu_grid import check, grid, grid_ctx, permuted, run  # noqa: F401
from xrt_rs import synth

pytestmark = pytest.mark.gpu


# Rows and columns of a tile in use from 32 to 256 in either orientation, remainders of
# one and of all but one, ray blocks that neither segments nor splits divide.
@pytest.mark.parametrize("n_outer,n_inner,n,dist,energy", [
    (256, 256, 4000, 600.0, 12_000.0), (257, 255, 4001, 300.0, 20_000.0),
    (257, 255, 4001, 450.0, 9_000.0), (33, 300, 3017, 300.0, 9_000.0),
    (300, 33, 3017, 450.0, 9_000.0), (64, 64, 1025, 400.0, 12_000.0),
    (513, 129, 5555, 400.0, 12_000.0), (130, 97, 40_033, 600.0, 12_000.0),
    (255, 510, 33_333, 350.0, 12_000.0), (255, 510, 33_333, 600.0, 20_000.0),
    (385, 300, 4000, 300.0, 9_000.0)])
@pytest.mark.parametrize("columns", [1, 2])
def test_tiles_and_remainders(grid_ctx, oracle, n_outer, n_inner, n, dist, energy, columns):
    rays = synth.gaussian_aperture(n, 0.1, energy, 2e4, seed=n_inner)
    if columns == 2:
        rng = np.random.default_rng(n)
        rays.update(ep_re=rng.normal(0, 1, n), ep_im=rng.normal(0, 1, n))
    pix = grid(np.linspace(-0.5, 0.5, n_outer), np.linspace(-0.4, 0.4, n_inner), dist, "xyz")
    out, st = check(grid_ctx, oracle, rays, pix)
    assert st["one_polarization"] == (columns == 1)


@pytest.mark.parametrize("axes", ["yxz", "zxy", "yzx"])
def test_axis_orders(grid_ctx, oracle, axes):
    rays = synth.gaussian_aperture(3000, 0.1, 12_000.0, 2e4, seed=1)
    pix = grid(np.linspace(-0.5, 0.4, 150), np.linspace(-0.3, 0.4, 90), 500.0, axes)
    check(grid_ctx, oracle, permuted(rays, axes), pix)


def test_general_normals(grid_ctx, oracle):
    """The obliquity factor varies along a tile."""
    rays, _ = cases.random_case(6000, 1, seed=3, general_normals=True, energy=14_000.0)
    check(grid_ctx, oracle, rays, synth.grid_screen(120, 120, 0.5, 700.0))


# A focus on a tile's corner beside the rays' axis, where E is its bound for every ray
# (0.019 to 0.03): coherent, so without the operands' random roundings, 1e-5 + 6.4e-6.
@pytest.mark.parametrize("fx,fy,dist,energy,half", [
    (5.9, 5.9, 1000.0, 10_000.0, 0.2), (7.4, 7.4, 1000.0, 10_000.0, 0.2),
    (3.0, 30.0, 2000.0, 20_000.0, 0.3), (60.0, -60.0, 4000.0, 9_000.0, 0.25)])
def test_focus_on_a_tile_corner(grid_ctx, oracle, fx, fy, dist, energy, half):
    rng = np.random.default_rng(3)
    n = 16384
    x, y = rng.uniform(-0.05, 0.05, n), rng.uniform(-0.05, 0.05, n)
    k = energy / 1973.2697177417986 * 1e7
    es = np.exp(-1j * k * np.sqrt((fx - x) ** 2 + (fy - y) ** 2 + dist ** 2))
    rays = cases.rays_from(x, y, 0.0, es=es, ep=0.5 * es, energy=energy)
    v = np.linspace(-half, half, 512)
    pix = grid(fx + v, fy + v, dist, "xyz")
    out, st = run(grid_ctx, rays, pix)
    assert st["sweep"] == 3
    i, j = np.meshgrid(np.arange(236, 276), np.arange(236, 276), indexing="ij")
    idx = (i * 512 + j).ravel()
    sub = {c: np.ascontiguousarray(pix[c][idx]) for c in "xyz"}
    err = cases.rel_l2([o[idx] for o in out], oracle.kahan_ld(*cases.as_lists(rays, sub)))
    print(f"focus at ({fx}, {fy}, {dist}): {err:.2e} tiles {st['n_tiles']}")
    assert err < 1e-5 + 6.4e-6


def test_stalled_stage_times_out_and_context_recovers():
    rays = synth.gaussian_aperture(60_000, 0.1, 12_000.0, 2e4, seed=13)
    pix = synth.grid_screen(256, 256, 0.5, 900.0)
    ctx = xrt_rs.GpuContext.new(0)
    try:
        ref, st = run(ctx, rays, pix)
        assert st["sweep"] == 3
        ctx.set_option("wait_limit", 4096)
        ctx.set_option("inject_stall", 16)
        with pytest.raises(xrt_rs.XkError) as ei:
            run(ctx, rays, pix)
        assert ei.value.code == xrt_rs._lib.XK_ERR_TIMEOUT
        ctx.set_option("wait_limit", float(1 << 24))
        out, _ = run(ctx, rays, pix)
        assert all(np.array_equal(x, y) for x, y in zip(out, ref))
    finally:
        ctx.close()
