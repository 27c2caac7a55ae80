"""Rectangular screens from a millimetre to a hundred metres behind the rays.

The product's first-order operands are f16 numbers; their sizes go with the
cube of the distance, so screens of micrometres close to an aperture and of
decimetres far from it test both ends of f16's range.

Tolerance: that of the product (160 accumulation steps truncated at 2^-24, the
first-order operands' 2^-11 of E, the 2^-22 split): 1e-5 of the field's norm.
"""
import numpy as np
import pytest

import cases
import xrt_rs
from test_gpu_grid import TOL, check, grid, grid_ctx  # noqa: F401

pytestmark = pytest.mark.gpu


def square_aperture(n, half, energy, dist, seed):
    """Uniform rays, half of them focused on the screen's centre."""
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(-half, half, n), rng.uniform(-half, half, n)
    k = energy / 1973.2697177417986 * 1e7
    phase = np.where(rng.random(n) < 0.5, -k * (x * x + y * y) / (2 * dist),
                     rng.uniform(0, 2 * np.pi, n))
    return cases.rays_from(x, y, 0.0, es=np.exp(1j * phase), ep=0.1 * np.exp(1j * phase),
                           energy=energy)


# energy [eV], distance, aperture half width, screen half width [mm]
@pytest.mark.parametrize("energy,dist,aperture,screen", [
    (10_000.0, 1.0, 0.01, 0.001), (10_000.0, 2.0, 0.02, 0.002), (30_000.0, 1.0, 0.006, 0.0006),
    (30_000.0, 5.0, 0.02, 0.002), (60_000.0, 5.0, 0.02, 0.001), (10_000.0, 5.0, 0.03, 0.004)])
def test_micrometre_screens(grid_ctx, oracle, energy, dist, aperture, screen):
    rays = square_aperture(6000, aperture, energy, dist, seed=int(dist))
    v = np.linspace(-screen, screen, 128)
    check(grid_ctx, oracle, rays, grid(v, 0.9 * v, dist, "xyz"))


@pytest.mark.parametrize("energy,dist,aperture,screen", [
    (100.0, 1e5, 100.0, 100.0), (100.0, 5e4, 60.0, 50.0), (200.0, 5e4, 50.0, 50.0),
    (500.0, 5e4, 20.0, 20.0), (1000.0, 1e5, 40.0, 30.0), (1000.0, 5e4, 20.0, 15.0)])
def test_soft_x_rays_at_tens_of_metres(grid_ctx, oracle, energy, dist, aperture, screen):
    rays = square_aperture(6000, aperture, energy, dist, seed=int(energy))
    v = np.linspace(-screen, screen, 128)
    check(grid_ctx, oracle, rays, grid(v, 0.9 * v, dist, "xyz"))


def test_product_is_the_same_in_every_length_unit(grid_ctx):
    """All lengths times 2^6 at 2^-6 of the energy: every phase and factor of the
    product is the same number, so is the field but for the 1 / length."""
    rays = square_aperture(5000, 0.3, 8192.0, 1500.0, seed=4)
    pix = grid(np.linspace(-0.4, 0.4, 96), np.linspace(-0.3, 0.3, 80), 1500.0, "xyz")
    run = lambda r, p: xrt_rs.diffraction_integral(*cases.as_lists(r, p), path="f32pr",
                                                   ctx=grid_ctx, return_stats=True)
    out, st = run(rays, pix)
    big = dict(rays, **{k: rays[k] * 64.0 for k in "xyz"}, energy=rays["energy"] / 64.0)
    out2, st2 = run(big, {k: v * 64.0 for k, v in pix.items()})
    assert st["sweep"] == st2["sweep"] == 3
    # i k / (4 pi) / |p - r|: 2^-6 in k and 2^-6 in 1 / length.
    assert cases.rel_l2([o * 4096.0 for o in out2], out) < 1e-9
