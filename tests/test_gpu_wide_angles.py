"""Rays with depth seen at angles of tenths of a radian: cells that are as wide as the
length along the beam allows must not run through the whole depth.

Tolerance: the path's 1e-4 requested, of which the general kernel's worst fields use a
sixth (1.6e-5, test_gpu_precision.py).
"""
import numpy as np
import pytest

import cases
import xrt_rs

pytestmark = pytest.mark.gpu


def check(ctx, oracle, rays, pix, rng):
    out, st = xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=ctx,
                                          return_stats=True)
    assert st["path"] == xrt_rs.XK_PATH_F32PR
    idx = rng.integers(0, len(pix["x"]), 40)
    sub = {c: np.ascontiguousarray(pix[c][idx]) for c in "xyz"}
    err = cases.rel_l2([o[idx] for o in out], oracle.kahan_ld(*cases.as_lists(rays, sub)))
    print(f"{err:.2e}, {st['n_chunks']} chunks, sweep {st['sweep']}, {st['phase_bound_rad']:.0f}")
    assert err < 1.6e-5


@pytest.mark.parametrize("seed", range(80))
def test_micrometre_screens_at_millimetres(ctx, oracle, seed):
    """Screens of micrometres, 5 to 40 mm from rays half as wide."""
    rng = np.random.default_rng(seed)
    n, m = 4000, 600
    energy, dist = rng.uniform(5e3, 3e4), rng.uniform(5, 40)
    width, depth = dist * rng.uniform(0.3, 0.8), dist * rng.uniform(0.01, 0.08)
    screen, off = dist / energy * rng.uniform(0.5, 4), dist * rng.uniform(0, 0.4)
    x, z = rng.uniform(-width, width, n), rng.uniform(-depth, depth, n)
    es = np.exp(1j * rng.uniform(0, 2 * np.pi, n))
    rays = cases.rays_from(x, 0.01 * z, z, es=es, ep=0.3 * es, energy=energy)
    pix = cases.pixels_from(off + rng.uniform(-screen, screen, m),
                            off + rng.uniform(-screen, screen, m), dist)
    check(ctx, oracle, rays, pix, rng)


@pytest.mark.parametrize("energy,dist,width,depth,screen,off", [
    (10_000.0, 100.0, 8.0, 0.5, 0.002, 8.0), (240.0, 4.0, 0.3, 0.3, 0.2, 0.3),
    (1_000.0, 50.0, 4.0, 2.0, 0.003, 6.0), (20_000.0, 300.0, 40.0, 5.0, 0.001, 30.0)])
def test_two_polarizations(ctx, oracle, energy, dist, width, depth, screen, off):
    rng = np.random.default_rng(int(dist))
    n, m = 4000, 600
    x, z = rng.uniform(-width, width, n), rng.uniform(-depth, depth, n)
    rays = cases.rays_from(x, 0.01 * z, z, es=np.exp(1j * rng.uniform(0, 2 * np.pi, n)),
                           ep=np.exp(1j * rng.uniform(0, 2 * np.pi, n)), energy=energy)
    pix = cases.pixels_from(off + rng.uniform(-screen, screen, m),
                            off + rng.uniform(-screen, screen, m), dist)
    check(ctx, oracle, rays, pix, rng)
