"""The general kernel a few millimetres from the rays.

The residual phase B of a pair leaves out B^2 / (2 k d) rad (the path's own change
in the denominator of the expansion). The planner keeps that within half the
tolerance; FP32 rounding of the residual phase adds up to 1.6e-5.
"""
import numpy as np
import pytest

import cases
import xrt_rs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("energy,dist,aperture,screen", [
    (10_000.0, 1.0, 0.01, 0.001), (10_000.0, 2.0, 0.02, 0.002), (30_000.0, 1.0, 0.006, 0.0006),
    (1_000.0, 2.0, 0.02, 0.02), (10_000.0, 5.0, 0.03, 0.004), (10_000.0, 20.0, 0.05, 0.05)])
@pytest.mark.parametrize("polarizations", [1, 2])
def test_millimetres_from_an_aperture(ctx, oracle, energy, dist, aperture, screen, polarizations):
    rng = np.random.default_rng(int(dist))
    n, m = 4000, 700
    x, y = rng.uniform(-aperture, aperture, n), rng.uniform(-aperture, aperture, n)
    es = np.exp(1j * rng.uniform(0, 2 * np.pi, n))
    ep = 0.3 * es if polarizations == 1 else np.exp(1j * rng.uniform(0, 2 * np.pi, n))
    rays = cases.rays_from(x, y, 0.0, es=es, ep=ep, energy=energy)
    pix = cases.pixels_from(rng.uniform(-screen, screen, m), rng.uniform(-screen, screen, m), dist)
    out, st = xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=ctx,
                                          return_stats=True)
    assert st["path"] == xrt_rs.XK_PATH_F32PR and st["sweep"] in (0, 1, 2)
    err = cases.rel_l2(out, oracle.kahan_ld(*cases.as_lists(rays, pix)))
    print(f"{energy} eV {dist} mm: {err:.2e}, residual phase {st['phase_bound_rad']:.0f} rad")
    assert err < 0.5e-4 + 1.6e-5
