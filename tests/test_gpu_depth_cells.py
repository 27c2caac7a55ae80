"""Rays and screens that are long along the beam (mirrors at grazing incidence):
ray cells get their own length along it, and on deep screens the tiles are cut
on one transverse scale.

Tolerance: 1.45e-7 per rad of residual-phase bound on the worst fields
(kPhasePerTolerance), 60 rad in the widest tile of a deep screen (8.7e-6) and
0.3 of the budget on flat ones (83 rad, 1.2e-5).
"""
import numpy as np
import pytest

import cases
import xrt_rs
from xrt_rs import synth

pytestmark = pytest.mark.gpu

TH = 3e-3


def mirror_rays(n, dist, energy, seed, length=15.0):
    rng = np.random.default_rng(seed)
    x, y = rng.normal(0, 0.2, n), rng.normal(0, length, n)
    rays = cases.rays_from(x, y, y * y * TH / (4 * dist), energy=energy,
                           es=np.exp(1j * rng.uniform(0, 6, n)),
                           ep=0.4 * np.exp(1j * rng.uniform(0, 6, n)))
    rays["ny"] = -y * TH / (2 * dist)
    rays["nl"] = np.full(n, TH)
    return rays


def second_mirror(m, dist, seed):
    rng = np.random.default_rng(seed)
    py = rng.normal(0, 20.0, m)
    return cases.pixels_from(rng.normal(0, 0.3, m), dist + py,
                             TH * dist + TH * py + py * py * TH / (4 * dist))


@pytest.mark.parametrize("n,m,dist,energy", [(4000, 5000, 3000.0, 9000.0),
                                              (9001, 257, 9000.0, 6000.0),
                                              (1500, 3000, 2000.0, 20000.0)])
def test_mirror_to_mirror(ctx, oracle, n, m, dist, energy):
    rays, pix = mirror_rays(n, dist, energy, n), second_mirror(m, dist, m)
    out, st = xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=ctx,
                                          return_stats=True)
    assert st["path"] == xrt_rs.XK_PATH_F32PR and st["phase_bound_rad"] <= 60.0 + 1e-9
    sub, idx = synth.subsample_screen(pix, 200, seed=1)
    ref = oracle.kahan_ld(*cases.as_lists(rays, sub))
    err = cases.rel_l2([o[idx] for o in out], ref)
    print(f"mirror to mirror {err:.2e} chunks={st['n_chunks']}")
    assert err < 8.7e-6


@pytest.mark.parametrize("screen", ["line", "scattered", "tilted"])
@pytest.mark.parametrize("length", [15.0, 0.5])
def test_mirror_to_flat_screens(ctx, oracle, screen, length):
    dist = 6000.0
    rays = mirror_rays(6000, dist, 11000.0, 3, length)
    rng = np.random.default_rng(5)
    if screen == "line":
        pix = cases.pixels_from(np.linspace(-1, 1, 3000), dist, TH * dist)
    else:
        x, z = rng.uniform(-1, 1, 3000), rng.uniform(-1, 1, 3000)
        depth = 0.0 if screen == "scattered" else 0.4 * z
        pix = cases.pixels_from(x, dist + depth, TH * dist + z)
    out, st = xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=ctx,
                                          return_stats=True)
    assert st["path"] == xrt_rs.XK_PATH_F32PR
    sub, idx = synth.subsample_screen(pix, 200, seed=1)
    ref = oracle.kahan_ld(*cases.as_lists(rays, sub))
    err = cases.rel_l2([o[idx] for o in out], ref)
    print(f"{screen} {length} {err:.2e} chunks={st['n_chunks']} bound={st['phase_bound_rad']:.0f}")
    assert err < 1.45e-7 * st["phase_bound_rad"] + 4e-7
