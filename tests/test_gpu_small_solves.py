"""Solves of few screen tiles: their rays are cut into many small items (down
to 16 rays) so that every warp has one, and the items' sums are added by 16
rows of threads. Sizes around one and several rounds of items and around the
rows' remainders, lines and scattered points, against the extended-precision
oracle (the path's tolerance), twice bit for bit."""
import numpy as np
import pytest

import cases
import xrt_rs
from xrt_rs import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rays", [16, 255, 256, 257, 4111, 28416, 70001])
@pytest.mark.parametrize("n_pix", [1, 256, 257, 2600])
def test_few_tiles(ctx, oracle, n_rays, n_pix):
    rays = synth.gaussian_aperture(n_rays, 0.05, 10_000.0, 30_000.0, seed=n_rays)
    pix = synth.line_screen(n_pix, 0.5, 1000.0)
    run = lambda: xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=ctx,
                                              return_stats=True)
    out, st = run()
    assert st["path"] == xrt_rs.XK_PATH_F32PR and st["groups"] <= max(1, n_rays // 16)
    again, _ = run()
    assert all(np.array_equal(a, b) for a, b in zip(out, again))
    sub, idx = synth.subsample_screen(pix, 40, seed=n_pix)
    ref = oracle.kahan_ld(*cases.as_lists(rays, sub))
    assert cases.rel_l2([o[idx] for o in out], ref) < 1e-4


def test_screen_with_and_without_depth_sort_alike(ctx, oracle):
    """The tile sort leaves out the depth bits of a flat screen."""
    rays, pix = cases.random_case(3000, 3000, seed=4)
    deep = dict(pix, z=pix["z"] + np.random.default_rng(1).uniform(0, 1.0, 3000))
    for p in (pix, deep):
        out = xrt_rs.diffraction_integral(*cases.as_lists(rays, p), path="f32pr", ctx=ctx)
        sub, idx = synth.subsample_screen(p, 200, seed=2)
        ref = oracle.kahan_ld(*cases.as_lists(rays, sub))
        assert cases.rel_l2([o[idx] for o in out], ref) < 1e-4
