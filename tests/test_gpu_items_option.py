"""The "items_per_warp" option decides the ray groups of solves with few tiles as well."""
import pytest

import cases
import xrt_rs
from xrt_rs import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pix,items", [(256, 1), (25_600, 1), (25_600, 2), (25_600, 5)])
def test_a_set_number_of_items_stands(ctx, n_pix, items):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, tiles = 10_000, n_pix // 256
    rays = synth.gaussian_aperture(n, 0.05, 10_000.0, 30_000.0, seed=1)
    pix = synth.line_screen(n_pix, 0.5, 1000.0)
    run = lambda: xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=ctx,
                                              return_stats=True)
    out, st = run()
    try:
        ctx.set_option("items_per_warp", items)
        got, st2 = run()
    finally:
        ctx.set_option("items_per_warp", 16)
    # Twelve resident warps per SM; items of at least four stages of 56 rays.
    assert st2["groups"] == min(-(-12 * sms * items // tiles), n // 224)
    assert cases.rel_l2(got, out) < 1e-5
    assert run()[1]["groups"] == st["groups"]
