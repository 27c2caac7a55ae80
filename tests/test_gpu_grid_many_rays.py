"""Many rays on a screen of so many tiles that each is one split: FP32 partials take
hundreds of segments, launches add up in FP64.

Tolerance: `seg` x 16 accumulation steps truncated at 2^-24, of which a third is common to
all points' scale (test_gpu_grid.py), 3.5e-7 of the phasors, and sqrt(512) roundings of
2^-24 / sqrt(12) of the sum (4e-7).
"""
import numpy as np
import pytest

import cases
import xrt_rs
from test_gpu_grid import grid_ctx  # noqa: F401
from xrt_rs import synth

pytestmark = pytest.mark.gpu


# Residual phases of 10 and 18 rad: segments of one and of three blocks.
@pytest.mark.parametrize("dist,seg", [(5400.0, 1), (3000.0, 3)])
def test_one_split_and_many_segments(grid_ctx, oracle, dist, seg):
    rng = np.random.default_rng(seg)
    n = (1 << 20) - 7
    ph = rng.uniform(0, 2 * np.pi, n)
    rays = cases.rays_from(rng.normal(0, 0.1, n), rng.normal(0, 0.1, n), 0.0, es=np.exp(1j * ph),
                           ep=0.2 * np.exp(1j * ph), energy=1000.0)
    pix = synth.grid_screen(2048, 2048, 1.0, dist)
    out, st = xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=grid_ctx,
                                          return_stats=True)
    assert st["sweep"] == 3
    sub, idx = synth.subsample_screen(pix, 64, seed=5)
    err = cases.rel_l2([o[idx] for o in out], oracle.kahan_ld(*cases.as_lists(rays, sub)))
    print(f"{seg} blocks a segment, {st['groups']} splits: {err:.2e}")
    assert err < 16 * seg * 2.0 ** -24 * 2 / 3 + 3.5e-7 + 4e-7
