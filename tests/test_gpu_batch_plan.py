"""Planning of many solves: the planner's first kernels serve 16 of them per launch
and skip those routed before. Counts around one and two launches, rectangular and
line screens and solves without rays among them; every result equals the solve's own,
bit for bit."""
import numpy as np
import pytest

import cases
import xrt_rs
from xrt_rs import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 16, 17, 33])
def test_batch_of(ctx, count):
    solves = []
    for i in range(count):
        rays = synth.gaussian_aperture(1024 + 37 * i, 0.1, 9000.0, 3e4, seed=i)
        pix = synth.grid_screen(40, 30 + i, 0.5, 2000.0) if i % 3 else \
            synth.line_screen(200 + i, 0.5, 1500.0)
        solves.append((cases.rays_from([]) if i == 5 else rays, pix))
    outs = xrt_rs.Batch(solves, path="f32pr", ctx=ctx).run()
    for i, ((rays, pix), got) in enumerate(zip(solves, outs)):
        alone = xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=ctx)
        assert all(np.array_equal(a, b) for a, b in zip(got, alone)), i
