"""Screens that are deep along the beam: the ray cells' size follows from the mean extent of
the tiles, whose sum must not depend on the order in which the tiles' warps finish."""
import numpy as np
import pytest

import cases
import xrt_rs
from test_gpu_depth_cells import mirror_rays, second_mirror

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(20_000, 50_021), (9001, 257)])
def test_reruns_and_batches_are_bitwise_the_same(ctx, n, m):
    rays, pix = mirror_rays(n, 3000.0, 9000.0, n), second_mirror(m, 3000.0, m)
    run = lambda: xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=ctx,
                                              return_stats=True)
    out, st = run()
    for _ in range(15):
        again, st2 = run()
        assert st2["n_chunks"] == st["n_chunks"]
        assert st2["phase_bound_rad"] == st["phase_bound_rad"]
        assert all(np.array_equal(a, b) for a, b in zip(out, again))
    batch = xrt_rs.Batch([(rays, pix)] * 3, path="f32pr", ctx=ctx)
    for got in batch.run():
        assert all(np.array_equal(a, b) for a, b in zip(out, got))
    batch.close()
