"""A stalled Fresnel product ends after a few of its bounded waits, however many ray blocks
are left: every role leaves when one of its waits has run out.

The "fresnel_stall" hook makes the first stage's barrier expect an arrival that nobody
makes. At 4096 polls a wait takes milliseconds; a role that waited again for each of its
blocks (some hundred here) would take a hundred times that.
"""
import time

import numpy as np
import pytest

import xrt_rs
from xrt_rs import FresnelScreen, _lib

pytestmark = pytest.mark.gpu


# One CTA per tile, CTA pairs, pairs on 256 points (4 x 128 rows, 2 x 256 points).
@pytest.mark.parametrize("n,nx,nz,tiles", [(60_000, 64, 64, 1), (60_000, 100, 200, 2),
                                            (60_000, 512, 512, 8)])
def test_every_role_leaves(n, nx, nz, tiles):
    rng = np.random.default_rng(nz)
    x, z = rng.normal(0, 0.05, n), rng.normal(0, 0.05, n)
    es = np.exp(1j * rng.uniform(-np.pi, np.pi, n))
    sc = FresnelScreen(-0.2, 0.2, nx, -0.2, 0.2, nz)
    ctx = xrt_rs.GpuContext.new(0)
    try:
        run = lambda: xrt_rs.fresnel_propagate(x, z, es, 10000.0, 1000.0, sc, ctx=ctx,
                                               return_stats=True)
        ref, st = run()
        assert st["n_tiles"] == tiles
        ctx.set_option("wait_limit", 4096)
        ctx.set_option("fresnel_stall", 1)
        t0 = time.perf_counter()
        with pytest.raises(xrt_rs.XkError) as ei:
            run()
        dt = time.perf_counter() - t0
        print(f"{nx} x {nz}: {dt * 1e3:.1f} ms, {st['groups']} splits")
        assert ei.value.code == _lib.XK_ERR_TIMEOUT
        assert dt < 0.5
        ctx.set_option("wait_limit", float(1 << 24))
        assert np.array_equal(run()[0].amplitude, ref.amplitude)
    finally:
        ctx.close()
