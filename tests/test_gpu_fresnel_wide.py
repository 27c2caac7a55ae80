"""Fresnel products on 256-point tiles (more than 128 rows, 1e10 pairs and up).

Tolerance: 160 accumulation steps per segment truncated at 2^-24 (6.4e-6 at most,
5e-6 on average over the K splits) and the 2^-22 split of the phasors: 1e-5.
"""
import numpy as np
import pytest

import xrt_rs
from xrt_rs import FresnelScreen

pytestmark = pytest.mark.gpu


# One tile with 1 to 128 points of its second half used, last tiles of one row, many
# tiles with one split, ray blocks that no segment divides, and 257 points, which
# 128-point tiles pad less.
@pytest.mark.parametrize("n,nx,nz", [(153000, 129, 200), (153011, 256, 129), (80001, 257, 256),
                                      (77011, 255, 257), (40033, 500, 512), (2750, 2000, 2048)])
def test_wide_tiles_against_f64(ctx, n, nx, nz):
    rng = np.random.default_rng(n)
    x, z = rng.normal(0, 0.1, n), rng.normal(0, 0.1, n)
    es = rng.uniform(0.2, 1.0, n) * np.exp(1j * rng.uniform(-np.pi, np.pi, n))
    sc = FresnelScreen(-0.5, 0.4, nx, -0.3, 0.5, nz)
    got, st = xrt_rs.fresnel_propagate(x, z, es, 10000.0, 1000.0, sc, ctx=ctx, return_stats=True)
    wide, narrow = -(-nx // 256), -(-nx // 128)
    assert st["n_tiles"] == -(-nz // 256) * 2 * (wide if 0.9 * 2 * wide < narrow else narrow)
    ref = xrt_rs.fresnel_propagate(x, z, es, 10000.0, 1000.0, sc, path="f64", ctx=ctx)
    err = np.linalg.norm(got.amplitude - ref.amplitude) / np.linalg.norm(ref.amplitude)
    print(f"{n} rays, {nx} x {nz}: {err:.2e}, {st['n_tiles']} tiles x {st['groups']} splits")
    assert err < 1e-5
