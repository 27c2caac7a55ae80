"""XK_PATH_F64 where its kernel changes form.

The pair kernel evaluates root, reciprocal and sin/cos itself inside
2^-198 <= |p - r|^2 < 2^777 and |k |p - r|| < 2^50, and by the library outside;
its phase must be the oracle's to the last bit on both sides (at 2^49 rad one
ulp of the path already moves the phase by 0.1 rad). The ranges' partial sums
are added eight at a time with a remainder.

Tolerance: the terms carry at most a dozen roundings of 2^-53 and a sine and
cosine good to two ulp, so 1e-14 of the field's norm; 1e-13 with the sums.
"""
import numpy as np
import pytest

import cases
import xrt_rs

pytestmark = pytest.mark.gpu

TOL = 1e-13


def _check(ctx, oracle, rays, pix):
    rl, pl = cases.as_lists(rays, pix)
    ref = oracle.kahan_f64(rl, pl)
    out = xrt_rs.diffraction_integral(rl, pl, path="f64", ctx=ctx)
    assert cases.rel_l2(out, ref) < TOL


# |p - r| [mm] on both sides of 2^-99 (1.6e-30), of the skip at 1e-30, and up
# to beyond 2^388; energies that put the phase on both sides of 2^50.
@pytest.mark.parametrize("scale,energy", [
    (1e-31, 1e4), (1.2e-30, 1e4), (1.7e-30, 1e4), (1e-12, 1e4), (1e3, 1e4), (2e4, 3e4),
    (1e6, 1e8), (2e6, 1e8), (4e6, 1e8), (1e9, 1e9), (1e100, 1e-90), (1e120, 1e-110)])
def test_pair_ranges(ctx, oracle, scale, energy):
    rng = np.random.default_rng(3)
    rays = cases.rays_from([0.0], [0.0], [0.0], es=0.7 - 0.4j, ep=0.2 + 0.9j, energy=energy,
                           n=(0.1, -0.2, 0.97))
    u = rng.normal(0, 1, (3, 2049))
    u *= scale * rng.uniform(0.6, 1.4, 2049) / np.linalg.norm(u, axis=0)
    _check(ctx, oracle, rays, cases.pixels_from(u[0], u[1], u[2]))


@pytest.mark.parametrize("ranges", [1, 2, 7, 8, 9, 16, 23])
def test_range_sums(ctx, oracle, ranges):
    rays, pix = cases.random_case(32 * ranges - 5, 3, seed=ranges, general_normals=True)
    _check(ctx, oracle, rays, pix)
