"""XK_PATH_F64 on both sides of |p - r|^2 = 2^817 (1e123 mm), where its kernel hands over to
the library's root, division and sine (tests/test_gpu_f64_edges.py has the other bounds and
the tolerance)."""
import numpy as np
import pytest

import cases
from test_gpu_f64_edges import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,energy", [(1e121, 1e-111), (9e122, 1e-112), (1.1e123, 1e-113),
                                           (1e125, 1e-115), (1e150, 1e-140)])
def test_huge_paths(ctx, oracle, scale, energy):
    rng = np.random.default_rng(5)
    rays = cases.rays_from([0.0], [0.0], [0.0], es=0.7 - 0.4j, ep=0.2 + 0.9j, energy=energy,
                           n=(0.1, -0.2, 0.97))
    u = rng.normal(0, 1, (3, 2049))
    u *= scale * rng.uniform(0.6, 1.4, 2049) / np.linalg.norm(u, axis=0)
    _check(ctx, oracle, rays, cases.pixels_from(u[0], u[1], u[2]))
