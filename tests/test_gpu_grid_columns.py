"""The product's two amplitude columns, one far weaker than the other: either keeps its
own accuracy (the tolerance of the product, 1e-5, of that column's norm)."""
import numpy as np
import pytest

import cases
import xrt_rs
from test_gpu_grid import TOL, grid, grid_ctx, run  # noqa: F401

pytestmark = pytest.mark.gpu


def column_errors(ctx, oracle, rays):
    pix = grid(np.linspace(-0.5, 0.5, 48), np.linspace(-0.4, 0.4, 40), 2000.0, "xyz")
    out, st = run(ctx, rays, pix)
    assert st["sweep"] == 3
    ref = oracle.kahan_ld(*cases.as_lists(rays, pix))
    err = []
    for a, b in zip(cases.field_c(out), cases.field_c(ref)):
        err.append(float(np.linalg.norm(a - b) / np.linalg.norm(b)))
    return err, st


@pytest.mark.parametrize("ratio", [1e-4, 1e-7, 1e-8, 1e-10, 1e10])
def test_each_column_by_itself(grid_ctx, oracle, ratio):
    """Ep `ratio` times Es, with phases of its own."""
    rng = np.random.default_rng(2)
    n = 4000
    ph = rng.uniform(0, 2 * np.pi, (2, n))
    rays = cases.rays_from(rng.normal(0, 0.1, n), rng.normal(0, 0.1, n), 0.0,
                           es=np.exp(1j * ph[0]), ep=ratio * np.exp(1j * ph[1]))
    (es, ep), st = column_errors(grid_ctx, oracle, rays)
    print(f"ratio {ratio:g}: es {es:.2e} ep {ep:.2e}")
    assert st["one_polarization"] == 0 and es < TOL and ep < TOL


@pytest.mark.parametrize("ratio", [1e-9, 1e9])
def test_one_polarization_of_any_ratio(grid_ctx, oracle, ratio):
    rng = np.random.default_rng(3)
    n = 4000
    a = rng.uniform(0.5, 1.0, n) * np.exp(1j * rng.uniform(0, 2 * np.pi, n))
    rays = cases.rays_from(rng.normal(0, 0.1, n), rng.normal(0, 0.1, n), 0.0, es=a, ep=ratio * a)
    (es, ep), st = column_errors(grid_ctx, oracle, rays)
    print(f"one polarization, ratio {ratio:g}: es {es:.2e} ep {ep:.2e}")
    assert st["one_polarization"] == 1 and es < TOL and ep < TOL


@pytest.mark.parametrize("zero", ["es", "ep"])
def test_a_column_of_zeros(grid_ctx, oracle, zero):
    """Both columns summed although one is zero."""
    grid_ctx.set_option("polarization", 0)
    rng = np.random.default_rng(4)
    a = np.exp(1j * rng.uniform(0, 6, 3000))
    rays = cases.rays_from(rng.normal(0, 0.1, 3000), rng.normal(0, 0.1, 3000), 0.0,
                           **{zero: 0j, "ep" if zero == "es" else "es": a})
    pix = grid(np.linspace(-0.5, 0.5, 48), np.linspace(-0.4, 0.4, 40), 2000.0, "xyz")
    out, st = run(grid_ctx, rays, pix)
    assert st["sweep"] == 3 and st["one_polarization"] == 0
    got = cases.field_c(out)
    ref = cases.field_c(oracle.kahan_ld(*cases.as_lists(rays, pix)))
    k = 0 if zero == "es" else 1
    assert not np.any(got[k])
    assert np.linalg.norm(got[1 - k] - ref[1 - k]) < TOL * np.linalg.norm(ref[1 - k])
