"""Rectangular screens as a tensor-core product (stats sweep 3).

Every form the rule accepts is compared with the extended-precision oracle and
with the general kernel (option grid_product 0), which remains the path of
every form it refuses. Tolerance of the product: 160 accumulation steps
truncated at 2^-24 (6.4e-6 at most, 2e-6 on average), the dropped second order
of exp(iE) and the 2^-22 split: 1e-5 of the field's norm.
"""
import numpy as np
import pytest

import cases
import xrt_rs
from xrt_rs import synth

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.fixture
def grid_ctx(ctx):
    yield ctx
    for name, value in (("grid_product", 1), ("polarization", -1), ("sweep", -1),
                        ("tolerance", 1e-4)):
        ctx.set_option(name, value)


def run(ctx, rays, pix):
    return xrt_rs.diffraction_integral(*cases.as_lists(rays, pix), path="f32pr", ctx=ctx,
                                       return_stats=True)


def grid(outer, inner, other, axes):
    """Points outer x inner (inner fastest); axes: coordinates of outer, inner, other."""
    cols = [np.repeat(outer, len(inner)), np.tile(inner, len(outer)),
            np.full(len(outer) * len(inner), other)]
    return {k: cols[axes.index(k)].astype(np.float64) for k in "xyz"}


def permuted(rays, axes):
    """Aperture rays (plane z = 0, normal z) with x, y, z renamed to the axes."""
    out = dict(rays)
    for a, b in zip("xyz", axes):
        out[b], out["n" + b] = rays[a], rays["n" + a]
    return out


def check(ctx, oracle, rays, pix, want=3, tol=TOL):
    out, st = run(ctx, rays, pix)
    assert st["path"] == xrt_rs.XK_PATH_F32PR and st["sweep"] == want, st
    ctx.set_option("grid_product", 0)
    gen, gst = run(ctx, rays, pix)
    ctx.set_option("grid_product", 1)
    assert gst["sweep"] in (0, 1, 2)
    assert gst["one_polarization"] == st["one_polarization"]
    sub, idx = synth.subsample_screen(pix, 96, seed=5)
    exact = oracle.kahan_ld(*cases.as_lists(rays, sub))
    err = cases.rel_l2([o[idx] for o in out], exact)
    err_gen = cases.rel_l2([o[idx] for o in gen], exact)
    print(f"product {err:.2e} general {err_gen:.2e} bound {st['phase_bound_rad']:.1f}")
    assert err < (tol if want == 3 else 1e-4)
    assert cases.rel_l2(out, gen) < tol + 3e-5  # the general kernel's own worst error
    return out, st


@pytest.mark.parametrize("axes", ["xyz", "yxz", "xzy", "zxy", "yzx", "zyx"])
def test_axis_orders(grid_ctx, oracle, axes):
    rays = synth.gaussian_aperture(5000, 0.08, 9000.0, 3e4, seed=1)
    pix = grid(np.linspace(-0.6, 0.5, 70), np.linspace(-0.3, 0.4, 45), 1800.0, axes)
    check(grid_ctx, oracle, permuted(rays, axes), pix)


# Tile edges: 256 rows x 128 columns in either orientation, and the smallest.
@pytest.mark.parametrize("n_outer,n_inner", [(2, 700), (700, 2), (128, 129), (129, 128),
                                              (256, 257), (257, 256), (255, 127), (33, 32),
                                              (385, 300)])
def test_tile_edges(grid_ctx, oracle, n_outer, n_inner):
    rays = synth.gaussian_aperture(3000, 0.1, 12000.0, 2e4, seed=2)
    pix = grid(np.linspace(-0.5, 0.5, n_outer), np.linspace(-0.4, 0.4, n_inner), 3000.0, "xyz")
    check(grid_ctx, oracle, rays, pix)


# Tiles of 256 x 256 points, taken from 4.3e9 padded pairs on: the smallest (129
# columns), last tiles of one, of half and of half and one columns in either
# orientation, ray blocks that do not divide into segments or splits.
@pytest.mark.parametrize("n_outer,n_inner,n,pol", [(256, 129, 70011, 1), (129, 256, 70050, 2),
                                                    (200, 257, 40001, 2), (384, 250, 40033, 1),
                                                    (385, 131, 50000, 1), (512, 255, 35000, 2)])
def test_wide_tiles(grid_ctx, oracle, n_outer, n_inner, n, pol):
    rays = synth.gaussian_aperture(n, 0.1, 12000.0, 2e4, seed=21)
    if pol == 2:
        rng = np.random.default_rng(n)
        rays.update(ep_re=rng.normal(0, 1, n), ep_im=rng.normal(0, 1, n))
    pix = grid(np.linspace(-0.5, 0.5, n_outer), np.linspace(-0.4, 0.4, n_inner), 3000.0, "xyz")
    out, st = check(grid_ctx, oracle, rays, pix)
    assert st["one_polarization"] == (pol == 1)


# Screens near enough that a full tile's mixed phase is past the first order: tiles
# use 32 to 256 of their rows and 32 to 128 of their columns, with remainders.
@pytest.mark.parametrize("n_outer,n_inner,n,dist,energy", [
    (385, 300, 4000, 350.0, 12000.0), (130, 97, 4000, 420.0, 12000.0),
    (64, 200, 3000, 300.0, 12000.0), (300, 33, 3000, 330.0, 12000.0),
    (96, 96, 2000, 350.0, 9000.0), (387, 119, 60000, 436.0, 11756.0)])
def test_tiles_in_part(grid_ctx, oracle, n_outer, n_inner, n, dist, energy):
    rays = synth.gaussian_aperture(n, 0.1, energy, 2e4, seed=n_inner)
    pix = grid(np.linspace(-0.5, 0.5, n_outer), np.linspace(-0.4, 0.4, n_inner), dist, "xyz")
    check(grid_ctx, oracle, rays, pix)


def test_mostly_padding_takes_the_general_kernel(grid_ctx, oracle):
    """A screen that fills a 32nd of its tile, with many rays."""
    rays = synth.gaussian_aperture(1_500_000, 0.1, 10000.0, 3e4, seed=14)
    check(grid_ctx, oracle, rays, synth.grid_screen(32, 33, 0.5, 2000.0), want=2)


# Blocks of 32 rays, segments of ten, splits of at least ten blocks.
@pytest.mark.parametrize("n", [1024, 1025, 1055, 10 * 32 + 1024, 20011])
def test_ray_remainders(grid_ctx, oracle, n):
    rays = synth.gaussian_aperture(n, 0.1, 10000.0, 3e4, seed=n)
    check(grid_ctx, oracle, rays, synth.grid_screen(40, 51, 0.5, 2000.0))


@pytest.mark.parametrize("shape", ["decreasing", "uneven", "shuffled", "negative_zero"])
def test_axis_values(grid_ctx, oracle, shape):
    rng = np.random.default_rng(4)
    o, i = np.linspace(-0.5, 0.5, 64), np.linspace(-0.2, 0.3, 50)
    if shape == "decreasing":
        o, i = o[::-1].copy(), i[::-1].copy()
    elif shape == "uneven":
        o, i = np.sort(rng.uniform(-0.5, 0.5, 64)), np.sort(rng.uniform(-0.2, 0.3, 50))
    elif shape == "shuffled":
        o, i = rng.permutation(o), rng.permutation(i)
    pix = grid(o, i, 2500.0, "xyz")
    if shape == "negative_zero":
        pix["y"][np.abs(pix["y"]) < 1e-3] = 0.0
        pix["y"] = np.where((pix["y"] == 0.0) & (np.arange(len(pix["y"])) % 100 < 50), -0.0,
                            pix["y"])
    rays = synth.gaussian_aperture(4000, 0.1, 10000.0, 3e4, seed=7)
    check(grid_ctx, oracle, rays, pix)


def test_two_polarizations_and_general_normals(grid_ctx, oracle):
    """Per-ray normals tilt the obliquity factor along the tile by up to 1e-3."""
    rays, _ = cases.random_case(6000, 1, seed=3, general_normals=True)
    out, st = check(grid_ctx, oracle, rays, synth.grid_screen(61, 47, 0.5, 2200.0))
    assert st["one_polarization"] == 0


@pytest.mark.parametrize("kind", ["es_zero", "ep_complex", "ep_zero"])
def test_one_polarization_columns(grid_ctx, oracle, kind):
    rays = synth.gaussian_aperture(4000, 0.1, 10000.0, 3e4, seed=8)
    es = rays["es_re"] + 1j * rays["es_im"]
    ep = {"es_zero": es, "ep_complex": (0.3 - 0.7j) * es, "ep_zero": 0 * es}[kind]
    if kind == "es_zero":
        es = 0 * es
    rays.update(es_re=es.real, es_im=es.imag, ep_re=ep.real, ep_im=ep.imag)
    rays = {k: np.ascontiguousarray(v) for k, v in rays.items()}
    out, st = check(grid_ctx, oracle, rays, synth.grid_screen(48, 48, 0.5, 2000.0))
    assert st["one_polarization"] == 1
    if kind == "es_zero":
        assert not np.any(out[0]) and not np.any(out[1])
    if kind == "ep_zero":
        assert not np.any(out[2]) and not np.any(out[3])


def test_mirror_rays_at_grazing_incidence(grid_ctx, oracle):
    """Rays spread 60 mm along the beam: their distances differ by 1 %, the
    quadratic phase by turns, the obliquity factor by 2 % along a tile."""
    rng = np.random.default_rng(6)
    n, dist, th = 5000, 10000.0, 3e-3
    x, y = rng.normal(0, 0.2, n), rng.normal(0, 15.0, n)
    rays = cases.rays_from(x, y, y * y * th / (4 * dist), es=np.exp(1j * rng.uniform(0, 6, n)),
                           ep=0.4 * np.exp(1j * rng.uniform(0, 6, n)))
    rays["ny"] = -y * th / (2 * dist)
    rays["nl"] = np.full(n, th) + rng.normal(0, 1e-5, n)
    pix = grid(np.linspace(-1, 1, 60), th * dist + np.linspace(-1, 1, 45), dist, "xzy")
    check(grid_ctx, oracle, rays, pix)


@pytest.mark.parametrize("scale", [1e-25, 1e25])
def test_amplitude_range(grid_ctx, scale):
    rays = synth.gaussian_aperture(3000, 0.1, 10000.0, 3e4, seed=9)
    pix = synth.grid_screen(40, 40, 0.5, 2000.0)
    base, st = run(grid_ctx, rays, pix)
    for k in ("es_re", "es_im", "ep_re", "ep_im"):
        rays[k] = rays[k] * scale
    out, st2 = run(grid_ctx, rays, pix)
    assert st["sweep"] == st2["sweep"] == 3
    assert cases.rel_l2(out, [b * scale for b in base]) < 1e-6


@pytest.mark.parametrize("energy,dist,sigma", [(1000.0, 8400.0, 0.1), (1000.0, 4200.0, 0.1),
                                                (30000.0, 20000.0, 0.2), (30000.0, 4000.0, 0.1)])
def test_energy_distance_corners(grid_ctx, oracle, energy, dist, sigma):
    """At 1 keV the residual phases of the whole ray set are 14 and 27 rad."""
    rays = synth.gaussian_aperture(20000, sigma, energy, 3e4, seed=11)
    check(grid_ctx, oracle, rays, synth.grid_screen(99, 99, 1.0, dist))


@pytest.mark.parametrize("dist,sweep", [(20000.0, 2), (14000.0, 3), (8400.0, 3)])
def test_small_residual_phases(grid_ctx, oracle, dist, sweep):
    """Where the general kernel's residual phases are a few radians its error
    is below 1e-6: the product has to be as good (short segments), or is not
    taken. 48 truncations of 2^-24 at most, and 3.5e-7 without any."""
    rays = synth.gaussian_aperture(20000, 0.1, 1000.0, 3e4, seed=11)
    check(grid_ctx, oracle, rays, synth.grid_screen(99, 99, 1.0, dist), want=sweep,
          tol=48 * 2.0 ** -24 * 2 / 3 + 3.5e-7)


@pytest.mark.parametrize("form", ["rotated", "one_point_off", "swapped_points", "short", "line",
                                  "near", "coarse_tile", "tolerance", "sweep", "budget"])
def test_refused_forms_take_the_general_kernel(grid_ctx, oracle, form):
    rays = synth.gaussian_aperture(3000, 0.1, 10000.0, 3e4, seed=12)
    pix = synth.grid_screen(40, 40, 0.5, 2000.0)
    if form == "rotated":
        c, s = np.cos(0.3), np.sin(0.3)
        pix["x"], pix["y"] = c * pix["x"] - s * pix["y"], s * pix["x"] + c * pix["y"]
    elif form == "one_point_off":
        pix["z"][777] = np.nextafter(pix["z"][777], 1e9)
    elif form == "swapped_points":
        pix["x"][[5, 900]] = pix["x"][[900, 5]]
    elif form == "short":
        pix = {k: v[:-1].copy() for k, v in pix.items()}
    elif form == "line":
        pix = synth.line_screen(1600, 0.5, 2000.0)
    elif form == "near":
        pix = synth.grid_screen(40, 40, 0.5, 150.0)
    elif form == "coarse_tile":
        pix = synth.grid_screen(40, 40, 8.0, 2000.0)
    elif form == "tolerance":
        grid_ctx.set_option("tolerance", 2e-5)
    elif form == "sweep":
        grid_ctx.set_option("sweep", 1)
    elif form == "budget":
        grid_ctx.set_option("phase_budget", 100.0)
    try:
        out, st = run(grid_ctx, rays, pix)
        assert st["path"] == xrt_rs.XK_PATH_F32PR and st["sweep"] in (0, 1, 2), st
    finally:
        grid_ctx.set_option("phase_budget", 512.0)
    sub, idx = synth.subsample_screen(pix, 64, seed=1)
    exact = oracle.kahan_ld(*cases.as_lists(rays, sub))
    assert cases.rel_l2([o[idx] for o in out], exact) < 1e-4


def test_batch_and_repeat_are_bitwise_the_single_solve(grid_ctx):
    solves = []
    for i, (n, a, b) in enumerate([(3000, 40, 40), (20011, 65, 130), (1500, 33, 300)]):
        solves.append((synth.gaussian_aperture(n, 0.1, 10000.0, 3e4, seed=i),
                       grid(np.linspace(-.5, .5, a), np.linspace(-.4, .4, b), 2000.0, "xyz")))
    solves.insert(1, synth.config0(seed=1))
    for graph in (True, False):
        batch = xrt_rs.Batch(solves, path="f32pr", ctx=grid_ctx, graph=graph)
        for _ in range(2):
            outs = batch.run()
            for i, ((rays, pix), got) in enumerate(zip(solves, outs)):
                alone, st = run(grid_ctx, rays, pix)
                assert batch.plan(i)["sweep"] == st["sweep"] == (2 if i == 1 else 3)
                assert all(np.array_equal(x, y) for x, y in zip(got, alone)), i
        batch.close()


def test_stalled_stage_times_out_and_context_recovers():
    """The inject_stall hook on a solve that takes the product: no MMA is
    issued, every wait is bounded, the next call is bitwise the clean one."""
    rays = synth.gaussian_aperture(3000, 0.1, 10000.0, 3e4, seed=13)
    pix = synth.grid_screen(40, 40, 0.5, 2000.0)
    ctx = xrt_rs.GpuContext.new(0)
    try:
        ref, st = run(ctx, rays, pix)
        assert st["sweep"] == 3
        ctx.set_option("wait_limit", 4096)
        ctx.set_option("inject_stall", 16)
        with pytest.raises(xrt_rs.XkError) as ei:
            run(ctx, rays, pix)
        assert ei.value.code == xrt_rs._lib.XK_ERR_TIMEOUT
        ctx.set_option("wait_limit", float(1 << 24))
        out, _ = run(ctx, rays, pix)
        assert all(np.array_equal(x, y) for x, y in zip(out, ref))
    finally:
        ctx.close()
