"""What a whole solve leaves out of its half-passes changes nothing.  A solve skips the planes of
settled neighbours and drops refinement trials after the sources that can bound them; a half-pass on
caller maps (hp_propagate_pass) does neither, it scores every distinct neighbour and every trial whole.
So a solve must equal initialisation, cost and its half-passes called one by one, bit for bit (tolerance
0: the same arithmetic on every cost that decides), for every source count and top_k (which set how many
sources bound a trial), windows inside and across the source's border, and ragged tiles."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import cam_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(hp, scene_mod):
    s = scene_mod.multi_object(seed=4, w=203, h=133, n_views=9, n_src=8, f=160.0)  # ragged: 203 = 3 x 64 + 11
    ctx = hp.Context(0)
    yield s, ctx, [ctx.upload(v.image) for v in s.views]
    ctx.close()


@pytest.mark.parametrize("precision,tile_h", [(0, 0), (1, 8), (1, 4)])
@pytest.mark.parametrize("sources,top_k,radius,stride,steps", [
    (8, 3, 7, 2, 2), (6, 3, 5, 1, 2), (4, 2, 3, 2, 4), (3, 3, 7, 1, 1), (2, 3, 5, 2, 2), (5, 1, 1, 1, 2), (1, 3, 5, 1, 0)])
def test_solve_equals_its_half_passes(hp, setup, precision, tile_h, sources, top_k, radius, stride, steps):
    s, ctx, ids = setup
    r, iterations = 2, 5
    srcs = s.sources[r][:sources]
    job = hp.make_job(ids[r], [ids[i] for i in srcs], hp.make_camera(*cam_of(s, r)),
                      [hp.make_camera(*cam_of(s, i)) for i in srcs], *s.depth_range, seed=7, view_id=r,
                      iterations=iterations)
    params = hp.default_params(radius=radius, stride=stride, top_k=top_k, precision=precision, refine_steps=steps,
                               tile_h=tile_h)
    whole, d, n, c = hp.host_maps(s.height, s.width)
    ctx.solve([job], params, [whole])
    maps, d2, n2, c2 = hp.host_maps(s.height, s.width)
    ctx.init_hypotheses(job, params, maps)
    ctx.ncc_cost(job, params, maps)
    for it in range(iterations):
        for color in (0, 1):
            ctx.propagate_pass(job, params, maps, it, color)
    assert np.array_equal(d, d2) and np.array_equal(n, n2) and np.array_equal(c, c2)
    assert (c >= 0).all() and not np.signbit(c).any()


def test_a_half_pass_keeps_the_callers_costs_as_they_are(hp, setup):
    """Costs of pixels a half-pass does not visit come back as given, whatever their sign."""
    s, ctx, ids = setup
    job = hp.make_job(ids[0], [ids[1]], hp.make_camera(*cam_of(s, 0)), [hp.make_camera(*cam_of(s, 1))],
                      *s.depth_range, seed=7, view_id=0, iterations=1)
    params = hp.default_params(radius=3, stride=1)
    maps, d, n, c = hp.host_maps(s.height, s.width)
    ctx.init_hypotheses(job, params, maps)
    c[:] = np.random.default_rng(0).uniform(-2, 2, c.shape).astype(np.float32)
    before = c.copy()
    ctx.propagate_pass(job, params, maps, 1, 0)
    ys, xs = np.mgrid[0:s.height, 0:s.width]
    other = ((xs + ys) & 1) == 1
    assert np.array_equal(c[other], before[other]) and (c[~other] <= before[~other]).all()
