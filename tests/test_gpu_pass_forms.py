"""The forms a launch of half-passes takes (units on whole or half tiles, items scored whole) give the
same bits: a job solved alone, in batches that take the other forms, and in a persistent plan, for every
window, both precisions and tile heights, and source counts on both sides of the lines between the forms.
And a solve whose launches are whole tiles, or half tiles that fill the GPU, equals its half-passes on
caller maps, which leave nothing out (tolerance 0: the same arithmetic on every cost that decides).

The forms follow from the tiles a launch has for each SM, so the batch sizes are chosen by the device's
SM count, and `_form` restates the rule to assert that the intended ones run."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import cam_of

pytestmark = pytest.mark.gpu

W, H = 203, 130  # 4 x 17 tiles; the last row of tiles has two rows of pixels, so its lower halves none
TILES = 4 * 17
WHOLE_SAMPLES = {0: 27, 1: 100}  # by precision


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _form(precision, radius, stride, sources, tiles, sms):
    samples = ((2 * radius) // stride + 1) ** 2 * sources
    if 2 * tiles <= 3 * sms:
        return "roomy"
    if samples <= WHOLE_SAMPLES[precision]:
        return "whole"
    if precision == 0:
        most = min(8, samples / (100 if sources == 2 else 24))
    else:
        most = 2.2 if sources < 3 else min(8, max(2.2, samples * sources / 175))
    past = tiles % sms
    return "split" if 0 < 2 * past <= sms and tiles <= most * sms else "units"


def _batches(sms):
    """A batch size whose halves spread no better, and one whose do (both past the roomy line)."""
    past = {k: 2 * ((TILES * k) % sms) for k in range(1, 40) if 2 * TILES * k > 3 * sms}
    plain = min(k for k, p in past.items() if p == 0 or p > sms)
    spread = min(k for k, p in past.items() if 0 < p <= sms and TILES * k >= 2 * sms)
    return plain, spread


@pytest.fixture(scope="module")
def small(hp, scene_mod):
    s = scene_mod.multi_object(seed=4, w=W, h=H, n_views=9, n_src=8, f=160.0)
    ctx = hp.Context(0)
    yield s, ctx, [ctx.upload(v.image) for v in s.views]
    ctx.close()


def _job(hp, s, ids, r, sources, iterations):
    srcs = s.sources[r][:sources]
    return hp.make_job(ids[r], [ids[i] for i in srcs], hp.make_camera(*cam_of(s, r)),
                       [hp.make_camera(*cam_of(s, i)) for i in srcs], *s.depth_range, seed=7, view_id=r,
                       iterations=iterations)


@pytest.mark.parametrize("precision,tile_h", [(0, 0), (1, 8), (1, 4)])
@pytest.mark.parametrize("radius,stride", [(r, s) for r in range(1, 8) for s in (1, 2)])
@pytest.mark.parametrize("sources", [1, 2, 4])
def test_every_form_gives_the_same_bits(hp, small, precision, tile_h, radius, stride, sources):
    s, ctx, ids = small
    params = hp.default_params(radius=radius, stride=stride, precision=precision, tile_h=tile_h)
    job = _job(hp, s, ids, 4, sources, 3)
    maps, d, n, c = hp.host_maps(H, W)
    ctx.solve([job], params, [maps])

    def same(outs):
        return all(np.array_equal(a, d) and np.array_equal(b, n) and np.array_equal(e, c) for _, a, b, e in outs)

    for k in _batches(_sms()):
        outs = [hp.host_maps(H, W) for _ in range(k)]
        ctx.solve([job] * k, params, [o[0] for o in outs])
        assert same(outs)
        outs = [hp.host_maps(H, W) for _ in range(k)]
        with hp.Plan(ctx, [job] * k, params, [o[0] for o in outs],
                     hp.plan_options(schedule=hp.SCHEDULE_PERSISTENT)) as plan:
            plan.run()
        assert same(outs)


def test_the_batches_take_every_form():
    sms = _sms()
    plain, spread = (TILES * k for k in _batches(sms))
    for p in (0, 1):
        forms = {_form(p, r, s, n, t, sms)
                 for r in range(1, 8) for s in (1, 2) for n in (1, 2, 4) for t in (TILES, plain, spread)}
        assert forms == {"roomy", "whole", "units", "split"}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("w,h,spread", [(571, 205, False), (571, 301, True)])
@pytest.mark.parametrize("sources,top_k,radius,stride", [
    (8, 3, 7, 2), (6, 3, 5, 1), (3, 3, 5, 1), (3, 1, 3, 1), (2, 3, 7, 2), (2, 2, 2, 1), (1, 3, 5, 1)])
def test_solve_equals_its_half_passes_where_smaller_launches_end(hp, scene_mod, precision, w, h, spread, sources,
                                                                 top_k, radius, stride):
    sms, tiles, iterations = _sms(), ((w + 63) // 64) * ((h + 7) // 8), 4
    form = _form(precision, radius, stride, sources, tiles, sms)
    if sms == 148:  # 234 tiles spread no better in halves, 342 do
        samples = ((2 * radius) // stride + 1) ** 2 * sources
        assert form in (("whole",) if samples <= WHOLE_SAMPLES[precision] else ("units", "split") if spread else ("units",))
    s = scene_mod.multi_object(seed=5, w=w, h=h, n_views=9, n_src=8, f=0.8 * w)
    params = hp.default_params(radius=radius, stride=stride, top_k=top_k, precision=precision)
    with hp.Context(0) as ctx:
        ids = [ctx.upload(v.image) for v in s.views]
        job = _job(hp, s, ids, 4, sources, iterations)
        whole, d, n, c = hp.host_maps(h, w)
        ctx.solve([job], params, [whole])
        maps, d2, n2, c2 = hp.host_maps(h, w)
        ctx.init_hypotheses(job, params, maps)
        ctx.ncc_cost(job, params, maps)
        for it in range(iterations):
            for color in (0, 1):
                ctx.propagate_pass(job, params, maps, it, color)
    assert np.array_equal(d, d2) and np.array_equal(n, n2) and np.array_equal(c, c2)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("radius,stride,sources", [(1, 1, 3), (3, 2, 4), (4, 2, 3), (5, 1, 2), (7, 2, 6), (7, 1, 2)])
def test_persistent_launches_of_many_tiles(hp, small, precision, radius, stride, sources):
    """Past 8 tiles an SM, persistent launches take their kernels for many tiles: plan and server."""
    s, ctx, ids = small
    k = 8 * _sms() // TILES + 1
    assert TILES * k > 8 * _sms()
    params = hp.default_params(radius=radius, stride=stride, precision=precision)
    job = _job(hp, s, ids, 4, sources, 3)
    maps, d, n, c = hp.host_maps(H, W)
    ctx.solve([job], params, [maps])
    outs = [hp.host_maps(H, W) for _ in range(k)]
    with hp.Plan(ctx, [job] * k, params, [o[0] for o in outs],
                 hp.plan_options(schedule=hp.SCHEDULE_PERSISTENT)) as plan:
        plan.run()
    served = [hp.host_maps(H, W) for _ in range(k)]
    with hp.Server(ctx, params) as server:
        for o in served:
            server.submit(job, o[0])
        server.drain()
        server.poll()
    for _, a, b, e in outs + served:
        assert np.array_equal(a, d) and np.array_equal(b, n) and np.array_equal(e, c)
