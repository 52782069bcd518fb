"""Fusion past the line where its CTAs take four steps (1024 pixels): the engine equals the oracle bit for
bit (tolerance 0, the same FP32 operation order) for views that end inside a CTA's second, third and fourth
step, on host and device maps, and on one context whose workspace serves calls of other layouts between."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import cam_of
from test_fuse import _gt_maps, _same

pytestmark = pytest.mark.gpu

SIZES = [(1033, 601, 3), (517, 303, 1), (519, 305, 1)]  # width, height, views; pixels % 1024: 289, 1003, 599


@pytest.fixture(scope="module")
def uneven(scene_mod):
    """Five views of three sizes of one scene: maps and cameras."""
    maps, cams, at = [], [], 0
    for w, h, n in SIZES:
        s = scene_mod.plane_sphere(w=w, h=h)
        m = _gt_maps(s, noise=0.001, seed=w)
        maps += m[at:at + n]
        cams += [cam_of(s, i) for i in range(at, at + n)]
        at += n
    return maps, cams


def _fuse(hp, ctx, maps, cams, neighbors=None, device=False, **kw):
    import torch
    cols = list(zip(*maps))
    if device:
        cols = [[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in c] for c in cols]
    cloud = ctx.fuse([hp.make_camera(*c) for c in cams], cols[0], cols[1], cols[2], cols[3], neighbors,
                     hp.fuse_params(**kw))
    out = (cloud.positions, cloud.normals, cloud.colors)
    return tuple(a.cpu().numpy() for a in out) if device else out


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("kw", [{}, {"min_views": 1, "min_confidence": 0.7}, {"min_views": 3, "max_depth_rel": 0.05}])
def test_four_step_ctas_match_the_oracle(hp, po, uneven, device, kw):
    import torch
    maps, cams = uneven
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert sum(m[0].size for m in maps) >= 2 * sms * 6 * 1024
    with hp.Context(0) as ctx:
        got = _fuse(hp, ctx, maps, cams, device=device, **kw)
    want = po.fuse(maps, cams, **kw)
    assert len(want[0]) > 50_000 and _same(got, want)


def test_a_context_serves_large_and_small_calls_in_turn(hp, po, scene_mod, uneven):
    maps, cams = uneven
    s = scene_mod.plane_sphere(w=97, h=61)
    small, small_cams = _gt_maps(s, noise=0.001, seed=2), [cam_of(s, i) for i in range(len(s.views))]
    nb = [[4, 1], [3, 0, 2], [0], [2, 1], []]
    large_want, large_nb_want = po.fuse(maps, cams), po.fuse(maps, cams, neighbors=nb, min_views=1)
    small_want, two_want = po.fuse(small, small_cams), po.fuse(small[:2], small_cams[:2])
    with hp.Context(0) as ctx:
        for _ in range(2):
            assert _same(_fuse(hp, ctx, small, small_cams), small_want)
            assert _same(_fuse(hp, ctx, maps, cams), large_want)
            assert _same(_fuse(hp, ctx, small[:2], small_cams[:2]), two_want)
            assert _same(_fuse(hp, ctx, maps, cams, neighbors=nb, min_views=1), large_nb_want)
    assert len(small_want[0]) and len(two_want[0]) and len(large_nb_want[0])
