"""Fusion at the edges of its CTAs (1024 pixels of one view) and of its count scan: the engine equals
the oracle bit for bit (tolerance 0, the same FP32 operation order) for views one pixel short of, at and
past whole CTAs, neighbour lists in any order and with repeats, and every number of views required."""
from __future__ import annotations

import numpy as np
import pytest

from test_fuse import _engine, _gt_maps, _same
from conftest import cam_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(33, 31), (32, 32), (41, 25), (64, 48), (8, 3)])
@pytest.mark.parametrize("min_views", [1, 2, 4])
def test_engine_matches_oracle_at_block_edges(hp, po, scene_mod, w, h, min_views):
    s = scene_mod.plane_sphere(w=w, h=h)
    maps = _gt_maps(s, noise=0.001, seed=w)
    nb = [[4, 1, 3, 1], [3, 0, 2], [0, 4, 1, 1, 3], [], [2, 3, 0, 1]]
    kw = dict(min_views=min_views, max_depth_rel=0.05, max_reproj_px=3.0, min_normal_cos=0.0)
    with hp.Context(0) as ctx:
        got = _engine(hp, ctx, s, maps, neighbors=nb, **kw)
    want = po.fuse(maps, [cam_of(s, i) for i in range(len(maps))], neighbors=nb, **kw)
    assert _same(got, want)
    assert min_views > 2 or len(want[0]) > 0


def test_count_scan_past_one_tile(hp, po, scene_mod):
    """More CTAs than the scan takes at once (8192 counts): many small views, each its own CTA."""
    s = scene_mod.plane_sphere(w=8, h=6)
    maps = (_gt_maps(s, noise=0.001, seed=1) * 1700)[:8300]
    cams = [cam_of(s, i % len(s.views)) for i in range(len(maps))]
    nb = [[] for _ in maps]
    import types
    fake = types.SimpleNamespace(views=[types.SimpleNamespace(cam=s.views[i % len(s.views)].cam)
                                        for i in range(len(maps))])
    with hp.Context(0) as ctx:
        got = _engine(hp, ctx, fake, maps, neighbors=nb, min_views=1)
    want = po.fuse(maps, cams, neighbors=nb, min_views=1)
    assert len(want[0]) > 8192 and _same(got, want)
