"""Claimed cache entries join their table's list once each, also where the lanes
of a warp claim from several scenes' tables at once and after probe loops of
different lengths: a batch of small views over three scenes, whose paths mix in
the shading warps, leaves the same counts and decayed sums when the decay visits
the list (large table) as when it sweeps the table (small one).  An entry missing
from the list would keep its sums, one listed twice would lose half of them."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def caches(ve, hash_log2, frames, size):
    words, depth, mats, _, _ = helpers.small_setup()
    eye, d = helpers.workloads().small_camera()
    with ve.Renderer(hash_log2=hash_log2, hash_probes=256) as r:
        r.set_materials(mats)
        sids = [r.upload_scene(words, depth) for _ in range(3)]
        dropped = 0
        for f in range(frames):
            views = []
            for k in range(36):
                cam = ve.camera_ubo(eye + np.float32([0.5 * k, 0.0, 0.25 * f]), d, 50.0 + k, size[0] / size[1])
                views.append((sids[k % 3], cam,
                              ve.FrameConfig(width=size[0], height=size[1], spp=2, bounces=2, frame_index=f,
                                             decay=0.5)))
            r.render_batch(views, outputs=())
            dropped += r.stats()["deposits_dropped"]
        return [r.cache_dump(s) for s in sids], dropped


@pytest.mark.parametrize("size", [(7, 5), (16, 16), (33, 9)])
@pytest.mark.parametrize("frames", [1, 4])
def test_mixed_scenes_in_a_warp(ve, size, frames):
    listed, dropped = caches(ve, 18, frames, size)
    assert not dropped
    used = max(len(v) for v, _, _ in listed)
    assert 100 < used <= (1 << 18) // 4
    small = max(8, (min(len(v) for v, _, _ in listed) * 2).bit_length())  # at most half full, above a quarter
    swept, dropped = caches(ve, small, frames, size)
    assert not dropped
    for (v, c, x), (v2, c2, x2) in zip(listed, swept):
        assert np.array_equal(v, v2) and np.array_equal(c, c2)
        # float sums of a few hundred terms of one sign in another order
        np.testing.assert_allclose(x, x2, rtol=1e-4, atol=1e-6)
