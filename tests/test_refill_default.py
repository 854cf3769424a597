"""The trace refill threshold left at its default (one per kind of walk) against
set ones: the configuration reads back, and frames of a flat scene, of a deep
one (general walk) and of both in a batch keep every path's deposit."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def test_default_and_set_thresholds(ve):
    words, depth, mats, cam, fc = helpers.small_setup()
    fc.width, fc.height, fc.spp, fc.bounces, fc.flags = 97, 63, 2, 2, ve.FRAME_PATH_RGB
    rng = np.random.default_rng(7)
    L = 1 << 11
    v = np.zeros((60000, 4), np.uint32)
    v[:, 0], v[:, 2] = rng.integers(900, 1100, 60000), rng.integers(900, 1100, 60000)
    v[:, 1] = 1000 + (v[:, 0] // 7 + v[:, 2] // 5) % 9
    v[:, 3] = rng.integers(1, 9, 60000)
    eye = np.array([860.0, 1060.0, 870.0], np.float32)
    deep_cam = ve.camera_ubo(eye, ve.look_at(eye, (1000, 1000, 1000)), 60.0, 97 / 63)
    assert v[:, :3].max() < L
    with ve.Renderer(hash_log2=16) as r:
        r.set_materials(mats)
        flat, deep = r.upload_scene(words, depth), r.build_scene(v, 11)
        views = [(flat, cam, fc), (deep, deep_cam, fc)]
        ref = None
        for threshold in (0, 1, 20, 24, 32, 0):
            r.set_launch_config(0, 0, threshold)
            assert r.launch_config()["refill_threshold"] == (threshold or 24)
            outs = [r.render(*w, outputs=("gbuffer", "path_rgb")) for w in views]
            outs += r.render_batch(views, outputs=("gbuffer", "path_rgb"))
            got = [o[k].view(np.uint32) for o in outs for k in ("gbuffer", "path_rgb")]
            assert all((o["gbuffer"][..., 3] != 0).sum() > 500 for o in outs)
            if ref is None:
                ref = [g.copy() for g in got]
            assert all(np.array_equal(a, b) for a, b in zip(got, ref)), threshold
