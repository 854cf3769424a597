"""The shade kernel of large batches (k_shade_rows) against the other one: a view
rendered alone (k_shade) and beside another that takes the batch to, just below
and above the number of path slots from which k_shade_rows is taken gives the
same GBuffer and the same deposit for every path, bit for bit, and the same
deposit counts in the cache; path counts off the rows' multiples included."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

SLOTS = 3 << 19  # path slots of a batch from which k_shade_rows is taken


@pytest.mark.parametrize("extra", [-1, 0, 1, 33, 4097])
@pytest.mark.parametrize("bounces", [0, 1, 4])
def test_view_alone_and_in_a_large_batch(ve, extra, bounces):
    words, depth, mats, cam, fc = helpers.small_setup()
    fc.width, fc.height, fc.spp, fc.bounces, fc.flags = 131, 97, 3, bounces, ve.FRAME_PATH_RGB
    fill = SLOTS + extra - fc.width * fc.height * fc.spp  # one-sample paths, mostly of pixels that hit nothing
    w = 1031
    h = fill // w
    rest = fill - w * h
    away = ve.camera_ubo([64.0, 200.0, -40.0], [0.0, 1.0, 0.0], 70.0, 1.0)
    views = [(0, cam, fc), (1, away, ve.FrameConfig(width=w, height=h, spp=1, bounces=bounces))]
    if rest:
        views.append((1, cam, ve.FrameConfig(width=rest, height=1, spp=1, bounces=bounces)))
    with ve.Renderer(hash_log2=16) as r:
        r.set_materials(mats)
        sids = [r.upload_scene(words, depth) for _ in range(2)]
        alone = r.render(sids[0], cam, fc, outputs=("gbuffer", "path_rgb"))
        vids, counts, _ = r.cache_dump(sids[0])
        r.cache_reset(sids[0])
        outs = r.render_batch([(sids[s], c, f) for s, c, f in views], outputs=("gbuffer", "path_rgb"))
        vids2, counts2, _ = r.cache_dump(sids[0])
    assert np.array_equal(outs[0]["gbuffer"], alone["gbuffer"])
    assert np.array_equal(outs[0]["path_rgb"].view(np.uint32), alone["path_rgb"].view(np.uint32))
    assert np.array_equal(vids, vids2) and np.array_equal(counts, counts2) and counts.sum() > 1000
