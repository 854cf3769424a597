"""k_shade_rows with two, three and four rows of paths per warp (ordering across
rows, the next row's state copied in ahead, one append for all rows) against
k_shade: views whose rays nearly all hit, alone below the path slots from which
k_shade_rows is taken and together above them, give the same GBuffer and the
same deposit for every path, bit for bit, and the same deposit counts.  A smaller
grid (fewer warps) reaches the same rows with fewer paths."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

SLOTS = 3 << 19  # path slots of a batch from which k_shade_rows is taken
SMS, WARPS_PER_BLOCK, BLOCKS = 148, 8, 4


def rows(live, blocks):
    return min(max(live // (SMS * (blocks or BLOCKS) * WARPS_PER_BLOCK * 96), 1), 4)


@pytest.mark.parametrize("blocks,sizes,want", [
    (1, [(601, 401)], 2), (1, [(701, 503)], 3), (1, [(811, 607)], 4), (1, [(1009, 997)], 4),
    (0, [(1021, 953)], 2), (0, [(1009, 701), (997, 809)], 3), (0, [(1021, 947), (1013, 1019)], 4)])
@pytest.mark.parametrize("bounces", [1, 3])
def test_rows_against_k_shade(ve, blocks, sizes, want, bounces):
    words, depth, mats, cam, small = helpers.small_setup()
    L = float(1 << depth)
    small.width, small.height, small.spp, small.bounces, small.flags = 131, 97, 3, bounces, ve.FRAME_PATH_RGB
    views = [(0, cam, small)]
    for k, (w, h) in enumerate(sizes):  # from above the middle, straight down: ground in every pixel
        eye = np.array([L / 2 + 3 * k, 120.0, L / 2 - 2 * k], np.float32)
        down = ve.camera_ubo(eye, ve.look_at(eye, (L / 2, 0.0, L / 2 + 1.0)), 40.0, w / h)
        views.append((1, down, ve.FrameConfig(width=w, height=h, spp=1, bounces=bounces, primary_controlchecks=200,
                                              bounce_controlchecks=200, flags=ve.FRAME_PATH_RGB)))
    slots = sum(f.width * f.height * f.spp for _, _, f in views)
    if slots < SLOTS:  # paths of pixels that hit nothing
        away = ve.camera_ubo([64.0, 200.0, -40.0], [0.0, 1.0, 0.0], 70.0, 1.0)
        views.append((1, away, ve.FrameConfig(width=1024, height=-(-(SLOTS - slots) // 1024), spp=1, bounces=bounces)))
    with ve.Renderer(hash_log2=18) as r:
        r.set_materials(mats)
        sids = [r.upload_scene(words, depth) for _ in range(2)]
        r.set_launch_config(0, blocks, 0)
        alone, live = [], 0
        for s, c, f in views[: 1 + len(sizes)]:
            assert f.width * f.height * f.spp < SLOTS
            alone.append({k: v.copy() for k, v in r.render(sids[s], c, f, outputs=("gbuffer", "path_rgb")).items()})
            live += int((alone[-1]["gbuffer"][..., 3] != 0).sum()) * f.spp
        assert rows(live * 0.97, blocks) == want  # (paths that end at their first hit are few)
        counts = [r.cache_dump(s)[:2] for s in sids]
        for s in sids:
            r.cache_reset(s)
        outs = r.render_batch([(sids[s], c, f) for s, c, f in views], outputs=("gbuffer", "path_rgb"))
        for o, a in zip(outs, alone):
            assert np.array_equal(o["gbuffer"], a["gbuffer"])
            assert np.array_equal(o["path_rgb"].view(np.uint32), a["path_rgb"].view(np.uint32))
        for s, (vids, n) in zip(sids, counts):
            v, m, _ = r.cache_dump(s)
            assert np.array_equal(v, vids) and np.array_equal(m, n) and n.sum() > 1000
