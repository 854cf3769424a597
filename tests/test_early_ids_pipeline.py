"""Voxel-id and hit-node images that leave after the primary pass, behind frames
that nobody waited for: in a pipelined renderer both frame sets write the same
images, and a frame without outputs may still be on its way when the next one's
primary pass runs.  The ids read back are those of the frame's own GBuffer,
after any number of such frames (either frame set), with and without
asynchronous outputs asked for.  Exact."""
import dataclasses

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("async_before", [False, True])
@pytest.mark.parametrize("want", [("voxel_id",), ("hit_node", "rgb"), ("gbuffer", "voxel_id", "hit_node")])
def test_ids_behind_frames_in_flight(ve, want, async_before):
    words, depth, mats, _, fc = helpers.small_setup()
    eye, d = helpers.workloads().small_camera()
    fc.width, fc.height, fc.bounces = 1024, 768, 1
    cams = [ve.camera_ubo(eye + np.float32(3 * k), d, 70.0, 1024 / 768) for k in range(3)]
    slow = dataclasses.replace(fc, spp=4, bounces=4, flags=ve.FRAME_ASYNC_OUTPUTS if async_before else 0)
    with ve.Renderer(hash_log2=18, pipeline=True) as r:
        r.set_materials(mats)
        sid = r.upload_scene(words, depth)
        true = [r.render(sid, c, fc, outputs=("gbuffer",))["gbuffer"] for c in cams]
        assert not np.array_equal(true[0], true[1]) and not np.array_equal(true[1], true[2])
        for k in range(12):
            for _ in range(1 + k % 3):
                r.render(sid, cams[(k + 1) % 3], slow, outputs=())
            out = r.render(sid, cams[k % 3], fc, outputs=want)
            for name, channel in (("voxel_id", 3), ("hit_node", 2)):
                if name in want:
                    assert np.array_equal(out[name], true[k % 3][..., channel]), (k, name)
