"""Voxel-id and hit-node images that leave after the primary pass (large plain
frames into pinned arrays) are the GBuffer's fields: around the size from which
they do, in batches, with and without frame pipelining, for frames that do not
qualify (no bounce) and after asynchronous frames on the same buffers.  Exact."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

WANT = ("gbuffer", "voxel_id", "hit_node", "rgb")


def check(out):
    assert np.array_equal(out["voxel_id"], out["gbuffer"][..., 3])
    assert np.array_equal(out["hit_node"], out["gbuffer"][..., 2])
    assert out["voxel_id"].any() and np.isfinite(out["rgb"]).all()


@pytest.mark.parametrize("pipeline", [False, True])
@pytest.mark.parametrize("size", [(512, 511), (512, 512), (513, 512), (724, 725), (1023, 1025)])
def test_ids_equal_the_gbuffer(ve, size, pipeline):
    words, depth, mats, cam, fc = helpers.small_setup()
    wl = helpers.workloads()
    eye, d = wl.small_camera()
    with ve.Renderer(hash_log2=18, pipeline=pipeline) as r:
        r.set_materials(mats)
        sid = r.upload_scene(words, depth)
        fc.width, fc.height = size
        for k, bounces in enumerate((1, 1, 0, 2)):
            fc.bounces, fc.frame_index = bounces, k
            cam = ve.camera_ubo(eye + np.float32(k), d, 70.0, size[0] / size[1])
            check(r.render(sid, cam, fc, outputs=WANT))
            only = r.render(sid, cam, fc, outputs=("hit_node",))["hit_node"]
            assert np.array_equal(only, r.render(sid, cam, fc, outputs=WANT)["gbuffer"][..., 2])
        small = ve.FrameConfig(width=64, height=48, spp=1, bounces=1)
        views = [(sid, cam, fc), (sid, cam, small), (sid, cam, fc)]
        for out in r.render_batch(views, outputs=WANT):
            check(out)


def test_ids_after_asynchronous_frames(ve):
    torch = pytest.importorskip("torch")
    words, depth, mats, cam, fc = helpers.small_setup()
    fc.width, fc.height = 1024, 768
    with ve.Renderer(hash_log2=18, pipeline=True) as r:
        r.set_materials(mats)
        sid = r.upload_scene(words, depth)
        ids = [torch.zeros((768, 1024), dtype=torch.int32).pin_memory().numpy().view(np.uint32) for _ in range(3)]
        plain = r.render(sid, cam, fc, outputs=WANT)
        fc.flags = ve.FRAME_ASYNC_OUTPUTS
        for k in range(3):
            r.render_into(sid, cam, fc, {"voxel_id": ids[k]})
        fc.flags = 0
        out = r.render(sid, cam, fc, outputs=WANT)
        r.synchronize()
    check(out)
    for a in (*ids, out["voxel_id"]):
        assert np.array_equal(a, plain["voxel_id"])
