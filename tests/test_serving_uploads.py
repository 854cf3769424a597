"""Scenes are uploaded, edited and released on a context whose server has
requests in flight: the server's worker reads nothing of the host's scene table,
which these calls extend.  Images equal those rendered before."""
import dataclasses

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def test_scene_calls_beside_a_running_server(ve):
    words, depth, mats, cam, fc = helpers.small_setup()
    fc = dataclasses.replace(fc, width=320, height=240, spp=4, bounces=3)
    rng = np.random.default_rng(11)
    deep = helpers.random_voxels(rng, 6, 0.02)
    deep[:, :3] += 1000  # depth 11: no table to the leaves
    eye = np.array([1032.0, 1090.0, 980.0], np.float32)
    deep_cam = ve.camera_ubo(eye, ve.look_at(eye, (1032, 1032, 1032)), 60.0, 320 / 240)
    with ve.Renderer(hash_log2=16) as r:
        r.set_materials(mats)
        jobs = [(r.upload_scene(words, depth), cam, fc), (r.build_scene(deep, 11), deep_cam, fc)]
        ref = [r.render(*j, outputs=("voxel_id",))["voxel_id"].copy() for j in jobs]
        assert all((v != 0).sum() > 1000 for v in ref)
        with ve.Server(r, pixel_capacity=1 << 20, path_capacity=1 << 22, max_requests=8) as srv:
            ids, extra = [], []
            for k in range(60):
                ids.append((k % 2, srv.submit(*jobs[k % 2])))
                extra.append(r.upload_scene(words, depth, keep_normals=bool(k % 3)))
                if k % 4 == 3:
                    r.release_scene(extra.pop(0))
            for which, i in ids:
                assert np.array_equal(srv.wait(i)["voxel_id"], ref[which])
