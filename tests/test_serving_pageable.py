"""Requests of one size that finish in the same step, into pageable arrays above
the driver's staging size: the worker's copies wait for one another's completion
calls while the program waits for the requests in turn.  Nothing waits for good,
and the images are the plain render's."""
import dataclasses

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("requests", [8, 40])
def test_waiting_while_pageable_copies_run(ve, requests):
    words, depth, mats, cam, fc = helpers.small_setup()
    fc = dataclasses.replace(fc, width=320, height=240, spp=2, bounces=2)
    with ve.Renderer(hash_log2=16) as r:
        r.set_materials(mats)
        sid = r.upload_scene(words, depth)
        ref = r.render(sid, cam, fc, outputs=("voxel_id",))["voxel_id"].copy()
        with ve.Server(r, pixel_capacity=1 << 20, path_capacity=1 << 22, max_requests=8) as srv:
            ids = [srv.submit(sid, cam, fc) for _ in range(requests)]
            for i in ids:
                assert np.array_equal(srv.wait(i, timeout_ms=20000)["voxel_id"], ref)
