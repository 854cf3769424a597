"""A batch in which only some views ask for asynchronous outputs is asynchronous
as a whole: none of its arrays may be a recycled pinned block, whose copy would
still be on its way when the call returns (and when the program has dropped the
array and the block serves another call)."""
import dataclasses
import types

import numpy as np
import pytest

import helpers


def bare_renderer(ve):
    """A renderer over a library whose calls do nothing (no GPU)."""
    r = object.__new__(ve.Renderer)
    r._lib = types.SimpleNamespace(ve_render=lambda *a: 0, ve_render_batch=lambda *a: 0)
    r._h = None
    return r


@pytest.mark.parametrize("flagged", [(), (0,), (2,), (0, 1, 2)])
def test_pooled_arrays_only_for_synchronous_calls(ve, monkeypatch, flagged):
    pooled = []

    def empty(shape, dtype):
        pooled.append(np.zeros(shape, dtype))
        return pooled[-1]

    monkeypatch.setattr(ve._results, "empty", empty)
    cam = np.zeros(16, np.float32)
    fcs = [ve.FrameConfig(width=200, height=100, flags=ve.FRAME_ASYNC_OUTPUTS if k in flagged else 0) for k in range(3)]
    r = bare_renderer(ve)
    outs = r.render_batch([(0, cam, fc) for fc in fcs], outputs=("voxel_id", "rgb"))
    got = [a for o in outs for a in o.values()]
    assert len(got) == 6
    assert len(pooled) == (0 if flagged else 6)
    pooled.clear()
    for k, fc in enumerate(fcs):
        r.render(0, cam, fc, outputs=("voxel_id",))
    assert len(pooled) == 3 - len(flagged)


@pytest.mark.gpu
def test_mixed_batches_dropped_and_held(ve):
    words, depth, mats, cam, fc = helpers.small_setup()
    fc.width, fc.height = 640, 480
    eye, d = helpers.workloads().small_camera()
    other = ve.camera_ubo(eye + np.float32(5), d, 70.0, 640 / 480)
    flagged = dataclasses.replace(fc, flags=ve.FRAME_ASYNC_OUTPUTS)
    with ve.Renderer(hash_log2=18) as r:
        r.set_materials(mats)
        sid = r.upload_scene(words, depth)
        a = r.render(sid, cam, fc, outputs=("voxel_id",))["voxel_id"].copy()
        b = r.render(sid, other, fc, outputs=("voxel_id",))["voxel_id"].copy()
        assert not np.array_equal(a, b)
        for _ in range(5):
            r.render_batch([(sid, cam, flagged), (sid, other, fc)], outputs=("voxel_id", "rgb"))  # dropped at once
            held = r.render(sid, cam, fc, outputs=("voxel_id",))["voxel_id"]
            mixed = r.render_batch([(sid, other, fc), (sid, cam, flagged)], outputs=("voxel_id",))
            r.synchronize()
            assert np.array_equal(held, a)
            assert np.array_equal(mixed[0]["voxel_id"], b) and np.array_equal(mixed[1]["voxel_id"], a)
