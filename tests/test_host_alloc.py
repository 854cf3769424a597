"""Pinned blocks of ve_host_alloc: a forked child keeps its own copy of a result
whose block the parent goes on using (as of an ordinary array), and only blocks
can be freed, once."""
import ctypes
import os
import time

import numpy as np
import pytest

import helpers


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore:.*fork.*")
@pytest.mark.parametrize("size", [(301, 200), (1024, 768)])
def test_a_forked_child_keeps_its_copy(ve, size):
    words, depth, mats, cam, fc = helpers.small_setup()
    fc.width, fc.height = size
    eye, d = helpers.workloads().small_camera()
    other = ve.camera_ubo(eye + np.float32(9), d, 70.0, size[0] / size[1])
    n = size[0] * size[1] * 4
    with ve.Renderer(hash_log2=16) as r:
        r.set_materials(mats)
        sid = r.upload_scene(words, depth)
        first, second = (r.render(sid, c, fc, outputs=("voxel_id",))["voxel_id"].copy() for c in (cam, other))
        assert not np.array_equal(first, second)
        p = ctypes.c_void_p()
        assert ve.load_library().ve_host_alloc(n, ctypes.byref(p)) == ve.VE_OK
        image = np.frombuffer((ctypes.c_char * n).from_address(p.value), np.uint32).reshape(size[1], size[0])
        r.render_into(sid, cam, fc, {"voxel_id": image})
        read, write = os.pipe()
        pid = os.fork()
        if pid == 0:  # host memory only, and no way back into the test
            code = 3
            try:
                os.read(read, 1)
                code = 0 if np.array_equal(image, first) else 4
            finally:
                os._exit(code)
        try:
            image[0, 0] ^= 1  # by the host and by the GPU
            r.render_into(sid, other, fc, {"voxel_id": image})
            assert np.array_equal(image, second)
        finally:
            os.write(write, b"x")
            end = time.monotonic() + 30
            done, status = os.waitpid(pid, os.WNOHANG)
            while not done and time.monotonic() < end:
                time.sleep(0.01)
                done, status = os.waitpid(pid, os.WNOHANG)
            if not done:
                os.kill(pid, 9)
                os.waitpid(pid, 0)
        assert done and os.WIFEXITED(status) and os.WEXITSTATUS(status) == 0
        del image
        assert ve.load_library().ve_host_free(p) == ve.VE_OK
        assert ve.load_library().ve_host_free(p) != ve.VE_OK  # no longer a block


@pytest.mark.gpu
def test_blocks_made_and_freed_by_a_fresh_thread(ve):
    """A thread that has made no CUDA call takes a renderer's device."""
    import threading

    words, depth, mats, cam, fc = helpers.small_setup()
    fc.width, fc.height = 300, 200
    rc = []

    def work():
        p = ctypes.c_void_p()
        rc.append(ve.load_library().ve_host_alloc(300 * 200 * 4, ctypes.byref(p)))
        image = np.frombuffer((ctypes.c_char * (300 * 200 * 4)).from_address(p.value), np.uint32).reshape(200, 300)
        r.render_into(sid, cam, fc, {"voxel_id": image})
        rc.append(np.array_equal(image, want))
        del image
        t = threading.Thread(target=lambda: rc.append(ve.load_library().ve_host_free(p)))
        t.start()
        t.join(60)

    with ve.Renderer(hash_log2=16) as r:
        r.set_materials(mats)
        sid = r.upload_scene(words, depth)
        want = r.render(sid, cam, fc, outputs=("voxel_id",))["voxel_id"].copy()
        t = threading.Thread(target=work)
        t.start()
        t.join(60)
    assert rc == [ve.VE_OK, True, ve.VE_OK]
