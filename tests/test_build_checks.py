"""ve_scene_build's checks of its voxel list run in the key pass: one wrong row
anywhere is refused with the status of the host check it replaces, and the next
build on the context is unaffected (words against OctreeCPU + Octree.set)."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

BAD = [(0, 64), (1, 64), (2, 1 << 31), (3, 0), (3, 128), (3, 0xFFFFFFFF)]  # (column, value) at depth 6


@pytest.mark.parametrize("n", [1, 255, 256, 257, 40001])
def test_wrong_rows_are_refused(ve, n):
    rng = np.random.default_rng(n)
    good = np.empty((n, 4), np.uint32)
    good[:, :3] = rng.integers(0, 64, (n, 3))
    good[:, 3] = rng.integers(1, 128, n)
    cpu = ve.OctreeCPU(6)
    cpu.insert_many(good)
    tree = ve.Octree(6)
    tree.set(cpu)
    want = tree.words()
    with ve.Renderer(hash_log2=8) as r:
        for col, value in BAD:
            for row in {0, n // 2, n - 1}:
                v = good.copy()
                v[row, col] = value
                with pytest.raises(ve.VeError) as e:
                    r.build_scene(v, 6)
                assert e.value.code == ve.VE_ERR_INVALID
        for _ in range(2):
            sid = r.build_scene(good, 6, keep_normals=True)
            got = r.download_scene(sid)
            assert np.array_equal(got, want[: got.size]) and not want[got.size:].any()
            r.release_scene(sid)
