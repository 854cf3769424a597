"""The temporal decay visits the list of claimed cache entries while it is short
and sweeps the table otherwise: the same frames through tables on both sides of
that line leave the same counts and sums (a lane adds its deposits in the same
order; atomics of different warps may swap, so the sums may differ by rounding:
a few hundred additions of one sign, 1e-4 relative)."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def frames(ve, hash_log2, reset=False):
    words, depth, mats, cam, fc = helpers.small_setup()
    fc.width, fc.height, fc.spp, fc.bounces, fc.decay = 72, 56, 2, 1, 0.5
    with ve.Renderer(hash_log2=hash_log2, hash_probes=256) as r:
        r.set_materials(mats)
        sid = r.upload_scene(words, depth)
        dropped = 0
        for k in range(5):
            if reset and k == 1:
                r.cache_reset(sid)  # the list is empty with the table
                for q in range(k):
                    fc.frame_index = q
                    r.render(sid, cam, fc, outputs=())
            fc.frame_index = k
            r.render(sid, cam, fc, outputs=())
            dropped += r.stats()["deposits_dropped"]
        return (*r.cache_dump(sid), dropped)


@pytest.mark.parametrize("hash_log2", [12, 13, 14, 15, 16])
@pytest.mark.parametrize("reset", [False, True])
def test_list_and_sweep_decay_alike(ve, hash_log2, reset):
    vids, counts, vals, dropped = frames(ve, hash_log2, reset)
    ref_vids, ref_counts, ref_vals, _ = frames(ve, 20)
    if dropped:
        pytest.skip("the table is too small for the frames' voxels")
    assert np.array_equal(vids, ref_vids) and np.array_equal(counts, ref_counts)
    np.testing.assert_allclose(vals, ref_vals, rtol=1e-4, atol=1e-6)


def test_both_sides_of_the_line_are_reached(ve):
    vids, _, _, dropped = frames(ve, 13)
    assert not dropped and (1 << 13) / 4 < len(vids) < (1 << 16) / 4, (len(vids), dropped)
