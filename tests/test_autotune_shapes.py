"""The autotuner tries only shapes that the views' kernels can take: trace
blocks per SM above an instance's occupancy are clamped to it, so a trial of
them repeats a shape and noise would pick.  A shape left at the occupancy
maximum leaves every other instance at its own."""
import pytest

import helpers

pytestmark = pytest.mark.gpu

MAX_ONE, MAX_ANY = 8, 6  # resident trace blocks per SM: one flat scene; other batches


@pytest.mark.parametrize("views", ["one", "two", "emissive"])
def test_trials_below_the_occupancy_or_the_maximum(ve, views):
    words, depth, mats, cam, fc = helpers.small_setup()
    fc.width, fc.height, fc.spp, fc.bounces = 160, 120, 1, 1
    if views == "emissive":
        fc.flags = ve.FRAME_EMISSIVE
    with ve.Renderer(hash_log2=16) as r:
        r.set_materials(mats)
        sids = [r.upload_scene(words, depth) for _ in range(2)]
        batch = [(sids[0], cam, fc)] + ([(sids[1], cam, fc)] if views == "two" else [])
        seen = set()
        for _ in range(6):
            r.set_launch_config()
            best = r.autotune(batch, frames_per_trial=1)
            assert r.launch_config() == best
            assert 1 <= best["trace_blocks_per_sm"] <= MAX_ONE and 1 <= best["shade_blocks_per_sm"] <= 8
            seen.add(best["trace_blocks_per_sm"])
        if views == "two":
            assert not seen & set(range(MAX_ANY, MAX_ONE)), seen
