"""A large pass runs as two halves of its paths on streams of their own (PassJobN::run_halves): the paths,
and so the work counters and the image, are those of the undivided pass (timing=True runs it undivided)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("screen,spp,pool", [((512, 512), 36, 0), ((513, 511), 36, 0), ((640, 411), 64, (1 << 23) + 1)])
def test_halves_trace_the_paths_of_the_undivided_pass(require_gpu, screen, spp, pool):
    """9.4 M paths (an even and an odd number of them) in the automatic pool, and 16.8 M in one of an odd size."""
    from math_b200 import ntrace, scenes

    spec = scenes.config("n3_small")
    P = spec["projector"]
    s = scenes.build_scene(spec)
    s.set_projector(ntrace.PARALLEL, P["org"], P["dir"], P["axes"], 8.0 / max(screen), screen)
    s.build()
    got = s.render(spp, max_depth=5, seed=4, pool_paths=pool)
    img = s.image()[0]
    s.clear()
    want = s.render(spp, max_depth=5, seed=4, pool_paths=pool, timing=True)
    ref = s.image()[0]
    for k in ("paths", "rays", "shadow_rays", "facet_tests", "box_steps", "descent_levels", "shadow_facet_tests",
              "shadow_box_steps", "shadow_descent_levels"):
        assert got[k] == want[k], k
    # the same FP64 contributions per pixel in another order
    assert np.sqrt(((img - ref) ** 2).sum() / (ref ** 2).sum()) < 1e-12
