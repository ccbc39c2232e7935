"""GPU: detection batches in five to eight parts (workspaces and host threads), with
parts of unequal size and images whose bytes start at any address: every image's
features are the oracle's, in image order, and those of the image alone."""
import numpy as np
import pytest

import oracle as O
from skylens_match import features as F
from skylens_match import synth
from test_gpu_features import check_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w,h", [(15, 65, 47), (16, 64, 48), (17, 97, 61), (23, 49, 33), (24, 83, 59), (25, 63, 45)])
@pytest.mark.parametrize("rgb", [True, False])
def test_batches_in_five_to_eight_parts(matcher, n, w, h, rgb):
    views = synth.scene_views(n, w, h, seed=n)
    gray = np.stack([O.gray_from_rgb8(v) for v in views])
    cfg = F.detector_config(upscale_below=0 if n % 2 else 800)
    got = F.detect_and_describe(matcher, views if rgb else gray, cfg)
    assert len(got) == n
    for k in range(n):
        check_equal(got[k], gray[k], cfg)
    alone = F.detect_and_describe(matcher, (views if rgb else gray)[n - 1], cfg)[0]
    assert np.array_equal(alone[0], got[n - 1][0]) and np.array_equal(alone[1], got[n - 1][1])
    assert sum(len(g[0]) for g in got) > n
