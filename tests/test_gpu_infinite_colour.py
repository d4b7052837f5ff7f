"""A Gaussian of infinite colour is blended into the pixels that take it and leaves
the others of its tile as they were: the image equals the oracle's, infinities
included, in every form of the forward (an 8x8 block per CTA, with and without
checkpoints, the other tile shapes). Negative infinity and NaN count as black."""
import numpy as np
import pytest

from _parity import assert_forward_parity, oracle_forward, run_gpu_forward
from rustscan_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,tile", [(64, 48, (16, 16)), (400, 300, (16, 16)), (1056, 1040, (16, 16)),
                                      (64, 48, (8, 8)), (64, 48, (32, 8))])
def test_infinite_colour(gsr_ctx_factory, w, h, tile):
    from rustscan_b200 import host_splats_to_device

    sc = S.small_scene(n=4000, degree=0, width=w, height=h, seed=7)
    for i, (value, channel) in enumerate([(np.inf, 0), (np.inf, 1), (np.inf, 2), (-np.inf, 0), (np.nan, 1)]):
        sc.sh[i::400, 0, channel] = value
    cam = sc.cameras[0]
    ctx = gsr_ctx_factory(max_splats=sc.n, max_pixels=w * h, tile=tile)
    _, g = run_gpu_forward(ctx, host_splats_to_device(sc), [cam])
    o = oracle_forward(sc, cam, tile=tile)
    assert np.isposinf(o.image[..., :3]).any() and np.isfinite(o.image[..., :3]).any()
    assert_forward_parity(g[0], o)
