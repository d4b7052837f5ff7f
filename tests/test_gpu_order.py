"""Depth order and intersection offsets at the edges of the one-launch sort
of small views: chunk boundaries of its 16 CTAs, a single Gaussian, equal
depths (ties go to the lower index), views of uneven visible counts in one
launch (one of them empty), and the first size past its limit, which takes
the radix passes. Bit-exact against the oracle."""
import numpy as np
import pytest

from _parity import assert_forward_parity, oracle_forward, run_gpu_forward
from rustscan_b200 import scenes as S

pytestmark = pytest.mark.gpu

LIMIT = 16 * 1024 * 13


def _scene(n, depths):
    rng = np.random.Generator(np.random.PCG64(5 + n))
    tr = np.zeros((n, 10), np.float32)
    tr[:, 0:2] = rng.uniform(-1.0, 1.0, (n, 2))
    tr[:, 2] = {"spread": rng.uniform(-1.0, 1.0, n), "equal": 0.25,
                "few": rng.integers(0, 3, n) * np.float32(0.5)}[depths]
    tr[:, 3] = 1.0
    tr[:, 7:10] = -6.0
    sh = rng.uniform(-1.0, 1.0, (n, 1, 3)).astype(np.float32)
    cams = [S.camera_from_rt(np.eye(3), np.array([x, 0.0, 3.0]), 64, 64, 32, 32, 64, 64) for x in (0.0, 1.2, 40.0)]
    return S.Scene(tr, sh, rng.standard_normal(n).astype(np.float32), 0, cams, "order")


@pytest.mark.parametrize("n,depths", [(1, "spread"), (1023, "equal"), (1025, "few"), (16384, "spread"),
                                      (16385, "few"), (32769, "spread"), (65537, "equal"), (131073, "few"),
                                      (180225, "spread"), (LIMIT, "spread"), (LIMIT + 1, "few")])
def test_depth_order_edges(gsr_ctx_factory, n, depths):
    from rustscan_b200 import host_splats_to_device

    sc = _scene(n, depths)
    ctx = gsr_ctx_factory(max_splats=n, max_views=3, max_pixels=64 * 64)
    _, g = run_gpu_forward(ctx, host_splats_to_device(sc), sc.cameras)
    for v, cam in enumerate(sc.cameras):
        assert_forward_parity(g[v], oracle_forward(sc, cam))
    assert int(g[2]["counts"][0]) == 0
