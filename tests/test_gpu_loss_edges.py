"""Loss gradient at the edges of the 32x32 tiles: images whose last row or column
is the first of a tile, the last of one or in between, so that the border's
weights and the zero halo fall on every side of a tile's boundary."""
import numpy as np
import pytest

from _parity import assert_grad_close
from oracle import oracle as O
from rustscan_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hw", [(32, 33), (33, 32), (36, 37), (37, 38), (65, 31), (31, 65), (6, 100), (70, 5), (101, 97)])
def test_loss_gradient_at_tile_edges(gsr_ctx_factory, hw):
    import torch

    H, W = hw
    rng = np.random.default_rng(H * 1000 + W)
    pred = rng.uniform(0, 1, (H, W, 4)).astype(np.float32)
    tgt = np.clip(pred[..., :3] + rng.normal(0, 0.1, (H, W, 3)), 0, 1).astype(np.float32)
    cam = S.camera_from_rt(np.eye(3), np.zeros(3), 50, 50, W / 2, H / 2, W, H)
    ctx = gsr_ctx_factory(max_splats=16, max_pixels=H * W)
    loss, vp = ctx.loss(torch.as_tensor(pred, device="cuda"), torch.as_tensor(tgt, device="cuda"), [cam])
    torch.cuda.synchronize()
    ol, ov = O.loss(pred, tgt)
    assert abs(float(loss[0]) - ol) <= 1e-5 * max(1.0, abs(ol))
    assert_grad_close(vp.cpu().numpy(), ov, what="d loss / d pred")
