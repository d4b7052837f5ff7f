"""The training step's 2D-gradient statistic is the mean of the absolute mean
gradient's components, divided with correct rounding: equal, bit for bit, to
that of the gradients which the same step's backward returns."""
import numpy as np
import pytest

from rustscan_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [0, 3])
def test_grad_2d_division(gsr_ctx_factory, degree):
    import torch

    from rustscan_b200 import Trainer, host_splats_to_device

    sc = S.small_scene(n=3000, degree=degree, width=96, height=72, seed=60 + degree)
    target = torch.rand(96 * 72 * 3, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    ctx = gsr_ctx_factory(max_splats=sc.n, max_pixels=96 * 72, deterministic=True)
    splats = host_splats_to_device(sc)
    flat, _, _ = ctx.render_forward(splats, sc.cameras)
    _, v = ctx.loss(flat, target, sc.cameras)
    g = np.abs(ctx.render_backward(splats, v)["v_transforms"].cpu().numpy()[:, :3])
    trainer = Trainer(ctx, splats)
    trainer.train_step(sc.cameras, target, 1)
    want = (g[:, 0] + g[:, 1] + g[:, 2]) / np.float32(3.0)
    assert np.count_nonzero(want) > 500
    np.testing.assert_array_equal(trainer.densify[0].cpu().numpy(), want)
