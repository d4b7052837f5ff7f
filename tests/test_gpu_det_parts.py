"""Deterministic mode's partial sums of intersections that no pixel took are zero
whatever an earlier backward left in their place: gradients of a scene on a context
that has rendered another one equal those on a fresh context bit for bit, and the
oracle's within the parity bar, in every tile shape and with and without segments
(4290 tiles of 16x16 have none)."""
import numpy as np
import pytest

from _parity import assert_grad_parity, oracle_forward, run_gpu_forward
from rustscan_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", ["default", "grid"])
@pytest.mark.parametrize("w,h,tile", [(96, 80, (8, 8)), (96, 80, (32, 8)), (96, 80, (16, 16)), (1056, 1040, (16, 16))])
def test_parts_do_not_carry_over(gsr_ctx_factory, w, h, tile, schedule):
    import torch

    from rustscan_b200 import host_splats_to_device

    # Opaque Gaussians in front: most list entries lie behind saturated pixels.
    first, second = (S.small_scene(n=6000, degree=0, width=w, height=h, seed=s) for s in (3, 4))
    second.raw_opacity[:] += 3.0
    first.raw_opacity[:] -= 3.0
    kw = dict(max_splats=6000, max_pixels=w * h, tile=tile, deterministic=True, schedule=schedule)
    up = S.upstream_grad(h, w, seed=1)
    v = torch.as_tensor(up.reshape(-1), device="cuda")
    used, fresh, res = gsr_ctx_factory(**kw), gsr_ctx_factory(**kw), []
    for ctx, scenes in ((used, (first, second)), (fresh, (second,))):
        for sc in scenes:
            splats = host_splats_to_device(sc)
            run_gpu_forward(ctx, splats, sc.cameras)
            g = ctx.render_backward(splats, v)
        torch.cuda.synchronize()
        res.append({k: g[k].cpu().numpy() for k in ("v_transforms", "v_sh", "v_raw_opacity")})
    cam = second.cameras[0]
    b32 = oracle_forward(second, cam, tile=tile).backward(up, mode=0)
    b64 = oracle_forward(second, cam, tile=tile, f64=True).backward(up, mode=0)
    for k, a in res[0].items():
        np.testing.assert_array_equal(a, res[1][k])
        assert_grad_parity(a, b32[k], b64[k], what=k)
