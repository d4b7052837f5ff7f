"""Launches of many tiles with one long list: a tile that gets through more than
4096 entries is walked by the backward as four 8x8 blocks. Just below, just above
and well above that length: forward bit-exact where the oracle is, gradients
within the parity bar of the FP32 / FP64 oracles; in deterministic mode, which
keeps such a tile whole, bitwise repeatable too."""
import numpy as np
import pytest

from _parity import assert_forward_parity, assert_grad_parity, oracle_forward, run_gpu_forward
from rustscan_b200 import scenes as S

pytestmark = pytest.mark.gpu

W, H = 1056, 1040  # 66 x 65 tiles


def _scene(n, W=W, H=H, tx=20, ty=30):
    """n small faint Gaussians inside tile (tx, ty), 200 larger ones anywhere."""
    rng = np.random.default_rng(n)
    f, z = 1000.0, 2.0 + 2.0 * rng.random(n + 200)
    u = np.concatenate([tx * 16 + 1 + 14 * rng.random(n), W * rng.random(200)])
    v = np.concatenate([ty * 16 + 1 + 14 * rng.random(n), H * rng.random(200)])
    tr = np.zeros((n + 200, 10), np.float32)
    tr[:, 0], tr[:, 1], tr[:, 2] = (u - W / 2) * z / f, (v - H / 2) * z / f, z
    tr[:, 3:7] = rng.standard_normal((n + 200, 4))
    tr[:n, 7:10] = np.log(0.0015) + 0.2 * rng.standard_normal((n, 3))
    tr[n:, 7:10] = np.log(0.03) + 0.3 * rng.standard_normal((200, 3))
    op = np.concatenate([rng.uniform(-4.2, -3.0, n), rng.uniform(-1, 1, 200)]).astype(np.float32)
    sh = rng.uniform(-1, 1, (n + 200, 1, 3)).astype(np.float32)
    cam = S.camera_from_rt(np.eye(3), np.zeros(3), f, f, W / 2, H / 2, W, H)
    return S.Scene(tr, sh, op, 0, [cam])


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("n", [4090, 4110, 9000])
def test_long_tile_parity(gsr_ctx_factory, n, deterministic):
    import torch

    from rustscan_b200 import host_splats_to_device

    sc = _scene(n)
    ctx = gsr_ctx_factory(max_splats=sc.n, max_pixels=W * H, deterministic=deterministic)
    splats = host_splats_to_device(sc)
    up = S.upstream_grad(H, W, seed=n)
    res = []
    for _ in range(2 if deterministic else 1):
        _, g = run_gpu_forward(ctx, splats, sc.cameras)
        gr = ctx.render_backward(splats, torch.as_tensor(up.reshape(-1), device="cuda"))
        torch.cuda.synchronize()
        res.append({k: gr[k].cpu().numpy() for k in ("v_transforms", "v_sh", "v_raw_opacity")})
    o = oracle_forward(sc, sc.cameras[0])
    assert_forward_parity(g[0], o)
    b32, b64 = o.backward(up, mode=0), oracle_forward(sc, sc.cameras[0], f64=True).backward(up, mode=0)
    for k, a in res[0].items():
        assert_grad_parity(a, b32[k], b64[k], what=f"{n} {k}")
        np.testing.assert_array_equal(a, res[-1][k])


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("w,h,n", [(64, 48, 4000), (64, 48, 9000), (400, 300, 6000), (1024, 1000, 3000), (1024, 1000, 12000)])
def test_long_list_of_few_tiles_parity(gsr_ctx_factory, w, h, n, deterministic):
    """Launches of at most 4096 tiles, whose lists are cut into segments that grow
    along the list: one list far longer than the short segments cover, with 64,
    33 and 4 segments a tile, and a last segment of more than 4096 entries."""
    import torch

    from rustscan_b200 import host_splats_to_device

    sc = _scene(n, w, h, w // 32, h // 32)
    ctx = gsr_ctx_factory(max_splats=sc.n, max_pixels=w * h, deterministic=deterministic)
    splats = host_splats_to_device(sc)
    up = S.upstream_grad(h, w, seed=n)
    _, g = run_gpu_forward(ctx, splats, sc.cameras)
    gr = ctx.render_backward(splats, torch.as_tensor(up.reshape(-1), device="cuda"))
    torch.cuda.synchronize()
    o = oracle_forward(sc, sc.cameras[0])
    assert_forward_parity(g[0], o)
    b32, b64 = o.backward(up, mode=0), oracle_forward(sc, sc.cameras[0], f64=True).backward(up, mode=0)
    for k in ("v_transforms", "v_sh", "v_raw_opacity"):
        assert_grad_parity(gr[k].cpu().numpy(), b32[k], b64[k], what=f"{w}x{h} {n} {k}")
