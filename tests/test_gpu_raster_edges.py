"""The raster kernels at the sizes where their batching can go wrong: list
lengths around the unroll, a ballot word, a batch and many batches, over
Gaussians that cover a whole tile and over needles and dots that reach only
some of its 8x8 blocks. The forward is bit-exact against the oracle (the
block culling may drop no contributor) and the gradients meet the parity bar;
not those of the needles, whose conics are so ill-conditioned in FP32 that the
FP32 and FP64 oracles themselves differ by up to 7e-3 there."""
import numpy as np
import pytest

from _parity import assert_forward_parity, assert_grad_parity, oracle_forward, run_gpu_forward
from rustscan_b200 import scenes as S

pytestmark = pytest.mark.gpu


def _scene(n, kind, width, height):
    rng = np.random.Generator(np.random.PCG64(77 + n))
    tr = np.zeros((n, 10), np.float32)
    tr[:, 0:2] = rng.uniform(-0.5, 0.5, (n, 2))
    tr[:, 2] = rng.uniform(0.0, 1.0, n)
    q = rng.standard_normal((n, 4))
    tr[:, 3:7] = q / np.linalg.norm(q, axis=1, keepdims=True)
    if kind == "wide":
        tr[:, 7:10] = -0.5
    elif kind == "dots":
        tr[:, 7:10] = -5.5
    else:  # needles: one long axis
        tr[:, 7:10] = -6.0
        tr[np.arange(n), 7 + rng.integers(0, 3, n)] = -1.0
    # Faint where every pixel meets every Gaussian, so that long lists do not saturate early.
    op = np.full(n, -5.0 if kind == "wide" else -2.0, np.float32)
    sh = rng.uniform(-0.5, 1.5, (n, 1, 3)).astype(np.float32)
    cam = S.camera_from_rt(np.eye(3), np.array([0.0, 0.0, 3.0]), 3.0 * width, 3.0 * width, width / 2, height / 2, width,
                           height)
    return S.Scene(tr, sh, op, 0, [cam], f"edge-{kind}")


@pytest.mark.parametrize("kind", ["wide", "needles", "dots"])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 32, 33, 64, 65, 128, 129, 1000, 6000])
def test_list_lengths(gsr_ctx_factory, n, kind):
    import torch

    from rustscan_b200 import host_splats_to_device

    w, h = (16, 16) if n % 2 else (21, 19)
    sc = _scene(n, kind, w, h)
    ctx = gsr_ctx_factory(max_splats=n, max_pixels=w * h)
    splats = host_splats_to_device(sc)
    _, g = run_gpu_forward(ctx, splats, sc.cameras)
    o = oracle_forward(sc, sc.cameras[0])
    assert_forward_parity(g[0], o)
    if kind == "needles":
        return
    up = S.upstream_grad(h, w, seed=n)
    got = ctx.render_backward(splats, torch.as_tensor(up, device="cuda"))
    torch.cuda.synchronize()
    ob = o.backward(up, mode=0)
    od = oracle_forward(sc, sc.cameras[0], f64=True).backward(up, mode=0)
    for k in ("v_transforms", "v_sh", "v_raw_opacity"):
        assert_grad_parity(got[k].cpu().numpy(), ob[k], od[k], what=k)


@pytest.mark.parametrize("schedule", ["default", "grid", "persistent"])
@pytest.mark.parametrize("n,w,h", [(700, 33, 31), (3000, 16, 40), (40_000, 512, 500), (32_767, 512, 512),
                                   (40_000, 513, 512)])
def test_split_tiles(gsr_ctx_factory, n, w, h, schedule):
    """Launches around the line where each 8x8 block is blended in a CTA of its
    own (1024 tiles, 32 Gaussians a tile), with partial tiles, in every
    schedule and with an odd view capacity, so that the views' hit bits start
    at odd addresses."""
    import torch

    from rustscan_b200 import host_splats_to_device

    sc = _scene(n, "dots", w, h)
    cams = sc.cameras if w * h > 4000 else sc.cameras * 3
    ctx = gsr_ctx_factory(max_splats=n, max_views=len(cams), max_pixels=w * h, max_isects=400_003, schedule=schedule)
    splats = host_splats_to_device(sc)
    _, g = run_gpu_forward(ctx, splats, cams)
    o = oracle_forward(sc, cams[0])
    for view in g:
        assert_forward_parity(view, o)
    up = S.upstream_grad(h, w, seed=n)
    v = torch.as_tensor(np.concatenate([up.reshape(-1)] * len(cams)), device="cuda")
    got = ctx.render_backward(splats, v)
    torch.cuda.synchronize()
    ob = o.backward(up, mode=0)
    od = oracle_forward(sc, cams[0], f64=True).backward(up, mode=0)
    for k in ("v_transforms", "v_sh", "v_raw_opacity"):
        assert_grad_parity(got[k].cpu().numpy() / len(cams), ob[k], od[k], what=k)
