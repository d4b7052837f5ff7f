"""The projection's layouts of SH rows against the oracle: every degree in FP32
and BF16 storage (rows of whole 16- or 8-byte units and others), SH arrays that
start off a unit's boundary, one view and several (instances of their own),
scenes of one Gaussian, one short of a block, a block and one more."""
import pytest

from _parity import assert_forward_parity, oracle_forward, run_gpu_forward
from rustscan_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("degree", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("offset", [0, 1, 4])
def test_sh_row_layouts(gsr_ctx_factory, degree, bf16, offset):
    import torch

    from rustscan_b200 import DeviceSplats, host_splats_to_device

    for n, views in ((1, 1), (255, 2), (257, 1), (513, 3)):
        sc = S.small_scene(n=n, degree=degree, width=72, height=56, seed=5 * degree + n, views=views)
        dtype = torch.bfloat16 if bf16 else torch.float32
        d = host_splats_to_device(sc, sh_dtype=dtype)
        flat = torch.zeros(d.sh_coeffs.numel() + offset, dtype=dtype, device="cuda")
        flat[offset:] = d.sh_coeffs.reshape(-1)
        splats = DeviceSplats(d.transforms, flat[offset:].view(d.sh_coeffs.shape), d.raw_opacities, degree)
        ref = S.Scene(sc.transforms, d.sh_coeffs.float().cpu().numpy(), sc.raw_opacity, degree, sc.cameras)
        ctx = gsr_ctx_factory(max_splats=n, max_views=views, max_pixels=72 * 56, sh_dtype="bf16" if bf16 else "f32")
        _, g = run_gpu_forward(ctx, splats, sc.cameras)
        for v, cam in enumerate(sc.cameras):
            assert_forward_parity(g[v], oracle_forward(ref, cam))
