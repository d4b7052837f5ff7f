"""The workloads whose time this framework is judged by: one pass of each
through the public entry points, over the sizes the repository's scenes,
tests and benchmark use.

listed() names a dozen of them, draw() gives others of the same ranges,
prepare() makes the inputs a user's program would hold (on the GPU, from the
seed alone), run() does one pass, work() counts what a pass cannot do without
and exact() gives the results in 64 bits from plain torch, where that is
affordable.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as TF

import rustscan_b200 as gsr
from rustscan_b200 import scenes
from rustscan_b200.frames import DecodedFrame

C0 = scenes.SH_C0
# Learning rates of a long run's end: every group has decayed to a hundredth,
# so that repeated passes over one state keep rendering much the same scene.
RATES = dict(position_final=1.6e-6, rotation_final=1e-5, scale_final=5e-5, color_final=2.5e-5, opacity_final=5e-4)
TOTAL_STEPS = 30000
FIRST_STEP = 29000  # Adam's step count of the resumed run


# ---- the cases --------------------------------------------------------------
def _case(name, op, n, degree, width, height, **more):
    return dict(name=name, op=op, n=n, degree=degree, width=width, height=height, views=1, uneven=False, bf16=False,
                fp64_conic=False, deterministic=False) | more


def listed():
    return [
        # A viewer's frame of a small scene: the smallest call, all latency.
        _case("render_16k_256", "render", 16384, 0, 256, 256),
        # An evaluation image, quantised and brought to the host; a ragged size.
        _case("evaluate_300k_957x541", "evaluate", 300_000, 3, 957, 541),
        # The differentiable render op (autograd) on a small colour-only scene.
        _case("op_16k_256", "op", 16384, 0, 256, 256),
        # The op on a VGA view of a mid-sized scene, one pixel short of whole tiles.
        _case("op_200k_639x479", "op", 200_000, 3, 639, 479),
        # The op in its mixed-precision form on the largest scene and view.
        _case("op_3M_1080p_bf16", "op", 3_000_000, 3, 1920, 1080, bf16=True, fp64_conic=True),
        # A hand-written training loop: op, loss, backward and optimizer as separate calls.
        _case("plain_500k_720p", "plain", 500_000, 3, 1280, 720),
        # The reference's own habit: one small view a step.
        _case("train_74k_320x240", "train", 74_000, 3, 320, 240),
        # The benchmark's batched step.
        _case("train_1M_8x720p", "train", 1_000_000, 3, 1280, 720, views=8),
        # An uneven batch of near and far views of several resolutions, BF16 storage.
        _case("train_2M_16_uneven_bf16", "train", 2_000_000, 3, 1920, 1080, views=16, uneven=True, bf16=True),
        # Steps fed with decoded 8-bit frames from the host, larger than the training size.
        _case("frames_300k_4x800x450", "frames", 300_000, 3, 800, 450, views=4),
        # The scan and the stable sort as primitives of their own.
        _case("primitives_3M", "primitives", 3_000_001, 0, 0, 0),
        # One densification round: splits, copies and prunes applied on the device.
        _case("topology_100k", "topology", 100_000, 3, 0, 0),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def size(lo, hi):
        w = log(lo, hi)
        return w, max(int(w * rng.choice((0.5625, 0.625, 0.75, 1.0))) - rng.randrange(3), 16)

    op = rng.choice(("render", "evaluate", "op", "op", "plain", "train", "train", "train", "frames", "primitives",
                     "topology"))
    degree = rng.choice((0, 1, 2, 3, 3, 3, 4))
    bf16 = rng.random() < 0.3
    if op == "render":
        w, h = size(120, 1000)
        c = _case("", op, log(4000, 300_000), degree, w, h)
    elif op == "evaluate":
        w, h = size(240, 1400)
        c = _case("", op, log(30_000, 700_000), degree, w, h)
    elif op == "op":
        w, h = size(160, 1400)
        c = _case("", op, log(8000, 1_500_000), degree, w, h, bf16=bf16, fp64_conic=bf16,
                  deterministic=rng.random() < 0.15)
    elif op == "plain":
        w, h = size(240, 1300)
        c = _case("", op, log(20_000, 700_000), degree, w, h, bf16=bf16)
    elif op == "train":
        w, h = size(240, 1280)
        c = _case("", op, log(20_000, 900_000), degree, w, h, views=rng.choice((1, 1, 2, 3, 5, 8)), bf16=bf16,
                  uneven=rng.random() < 0.25)
    elif op == "frames":
        w, h = size(240, 800)
        c = _case("", op, log(20_000, 300_000), degree, w, h, views=rng.choice((1, 2, 4)), bf16=bf16)
    elif op == "primitives":
        c = _case("", op, log(1000, 8_000_000), 0, 0, 0)
    else:
        c = _case("", op, log(2000, 100_000), degree, 0, 0, bf16=bf16)
    del c["name"]
    return c


# ---- inputs -----------------------------------------------------------------
def _dtype(case):
    return torch.bfloat16 if case["bf16"] else torch.float32


def _gaussians(case, seed):
    """The distributions of scenes.py, drawn on the GPU: eight blobs in a 4 m
    cube (a uniform cube for degree-0 scenes), log-scales N(-4, 0.5), DC from
    uniform RGB, higher bands N(0, 0.05), opacity logits N(0, 1); 5% flattened
    where the FP64 conic is asked for."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, K = case["n"], (case["degree"] + 1) ** 2

    def normal(*s):
        return torch.randn(s, generator=g, device="cuda")

    def uniform(*s):
        return torch.rand(s, generator=g, device="cuda")

    if case["degree"] == 0:
        means = 2.0 * uniform(n, 3) - 1.0
    else:
        centres = 4.0 * uniform(8, 3) - 2.0
        means = centres[torch.randint(0, 8, (n,), generator=g, device="cuda")] + 0.3 * normal(n, 3)
    quats = normal(n, 4)
    scales = -4.0 + 0.5 * normal(n, 3)
    if case["fp64_conic"]:
        flat = torch.nonzero(uniform(n) < 0.05).flatten()
        scales[flat, torch.randint(0, 3, flat.shape, generator=g, device="cuda")] = -9.0
    transforms = torch.cat([means, quats / quats.norm(dim=1, keepdim=True), scales], dim=1).contiguous()
    sh = 0.05 * normal(n, K, 3)
    sh[:, 0] = (uniform(n, 3) - 0.5) / C0
    return gsr.DeviceSplats(transforms, sh.to(_dtype(case)), normal(n), case["degree"])


def _cameras(case, seed):
    """Cameras on a sphere of radius 4 looking at the origin; an uneven batch
    mixes distances 1.5 to 8 and the size's halves and thirds."""
    rng = np.random.default_rng(seed)
    cams = []
    for v in range(case["views"]):
        d = rng.standard_normal(3)
        d /= np.linalg.norm(d)
        w, h, r = case["width"], case["height"], 4.0
        if case["uneven"]:
            part = (1, 1.5, 3, 6)[(v + int(rng.integers(4))) % 4]
            w, h, r = max(int(w / part), 16), max(int(h / part), 16), float(rng.uniform(1.5, 8.0))
        f = 0.82 * w
        cams.append(scenes.look_at(r * d, (0, 0, 0), f, f, (w - 1) / 2, (h - 1) / 2, w, h))
    return cams


def _image(g, h, w):
    """A picture to train against: smooth structure plus fine grain, in [0, 1]."""
    low = torch.rand((1, 3, max(h // 24, 2), max(w // 24, 2)), generator=g, device="cuda")
    x = TF.interpolate(low, size=(h, w), mode="bicubic", align_corners=False)[0].permute(1, 2, 0)
    return (x + 0.05 * torch.randn((h, w, 3), generator=g, device="cuda")).clamp(0.0, 1.0).contiguous()


def _context(case, splats, cams):
    """A context whose intersection capacity fits these views, found as a
    program finds it: render once and grow."""
    ctx = gsr.Context(max_splats=case["n"], max_views=len(cams), max_pixels=max(c.width * c.height for c in cams),
                      sh_dtype=_dtype(case), fp64_conic=case["fp64_conic"], deterministic=case["deterministic"])
    for _ in range(4):
        try:
            ctx.render_forward(splats, cams)
            return ctx
        except gsr.GsrError as e:
            if e.status != 3:
                raise
            ctx.reserve_isects(int(e.required * 1.15) + 1024)
    raise RuntimeError("could not fit the intersection capacity")


def _moments(opt, seed):
    """Adam's state as a resumed run finds it."""
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    for m, v in ((opt.m_tr, opt.v_tr), (opt.m_sh, opt.v_sh), (opt.m_op, opt.v_op)):
        m.copy_(1e-6 * torch.randn(m.shape, generator=g, device="cuda"))
        v.copy_(1e-11 * (0.05 + torch.rand(v.shape, generator=g, device="cuda")))
    opt.step = FIRST_STEP


def _plan(case, seed):
    """A densification plan: a tenth of the splats split in two, a twentieth
    pruned, the rest kept."""
    rng, n, T = np.random.default_rng(seed + 5), case["n"], gsr.TopologyPlan
    order, sample = rng.permutation(n).tolist(), rng.standard_normal(n).tolist()
    split, kept = order[:n // 10], sorted(order[n // 10:n - n // 20])
    rows = [(i, T.REFINE_EXISTING, sample[i]) for i in split] + [(i, T.EXISTING, 0.0) for i in kept]
    rows += [(i, T.REFINE_NEW, sample[i]) for i in split]
    return T(rows, refine_decay=(0.004, 0.002, 0.5))


def prepare(case, seed):
    op = case["op"]
    if op == "primitives":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = case["n"]
        # Depth-like keys (positive floats' bits) and tile counts, as the render path sorts and scans them.
        keys = (0.7 + 7.0 * torch.rand(n, generator=g, device="cuda")).view(torch.int32)
        counts = torch.randint(0, 40, (n,), generator=g, device="cuda", dtype=torch.int32)
        return dict(op=op, ctx=gsr.Context(max_splats=n, max_pixels=1 << 16), keys=keys, counts=counts,
                    vals=torch.arange(n, device="cuda", dtype=torch.int32))
    splats = _gaussians(case, seed)
    if op == "topology":
        ctx = gsr.Context(max_splats=case["n"], max_pixels=1 << 16, sh_dtype=_dtype(case))
        return dict(op=op, ctx=ctx, splats=splats, plan=_plan(case, seed))
    cams = _cameras(case, seed)
    s = dict(op=op, splats=splats, cams=cams)
    if op == "evaluate":
        s["renderer"] = gsr.SplatEvaluationRenderer(case["width"], case["height"], max_splats=case["n"])
        return s
    s["ctx"] = ctx = _context(case, splats, cams)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    if op in ("op", "plain"):
        for t in (splats.transforms, splats.sh_coeffs, splats.raw_opacities):
            t.requires_grad_(True)
    if op == "op":
        c = cams[0]
        s["v_image"] = torch.randn((c.height, c.width, 4), generator=g, device="cuda")
        s["v_image"][..., 3] = 0.0
    elif op in ("plain", "train"):
        s["target"] = torch.cat([_image(g, c.height, c.width).reshape(-1) for c in cams])
    elif op == "frames":
        # Two sets of frames half again the training size, shown in turn.
        s["frames"] = [[DecodedFrame((_image(g, c.height * 3 // 2, c.width * 3 // 2) * 255.0).round().to(torch.uint8)
                                     .cpu().numpy()).rgb for c in cams] for _ in range(2)]
    lrs = gsr.LearningRates(**RATES)
    if op == "plain":
        s["opt"], s["lr"] = gsr.AdamScaled(ctx, splats, lrs), lrs.at(TOTAL_STEPS, TOTAL_STEPS)
        _moments(s["opt"], seed)
    elif op in ("train", "frames"):
        s["trainer"], s["turn"] = gsr.Trainer(ctx, splats, lrs, total_iterations=TOTAL_STEPS), 0
        _moments(s["trainer"].opt, seed)
    return s


# ---- one pass ---------------------------------------------------------------
def _op_backward(s, v_image_of):
    """The differentiable render of s and its backward; fresh gradients."""
    sp = s["splats"]
    for t in (sp.transforms, sp.sh_coeffs, sp.raw_opacities):
        t.grad = None
    out = gsr.render_splats_with_visibility(s["ctx"], sp, s["cams"][0])
    v, loss = v_image_of(out.image)
    out.image.backward(v)
    grads = dict(v_transforms=sp.transforms.grad, v_sh=sp.sh_coeffs.grad, v_raw_opacity=sp.raw_opacities.grad)
    return dict(image=out.image.detach(), visible=out.visible, stats=out.screen_grad_stats.grad, **grads), loss


def _optimizer_state(splats, opt):
    return dict(transforms=splats.transforms.detach(), sh=splats.sh_coeffs.detach(),
                opacity=splats.raw_opacities.detach(), mean_tr=opt.m_tr, square_tr=opt.v_tr, mean_sh=opt.m_sh,
                square_sh=opt.v_sh, mean_op=opt.m_op, square_op=opt.v_op)


def run(s):
    op = s["op"]
    if op == "render":
        return dict(image=s["ctx"].render_forward(s["splats"], s["cams"])[0])
    if op == "evaluate":
        return dict(rgb=s["renderer"].render(s["splats"], s["cams"][0]))
    if op == "op":
        return _op_backward(s, lambda image: (s["v_image"], None))[0]
    if op == "plain":
        ctx, sp, cams = s["ctx"], s["splats"], s["cams"]

        def loss_gradient(image):
            loss, v = ctx.loss(image.detach(), s["target"], cams)
            return v, loss

        out, loss = _op_backward(s, loss_gradient)
        grads = {k: out[k].float() if k == "v_sh" else out[k] for k in ("v_transforms", "v_sh", "v_raw_opacity")}
        s["opt"].step_device_splats(sp, grads, s["lr"])
        return dict(out, loss=loss, **_optimizer_state(sp, s["opt"]))
    if op == "train":
        loss = s["trainer"].train_step(s["cams"], s["target"], TOTAL_STEPS)
        return dict(loss=loss, densify=s["trainer"].densify, **_optimizer_state(s["splats"], s["trainer"].opt))
    if op == "frames":
        now, s["turn"] = s["frames"][s["turn"]], 1 - s["turn"]
        loss = s["trainer"].train_step_frames(s["cams"], now, TOTAL_STEPS, next_frames=s["frames"][s["turn"]])
        return dict(loss=loss, densify=s["trainer"].densify, **_optimizer_state(s["splats"], s["trainer"].opt))
    if op == "primitives":
        keys, vals = s["ctx"].radix_sort_by_key_u32(s["keys"], s["vals"])
        return dict(scan=s["ctx"].prefix_sum_u32(s["counts"]), keys=keys, vals=vals)
    out = gsr.apply_topology(s["ctx"], s["splats"], s["plan"])
    return dict(transforms=out.transforms, sh=out.sh_coeffs, opacity=out.raw_opacities)


# ---- what a pass cannot do without -------------------------------------------
def work(case):
    """Bytes: every input read once and every output written once. Operations:
    projection and colour per Gaussian and view, blending of the pairs of a
    Gaussian and a pixel (at most about a hundred per pixel until it
    saturates), the loss's blurs and Adam."""
    op, n, K = case["op"], case["n"], (case["degree"] + 1) ** 2
    if op == "primitives":
        return {"bytes": n * (8 + 16), "flops": n}
    row = 44 + 3 * K * (2 if case["bf16"] else 4)
    if op == "topology":
        return {"bytes": n * row + 1.05 * n * (row + 16), "flops": 200 * n}
    pixels = sum(c.width * c.height for c in _cameras(case, 0))
    per_view = pixels / case["views"]
    footprint = 30.0 * (0.018 * 0.82 * math.sqrt(per_view * 16 / 9) / 4.0) ** 2 + 15.0  # pixels a Gaussian reaches
    blends = min(100.0 * pixels, 0.7 * n * case["views"] * footprint)
    flops = case["views"] * n * (400 + 6 * K) + 25 * blends
    params = n * row
    if op in ("render", "evaluate"):
        return {"bytes": params + pixels * (16 if op == "render" else 12), "flops": flops}
    flops += case["views"] * n * (500 + 12 * K) + 60 * blends
    grads = n * 4 * (11 + 3 * K)
    if op == "op":
        return {"bytes": 2 * params + pixels * 32 + grads + n * 32, "flops": flops}
    flops += 500 * pixels + 12 * n * (11 + 3 * K)
    adam = 2 * params + 4 * grads
    if op == "plain":
        return {"bytes": adam + pixels * (32 + 12) + 2 * grads + n * 32, "flops": flops}
    return {"bytes": adam + pixels * (12 if op == "train" else 6.75) + 72 * n, "flops": flops}


# ---- the same results in 64 bits ---------------------------------------------
def _basis(degree, d):
    """Real spherical harmonics of the unit directions d, [n, K], signs as the splatting formats have them."""
    x, y, z = d.unbind(1)
    b = [torch.full_like(x, C0)]
    if degree > 0:
        a = 0.48860251190292
        b += [-a * y, a * z, -a * x]
    if degree > 1:
        b += [1.092548430592079 * x * y, -1.092548430592079 * y * z, 0.9461746957575601 * z * z - 0.3153915652525201,
              -1.092548430592079 * x * z, 0.5462742152960395 * (x * x - y * y)]
    if degree > 2:
        p, q = -2.285228997322329 * z * z + 0.4570457994644658, 1.445305721320277 * z
        b += [-0.5900435899266435 * y * (3 * x * x - y * y), 2 * q * x * y, p * y,
              z * (1.865881662950577 * z * z - 1.119528997770346), p * x, q * (x * x - y * y),
              -0.5900435899266435 * x * (x * x - 3 * y * y)]
    if degree > 3:
        c2, s2 = x * (x * x - 3 * y * y), y * (3 * x * x - y * y)
        t, u = z * (-4.683325804901025 * z * z + 2.007139630671868), 3.31161143515146 * z * z - 0.47308734787878
        w = -1.770130769779931 * z
        b += [0.6258357354491763 * (x * s2 + y * c2), w * s2, 2 * u * x * y, t * y,
              1.984313483298443 * z * b[12] - 1.006230589874905 * b[6], t * x, u * (x * x - y * y), w * c2,
              0.6258357354491763 * (x * c2 - y * s2)]
    return torch.stack(b, dim=1)


class _Render64:
    """One view in 64 bits: EWA projection, colour and front-to-back blending,
    tile by tile so that the pairs fit; gradients through autograd."""

    def __init__(self, splats, cam, blur=0.3):
        self.tr = splats.transforms.detach().double().requires_grad_(True)
        self.sh = splats.sh_coeffs.detach().double().requires_grad_(True)
        self.op = splats.raw_opacities.detach().double().requires_grad_(True)
        self.w, self.h, self.n = cam.width, cam.height, splats.num_splats()
        dev = dict(dtype=torch.float64, device="cuda")
        view = torch.tensor(np.asarray(cam.viewmat, np.float64).reshape(4, 4).T.copy(), **dev)
        R, t = view[:3, :3], view[:3, 3]
        f = torch.tensor([np.float32(cam.fx), np.float32(cam.fy)], **dev)
        pc = torch.tensor([np.float32(cam.cx), np.float32(cam.cy)], **dev)
        size = torch.tensor([self.w, self.h], **dev)
        mean = self.tr[:, :3]
        mc = mean @ R.T + t
        z = mc[:, 2]
        q = self.tr[:, 3:7] / self.tr[:, 3:7].norm(dim=1, keepdim=True)
        w, x, y, zz = q.unbind(1)
        rot = torch.stack([1 - 2 * (y * y + zz * zz), 2 * (x * y - w * zz), 2 * (x * zz + w * y),
                           2 * (x * y + w * zz), 1 - 2 * (x * x + zz * zz), 2 * (y * zz - w * x),
                           2 * (x * zz - w * y), 2 * (y * zz + w * x), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)
        m = R @ rot * self.tr[:, 7:10].exp()[:, None, :]
        rz = 1.0 / z.clamp(min=0.01)
        uv = torch.maximum(torch.minimum(mc[:, :2] * rz[:, None], (1.15 * size - pc) / f), (-0.15 * size - pc) / f)
        zero = torch.zeros_like(rz)
        J = torch.stack([f[0] * rz, zero, -f[0] * rz * uv[:, 0], zero, f[1] * rz, -f[1] * rz * uv[:, 1]], 1)
        jm = J.view(-1, 2, 3) @ m
        cov = jm @ jm.transpose(1, 2)
        a0, b0, c0 = cov[:, 0, 0], cov[:, 0, 1], cov[:, 1, 1]
        a1, c1 = a0 + blur, c0 + blur
        raw = (a0 * c0 - b0 * b0).clamp(min=0.0)
        comp = torch.where(raw > 0, (torch.where(raw > 0, raw, 1.0) / (a1 * c1 - b0 * b0)).sqrt(), 0.0)
        opacity = torch.sigmoid(self.op) * comp
        det = (a1 + 1e-6) * (c1 + 1e-6) - b0 * b0
        conic = torch.stack([(c1 + 1e-6) / det, -b0 / det, (a1 + 1e-6) / det], 1)
        xy = f * mc[:, :2] / z[:, None] + pc
        d = mean - torch.tensor(np.asarray(cam.campos, np.float64), **dev)
        basis = _basis(splats.sh_degree, d / d.norm(dim=1, keepdim=True))
        rgb = torch.einsum("nk,nkc->nc", basis, self.sh) + 0.5
        with torch.no_grad():
            thr = (opacity * 255.0).log()
            ext = torch.stack([(2 * thr * a1).clamp(min=0).sqrt(), (2 * thr * c1).clamp(min=0).sqrt()], 1)
            inside = ((xy + ext > 0) & (xy - ext < size)).all(dim=1)
            seen = torch.nonzero((z >= 0.01) & (z <= 1e10) & (opacity >= 1 / 255) & inside).flatten()
            self.seen = seen = seen[torch.argsort(z[seen], stable=True)]
            self.lo, self.hi, self.depth = (xy - ext)[seen], (xy + ext)[seen], z.detach()
        self.full = (xy, conic, opacity, rgb)
        self.leaf = [v.detach()[seen].requires_grad_(True) for v in self.full]

    def tiles(self, v_image=None):
        """The image, and with an upstream gradient also the leaves' gradients and the per-splat statistics."""
        image = torch.zeros((self.h, self.w, 4), dtype=torch.float64, device="cuda")
        self.count = torch.zeros(len(self.seen), dtype=torch.float64, device="cuda")
        self.absolute = torch.zeros((len(self.seen), 2), dtype=torch.float64, device="cuda")
        for ty in range(0, self.h, 16):
            row = torch.nonzero((self.hi[:, 1] > ty) & (self.lo[:, 1] < ty + 16)).flatten()
            for tx in range(0, self.w, 16):
                i = row[(self.hi[row, 0] > tx) & (self.lo[row, 0] < tx + 16)]
                if not len(i):
                    continue
                y1, x1 = min(ty + 16, self.h), min(tx + 16, self.w)
                py, px = torch.meshgrid(torch.arange(ty, y1, device="cuda") + 0.5,
                                        torch.arange(tx, x1, device="cuda") + 0.5, indexing="ij")
                with torch.set_grad_enabled(v_image is not None):
                    xy, conic, opacity, rgb = (leaf[i] for leaf in self.leaf)
                    dx = xy[:, :1] - px.reshape(1, -1)
                    dy = xy[:, 1:] - py.reshape(1, -1)
                    sigma = 0.5 * (conic[:, :1] * dx * dx + 2 * conic[:, 1:2] * dx * dy + conic[:, 2:] * dy * dy)
                    if v_image is not None:
                        sigma.retain_grad()
                    alpha = (opacity[:, None] * torch.exp(-sigma)).clamp(max=0.999)
                    with torch.no_grad():
                        valid = (sigma >= 0) & (alpha >= 1 / 255)
                        T = torch.cumprod(torch.where(valid, 1.0 - alpha, 1.0), 0)
                        valid &= torch.cat([torch.ones_like(T[:1]), T[:-1]]) >= 1e-4
                    alpha = torch.where(valid, alpha, 0.0)
                    T = torch.cumprod(torch.cat([torch.ones_like(dx[:1]), 1.0 - alpha]), 0)
                    pixels = torch.cat([(alpha * T[:-1]).T @ rgb.clamp(min=0.0), 1.0 - T[-1][:, None]], 1)
                image[ty:y1, tx:x1] = pixels.detach().view(y1 - ty, x1 - tx, 4)
                self.count[i] += valid.sum(1)
                if v_image is not None:
                    pixels.backward(v_image[ty:y1, tx:x1].reshape(-1, 4))
                    vs = sigma.grad
                    gx, gy = conic[:, :1] * dx + conic[:, 1:2] * dy, conic[:, 1:2] * dx + conic[:, 2:] * dy
                    self.absolute[i] += torch.stack([(vs * gx).abs().sum(1), (vs * gy).abs().sum(1)], 1).detach()
        return image

    def gradients(self):
        """Parameter gradients after tiles(v_image), the visible flags and the [n, 7] screen statistics."""
        grads = [torch.zeros_like(x) if x.grad is None else x.grad for x in self.leaf]
        torch.autograd.backward([v[self.seen] for v in self.full], grads)
        visible = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        visible[self.seen] = (self.count > 0).double()
        stats = torch.zeros((self.n, 7), dtype=torch.float64, device="cuda")
        stats[self.seen] = torch.cat([grads[0], self.absolute, (self.count * self.absolute.norm(dim=1))[:, None],
                                      self.count[:, None], (self.count * self.depth[self.seen])[:, None]], 1)
        return dict(v_transforms=self.tr.grad, v_sh=self.sh.grad, v_raw_opacity=self.op.grad, visible=visible,
                    stats=stats)


def _loss64(image, target):
    """0.8 L1 + 0.2 (1 - SSIM): 11 taps, sigma 1.5, replicated borders; the window holds 32-bit values."""
    k = np.exp(-np.arange(-5.0, 6.0) ** 2 / (2 * 1.5 * 1.5)).astype(np.float32)
    k = torch.tensor((k / k.sum(dtype=np.float32)).astype(np.float64), device="cuda")
    x, y = image[..., :3].permute(2, 0, 1)[:, None], target.double().permute(2, 0, 1)[:, None]

    def blur(t):
        t = TF.conv2d(TF.pad(t, (5, 5, 0, 0), mode="replicate"), k.view(1, 1, 1, 11))
        return TF.conv2d(TF.pad(t, (0, 0, 5, 5), mode="replicate"), k.view(1, 1, 11, 1))

    mx, my = blur(x), blur(y)
    sx, sy, sxy = blur(x * x) - mx * mx, blur(y * y) - my * my, blur(x * y) - mx * my
    ssim = (2 * mx * my + 1e-4) * (2 * sxy + 9e-4) / ((mx * mx + my * my + 1e-4) * (sx + sy + 9e-4))
    return 0.8 * (x - y).abs().mean() + 0.2 * (1.0 - ssim.mean())


def _adam64(s, opt, lr, grads, bf16):
    """One Adam step in 64 bits from the 32-bit state and constants; BF16 coefficients round once, as stored."""
    b1, b2, eps, step = float(lr.beta1), float(lr.beta2), float(lr.eps), opt.step + 1
    col = torch.tensor([lr.position] * 3 + [lr.rotation] * 4 + [lr.scale] * 3, dtype=torch.float64, device="cuda")
    out = {}
    for p, g, m, v, rate, names in (
            (s.transforms, grads["v_transforms"], opt.m_tr, opt.v_tr, col,
             ("transforms", "mean_tr", "square_tr")),
            (s.sh_coeffs, grads["v_sh"], opt.m_sh, opt.v_sh, float(lr.color),
             ("sh", "mean_sh", "square_sh")),
            (s.raw_opacities, grads["v_raw_opacity"], opt.m_op, opt.v_op, float(lr.opacity),
             ("opacity", "mean_op", "square_op"))):
        m = b1 * m.double() + (1 - b1) * g
        v = b2 * v.double() + (1 - b2) * g * g
        p = p.detach().double() - rate * (m / (1 - b1 ** step)) / ((v / (1 - b2 ** step)).sqrt() + eps)
        out |= dict(zip(names, (None if bf16 and names[0] == "sh" else p, m, v)))
    return out


def _topology64(s):
    """The plan's rows in 64 bits."""
    rows, sp = s["plan"].rows, s["splats"]
    src = torch.tensor([r[0] for r in rows], device="cuda")
    kind = torch.tensor([r[1] for r in rows], device="cuda")
    sample = torch.tensor(np.array([r[2] for r in rows], np.float32), device="cuda").double()
    t, o = sp.transforms.double()[src], torch.sigmoid(sp.raw_opacities.double()[src])
    split = kind != gsr.TopologyPlan.EXISTING
    sign = torch.where(kind == gsr.TopologyPlan.REFINE_NEW, 1.0, -1.0)
    scale = t[:, 7:].exp()
    q = t[:, 3:7] / t[:, 3:7].norm(dim=1, keepdim=True)
    v, u = scale * sample[:, None], q[:, 1:]
    c = torch.cross(u, v, dim=1)
    move = v + 2 * (q[:, :1] * c + torch.cross(u, c, dim=1))
    half = scale * torch.where(TF.one_hot(scale.argmax(1), 3) > 0, 0.5, 1.0)
    mean = torch.where(split[:, None], t[:, :3] + sign[:, None] * move, t[:, :3])
    scale = torch.where(split[:, None], half.clamp(min=1e-6), scale)
    lo = 1 / 255
    o = torch.where(split, (1 - (1 - o.clamp(lo, 1 - lo)).sqrt()).clamp(lo, 1 - lo), o)
    opacity_decay, scale_decay, at = s["plan"].refine_decay
    scale = scale * (1 - scale_decay * (1 - at))
    o = (o - opacity_decay * (1 - at)).clamp(1e-12, 1 - 1e-12)
    return dict(transforms=torch.cat([mean, t[:, 3:7], scale.log()], 1), sh=None, opacity=(o / (1 - o)).log())


def exact(case, seed):
    op = case["op"]
    if op == "primitives":
        return None  # whole numbers
    tiles = -(-case["width"] // 16) * -(-case["height"] // 16)
    if op != "topology" and (case["views"] > 1 or tiles > 2100 or case["n"] > 600_000 or op == "frames"):
        return None  # over 20 seconds
    s = prepare(case, seed)
    if op == "topology":
        return _topology64(s)
    cam, sp = s["cams"][0], s["splats"]
    r = _Render64(sp, cam)
    image = r.tiles()
    if op == "render":
        return dict(image=image.reshape(-1))
    if op == "evaluate":
        return dict(rgb=torch.round(image[..., :3].clamp(0, 1) * 255.0).div(255.0).reshape(-1))
    if op == "op":
        r.tiles(s["v_image"].double())
        g = r.gradients()
        if case["bf16"]:
            g["v_sh"] = None  # autograd rounds it to the storage type
        return dict(image=image, **g)
    shown = image.clone().requires_grad_(True)
    loss = _loss64(shown, s["target"].view(cam.height, cam.width, 3))
    (v,) = torch.autograd.grad(loss, shown)
    r.tiles(v)
    g = r.gradients()
    if op == "plain":
        if case["bf16"]:
            return dict(image=image, loss=loss.detach().reshape(1), v_transforms=g["v_transforms"],
                        v_raw_opacity=g["v_raw_opacity"], visible=g["visible"], stats=g["stats"])
        return dict(image=image, loss=loss.detach().reshape(1), **g, **_adam64(sp, s["opt"], s["lr"], g, False))
    st, vm = g["stats"], g["v_transforms"][:, :3]
    one = torch.ones_like(st[:, 0])
    densify = torch.stack([vm.abs().mean(1), st[:, :2].norm(dim=1), st[:, 2:4].norm(dim=1), st[:, 4], st[:, 5],
                           st[:, 6], g["v_sh"].abs().mean((1, 2)), one, one])
    opt = s["trainer"].opt
    return dict(loss=loss.detach().reshape(1), densify=densify,
                **_adam64(sp, opt, opt.lrs.at(TOTAL_STEPS - 1, TOTAL_STEPS), g, case["bf16"]))
