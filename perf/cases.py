"""The timed cases of this framework: whole calls and single blocks through its
public entry points, with inputs made on the GPU from a seed.

Kinds
  fit     one training step of a fit (Fitter.step): forward, backward, Adam
  batch   one step of many uneven fits together (Batch.step)
  render  one frame of the forward-only renderer (Renderer.render)
  layers  one step assembled from the layer calls (activation, projection,
          rasterizer, loss, their backward, Adam), as the drop-in layers and the
          initializer's training use them
  conv    one 3x3 convolution block of the initializer, forward and backward
  init    the initializer's network on a batch of images, decoded to splats

The scenes follow diffsplat_b200.scenes: "frustum" is the random start of the
plain fitters, "orbit" the surfaces seen from a circle of cameras of the viewer
workload.  Adam's epsilon is 1e-6 in the fits: a splat whose gradient is lost in
rounding then stays where it is instead of moving by a whole learning rate.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from diffsplat_b200 import _lib, api, initializer, nn, scenes

EPS = 1e-6
TILE = 16


def listed():
    return [
        # the plain small fit (256 x 256, 4096 splats): a step is all launches and latency
        {"name": "fit_256", "kind": "fit", "scene": "frustum", "width": 256, "height": 256,
         "focal": 256, "count": 4096, "sh": 0, "storage": "fp32"},
        # the reference's default fit: 1280 x 720, 60000 splats
        {"name": "fit_720p", "kind": "fit", "scene": "frustum", "width": 1280, "height": 720,
         "focal": 1000, "count": 60000, "sh": 0, "storage": "fp32"},
        # a fit with BF16 storage, of an image and a count that fill no tile and no block
        {"name": "fit_odd_bf16", "kind": "fit", "scene": "frustum", "width": 797, "height": 531,
         "focal": 700, "count": 30011, "sh": 1, "storage": "bf16"},
        # training a large scene: a million splats with SH 3 at 1920 x 1080
        {"name": "fit_1080p_sh3", "kind": "fit", "scene": "orbit", "width": 1920, "height": 1080,
         "focal": 1200, "count": 1_000_000, "sh": 3, "storage": "fp32"},
        # 16 uneven fits stepped together, BF16 storage (the batched fitter's default)
        {"name": "batch_16", "kind": "batch", "instances": 16, "least": 2000, "most": 200_000},
        # a preview: a small scene in a small image, where latency counts
        {"name": "render_256", "kind": "render", "scene": "frustum", "width": 256, "height": 256,
         "focal": 256, "count": 4096, "sh": 0, "storage": "fp32"},
        # the viewer: a million splats with SH 3 at 1920 x 1080
        {"name": "render_1080p_sh3", "kind": "render", "scene": "orbit", "width": 1920,
         "height": 1080, "focal": 1200, "count": 1_000_000, "sh": 3, "storage": "fp32"},
        # the layer calls at the size of the initializer's rendered loss (512 x 512, 16384)
        {"name": "layers_512", "kind": "layers", "scene": "frustum", "width": 512, "height": 512,
         "focal": 512, "count": 16384, "sh": 0},
        # third convolution of the initializer: 64 -> 128 channels, stride 2
        {"name": "conv_64_128_s2", "kind": "conv", "batch": 8, "height": 256, "width": 256,
         "cin": 64, "cout": 128, "stride": 2},
        # fifth convolution of the initializer at its training batch of 32
        {"name": "conv_256_256", "kind": "conv", "batch": 32, "height": 64, "width": 64,
         "cin": 256, "cout": 256, "stride": 1},
        # the initializer on a batch of targets, as it is evaluated and trained
        {"name": "init_512", "kind": "init", "size": 512, "batch": 16},
    ]


def _between(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "batch", "render", "render", "layers", "conv", "conv",
                       "init"])
    if kind in ("fit", "render", "layers"):
        scene = rng.choice(["frustum", "orbit"])
        width = _between(rng, 128, 1280)
        case = {"kind": kind, "scene": scene, "width": width,
                "height": max(96, int(width * rng.uniform(0.5, 1.0))),
                "focal": int(width * (rng.uniform(0.75, 1.0) if scene == "frustum" else 0.625)),
                "count": _between(rng, 2000, 60_000 if scene == "frustum" else 600_000),
                "sh": rng.choice([0, 1, 2, 3])}
        if kind != "layers":
            case["storage"] = rng.choice(["fp32", "fp32", "bf16"])
        return case
    if kind == "batch":
        return {"kind": kind, "instances": rng.randint(2, 16), "least": 2000,
                "most": _between(rng, 4000, 200_000)}
    if kind == "conv":
        case = {"kind": kind, "batch": rng.randint(1, 8), "height": _between(rng, 17, 130),
                "width": _between(rng, 17, 130), "stride": rng.choice([1, 2])}
        case["cin"], case["cout"] = rng.choice([(3, 32), (32, 64), (64, 128), (128, 256),
                                                (256, 256), (256, 56)])
        while _conv_flops(*(case[k] for k in ("batch", "height", "width", "stride")), 1, 1)[0] % 8:
            case["batch"] += 1  # the backward takes a multiple of 8 output pixels
        return case
    return {"kind": kind, "size": 8 * _between(rng, 16, 64), "batch": rng.randint(1, 8)}


# ---- inputs --------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda")


def _normal(g, mean, std, *shape):
    return mean + std * torch.randn(*shape, generator=g, device="cuda")


def _target(g, width, height):
    """A colour gradient with 2000 blobs per 1280 x 720 of area (sigma 2 to 40
    pixels) and a faint checkerboard, in steps of 1/255."""
    blobs = max(100, 2000 * width * height // (1280 * 720))
    u = torch.arange(width, device="cuda") + 0.5
    v = torch.arange(height, device="cuda") + 0.5
    cx, cy = _uniform(g, 0, width, blobs, 1), _uniform(g, 0, height, blobs, 1)
    sigma, colour = _uniform(g, 2, 40, blobs, 1), _uniform(g, 0, 1, blobs, 3) - 0.5
    gx = torch.exp(-0.5 * ((u[None] - cx) / sigma) ** 2)
    gy = torch.exp(-0.5 * ((v[None] - cy) / sigma) ** 2)
    image = torch.stack([(gy * (0.5 * colour[:, c:c + 1])).T @ gx for c in range(3)], -1)
    du, dv = u[None] / width, v[:, None] / height
    image[..., 0] += 0.15 + 0.5 * du
    image[..., 1] += 0.15 + 0.5 * dv
    image[..., 2] += 0.65 - 0.25 * (du + dv)
    checker = (torch.floor(u[None] / 8) + torch.floor(v[:, None] / 8)) % 2
    image += (0.1 * checker - 0.05)[..., None]
    return (torch.round(image.clamp(0, 1) * 255) / 255).contiguous()


def _frustum(g, count, width, height, focal, sh):
    """The plain fitters' random splats and their pinhole camera."""
    f = float(focal)
    P = torch.zeros(14 + 3 * scenes.sh_bands(sh), count, device="cuda")
    z = _uniform(g, 2, 6, count)
    P[0] = (_uniform(g, 0, width, count) - width / 2) * z / f
    P[1] = (_uniform(g, 0, height, count) - height / 2) * z / f
    P[2] = z
    P[3:6] = _normal(g, -3.0, 0.5, 3, count)
    q = _normal(g, 0, 1, 4, count)
    P[6:10] = q / q.norm(dim=0, keepdim=True)
    P[10:13] = (_uniform(g, 0, 1, 3, count) - 0.5) / scenes.SH_C0
    if sh:
        P[14:] = _normal(g, 0, 0.05, P.shape[0] - 14, count)
    return P, scenes.pinhole_pv(width, height, f, f, width / 2, height / 2), np.zeros(3, np.float32)


def _orbit(g, count, width, height, focal, sh, seed):
    """The viewer's scene (20 planes and spheres around the origin) and one camera
    of its circle."""
    P = torch.zeros(14 + 3 * scenes.sh_bands(sh), count, device="cuda")
    which = torch.randint(0, 20, (count,), generator=g, device="cuda")
    c = _normal(g, 0, 1, 20, 3)
    c = c / c.norm(dim=1, keepdim=True) * _uniform(g, 0, 6, 20, 1)
    a = _normal(g, 0, 1, 20, 3)
    a = a / a.norm(dim=1, keepdim=True)
    b = torch.linalg.cross(a, _normal(g, 0, 1, 20, 3))
    b = b / b.norm(dim=1, keepdim=True)
    half, radius = _uniform(g, 1, 4, 20, 1), _uniform(g, 0.5, 3, 20, 1)
    uv = _uniform(g, -1, 1, count, 2) * half[which]
    plane = uv[:, :1] * a[which] + uv[:, 1:] * b[which]
    ball = _normal(g, 0, 1, count, 3)
    ball = ball / ball.norm(dim=1, keepdim=True) * radius[which]
    pos = c[which] + torch.where((which % 2 == 0)[:, None], plane, ball)
    pos = pos + _normal(g, 0, 0.02, count, 3)
    P[0:3] = (pos * (10 / pos.norm(dim=1, keepdim=True)).clamp(max=1)).T
    P[3:6] = _normal(g, -4.5, 0.7, 3, count)
    q = _normal(g, 0, 1, 4, count)
    P[6:10] = q / q.norm(dim=0, keepdim=True)
    P[10:13] = _normal(g, 0, 0.5, 3, count)
    P[13] = _normal(g, 0, 1.5, count)
    if sh:
        P[14:] = _normal(g, 0, 0.05, P.shape[0] - 14, count)
    cams = scenes.orbit_cameras(16, width=width, height=height, fx=float(focal))
    pv, eye = cams[seed % 16]
    return P, pv, eye


def _scene(case, seed):
    g = _generator(seed)
    size = case["count"], case["width"], case["height"], case["focal"], case["sh"]
    if case["scene"] == "orbit":
        P, pv, eye = _orbit(g, *size, seed)
    else:
        P, pv, eye = _frustum(g, *size)
    return P, pv, eye, _target(g, case["width"], case["height"])


def _rates(case):
    """A tenth of the plain fitters' rates, as late in a fit; in the orbit scene the
    positions have settled."""
    base = scenes.REFERENCE_LRS if case["width"] >= 512 else scenes.PLAIN_SMALL_LRS
    position = 1.6e-5 if case["scene"] == "orbit" else base[0]
    return tuple(0.1 * r for r in (position, *base[1:]))


def _storage(case):
    return _lib.DS_STORAGE_BF16 if case["storage"] == "bf16" else _lib.DS_STORAGE_FP32


def _has_moments(case):
    """Whether a fit returns its Adam moments beside its weights: BF16 storage has no
    FP32 ones, and in the orbit scene the gradients of splats thinner than a pixel
    amplify the last bit of their weights."""
    return case["storage"] == "fp32" and case["scene"] == "frustum"


BATCH_RATES = tuple(0.1 * r for r in scenes.PLAIN_SMALL_LRS)


def _batch_sizes(case):
    """Sizes that are part of the case, not of the seed: image sizes in turn, counts
    spread evenly over their logarithm."""
    k = case["instances"]
    lo, hi = math.log(case["least"]), math.log(case["most"])
    counts = [int(math.exp(lo + (hi - lo) * ((i * 7) % k) / max(1, k - 1))) for i in range(k)]
    return [(*scenes.BATCH_SIZES[i % len(scenes.BATCH_SIZES)], counts[i]) for i in range(k)]


def _batch_scene(size, seed, k):
    g = _generator(seed * 1009 + k)
    width, height, count = size
    return (*_frustum(g, count, width, height, width, 0), _target(g, width, height))


def _conv_inputs(case, seed):
    g = _generator(seed)
    B, H, W, s = case["batch"], case["height"], case["width"], case["stride"]
    Ho, Wo = (H - 1) // s + 1, (W - 1) // s + 1
    layer = nn.Conv3x3(case["cin"], case["cout"], s, gelu=True,
                       gen=torch.Generator().manual_seed(seed))
    layer.b.copy_(_normal(g, 0, 0.05, case["cout"]))
    # activations are GELU outputs, their pre-activations follow
    z_prev = _normal(g, 0, 1, B, H, W, case["cin"]).to(torch.bfloat16)
    x = torch.nn.functional.gelu(z_prev.float(), approximate="tanh").to(torch.bfloat16)
    dz = _normal(g, 0, 1e-3, B, Ho, Wo, case["cout"]).to(torch.bfloat16)
    return layer, x, z_prev, dz


def _network(case, seed):
    net = initializer.Initializer(case["size"], seed)
    g = torch.Generator().manual_seed(seed + 1)
    head = net.head  # a fresh head is zero; a trained one is not
    w = torch.randn(head.w.shape, generator=g) * 0.02
    w[:, 9 * head.cin:] = 0
    head.w.copy_(w)
    head.w16.copy_(w.to(torch.bfloat16))
    for m in net.modules():
        m.b.copy_(torch.randn(m.b.shape, generator=g) * 0.05)
    g = _generator(seed)
    images = torch.stack([_target(g, case["size"], case["size"]) for _ in range(case["batch"])])
    return net, images


class State:
    """What a case keeps between its passes."""

    def __init__(self, **kept):
        self.__dict__.update(kept)


class Outputs(dict):
    """Views of an object's own device memory, which live as long as the object."""

    def __init__(self, owner, **views):
        super().__init__(views)
        self.owner = owner


def _groups(P, G, M, V, lrs):
    rows = [(0, 3, lrs[0]), (3, 6, lrs[1]), (6, 10, lrs[2]), (10, 13, lrs[3]), (13, 14, lrs[5])]
    if P.shape[0] > 14:
        rows.append((14, P.shape[0], lrs[4]))
    return [(P[a:b], G[a:b], M[a:b], V[a:b], lr) for a, b, lr in rows]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fit":
        P, pv, eye, target = _scene(case, seed)
        f = api.Fitter(case["width"], case["height"], case["count"], case["sh"],
                       lrs=_rates(case), storage=_storage(case), eps=EPS)
        f.set_params(P)
        f.set_target(target)
        f.set_camera(pv, eye)
        out = Outputs(f, params=f.params, image=f.image(), loss=f.loss_device())
        if _has_moments(case):
            out["m"], out["v"] = f.moments()
        return State(case=case, fitter=f, out=out)
    if kind == "batch":
        sizes = _batch_sizes(case)
        b = api.Batch(sizes, lrs=BATCH_RATES, max_isects=1 << 25, ppt=2, eps=EPS)
        for k, size in enumerate(sizes):
            P, pv, eye, target = _batch_scene(size, seed, k)
            b.set_params(k, P)
            b.set_target(k, target)
            b.set_camera(k, pv, eye)
        out = Outputs(b, params=b.params, images=[b.image(k) for k in range(len(sizes))])
        return State(case=case, batch=b, out=out)
    if kind == "render":
        P, pv, eye, _ = _scene(case, seed)
        r = api.Renderer(case["width"], case["height"], case["count"], case["sh"],
                         storage=_storage(case))
        r.set_params(P)
        return State(case=case, renderer=r, pv=pv, eye=eye)
    if kind == "layers":
        P, pv, eye, target = _scene(case, seed)
        r = api.Rasterizer(case["width"], case["height"], case["count"], 1 << 23)
        return State(case=case, raster=r, params=P, pv=pv, eye=eye, target=target, step=0,
                     m=torch.zeros_like(P), v=torch.zeros_like(P), lrs=_rates(case))
    if kind == "conv":
        layer, x, z_prev, dz = _conv_inputs(case, seed)
        return State(case=case, layer=layer, x=x, z_prev=z_prev, dz=dz, gemm=nn.Gemm())
    net, images = _network(case, seed)
    return State(case=case, net=net, images=images)


def run(s):
    kind = s.case["kind"]
    if kind == "fit":
        s.fitter.step()
        return s.out
    if kind == "batch":
        s.batch.step()
        return s.out
    if kind == "render":
        return Outputs(s.renderer, image=s.renderer.render(s.pv, s.eye))
    if kind == "layers":
        sh, P = s.case["sh"], s.params
        s3 = api.activ_forward(P, sh, s.eye)
        s2 = api.project_forward(s3, s.pv)
        image = s.raster.forward(s2)
        loss = api.mse_forward(image, s.target)
        g2 = s.raster.backward(s2, api.mse_backward(image, s.target))
        g3 = api.project_backward(s3, s.pv, g2)
        grad = api.activ_backward(P, s3, g3, sh, s.eye)
        s.step += 1
        api.adam_step(_groups(P, grad, s.m, s.v, s.lrs), s.step, eps=EPS)
        return {"image": image, "loss": loss, "grad2d": g2, "grad": grad, "params": P}
    if kind == "conv":
        z, y = s.layer.forward(s.gemm, s.x)
        # the first layer of the network has no layer below it to pass a gradient to
        dx = s.layer.backward(s.gemm, s.dz, s.z_prev, need_dx=s.case["cin"] > 3)
        return {"z": z, "y": y, "dx": dx, "gw": s.layer.gw, "gb": s.layer.gb}
    out = s.net.forward(s.images)
    return {"head": out, "params": s.net.decode(out)}


# ---- what a pass cannot do without ---------------------------------------------


def _depth(case):
    """About how many splats a pixel composites before it is opaque or the list
    ends: the splats' mean footprint (a disc of 2.5 sigma) over the image."""
    if case["scene"] == "orbit":
        sigma = math.exp(-4.5) * case["focal"] / 15.0
        return min(40.0, case["count"] * math.pi * (2.5 * sigma) ** 2 /
                   (case["width"] * case["height"]))
    sigma = math.exp(-3.0) * case["focal"] / 4.0
    return min(100.0, case["count"] * math.pi * (2.5 * sigma) ** 2 /
               (case["width"] * case["height"]))


def _splat_work(case, backward):
    pixels, n = case["width"] * case["height"], case["count"]
    values = (14 + 3 * scenes.sh_bands(case["sh"])) * n
    lit = pixels * _depth(case)  # (pixel, splat) pairs that contribute
    if not backward:
        width = 2 if case.get("storage") == "bf16" else 4
        return values * width + 12.0 * pixels, 24.0 * lit + 200.0 * n
    # masters and both moments read and written; image, target and result
    moved = 24.0 if case.get("storage") != "bf16" else 8.0 + 2.0 + 8.0
    return values * moved + 24.0 * pixels, 94.0 * lit + 800.0 * n


def _conv_flops(B, H, W, stride, cin, cout):
    pixels = B * ((H - 1) // stride + 1) * ((W - 1) // stride + 1)
    return pixels, 2.0 * pixels * cout * 9 * cin


def work(case):
    kind = case["kind"]
    if kind in ("fit", "layers", "render"):
        b, f = _splat_work(case, kind != "render")
        return {"bytes": b, "flops": f}
    if kind == "batch":
        b = f = 0.0
        for w, h, n in _batch_sizes(case):
            one = _splat_work({"width": w, "height": h, "focal": w, "count": n, "sh": 0,
                               "storage": "bf16", "scene": "frustum"}, True)
            b, f = b + one[0], f + one[1]
        return {"bytes": b, "flops": f}
    if kind == "conv":
        B, H, W, cin, cout = (case[k] for k in ("batch", "height", "width", "cin", "cout"))
        pixels, flops = _conv_flops(B, H, W, case["stride"], cin, cout)
        inner = cin > 3
        weights = 9 * cin * cout
        moved = 2.0 * B * H * W * cin * (3 if inner else 1) + 2.0 * pixels * cout * 3
        return {"bytes": moved + 2.0 * weights + 4.0 * (weights + 2 * cout),
                "flops": flops * (3 if inner else 2)}
    side, cin, flops, weights = case["size"], 3, 0.0, 0
    for cout, stride in zip(initializer.CHANNELS + (56,), initializer.STRIDES + (1,)):
        flops += _conv_flops(case["batch"], side, side, stride, cin, cout)[1]
        weights += 9 * cin * cout
        side, cin = (side - 1) // stride + 1, cout
    values = case["batch"] * side * side * 56
    return {"bytes": 12.0 * case["batch"] * case["size"] ** 2 + 2.0 * weights + 8.0 * values,
            "flops": flops}


# ---- the same results in 64 bits, in plain torch -------------------------------


def _rotation(q):
    w, x, y, z = q / q.norm(dim=0, keepdim=True).clamp(min=1e-6)
    return [[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
            [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
            [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]]


def _sh_basis(degree, d):
    x, y, z = d
    basis = []
    if degree >= 1:
        c = 0.4886025119029199
        basis += [-c * y, c * z, -c * x]
    if degree >= 2:
        c = 1.0925484305920792
        basis += [c * x * y, -c * y * z, 0.31539156525252 * (2 * z * z - x * x - y * y),
                  -c * x * z, 0.5462742152960396 * (x * x - y * y)]
    if degree >= 3:
        basis += [-0.5900435899266435 * y * (3 * x * x - y * y), 2.890611442640554 * x * y * z,
                  -0.4570457994644658 * y * (4 * z * z - x * x - y * y),
                  0.3731763325901154 * z * (2 * z * z - 3 * x * x - 3 * y * y),
                  -0.4570457994644658 * x * (4 * z * z - x * x - y * y),
                  1.445305721320277 * z * (x * x - y * y),
                  -0.5900435899266435 * x * (x * x - 3 * y * y)]
    return basis


def _splat2d(P, pv, eye, sh):
    """Screen splats [10, n] (ndc xyz, cov xx xy yy, rgb, opacity) of parameters,
    differentiable as the framework's backward is: the projection's Jacobian and
    the view direction count as constants."""
    pv = torch.as_tensor(np.asarray(pv, np.float64), device="cuda").view(4, 4)  # [column][row]
    at = P[0:3]
    clip = pv[:3].T @ at + pv[3][:, None]
    w = torch.where(clip[3] > 0, clip[3], torch.ones_like(clip[3]))
    ndc = clip[:3] / w
    J = ((pv[:3, None, :2].permute(2, 0, 1) * w.detach() -
          clip[:2].detach()[:, None] * pv[:3, 3][None, :, None]) / w.detach() ** 2)  # [2][3][n]
    R, scale = _rotation(P[6:10]), P[3:6].exp()
    M = torch.stack([torch.stack([R[i][k] * scale[k] for k in range(3)]) for i in range(3)])
    JM = torch.einsum("rin,ikn->rkn", J, M)
    cov = torch.einsum("rkn,skn->rsn", JM, JM)
    away = torch.as_tensor(np.asarray(eye, np.float64), device="cuda")[:, None] - at.detach()
    basis = _sh_basis(sh, away / away.norm(dim=0, keepdim=True).clamp(min=1e-6))
    bands = len(basis)
    colour = []
    for c in range(3):
        v = scenes.SH_C0 * P[10 + c]
        for k in range(bands):
            v = v + basis[k] * P[14 + c * bands + k]
        colour.append((v + 0.5).clamp(0, 1))
    S = torch.stack([*ndc, cov[0, 0], cov[0, 1], cov[1, 1], *colour, torch.sigmoid(P[13])])
    return S, clip[3] > 0


def _tile_lists(S, front, width, height):
    """Tiles' splat lists in depth order: (pairs' splats, first pair of each tile,
    pairs of each tile)."""
    x, y, z, xx, xy, yy = S[:6]
    ntx, nty = -(-width // TILE), -(-height // TILE)
    ex, ey = 3 * xx.clamp(min=0).sqrt(), 3 * yy.clamp(min=0).sqrt()
    ok = front & (x.abs() <= 1) & (y.abs() <= 1) & (z.abs() <= 1) & (xx * yy - xy * xy > 0)
    ok &= 2 * torch.maximum(ex, ey) >= max(2 / width, 2 / height)
    fx, fy = width / TILE, height / TILE
    x0 = ((x - ex + 1) * 0.5 * fx).floor().clamp(0, 1e6).long()
    x1 = ((x + ex + 1) * 0.5 * fx).floor().clamp(-1, ntx - 1).long()
    y0 = ((1 - y - ey) * 0.5 * fy).floor().clamp(0, 1e6).long()
    y1 = ((1 - y + ey) * 0.5 * fy).floor().clamp(-1, nty - 1).long()
    ok &= (x0 <= x1) & (y0 <= y1)
    order = torch.sort(z.float(), stable=True).indices  # equal 32-bit depths by index
    order = order[ok[order]]
    wide = (x1 - x0 + 1)[order]
    count = wide * (y1 - y0 + 1)[order]
    splat = torch.repeat_interleave(order, count)
    k = torch.arange(splat.numel(), device="cuda") - torch.repeat_interleave(
        count.cumsum(0) - count, count)
    wide = torch.repeat_interleave(wide, count)
    tile = (y0[splat] + k // wide) * ntx + x0[splat] + k % wide
    tile, by = torch.sort(tile, stable=True)
    length = torch.bincount(tile, minlength=ntx * nty)
    return splat[by], length.cumsum(0) - length, length


def _composite(S, lists, width, height, pixel_grad=None):
    """The image [H, W, 3]; with pixel_grad(image of the pixels, their indices) also
    the gradient [10, n] of the screen splats, by the framework's recurrence."""
    splat, first, length = lists
    ntx = -(-width // TILE)
    image = torch.zeros(height * width, 3, dtype=torch.float64, device="cuda")
    grad = torch.zeros_like(S) if pixel_grad else None
    order = torch.sort(length, descending=True).indices
    order = order[length[order] > 0]
    lengths = length[order].tolist()
    at = 0
    lane = torch.arange(TILE * TILE, device="cuda")
    while at < len(lengths):
        L = lengths[at]
        tiles = order[at:at + max(1, (1 << 24) // (L * TILE * TILE))]
        at += len(tiles)
        slot = torch.arange(L, device="cuda")
        real = slot[None] < length[tiles][:, None]
        g = splat[(first[tiles][:, None] + slot[None]).clamp(max=splat.numel() - 1)]  # [t, L]
        col = (tiles % ntx)[:, None] * TILE + lane[None] % TILE
        row = (tiles // ntx)[:, None] * TILE + lane[None] // TILE
        inside = (col < width) & (row < height)
        px = (2 * (col + 0.5) / width - 1)[:, None]  # [t, 1, 256]
        py = (1 - 2 * (row + 0.5) / height)[:, None]
        v = S[:, g]  # [10, t, L]
        det = v[3] * v[5] - v[4] * v[4]
        a, b, c = v[5] / det, -v[4] / det, v[3] / det
        dx, dy = v[0][..., None] - px, v[1][..., None] - py
        u, w = a[..., None] * dx + b[..., None] * dy, b[..., None] * dx + c[..., None] * dy
        sigma = 0.5 * (dx * u + dy * w)
        soft = v[9][..., None] * torch.exp(-sigma)
        alpha = soft.clamp(max=0.99)
        alpha = torch.where((sigma < 0) | (alpha < 1 / 255) | ~real[..., None],
                            torch.zeros_like(alpha), alpha)
        T = torch.cumprod(1 - alpha, 1)
        T = torch.cat([torch.ones_like(T[:, :1]), T[:, :-1]], 1)  # before each splat
        weight = torch.where(T > 1e-4, alpha * T, torch.zeros_like(T))
        rgb = torch.einsum("tlp,ctl->tpc", weight, v[6:9])
        where = (row * width + col)[inside]
        image[where] = rgb[inside]
        if not pixel_grad:
            continue
        gp = torch.zeros_like(rgb)
        gp[inside] = pixel_grad(rgb[inside], where)
        lit = torch.einsum("ctl,tpc->tlp", v[6:9], gp)
        behind = weight * lit
        behind = behind.sum(1, keepdim=True) - behind.cumsum(1)
        g_alpha = torch.where(weight > 0, T * (lit - behind), torch.zeros_like(T))
        s = torch.where(soft <= 0.99, soft * g_alpha, torch.zeros_like(T))
        parts = [-(s * u).sum(2), -(s * w).sum(2), torch.zeros_like(a), 0.5 * (s * u * u).sum(2),
                 (s * u * w).sum(2), 0.5 * (s * w * w).sum(2),
                 *torch.einsum("tlp,tpc->ctl", weight, gp), s.sum(2) / v[9]]
        for k, part in enumerate(parts):
            grad[k].index_add_(0, g[real], part[real])
    return image.view(height, width, 3), grad


def _exact_step(P, pv, eye, target, sh, lrs, bf16=False):
    """One training step from zero moments: image, loss, gradients, new parameters."""
    height, width = target.shape[:2]
    master = P.double()
    seen = P.double()
    if bf16:  # everything but the positions is rendered from a BF16 copy
        seen = torch.cat([seen[:3], P[3:].to(torch.bfloat16).double()])
    seen.requires_grad_(True)
    S, front = _splat2d(seen, pv, eye, sh)
    target = target.double().view(-1, 3)
    pixels = height * width
    with torch.no_grad():
        lists = _tile_lists(S, front, width, height)
        image, g2 = _composite(S.detach(), lists, width, height,
                               lambda rgb, at: 2.0 / pixels * (rgb - target[at]))
        loss = ((image.view(-1, 3) - target) ** 2).sum().view(1) / pixels
        g2 = torch.where(front[None], g2, torch.zeros_like(g2))
    grad, = torch.autograd.grad(S, seen, g2)
    rate = torch.empty(P.shape[0], 1, dtype=torch.float64, device="cuda")
    for k, (a, b) in enumerate([(0, 3), (3, 6), (6, 10), (10, 13), (14, P.shape[0]), (13, 14)]):
        rate[a:b] = lrs[k]
    new = master - rate * grad / (grad.abs() + EPS)
    return {"image": image, "loss": loss, "grad2d": g2, "grad": grad, "params": new}


def _taps(x, H, W, stride):
    """The nine shifted inputs of a padded 3x3 convolution, [B, Ho, Wo, C] each."""
    x = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    Ho, Wo = (H - 1) // stride + 1, (W - 1) // stride + 1
    return [x[:, ky:ky + stride * (Ho - 1) + 1:stride, kx:kx + stride * (Wo - 1) + 1:stride]
            for ky in range(3) for kx in range(3)]


def _exact_conv(x, w16, bias, cin, stride):
    w = w16.double()
    z = bias.double()
    for k, tap in enumerate(_taps(x, x.shape[1], x.shape[2], stride)):
        z = z + tap.double() @ w[:, k * cin:(k + 1) * cin].T
    return z


def _gelu_slope(z):
    z = z.double().requires_grad_(True)
    y = torch.nn.functional.gelu(z, approximate="tanh")
    return torch.autograd.grad(y.sum(), z)[0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "render":
        P, pv, eye, _ = _scene(case, seed)
        P = P.double() if case["storage"] == "fp32" else torch.cat(
            [P[:3].double(), P[3:].to(torch.bfloat16).double()])
        S, front = _splat2d(P, pv, eye, case["sh"])
        lists = _tile_lists(S, front, case["width"], case["height"])
        return {"image": _composite(S, lists, case["width"], case["height"])[0]}
    if kind in ("fit", "layers"):
        P, pv, eye, target = _scene(case, seed)
        e = _exact_step(P, pv, eye, target, case["sh"], _rates(case),
                        case.get("storage") == "bf16")
        if kind == "layers":
            return e
        out = {"params": e["params"], "image": e["image"], "loss": e["loss"]}
        if _has_moments(case):
            out["m"], out["v"] = 0.1 * e["grad"], 0.001 * e["grad"] ** 2
        return out
    if kind == "batch":
        steps = [_exact_step(*_batch_scene(size, seed, k), 0, BATCH_RATES, True)
                 for k, size in enumerate(_batch_sizes(case))]
        return {"params": torch.cat([e["params"] for e in steps], 1),
                "images": [e["image"] for e in steps]}
    if kind == "conv":
        layer, x, z_prev, dz = _conv_inputs(case, seed)
        B, H, W, cin, stride = (case[k] for k in ("batch", "height", "width", "cin", "stride"))
        z = _exact_conv(x, layer.w16, layer.b, cin, stride)
        flat = dz.double().view(-1, case["cout"])
        gw = torch.zeros(case["cout"], layer.kp, dtype=torch.float64, device="cuda")
        dx = torch.zeros(B, H + 2, W + 2, cin, dtype=torch.float64, device="cuda")
        into = _taps(dx[:, 1:-1, 1:-1], H, W, stride)  # shapes only
        for k, tap in enumerate(_taps(x, H, W, stride)):
            cols = slice(k * cin, (k + 1) * cin)
            gw[:, cols] = flat.T @ tap.double().reshape(-1, cin)
            ky, kx, (_, Ho, Wo, _) = k // 3, k % 3, into[k].shape
            dx[:, ky:ky + stride * (Ho - 1) + 1:stride, kx:kx + stride * (Wo - 1) + 1:stride] += (
                flat @ layer.w16.double()[:, cols]).view(B, Ho, Wo, cin)
        dx = dx[:, 1:-1, 1:-1] * _gelu_slope(z_prev)
        return {"z": z, "y": torch.nn.functional.gelu(z, approximate="tanh"),
                "dx": dx.contiguous() if cin > 3 else None, "gw": gw, "gb": flat.sum(0)}
    net, images = _network(case, seed)
    x = images.to(torch.bfloat16).double()
    for layer in net.layers:
        x = torch.nn.functional.gelu(_exact_conv(x, layer.w16, layer.b, layer.cin, layer.stride),
                                     approximate="tanh")
    out = _exact_conv(x, net.head.w16, net.head.b, net.head.cin, 1).view(-1, 56)
    o = out.view(case["batch"], -1, 14)  # splats of an image, 14 channels each
    p = o.clone()
    p[..., 0:3] = net.base.double().view(1, -1, 3) + o[..., 0:3] * torch.tensor(
        net.step, dtype=torch.float64, device="cuda")
    p[..., 3:6] = net.base_ls + o[..., 3:6]
    p[..., 6] = 1 + o[..., 6]
    return {"head": out, "params": p.view(-1, 14).T.contiguous()}
