"""The calls whose speed is tracked: inputs, one pass through the public entry
points, and reference values in 64 bits.

Kinds of case (``case["kind"]``):

* ``detect``: ``PySIFT.detectAndCompute(gray, gpu_output=True)`` of a device
  image, or, with ``host``, ``PySIFT.detect_arrays`` from and to host memory.
* ``batch``: ``PySIFT.detect_batch`` of images of uneven sizes.
* ``match``: one brute-force ratio-test matching of two descriptor sets
  (``match_u8_exact``, ``match_u8_split_fp8``, ``match_fp16``, ``match_i8``).
* ``stitch``: ``GPUPyStitch.stitch(img1, img2)`` to the cropped panorama.
* ``desc_grad``: differentiable descriptors, forward and backward.
* ``warp_grad``: differentiable warp + feather blend, forward and backward.

Detections and panoramas have as many rows as the image gives; ``run`` puts
them into buffers of a fixed size, as a program that stacks the results of
several images does.
"""
import functools
import math

import numpy as np
import torch

from pysift_b200 import PySIFT, grad, match, synthetic
from pysift_b200.stitch import GPUPyStitch

DEV = "cuda"
ASPECTS = ((4, 3), (3, 2), (16, 9))


def listed():
    return [
        # the smallest detection in use (a thumbnail): launches and latency
        dict(name="detect_320x240", kind="detect", H=240, W=320, options="default", host=False),
        # the plain detection configuration, host image in and host arrays out
        dict(name="detect_640x480_host", kind="detect", H=480, W=640, options="default", host=True),
        # the reference's golden-dump configuration (4 octaves, binary16
        # pyramid, DSP-5 descriptors) at an odd size
        dict(name="detect_1023x767_dsp5_fp16", kind="detect", H=767, W=1023, options="dsp5_fp16", host=False),
        # the largest image of the batch workload (12 Mpix, still doubled)
        dict(name="detect_4000x3000", kind="detect", H=3000, W=4000, options="default", host=False),
        # a batch of uneven images over the streams
        dict(name="batch_12_uneven", kind="batch", n=12, wmin=480, wmax=2000, graph=False),
        # a small pair of sets, int8 rows of the int8_matching option
        dict(name="match_i8_997x613", kind="match", mode="i8", N=997, M=613, D=64),
        # the precision/matching configuration
        dict(name="match_u8_8192", kind="match", mode="u8", N=8192, M=8192, D=128),
        # the stitch path's sets: PCA-64, fp16, uneven and off the tile grid
        dict(name="match_fp16_7919x5003", kind="match", mode="fp16", N=7919, M=5003, D=64),
        # the plain stitch configuration, device images
        dict(name="stitch_1280x960", kind="stitch", H=960, W=1280, ransac_iters=2048, host=False),
        # the upper end of the batched stitch's sizes, host images
        dict(name="stitch_2999x1999_host", kind="stitch", H=1999, W=2999, ransac_iters=4096, host=True),
        # the differentiation configuration, one image
        dict(name="desc_grad_1024x768", kind="desc_grad", H=768, W=1024, K=2000),
        dict(name="warp_grad_1024x768", kind="warp_grad", H=768, W=1024, C=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, wmin, wmax):
    """A width spread over the logarithm of the range, with its height; any parity."""
    w = _log(rng, wmin, wmax)
    aw, ah = ASPECTS[rng.randrange(3)]
    return min(wmax * 3 // 4, max(2, w * ah // aw + rng.randrange(3))), w


def draw(rng):
    kind = rng.choice(("detect", "detect", "detect", "batch", "match", "match", "match", "stitch", "stitch",
                       "desc_grad", "warp_grad"))
    if kind == "detect":
        options = rng.choice(("default", "default", "dsp5_fp16", "no_doubling"))
        H, W = _size(rng, 320, 2000 if options == "dsp5_fp16" else 4000)
        return dict(kind=kind, H=H, W=W, options=options, host=rng.random() < 0.3)
    if kind == "batch":
        lo = _log(rng, 320, 1000)
        return dict(kind=kind, n=rng.randint(3, 12), wmin=lo, wmax=_log(rng, lo, 2000), graph=rng.random() < 0.5)
    if kind == "match":
        mode = rng.choice(("u8", "u8", "fp16", "fp16", "i8", "split_fp8"))
        return dict(kind=kind, mode=mode, N=_log(rng, 500, 16000), M=_log(rng, 500, 16000),
                    D=128 if mode in ("u8", "split_fp8") else rng.choice((64, 64, 128)))
    if kind == "stitch":
        H, W = _size(rng, 640, 3000)
        return dict(kind=kind, H=H, W=W, ransac_iters=rng.choice((1500, 2048, 4096)), host=rng.random() < 0.5)
    H, W = _size(rng, 240, 1400)
    if kind == "desc_grad":
        return dict(kind=kind, H=H, W=W, K=_log(rng, 100, 2000))
    return dict(kind=kind, H=H, W=W, C=rng.choice((1, 3)))


# -- inputs ------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _gauss1(t, sigma=1.0):
    r = int(4 * sigma + 0.5)
    x = torch.arange(-r, r + 1, device=DEV, dtype=torch.float32)
    k = torch.exp(-0.5 * (x / sigma) ** 2)
    k = k / k.sum()
    t = torch.nn.functional.pad(t[None, None], (r, r, r, r), mode="reflect")
    t = torch.nn.functional.conv2d(t, k.view(1, 1, 1, -1))
    return torch.nn.functional.conv2d(t, k.view(1, 1, -1, 1))[0, 0]


def _scene(H, W, seed):
    """Rectangles (intensity 30-220), Gaussian blobs (sigma 2-25 px, amplitude
    +-80) and band-limited noise (sigma 1, std 6) on 128: the scene of
    pysift_b200.synthetic, drawn on the device; float32."""
    rng = np.random.default_rng([int(seed), 1])
    img = torch.full((H, W), 128.0, device=DEV)
    for _ in range(50):
        h, w = int(rng.uniform(8, max(9, H / 4))), int(rng.uniform(8, max(9, W / 4)))
        y, x = int(rng.uniform(0, H - h)), int(rng.uniform(0, W - w))
        img[y:y + h, x:x + w] = rng.uniform(30, 220)
    yy, xx = torch.arange(H, device=DEV).float(), torch.arange(W, device=DEV).float()
    for _ in range(200):
        s, a = rng.uniform(2, 25), rng.uniform(-80, 80)
        cy, cx = rng.uniform(0, H), rng.uniform(0, W)
        r = int(4 * s + 1)
        y0, y1, x0, x1 = max(0, int(cy) - r), min(H, int(cy) + r + 1), max(0, int(cx) - r), min(W, int(cx) + r + 1)
        gy = torch.exp(-(yy[y0:y1] - cy) ** 2 / (2 * s * s))
        gx = torch.exp(-(xx[x0:x1] - cx) ** 2 / (2 * s * s))
        img[y0:y1, x0:x1] += a * gy[:, None] * gx[None, :]
    noise = _gauss1(torch.randn((H, W), device=DEV, generator=_gen(seed)))
    return img + noise * (6.0 / noise.std())


def _u8(t):
    return t.round().clamp(0, 255).to(torch.uint8)


def _gray(H, W, seed):
    return _u8(_scene(H, W, seed))


def _homography(H, W, seed, shift=1.0):
    """View 1 -> view 2 of a stitch pair: 30-40 % overlap at shift = 1."""
    Hm = synthetic.random_homography(np.random.default_rng([int(seed), 2]), W, H)
    Hm[0, 2] *= shift
    return Hm


def _sample(img, Hm, H, W):
    """(C, h, w) image seen through the inverse of Hm on an H x W grid."""
    Hi = torch.from_numpy(np.linalg.inv(Hm)).to(DEV)
    v, u = torch.meshgrid(torch.arange(H, device=DEV).double(), torch.arange(W, device=DEV).double(), indexing="ij")
    p = Hi @ torch.stack([u.reshape(-1), v.reshape(-1), torch.ones(H * W, device=DEV, dtype=torch.float64)])
    h, w = img.shape[1:]
    g = torch.stack([2 * (p[0] / p[2]) / (w - 1) - 1, 2 * (p[1] / p[2]) / (h - 1) - 1], -1).float().view(1, H, W, 2)
    return torch.nn.functional.grid_sample(img[None], g, mode="bilinear", padding_mode="reflection",
                                           align_corners=True)[0]


def _views(H, W, seed):
    """Two overlapping BGR uint8 views of one scene, sensor noise of std 2."""
    Hm = _homography(H, W, seed)
    bw, bh = int(W * 2.2), int(H * 1.4)
    oy = (bh - H) // 2
    gains = np.random.default_rng([int(seed), 3]).uniform(0.8, 1.2, size=3)
    base = _scene(bh, bw, seed)
    big = torch.stack([(base * float(g)).clamp(0, 255) for g in gains])
    S = np.array([[1, 0, 0], [0, 1, -oy], [0, 0, 1]], np.float64)
    g = _gen(int(seed) + 1)
    views = [big[:, oy:oy + H, :W], _sample(big, Hm @ S, H, W)]
    return [_u8(v + 2 * torch.randn(v.shape, device=DEV, generator=g)).permute(1, 2, 0).contiguous() for v in views]


def _descriptors(N, M, seed):
    """uint8 128-d sets with the distribution of SIFT descriptors; half of the
    second set are copies of rows of the first within +-3 levels."""
    g = _gen(seed)

    def rows(n):
        v = torch.randn((n, 128), device=DEV, generator=g).square() + 1e-6   # gamma(1/2)
        v = (v / v.norm(dim=1, keepdim=True)).clamp(max=0.2)
        return (v / v.norm(dim=1, keepdim=True) * 512).round().clamp(0, 255)

    a, b = rows(N), rows(M)
    k = min(M // 2, N)
    src, dst = torch.randperm(N, device=DEV, generator=g)[:k], torch.randperm(M, device=DEV, generator=g)[:k]
    b[dst] = (a[src] + torch.randint(-3, 4, (k, 128), device=DEV, generator=g)).clamp(0, 255)
    return a.to(torch.uint8), b.to(torch.uint8), k


def _unit_rows(a, D):
    """Normalised rows of D dimensions, as the stitch's matcher takes them."""
    x = a.float() / 512
    if D < 128:
        q = torch.linalg.qr(torch.randn((128, 128), generator=torch.Generator().manual_seed(7)))[0][:, :D].to(DEV)
        x = (x - 0.06) @ q
    return x / x.norm(dim=1, keepdim=True)


def _table(H, W, K, seed):
    """K fixed keypoints [octave, scale index, row, column, angle in degrees]:
    most of them in the fine octaves, as a detection gives them."""
    rng = np.random.default_rng([int(seed), 4])
    top = max(1, min(4, int(math.log2(min(H, W) / 48.0)) + 1))
    o = np.minimum(rng.geometric(0.6, K) - 1, top - 1)
    si = rng.integers(1, 4, K)
    r = (rng.uniform(2, (H >> o) - 3)).astype(int)
    c = (rng.uniform(2, (W >> o) - 3)).astype(int)
    return torch.from_numpy(np.stack([o, si, r, c, rng.uniform(0, 360, K)], 1).astype(np.float64))


OPTIONS = {
    "default": {},
    "no_doubling": dict(double_image=False),
    "dsp5_fp16": dict(n_octaves=4, dsp=True, dsp_n_scales=5, fp16_pyramid=True),
}


@functools.lru_cache(maxsize=1)
def _detector(options, sizes):
    """The detector that a program keeps for its images (one set of sizes at a time here)."""
    return PySIFT(**OPTIONS[options])


def _batch_sizes(case):
    rng = np.random.default_rng([case["n"], case["wmin"], case["wmax"]])
    out = []
    for _ in range(case["n"]):
        w = int(rng.uniform(case["wmin"], case["wmax"] + 1))
        aw, ah = ASPECTS[int(rng.integers(0, 3))]
        out.append((w * ah // aw, w))
    return out


def _rows(H, W):
    """Output rows of a detection of an H x W image in the fixed-size buffers."""
    return int(min(32000, 256 + H * W // 32))


# -- one pass ------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "detect":
        H, W = case["H"], case["W"]
        img = _gray(H, W, seed)
        s.update(sift=_detector(case["options"], ((H, W),)), img=img.cpu().numpy() if case["host"] else img,
                 rows=_rows(H, W))
    elif kind == "batch":
        sizes = tuple(_batch_sizes(case))
        s.update(sift=_detector("default", sizes), rows=sum(_rows(*hw) for hw in sizes),
                 imgs=[_gray(h, w, seed * 1000 + i) for i, (h, w) in enumerate(sizes)])
    elif kind == "match":
        a, b, k = _descriptors(case["N"], case["M"], seed)
        s["k"] = k
        if case["mode"] in ("u8", "split_fp8"):
            fn = match.match_u8_exact if case["mode"] == "u8" else match.match_u8_split_fp8
            s.update(fn=fn, args=(a, b))
        else:
            x, y = _unit_rows(a, case["D"]), _unit_rows(b, case["D"])
            if case["mode"] == "fp16":
                s.update(fn=match.match_fp16, args=(x.half(), y.half()))
            else:
                s.update(fn=match.match_i8, args=(*match.quantize_i8(x), *match.quantize_i8(y)))
    elif kind == "stitch":
        H, W = case["H"], case["W"]
        v = _views(H, W, seed)
        # a stitcher keeps the PCA basis of its first pair: one for each pair here
        s.update(imgs=[x.cpu().numpy() for x in v] if case["host"] else v,
                 stitcher=GPUPyStitch(ransac_iters=case["ransac_iters"], inlier_thresh=4.0, save_output=False,
                                      verbose=False),
                 frame=torch.zeros((2 * H, 3 * W, 3), dtype=torch.uint8))
    elif kind == "desc_grad":
        x = (_scene(case["H"], case["W"], seed) / 255).clamp(0, 1)
        target = torch.rand((case["K"], 128), device=DEV, generator=_gen(seed)) * 0.2
        s.update(sift=PySIFT(double_image=False), x=x.requires_grad_(True), target=target,
                 table=_table(case["H"], case["W"], case["K"], seed))
    else:
        H, W = case["H"], case["W"]
        a, b, t, h8, geo = _warp_inputs(case, seed)
        s.update(a=a.requires_grad_(True), b=b.requires_grad_(True), h8=h8.requires_grad_(True), target=t, geo=geo)
        assert geo == grad.canvas_geometry((H, W), (H, W), _homography(H, W, H * W, 0.3))
    return s


def _warp_inputs(case, seed):
    H, W, C = case["H"], case["W"], case["C"]
    Hm = _homography(H, W, H * W, 0.3)  # one view change for each size: the canvas follows from it
    geo = _geometry(H, W, Hm)
    a = torch.stack([_scene(H, W, seed * 10 + c) for c in range(C)]) / 255
    b = _sample(a, Hm, H, W)
    t = torch.rand((geo[1], geo[0], C), device=DEV, generator=_gen(seed))
    h8 = torch.from_numpy(Hm.ravel()[:8].copy()).to(DEV)
    return a.permute(1, 2, 0).contiguous(), b.permute(1, 2, 0).contiguous(), t, h8, geo


def _geometry(H, W, Hm):
    """(width, height, ox, oy, round(ox), round(oy)) of the canvas of two H x W views."""
    q = Hm @ np.array([[0, 0, 1], [W, 0, 1], [W, H, 1], [0, H, 1]], np.float64).T
    x, y = np.concatenate([q[0] / q[2], [0, W, W, 0]]), np.concatenate([q[1] / q[2], [0, 0, H, H]])
    ox, oy = max(0.0, -x.min()), max(0.0, -y.min())
    return (int(np.ceil(x.max() + ox)) + 1, int(np.ceil(y.max() + oy)) + 1, float(ox), float(oy), int(round(ox)),
            int(round(oy)))


def _padded(t, rows):
    out = t.new_zeros((rows, *t.shape[1:]))
    out[:t.shape[0]] = t[:rows]
    return out


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "detect":
        if case["host"]:
            out = s["sift"].detect_arrays(s["img"])
            return {k: _padded(torch.from_numpy(v), s["rows"]) for k, v in out.items()}
        return tuple(_padded(t, s["rows"]) for t in s["sift"].detectAndCompute(s["img"], gpu_output=True))
    if kind == "batch":
        out = s["sift"].detect_batch(s["imgs"], graph=case["graph"])
        return tuple(_padded(torch.cat(t), s["rows"]) for t in zip(*out))
    if kind == "match":
        m = s["fn"](*s["args"], 0.75)
        return {"count": m["count"], "pairs": m["pairs"][:s["k"]], "dist": m["dist"][:s["k"]],
                "fwd_best": m["fwd_best"], "fwd_pass": m["fwd_pass"], "bwd_best": m["bwd_best"],
                "bwd_pass": m["bwd_pass"]}
    if kind == "stitch":
        pano = s["stitcher"].stitch(*s["imgs"])
        s["frame"][:pano.shape[0], :pano.shape[1]] = torch.from_numpy(pano)
        return s["frame"], pano.shape[0], pano.shape[1]
    if kind == "desc_grad":
        s["x"].grad = None
        d = grad.descriptors(s["x"], s["table"], s["sift"])
        ((d - s["target"]) ** 2).sum().backward()
        return d.detach(), s["x"].grad
    for k in ("a", "b", "h8"):
        s[k].grad = None
    out = grad.warp_blend(s["a"], s["b"], s["h8"], s["geo"])
    ((out - s["target"]) ** 2).sum().backward()
    return out.detach(), s["a"].grad, s["b"].grad, s["h8"].grad


# -- what a pass cannot do without -----------------------------------------------
def _detect_work(H, W, options):
    """The image in, the Gaussian levels of every octave written once (they
    exceed the chip's memory before the last one is read), keypoints and
    descriptors out; two separable passes of 6 sigma taps a level and about
    40 operations a sample of a keypoint's patch."""
    scale = 1 if options == "no_doubling" else 4
    octaves = 4 if options == "dsp5_fp16" else 5
    px = sum((H * W * scale) >> (2 * o) for o in range(octaves))
    n = min(10000, H * W // 100)
    return H * W + 4 * 6 * px + n * 532, px * 5 * 2 * 2 * 17 + n * 40 * 2500 * (5 if "dsp" in options else 1)


def work(case):
    kind = case["kind"]
    if kind == "detect":
        b, f = _detect_work(case["H"], case["W"], case["options"])
    elif kind == "batch":
        each = [_detect_work(h, w, "default") for h, w in _batch_sizes(case)]
        b, f = sum(e[0] for e in each), sum(e[1] for e in each)
    elif kind == "match":
        N, M, D = case["N"], case["M"], case["D"]
        b = (N + M) * (D * (2 if case["mode"] == "fp16" else 1) + 8) + 12 * min(M // 2, N)
        f = 2 * N * M * D
    elif kind == "stitch":
        H, W = case["H"], case["W"]
        b, f = _detect_work(H, W, "dsp5_fp16")
        # the views read twice (features, warp), the panorama (about 1.6 views) out
        b, f = 2 * b + 12 * H * W + int(4.8 * H * W), 2 * f + 2 * 8000 * 8000 * 64
    elif kind == "desc_grad":
        H, W, K = case["H"], case["W"], case["K"]
        px = sum((H * W) >> (2 * o) for o in range(4))
        # image and gradients; the levels once forward, once backward, their adjoints once
        b, f = 8 * H * W + 3 * 4 * 4 * px + K * 128 * 12, 3 * px * 4 * 2 * 2 * 17 + 3 * K * 40 * 2500
    else:
        H, W, C = case["H"], case["W"], case["C"]
        # two images and the output forward; the images, the output's gradient and two gradients backward
        b, f = 4 * C * H * W * (2 + 2 + 2 + 2 + 2), 60 * C * 2 * H * W
    return {"bytes": b, "flops": f}


# -- 64-bit values -----------------------------------------------------------------
def _mirror(n, r):
    i = torch.arange(-r, n + r, device=DEV)
    i = torch.where(i < 0, -i - 1, i)
    return torch.where(i >= n, 2 * n - 1 - i, i)


def _blur64(x, sigma):
    r = int(4 * sigma + 0.5)
    t = np.arange(-r, r + 1, dtype=np.float64)
    k = np.exp(-0.5 * (t / sigma) ** 2)
    k = torch.from_numpy(k / k.sum()).to(DEV)
    H, W = x.shape
    xi = x[:, _mirror(W, r)]
    h = sum(k[j] * xi[:, j:j + W] for j in range(2 * r + 1))
    hi = h[_mirror(H, r)]
    return sum(k[j] * hi[j:j + H] for j in range(2 * r + 1))


def _descriptor64(G, kp, ph):
    """4x4x8 gradient histograms of the (2 ph + 1)^2 patches at rows [row,
    column, angle], normalised, clipped at 0.2 and normalised again."""
    H, W = G.shape
    off = torch.arange(-ph, ph + 1, device=DEV)
    dr, dc = off.repeat_interleave(2 * ph + 1), off.repeat(2 * ph + 1)
    r, c = kp[:, :1].long() + dr, kp[:, 1:2].long() + dc
    ang = torch.deg2rad(kp[:, 2:3])
    xr = torch.cos(ang) * dc - torch.sin(ang) * dr
    yr = torch.sin(ang) * dc + torch.cos(ang) * dr
    xb, yb = xr * (2.0 / ph) + 1.5, yr * (2.0 / ph) + 1.5
    ok = (r >= 1) & (r < H - 1) & (c >= 1) & (c < W - 1) & (xb >= -0.5) & (xb < 3.5) & (yb >= -0.5) & (yb < 3.5)
    k, p = ok.nonzero(as_tuple=True)
    r, c, xr, yr, xb, yb, ang = r[k, p], c[k, p], xr[k, p], yr[k, p], xb[k, p], yb[k, p], ang[k, 0]
    dx, dy = G[r, c + 1] - G[r, c - 1], G[r + 1, c] - G[r - 1, c]
    m2 = dx * dx + dy * dy
    some = m2 > 0
    mag = torch.sqrt(torch.where(some, m2, torch.ones_like(m2))) * some
    ori = torch.rad2deg(torch.atan2(dy, dx) - ang) + 360.0
    ori = torch.where(ori >= 360.0, ori - 360.0, ori) / 45.0
    wm = mag * torch.exp(-(xr * xr + yr * yr) / (2.0 * (ph * 0.5657) ** 2))
    x0, y0, o0 = torch.floor(xb), torch.floor(yb), torch.floor(ori).detach()
    fx, fy, fo = xb - x0, yb - y0, ori - o0
    hist = torch.zeros(kp.shape[0] * 128, dtype=torch.float64, device=DEV)
    for j in (0, 1):
        for i in (0, 1):
            for o in (0, 1):
                b = (y0 + j).clamp(0, 3) * 32 + (x0 + i).clamp(0, 3) * 8 + torch.remainder(o0 + o, 8)
                wt = (fy if j else 1 - fy) * (fx if i else 1 - fx) * (fo if o else 1 - fo)
                hist = hist.index_add(0, k * 128 + b.long(), wt * wm)
    hist = hist.view(-1, 128)
    t = (hist / torch.sqrt((hist * hist).sum(1, keepdim=True) + 1e-14)).clamp(max=0.2)
    return t / torch.sqrt((t * t).sum(1, keepdim=True) + 1e-14)


def _exact_desc_grad(case, seed):
    H, W, K = case["H"], case["W"], case["K"]
    x = (_scene(H, W, seed) / 255).clamp(0, 1).double().requires_grad_(True)
    target = torch.rand((K, 128), device=DEV, generator=_gen(seed)) * 0.2
    table = _table(H, W, K, seed)
    kf = 2.0 ** (1 / 3)
    sig = [1.6 * kf ** i for i in range(6)]
    level = _blur64(x, math.sqrt(1.6 ** 2 - 0.5 ** 2))
    d = torch.zeros((K, 128), dtype=torch.float64, device=DEV)
    for o in range(int(table[:, 0].max()) + 1):
        for si in range(1, 4):
            level = _blur64(level, math.sqrt(sig[si] ** 2 - sig[si - 1] ** 2))
            sel = ((table[:, 0] == o) & (table[:, 1] == si)).nonzero()[:, 0].to(DEV)
            ph = int(max(4, np.round(np.float32(3.0 * sig[si] * math.sqrt(2) * 2.5))))
            if sel.numel():
                d = d.index_copy(0, sel, _descriptor64(level, table.to(DEV)[sel, 2:], ph))
        level = level[::2, ::2]
    ((d - target.double()) ** 2).sum().backward()
    return d.detach(), x.grad


def _exact_warp_grad(case, seed):
    H, W = case["H"], case["W"]
    a, b, target, h8, (cw, ch, ox, oy, iox, ioy) = _warp_inputs(case, seed)
    a, b, h8 = (t.double().requires_grad_(True) for t in (a, b, h8))
    Hi = torch.linalg.inv(torch.cat([h8, torch.ones(1, dtype=torch.float64, device=DEV)]).view(3, 3))
    v, u = torch.meshgrid(torch.arange(ch, device=DEV), torch.arange(cw, device=DEV), indexing="ij")
    X, Y = u - ox, v - oy
    den = Hi[2, 0] * X + Hi[2, 1] * Y + Hi[2, 2]
    den = torch.where(den >= 1e-10, den, torch.full_like(den, 1e-10))
    sx, sy = (Hi[0, 0] * X + Hi[0, 1] * Y + Hi[0, 2]) / den, (Hi[1, 0] * X + Hi[1, 1] * Y + Hi[1, 2]) / den
    in1 = (sx >= 0) & (sx <= W - 1) & (sy >= 0) & (sy <= H - 1)
    x0, y0 = torch.floor(sx).detach(), torch.floor(sy).detach()
    fx, fy = (sx - x0).unsqueeze(-1), (sy - y0).unsqueeze(-1)

    def px(i, j):
        return a[(y0 + j).clamp(0, H - 1).long(), (x0 + i).clamp(0, W - 1).long()]

    w1 = (1 - fy) * ((1 - fx) * px(0, 0) + fx * px(1, 0)) + fy * ((1 - fx) * px(0, 1) + fx * px(1, 1))
    d1 = 1 + torch.minimum(torch.minimum(sx, W - 1 - sx), torch.minimum(sy, H - 1 - sy)).unsqueeze(-1)
    x2, y2 = u - iox, v - ioy
    in2 = (x2 >= 0) & (x2 < W) & (y2 >= 0) & (y2 < H)
    i2 = b[y2.clamp(0, H - 1), x2.clamp(0, W - 1)]
    d2 = 1 + torch.minimum(torch.minimum(x2, W - 1 - x2), torch.minimum(y2, H - 1 - y2)).unsqueeze(-1)
    one, two = in1.unsqueeze(-1), in2.unsqueeze(-1)
    mixed = (w1 * d1 + i2 * d2) / torch.where(one & two, d1 + d2, torch.ones_like(d1))
    out = torch.where(one & two, mixed, torch.where(two, i2, torch.where(one, w1, torch.zeros_like(w1))))
    ((out - target.double()) ** 2).sum().backward()
    return out.detach(), a.grad, b.grad, h8.grad


def exact(case, seed):
    """Detections and panoramas are defined by comparisons of 32-bit values and
    the fp16 and int8 distances by rounded similarities: no 64-bit value."""
    if case["kind"] == "desc_grad":
        return _exact_desc_grad(case, seed)
    if case["kind"] == "warp_grad":
        return _exact_warp_grad(case, seed)
    if case["kind"] == "match" and case["mode"] in ("u8", "split_fp8"):
        a, b, k = _descriptors(case["N"], case["M"], seed)
        a, b = a.double(), b.double()
        d = (a * a).sum(1, keepdim=True) + (b * b).sum(1) - 2 * a @ b.t()

        def side(t):
            two, at = torch.topk(t, 2, dim=1, largest=False)
            return at[:, 0], (two[:, 1] > 0) & (two[:, 0] < 0.75 ** 2 * two[:, 1]), two[:, 0]

        (f, fp, d1), (g, gp, _) = side(d), side(d.t())
        i = torch.arange(case["N"], device=DEV)
        dist = torch.sqrt(d1[fp & gp[f] & (g[f] == i)])[:k]
        return {"count": None, "pairs": None, "dist": dist, "fwd_best": None, "fwd_pass": None, "bwd_best": None,
                "bwd_pass": None}
    return None
