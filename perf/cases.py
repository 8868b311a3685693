"""Performance cases of the framework: the calls its users make, over the sizes they make them at.

Families (``case["kind"]``):

* ``sncc``    spectral NCC of candidate poses in both views with the pose gradient (candidate screening, pose
              optimisation; parallel beam), ``sncc_eval`` the loss alone in one view (re-scoring at fine resolution);
* ``image``   the image-domain training step of the parallel-beam engine: render, image spectral NCC, pose gradient;
* ``numpy``   the fp64 NumPy-convention biplanar loss and gradient, host arrays in and out;
* ``pou``     the partition-of-unity cone-beam renderer, forward and pose-matrix gradient (or forward alone);
* ``rays``    the same renderer on explicit sources and detector points, gradients to both;
* ``loss``    the per-candidate biplanar registration loss on rendered images, gradients to the images.

Volumes are an attenuating body filled with random ellipsoids (a torso stand-in: every block of the cone-beam
renderer is active), poses are spread as candidate screening spreads them (+-10 degrees, +-5 mm), targets are
rendered at another pose with 2 % noise.  ``exact`` restates each call in float64 torch / NumPy.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "diff-fvr_b200"))

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
BYTES = {"f32": 4, "bf16": 2, "f16": 2}
SDD, SAD = 1020.0, 765.0
DEG = math.pi / 180.0


def listed():
    return [
        # one pose of an optimiser loop, plain f32: launch latency and host work
        dict(name="sncc_pose_f32", kind="sncc", api="autograd", n=128, res=128, poses=1, dtype="f32", sp=1.0),
        # candidate screening, the headline configuration
        dict(name="sncc_screen_f16", kind="sncc", api="fused", n=128, res=128, poses=64, dtype="f16", sp=1.0),
        # the same on a full-size CT, 512^3 spectrum, anisotropic spacing
        dict(name="sncc_ct512_f16", kind="sncc", api="fused", n=256, res=192, poses=256, dtype="f16", sp=0.8),
        # scoring candidates at fine detector resolution, no gradient
        dict(name="sncc_eval_bf16", kind="sncc_eval", n=128, res=512, poses=64, dtype="bf16", sp=1.0),
        # image-domain training step of the parallel engine
        dict(name="image_step_f32", kind="image", n=96, res=96, poses=64, dtype="f32", sp=1.0),
        # one objective + gradient evaluation of the fp64 registration driver
        dict(name="numpy_biplanar_f64", kind="numpy", n=96),
        # one pose of a cone-beam pose optimisation, the small block preset
        dict(name="pou_pose_bf16", kind="pou", grad=True, n=192, gz=2, gy=2, gx=2, block_res=64, poses=1, h=256, w=256,
             pix=1.0, dtype="bf16"),
        # cone-beam candidate screening on the isotropic block grid
        dict(name="pou_grid4_f32", kind="pou", grad=True, n=192, gz=4, gy=4, gx=4, block_res=64, poses=64, h=256,
             w=256, pix=0.8, dtype="f32"),
        # a fine detector on the small block preset
        dict(name="pou_det512_bf16", kind="pou", grad=True, n=192, gz=2, gy=2, gx=2, block_res=64, poses=64, h=512,
             w=512, pix=0.5, dtype="bf16"),
        # the "balanced" preset (block_res 80), a detector of odd size
        dict(name="pou_balanced_bf16", kind="pou", grad=True, n=160, gz=2, gy=4, gx=2, block_res=80, poses=24, h=211,
             w=247, pix=0.9, dtype="bf16"),
        # explicit source and detector points (a calibrated C-arm sweep), gradients to the geometry
        dict(name="rays_f32", kind="rays", n=128, gz=2, gy=2, gx=2, block_res=64, poses=8, h=144, w=120, pix=1.6,
             dtype="f32"),
        # the registration loss of 64 candidates in two views
        dict(name="reg_loss_f32", kind="loss", poses=64, h=256, w=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng):
    """Volume sides from 64 to 192, odd ones among them (a padded side's prime factors stay below 128)."""
    return _log(rng, 64, 127) if rng.random() < 0.5 else 2 * _log(rng, 40, 96)


def draw(rng):
    kind = rng.choice(["sncc", "sncc", "sncc_eval", "image", "numpy", "pou", "pou", "pou", "rays", "loss"])
    dt = rng.choice(["f32", "bf16", "f16"])
    sp = rng.choice([0.8, 1.0, 1.5])
    if kind == "sncc":
        return dict(kind=kind, api=rng.choice(["autograd", "fused"]), n=_side(rng), res=_log(rng, 64, 192),
                    poses=_log(rng, 1, 256), dtype=dt, sp=sp)
    if kind == "sncc_eval":
        res = _log(rng, 64, 512)
        return dict(kind=kind, n=_side(rng), res=res, poses=_log(rng, 1, min(256, (1 << 24) // res ** 2)),
                    dtype=dt, sp=sp)
    if kind == "image":
        return dict(kind=kind, n=_side(rng), res=2 * _log(rng, 24, 64), poses=_log(rng, 1, 64), dtype=dt, sp=sp)
    if kind == "numpy":
        return dict(kind=kind, n=2 * _log(rng, 24, 60))
    if kind == "loss":
        return dict(kind=kind, poses=_log(rng, 1, 64), h=_log(rng, 64, 256), w=_log(rng, 64, 256))
    grid = rng.choice([(1, 1, 1), (2, 2, 2), (2, 2, 2), (2, 4, 2), (3, 3, 3), (4, 4, 4)])
    br = rng.choice([32, 48, 64, 64, 80])
    n, pix = _log(rng, 96, 192), rng.choice([0.6, 0.8, 1.0, 1.6])
    shape = dict(n=n, gz=grid[0], gy=grid[1], gx=grid[2], block_res=br, pix=pix, dtype=dt)
    if kind == "rays":
        return dict(kind=kind, poses=_log(rng, 1, 8), h=_log(rng, 64, 160), w=_log(rng, 64, 160), **shape)
    h = _log(rng, 96, 512)
    w = h if rng.random() < 0.5 else _log(rng, 96, 512)
    # no drawn case samples more than the largest listed one (64 blocks x 64 poses)
    most = 64 * 64 * (128 ** 2 + 256 ** 2) // (math.prod(grid) * (4 * br ** 2 + h * w))
    return dict(kind=kind, grad=rng.random() < 0.75, poses=_log(rng, 1, max(1, min(64, most))), h=h, w=w, **shape)


# ---------------------------------------------------------------- inputs


def _dev():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


def _volume(n, seed):
    """Body ellipsoid (0.02 / mm) with 12 random ellipsoids inside, float32 [n, n, n] on the device."""
    rng = np.random.default_rng(seed)
    g = torch.arange(n, dtype=torch.float32, device=_dev())
    vol = torch.zeros((n, n, n), dtype=torch.float32, device=_dev())
    parts = [([0.5 * n] * 3, [0.47 * n] * 3, 0.02)]
    for _ in range(12):
        parts.append(([rng.uniform(0.3 * n, 0.7 * n) for _ in range(3)],
                      [rng.uniform(0.05 * n, 0.2 * n) for _ in range(3)], rng.uniform(0.0, 0.05)))
    for c, r, mu in parts:
        z, y, x = (((g - ci) / ri) ** 2 for ci, ri in zip(c, r))
        vol += mu * ((z[:, None, None] + y[None, :, None]) + x[None, None, :] <= 1.0)
    return vol


def _poses(n, seed):
    """[n, 6] float32: rotations U(+-10) degrees, translations U(+-5) mm."""
    rng = np.random.default_rng(seed)
    p = np.concatenate([rng.uniform(-10, 10, (n, 3)), rng.uniform(-5, 5, (n, 3))], 1)
    return torch.from_numpy(p.astype(np.float32)).to(_dev())


def _mats(n, seed):
    """Camera-to-world matrices [n, 4, 4] float32: source SAD mm from the isocentre, turned and shifted."""
    rng = np.random.default_rng(seed)
    rv = torch.from_numpy(rng.uniform(-10 * DEG, 10 * DEG, (n, 3)))
    tj = torch.from_numpy(rng.uniform(-5, 5, (n, 3)))
    k = torch.zeros((n, 3, 3), dtype=torch.float64)
    k[:, 0, 1], k[:, 0, 2], k[:, 1, 2] = -rv[:, 2], rv[:, 1], -rv[:, 0]
    rot = torch.matrix_exp(k - k.transpose(1, 2))
    m = torch.zeros((n, 4, 4), dtype=torch.float64)
    m[:, :3, :3] = rot
    m[:, :3, 3] = rot @ torch.tensor([0.0, 0.0, -SAD], dtype=torch.float64) + tj
    m[:, 3, 3] = 1.0
    return m.float().to(_dev())


def _noise(shape, seed):
    return torch.from_numpy(np.random.default_rng(seed).standard_normal(shape, dtype=np.float32)).to(_dev())


def _upstream(shape, seed):
    """The gradient a loss hands back: standard normal values made on the device."""
    g = torch.Generator(device=_dev())
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device=_dev())


def _k_inv(case):
    f = SDD / case["pix"]
    return torch.tensor([[1 / f, 0, -0.5 * case["w"] / f], [0, 1 / f, -0.5 * case["h"] / f], [0, 0, 1.0]],
                        dtype=torch.float32, device=_dev())


def _ray_inputs(case, seed):
    """Sources [N, 3] and detector points [N, H, W, 3] of the pose matrices' pinhole cameras."""
    m = _mats(case["poses"], seed + 1).double()
    k = _k_inv(case).double()
    h, w = case["h"], case["w"]
    yy, xx = torch.meshgrid(torch.arange(h, device=_dev()) + 0.5, torch.arange(w, device=_dev()) + 0.5, indexing="ij")
    cam = torch.stack([xx, yy, torch.ones_like(xx)], -1).double() @ k.T * SDD
    trg = torch.einsum("nij,hwj->nhwi", m[:, :3, :3], cam) + m[:, None, None, :3, 3]
    return m[:, :3, 3].float().contiguous(), trg.float().contiguous()


def _loss_images(case, seed):
    """Rendered-looking candidate images and references: smooth blobs, each candidate shifted a little."""
    h, w, n = case["h"], case["w"], case["poses"]
    rng = np.random.default_rng(seed)
    y = torch.arange(h, device=_dev(), dtype=torch.float32)[None, :, None]
    x = torch.arange(w, device=_dev(), dtype=torch.float32)[None, None, :]

    def blobs(shift):
        img = torch.zeros((shift.shape[0], h, w), device=_dev())
        for cy, cx, ry, rx, a in parts:
            q = ((y - cy * h - shift[:, :1, None]) / (ry * h)) ** 2 + ((x - cx * w - shift[:, 1:, None]) / (rx * w)) ** 2
            img += a * torch.clamp(1.0 - q, min=0.0).sqrt()
        return img[:, None].contiguous()

    out = []
    for v in range(2):
        parts = [(0.5, 0.5, 0.45, 0.45, 4.0)] + [tuple(rng.uniform((0.3, 0.3, 0.05, 0.05, 0.5), (0.7, 0.7, 0.2, 0.2, 2.0)))
                                                for _ in range(12)]
        shift = torch.from_numpy(rng.uniform(-12, 12, (n, 2)).astype(np.float32)).to(_dev())
        ref = blobs(torch.zeros((1, 2), device=_dev()))
        out += [blobs(shift), ref + 0.02 * ref.max() * _noise(ref.shape, seed + 3 + v)]
    return out


# ---------------------------------------------------------------- float64 restatement, plain torch


def _pad1(vol):
    return torch.nn.functional.pad(vol, (1, 1) * vol.dim())


def _interp(padded, pos):
    """Multilinear interpolation with zeros outside of a field padded by one zero on each side; ``pos`` are the
    coordinates, slowest axis first.  Differentiable in ``pos``."""
    out = None
    base, frac = [], []
    for p, n in zip(pos, padded.shape):
        f = torch.floor(p.detach())
        base.append(f.long() + 1)
        frac.append(p - f)
    flat = padded.reshape(-1)
    for c in range(1 << len(pos)):
        idx, wt = 0, 1.0
        for d, (b, t, n) in enumerate(zip(base, frac, padded.shape)):
            up = (c >> d) & 1
            idx = idx * n + (b + up).clamp(0, n - 1)
            wt = wt * (t if up else 1.0 - t)
        term = flat[idx] * wt
        out = term if out is None else out + term
    return out


def _linspace32(n):
    """The float32 grid torch.linspace(-1, 1, n) holds, in float64."""
    if n == 1:
        return torch.full((1,), -1.0, dtype=torch.float64, device=_dev())
    step = float(np.float32(2.0) / np.float32(n - 1))
    i = np.arange(n, dtype=np.float64)
    v = np.where(i < n // 2, -1.0 + step * i, 1.0 - step * (n - 1 - i)).astype(np.float32)
    return torch.from_numpy(v.astype(np.float64)).to(_dev())


def _spectrum(vol, pad=2.0):
    """fftshift(fftn(centred zero pad)), complex128, padded by one zero on each side."""
    p = [int(round(s * pad)) for s in vol.shape]
    full = torch.zeros(p, dtype=torch.float64, device=vol.device)
    lo = [(a - s) // 2 for a, s in zip(p, vol.shape)]
    full[lo[0]:lo[0] + vol.shape[0], lo[1]:lo[1] + vol.shape[1], lo[2]:lo[2] + vol.shape[2]] = vol.double()
    return _pad1(torch.fft.fftshift(torch.fft.fftn(full)))


def _axis_rot(a, i, j):
    c, s = torch.cos(a), torch.sin(a)
    r = [[torch.zeros_like(c) for _ in range(3)] for _ in range(3)]
    r[3 - i - j][3 - i - j] = torch.ones_like(c)
    r[i][i], r[j][j], r[i][j], r[j][i] = c, c, -s, s
    return torch.stack([torch.stack(x, -1) for x in r], -2)


def _slices(spec, poses, view, res, sp):
    """Phase-modulated central slices [C, res, res] of the parallel-beam convention."""
    yaw, pitch, roll = (poses[:, i] * DEG for i in range(3))
    rot = _axis_rot(yaw, 0, 1) @ _axis_rot(pitch, 2, 0) @ _axis_rot(roll, 1, 2)
    if view == "lateral":
        a = np.float32(90.0) * np.float32(math.pi / 180.0)
        c, s = float(np.cos(a)), float(np.sin(a))
        rot = rot @ torch.tensor([[c, -s, 0], [s, c, 0], [0, 0, 1.0]], dtype=torch.float64, device=poses.device)
    d, h, w = (x - 2 for x in spec.shape)
    half = torch.tensor([0.5 * (w - 1), 0.5 * (h - 1), 0.5 * (d - 1)], dtype=torch.float64, device=poses.device)
    lin = _linspace32(res)
    ku, kv = lin[None, :, None], lin[None, None, :]
    u, v = rot[:, 0] * half, rot[:, 1] * half
    pos = [half[k] + ku * u[:, k, None, None] + kv * v[:, k, None, None] for k in (2, 1, 0)]
    kap = -2.0 * math.pi / (res * sp + 1e-6)
    ph = kap * (ku * poses[:, 3, None, None] + kv * poses[:, 4, None, None])
    return _interp(spec, pos) * torch.complex(torch.cos(ph), torch.sin(ph))


def _high_pass(h, w, sigma=4.0):
    y = torch.linspace(-h / 2, h / 2, h, dtype=torch.float64, device=_dev())[:, None]
    x = torch.linspace(-w / 2, w / 2, w, dtype=torch.float64, device=_dev())[None]
    return 1.0 - torch.exp(-(x * x + y * y) / (2.0 * sigma ** 2))


def _ncc_c(a, b):
    """Re<a, b> / (|a| |b| + 1e-8) over the last two axes."""
    en = (a.abs().square().sum((-2, -1)) * b.abs().square().sum((-2, -1))).sqrt()
    return (a * b.conj()).real.sum((-2, -1)) / (en + 1e-8)


def _render(spec, poses, view, res, sp):
    s = _slices(spec, poses, view, res, sp)
    return torch.fft.ifft2(torch.fft.ifftshift(s, dim=(-2, -1))).real.clamp(min=0.0)[:, None]


def _targets(case, seed, vol):
    """Target images [1, 1, R, R] float32 of both views at another pose, 2 % noise."""
    spec, tp, out = _spectrum(vol), _poses(1, seed + 2).double(), []
    for k, v in enumerate(("ap", "lateral")):
        img = _render(spec, tp, v, case["res"], case["sp"])
        out.append((img + 0.02 * img.max() * _noise(img.shape, seed + 3 + k)).float())
    return out


def _target_spectra(case, seed, vol):
    return [(torch.fft.fftshift(torch.fft.fft2(t.double()), dim=(-2, -1)) * _high_pass(case["res"], case["res"]))
            .to(torch.complex64).contiguous() for t in _targets(case, seed, vol)]


def _windows(n, k, overlap):
    """Raised-cosine partition of unity of n voxels into k blocks, [k, n], and the block pitch."""
    w = torch.ones((k, n), dtype=torch.float64, device=_dev())
    step = n / k
    if k == 1:
        return w, step
    half, c = max(2.0, step * overlap), torch.arange(n, dtype=torch.float64, device=_dev()) + 0.5
    for i in range(k):
        if i > 0:
            w[i] *= torch.sin(0.5 * math.pi * ((c - (i * step - half)) / (2 * half)).clamp(0, 1)) ** 2
        if i < k - 1:
            w[i] *= torch.cos(0.5 * math.pi * ((c - ((i + 1) * step - half)) / (2 * half)).clamp(0, 1)) ** 2
    return w, step


def _blocks(case, vol, overlap=0.5):
    """(ds, P, generator of (centre [3], padded spectrum)) of the cone-beam renderer's blocks, 1 mm voxels."""
    n, br = case["n"], case["block_res"]
    grid = (case["gz"], case["gy"], case["gx"])
    wins, steps = zip(*(_windows(n, k, overlap) for k in grid))
    ov = [max(2, int(round(s * overlap))) if k > 1 else 0 for s, k in zip(steps, grid)]
    m = max(int(np.ceil(s + 2 * o)) for s, o in zip(steps, ov)) + (1 if max(grid) > 1 else 0)
    ds, p = m / br, 2 * br
    lo = (p - br) // 2
    half = (p // 2 - (lo + (br - 1) * 0.5)) * ds
    c = (torch.arange(br, dtype=torch.float64, device=_dev()) - (br - 1) / 2) / p
    comp = 1.0 / (torch.sinc(c) ** 2).clamp(min=0.05)

    def each():
        for i in np.ndindex(*grid):
            sup = []
            for w, k in zip(wins, i):
                nz = torch.nonzero(w[k].float() > 1e-6).flatten()
                sup.append((int(nz[0]), int(nz[-1]) + 1))
            (a0, b0), (a1, b1), (a2, b2) = sup
            sub = vol[a0:b0, a1:b1, a2:b2].double() * wins[0][i[0], a0:b0, None, None] * \
                wins[1][i[1], None, a1:b1, None] * wins[2][i[2], None, None, a2:b2]
            if float(sub.sum()) <= 1e-4:
                continue
            off = [(m - s) // 2 for s in sub.shape]
            cube = torch.zeros((m, m, m), dtype=torch.float64, device=_dev())
            cube[off[0]:off[0] + sub.shape[0], off[1]:off[1] + sub.shape[1], off[2]:off[2] + sub.shape[2]] = sub
            cube = torch.nn.functional.interpolate(cube[None, None], size=(br,) * 3, mode="trilinear",
                                                   align_corners=False)[0, 0] * ds
            full = torch.zeros((p, p, p), dtype=torch.float64, device=_dev())
            full[lo:lo + br, lo:lo + br, lo:lo + br] = cube * comp[:, None, None] * comp[:, None] * comp
            cen = torch.tensor([-0.5 * (n - 1) + a + (m - 1) * 0.5 - o + half for (a, _), o in zip(sup, off)])
            f = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(full)))
            yield cen.float().double().to(_dev()), _pad1(f)

    return ds, p, each


def _block_image(spec, u, v, ds, p):
    """Re fftshift(ifft2(ifftshift(central slice))) of one block for detector axes u, v [N, 3], [N, p, p]."""
    fr = torch.from_numpy(np.fft.fftshift(np.fft.fftfreq(p, d=ds)).astype(np.float32)).double().to(u.device) * (p * ds)
    pos = [p // 2 + fr[None, None, :] * u[:, k, None, None] + fr[None, :, None] * v[:, k, None, None] for k in range(3)]
    s = _interp(spec, pos)
    return torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(s, dim=(-2, -1))).real, dim=(-2, -1))


def _warp(img, px, py):
    """Bilinear samples of img [N, p, p] at px, py [N, ...], zeros outside."""
    n, p = img.shape[0], img.shape[-1]
    pad = torch.nn.functional.pad(img, (1, 1, 1, 1)).reshape(n, -1)
    x0, y0 = torch.floor(px.detach()), torch.floor(py.detach())
    tx, ty = px - x0, py - y0
    out = 0.0
    for dy in (0, 1):
        for dx in (0, 1):
            idx = (y0.long() + 1 + dy).clamp(0, p + 1) * (p + 2) + (x0.long() + 1 + dx).clamp(0, p + 1)
            wt = (tx if dx else 1.0 - tx) * (ty if dy else 1.0 - ty)
            out = out + pad.gather(1, idx.reshape(n, -1)).reshape(idx.shape) * wt
    return out


def _exact_cone(case, leaves, geometry, g):
    """Image and the leaves' gradients of the cone-beam renderer, one block at a time.  ``geometry(leaves)`` gives
    (src, u, v, n, rx, ry, ic), rays per unit distance along n."""
    vol = _volume(case["n"], case["_seed"])
    ds, p, each = _blocks(case, vol)
    img, grads = 0.0, [torch.zeros_like(x) for x in leaves]
    for cen, spec in each():
        with torch.set_grad_enabled(g is not None):
            xs = [x.detach().requires_grad_(g is not None) for x in leaves]
            src, u, v, n, rx, ry, ic = geometry(xs)
            diff = cen[None] - src
            d, cu, cv = ((diff * a).sum(-1)[:, None, None] for a in (n, u, v))
            part = _warp(_block_image(spec, u, v, ds, p), (d * rx - cu) / ds + p // 2, (d * ry - cv) / ds + p // 2) * ic
            if g is not None:
                for t, a in zip(grads, torch.autograd.grad(part, xs, g)):
                    t += a
        img = img + part.detach()
    return img, grads


def _exact_pou(case, seed):
    h, w, f = case["h"], case["w"], SDD / case["pix"]
    k = _k_inv(case).double()
    rx = (k[0, 0] * (torch.arange(w, device=_dev()) + 0.5) + k[0, 2]).expand(h, w)
    ry = (k[1, 1] * (torch.arange(h, device=_dev()) + 0.5) + k[1, 2])[:, None].expand(h, w)
    ic = (1.0 + rx * rx + ry * ry).sqrt().float().double()[None]
    rx, ry = rx.float().double()[None], ry.float().double()[None]
    base = torch.eye(3, dtype=torch.float64, device=_dev())

    def geometry(xs):
        r = xs[0][:, :3, :3]
        return xs[0][:, :3, 3], r @ base[0], r @ base[1], r @ base[2], rx, ry, ic

    n = case["poses"]
    g = _upstream((n, 1, h, w), seed + 5).double()[:, 0] if case["grad"] else None
    img, grads = _exact_cone({**case, "_seed": seed}, [_mats(n, seed + 1).double()], geometry, g)
    return [img[:, None]] + (grads if case["grad"] else [])


def _exact_rays(case, seed):
    src, trg = _ray_inputs(case, seed)

    def geometry(xs):
        s, t = xs
        e = torch.stack([t[:, 0, -1] - t[:, 0, 0], t[:, -1, 0] - t[:, 0, 0]], 1)
        e = e / (e.norm(dim=-1, keepdim=True) + 1e-12)
        u, v = e[:, 0], e[:, 1]
        n = torch.linalg.cross(v, u, dim=-1)
        n = n / (n.norm(dim=-1, keepdim=True) + 1e-12)
        n = torch.where(((t.mean((1, 2)) - s) * n).sum(-1, keepdim=True) < 0, -n, n)
        r = t - s[:, None, None]
        r = r / (r * r).sum(-1, keepdim=True).clamp(min=1e-12).sqrt()
        ic = 1.0 / (r * n[:, None, None]).sum(-1).clamp(min=0.1)
        return s, u, v, n, (r * u[:, None, None]).sum(-1) * ic, (r * v[:, None, None]).sum(-1) * ic, ic

    g = _upstream((case["poses"], case["h"], case["w"]), seed + 5).double()
    img, grads = _exact_cone({**case, "_seed": seed}, [src.double(), trg.double()], geometry, g)
    return [img] + grads


def _chunks(n, per):
    return [(i, min(n, i + per)) for i in range(0, n, per)]


def _exact_sncc(case, seed):
    vol = _volume(case["n"], seed)
    spec, poses, n = _spectrum(vol), _poses(case["poses"], seed + 1).double(), case["poses"]
    fts = _target_spectra(case, seed, vol)
    hp, grad = _high_pass(case["res"], case["res"]), case["kind"] == "sncc"
    loss, g = 0.0, torch.zeros_like(poses)
    for ft, view in list(zip(fts, ("ap", "lateral")))[:2 if grad else 1]:
        for a, b in _chunks(n, max(1, 2_000_000 // case["res"] ** 2)):
            with torch.set_grad_enabled(grad):
                p = poses[a:b].clone().requires_grad_(grad)
                ncc = _ncc_c(_slices(spec, p, view, case["res"], case["sp"]) * hp, ft[0].to(torch.complex128)).sum()
                if grad:
                    g[a:b] -= torch.autograd.grad(ncc, p)[0] / n
            loss = loss - ncc.detach() / n
        loss = loss + 1.0
    return [loss, g] if grad else [loss]


def _exact_image(case, seed):
    vol = _volume(case["n"], seed)
    spec, poses, n = _spectrum(vol), _poses(case["poses"], seed + 1).double(), case["poses"]
    t = _targets(case, seed, vol)[0].double()
    hp = _high_pass(case["res"], case["res"])
    ft = torch.fft.fftshift(torch.fft.fft2(t), dim=(-2, -1)) * hp
    imgs, loss, g = [], 1.0, torch.zeros_like(poses)
    for a, b in _chunks(n, max(1, 1_000_000 // case["res"] ** 2)):
        p = poses[a:b].clone().requires_grad_(True)
        img = _render(spec, p, "ap", case["res"], case["sp"])
        ncc = _ncc_c(torch.fft.fftshift(torch.fft.fft2(img), dim=(-2, -1)) * hp, ft).sum()
        g[a:b] = -torch.autograd.grad(ncc, p)[0] / n
        imgs.append(img.detach())
        loss = loss - ncc.detach() / n
    return [torch.cat(imgs), loss, g]


def _np_inputs(case, seed):
    rng = np.random.default_rng(seed + 1)
    vol = _volume(case["n"], seed).cpu().numpy().astype(np.float64)
    pose = np.concatenate([rng.uniform(-10, 10, 3), rng.uniform(-5, 5, 3)])
    tpose = np.concatenate([rng.uniform(-10, 10, 3), rng.uniform(-5, 5, 3)])
    spec = _np_spectrum(vol)
    ap, lat = (_np_slice(spec, tpose[:3], tpose[i], tpose[5], v) for i, v in ((3, "ap"), (4, "lateral")))
    return vol, pose, spec, ap.cpu().numpy(), lat.cpu().numpy()


def _np_spectrum(vol):
    n = vol.shape[0]
    p = 2 * n
    c = 1.0 / np.maximum(np.sinc((np.arange(n) - n / 2.0) / p) ** 2, 0.05)
    full = np.zeros((p, p, p))
    lo = (p - n) // 2
    full[lo:lo + n, lo:lo + n, lo:lo + n] = vol * c[:, None, None] * c[:, None] * c
    return torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(torch.from_numpy(full).to(_dev()))))


def _np_slice(spec, ang, tx, ty, view):
    """Order-1 central slice of a cubic spectrum with 'constant' borders and the phase ramp (NumPy convention)."""
    p = spec.shape[0]
    y, pt, r = (a * DEG for a in ang)
    rz = np.array([[1, 0, 0], [0, np.cos(y), -np.sin(y)], [0, np.sin(y), np.cos(y)]])
    ry = np.array([[np.cos(r), 0, np.sin(r)], [0, 1, 0], [-np.sin(r), 0, np.cos(r)]])
    rx = np.array([[np.cos(pt), -np.sin(pt), 0], [np.sin(pt), np.cos(pt), 0], [0, 0, 1]])
    rot = rz @ ry @ rx
    u, v = rot[:, 1 if view == "lateral" else 2], rot[:, 0]
    k = torch.arange(p, dtype=torch.float64, device=spec.device) - p / 2.0
    uu, vv = k[None, :], k[:, None]
    pos = [uu * u[i] + vv * v[i] + p / 2.0 for i in range(3)]
    ok = True
    for q in pos:
        ok = ok & (q >= 0) & (q <= p - 1)
    s = torch.where(ok, _interp(_pad1(spec), pos), 0.0)
    ph = -2.0 * math.pi * (uu * tx / p + vv * ty / p)
    return s * torch.complex(torch.cos(ph), torch.sin(ph))


def _exact_numpy(case, seed):
    _, pose, spec, *fts = _np_inputs(case, seed)
    p = spec.shape[0]
    k = torch.arange(p, dtype=torch.float64, device=spec.device) - p / 2.0
    loss, g = 0.0, np.zeros(6)
    for ft, view, i in zip(fts, ("ap", "lateral"), (3, 4)):
        t = torch.from_numpy(ft).to(spec.device)
        nt = t.abs().square().sum().sqrt()

        def ncc(s):
            return ((s * t.conj()).real.sum() / (s.abs().square().sum().sqrt() * nt))

        s = _np_slice(spec, pose[:3], pose[i], pose[5], view)
        q = ncc(s)
        ns = s.abs().square().sum().sqrt()
        r = (t - q * (nt / ns) * s) / (ns * nt)
        for slot, ax in ((i, k[None, :]), (5, k[:, None])):
            g[slot] -= 0.5 * float((-2j * math.pi * (ax / p) * s * r.conj()).real.sum())
        loss += 0.5 * (1.0 - float(q))
        for j in range(3):
            d = []
            for e in (0.2, -0.2):
                a = pose[:3].copy()
                a[j] += e
                d.append(float(ncc(_np_slice(spec, a, pose[i], pose[5], view))))
            g[j] -= 0.5 * (d[0] - d[1]) / 0.4
    return [loss, g]


def _exact_loss(case, seed):
    im_a, ref_a, im_b, ref_b = (x.double() for x in _loss_images(case, seed))
    kx = torch.tensor([[-1.0, 0, 1], [-2, 0, 2], [-1, 0, 1]], dtype=torch.float64, device=_dev())
    crop = max(4, case["w"] // 8)

    def conv(x, k):
        return torch.nn.functional.conv2d(x, k[None, None], padding=1)

    def ncc(a, b):
        a, b = a - a.mean((-2, -1), keepdim=True), b - b.mean((-2, -1), keepdim=True)
        den = (a.square().sum((-2, -1)) * b.square().sum((-2, -1))).clamp(min=1e-12).sqrt()
        return ((a * b).sum((-2, -1)) / den)[:, 0]

    def edge(a, b):
        cut = slice(crop, -crop)
        return 0.5 * sum(ncc(conv(a, k)[..., cut, cut], conv(b, k)[..., cut, cut]) for k in (kx, kx.T))

    def sim(a, b):
        e = edge(a, b)
        if case["w"] >= 96:
            box = torch.full((3, 3), 1 / 9, dtype=torch.float64, device=_dev())
            e = 0.75 * e + 0.25 * edge(conv(a, box), conv(b, box))
        return 0.75 * e + 0.25 * ncc(a, b)

    im_a.requires_grad_(True)
    im_b.requires_grad_(True)
    loss = 1.0 - 0.5 * (sim(im_a, ref_a) + sim(im_b, ref_b))
    return [loss.detach(), *torch.autograd.grad(loss.sum(), (im_a, im_b))]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sncc", "sncc_eval"):
        return _exact_sncc(case, seed)
    return {"image": _exact_image, "numpy": _exact_numpy, "pou": _exact_pou, "rays": _exact_rays,
            "loss": _exact_loss}[kind](case, seed)


# ---------------------------------------------------------------- what a program keeps, and its call


def _engine(case, seed):
    import fvr

    vol = _volume(case["n"], seed)
    sp = case["sp"]
    return vol, fvr.TorchDiffFVREngine(vol, spacing=(sp, sp, 1.5 * sp), pad_factor=2.0, dtype=DTYPES[case["dtype"]])


def _model(case, seed):
    from fvr.cone_beam_fvr import PerspectiveSlabFVR

    return PerspectiveSlabFVR.from_volume(_volume(case["n"], seed), vox_mm=1.0,
                                          grid_blocks=(case["gz"], case["gy"], case["gx"]),
                                          block_res=case["block_res"], overlap=0.5, dtype=DTYPES[case["dtype"]])


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("sncc", "sncc_eval", "image"):
        vol, s["engine"] = _engine(case, seed)
        s["poses"] = _poses(case["poses"], seed + 1).requires_grad_(kind != "sncc_eval")
        if kind == "image":
            s["target"] = _targets(case, seed, vol)[0]
        else:
            s["ft"] = _target_spectra(case, seed, vol)
    elif kind == "numpy":
        from fvr.diff_fvr import DifferentiableFourierVolumeRenderer
        from fvr.gradients import SpectralGradientEngine

        vol, s["pose"], _, s["ap"], s["lat"] = _np_inputs(case, seed)
        s["engine"] = SpectralGradientEngine(DifferentiableFourierVolumeRenderer(vol, pad_factor=2.0))
    elif kind == "loss":
        s["imgs"] = _loss_images(case, seed)
        for k in (0, 2):
            s["imgs"][k].requires_grad_(True)
    elif kind == "pou":
        s["model"] = _model(case, seed)
        s["lattice"] = s["model"].make_pinhole_lattice(_k_inv(case), SDD, case["h"], case["w"])
        s["mats"] = _mats(case["poses"], seed + 1).requires_grad_(case["grad"])
        s["g"] = _upstream((case["poses"], 1, case["h"], case["w"]), seed + 5)
    else:
        s["model"] = _model(case, seed)
        s["src"], s["trg"] = (x.requires_grad_(True) for x in _ray_inputs(case, seed))
        s["g"] = _upstream((case["poses"], case["h"], case["w"]), seed + 5)
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "sncc":
        if case["api"] == "fused":
            return list(s["engine"].spectral_ncc_value_and_grad(s["poses"], s["ft"], ("ap", "lateral")))
        loss = s["engine"].forward_spectral_ncc(s["poses"], s["ft"][0], "ap") + \
            s["engine"].forward_spectral_ncc(s["poses"], s["ft"][1], "lateral")
        return [loss.detach(), *torch.autograd.grad(loss, s["poses"])]
    if kind == "sncc_eval":
        with torch.no_grad():
            return [s["engine"].forward_spectral_ncc(s["poses"], s["ft"][0], "ap")]
    if kind == "image":
        img = s["engine"](s["poses"], view="ap", out_res=case["res"])
        loss = s["engine"].spectral_ncc_loss(img, s["target"])
        return [img.detach(), loss.detach(), *torch.autograd.grad(loss, s["poses"])]
    if kind == "numpy":
        return list(s["engine"].compute_biplanar_loss_and_gradients(s["pose"], s["ap"], s["lat"]))
    if kind == "loss":
        from fvr.registration import biplanar_loss_per_candidate

        a, ref_a, b, ref_b = s["imgs"]
        loss = biplanar_loss_per_candidate(a, b, ref_a, ref_b)
        return [loss.detach(), *torch.autograd.grad(loss.sum(), (a, b))]
    if kind == "pou":
        if not case["grad"]:
            with torch.no_grad():
                return [s["model"].forward_pinhole(s["mats"], s["lattice"])]
        img = s["model"].forward_pinhole(s["mats"], s["lattice"])
        return [img.detach(), *torch.autograd.grad(img, s["mats"], s["g"])]
    img = s["model"].project_rays_batched(s["src"], s["trg"])
    return [img.detach(), *torch.autograd.grad(img, (s["src"], s["trg"]), s["g"])]


def work(case):
    """Bytes: the part of the spectra that the slices' cells can touch, read once, and every other input and output
    once.  Operations: 8 corners (a complex multiply-add each, four of them with the three derivatives of the
    gradient), 5 N log2 N per transform of N points, 4 taps per detector pixel and block."""
    kind = case["kind"]
    n = case["poses"] if kind != "numpy" else 14
    if kind in ("sncc", "sncc_eval", "image"):
        r2, views, grad = case["res"] ** 2, 2 if kind == "sncc" else 1, kind != "sncc_eval"
        samples = views * n * r2
        touched = min((2 * case["n"]) ** 3, 8 * samples) * 2 * BYTES[case["dtype"]]
        flops = samples * (8 * 4 * (4 if grad else 1) + (60 if grad else 20))
        nbytes = touched + views * r2 * 12 + n * 48
        if kind == "image":
            flops += 4 * n * 5 * r2 * math.log2(r2)
            nbytes += n * r2 * 4
        return {"bytes": nbytes, "flops": flops}
    if kind == "numpy":
        p2 = (2 * case["n"]) ** 2
        return {"bytes": 16 * (min((2 * case["n"]) ** 3, 8 * n * p2) + 2 * p2), "flops": n * p2 * (8 * 4 + 30)}
    if kind == "loss":
        px = 2 * n * case["h"] * case["w"]
        return {"bytes": px * 8 + px // n * 4 + n * 4, "flops": px * 160}
    blocks, p, hw = case["gz"] * case["gy"] * case["gx"], 2 * case["block_res"], case["h"] * case["w"]
    grad = case.get("grad", True)
    samples = blocks * n * p * p // 2  # a real block's slice is known from half of it
    touched = min(blocks * p ** 3 // 2, 8 * samples) * 2 * BYTES[case["dtype"]]
    flops = samples * 8 * 4 * (5 if grad else 1) + blocks * n * 2.5 * p * p * math.log2(p * p) * (2 if grad else 1) + \
        blocks * n * hw * 8 * (3 if grad else 1)
    nbytes = touched + n * hw * 4 * (2 if grad else 1) + hw * 12 + n * 128
    if kind == "rays":
        nbytes += n * hw * 24
    return {"bytes": nbytes, "flops": flops}
