"""The calls this library is timed on: what a microscopist's program has it do, through the
public entry points, from one live camera region to the full sensor.

Every case has a ``kind``:

* ``stack``       Solver.reduce_noise on a device-resident photo-electron stack;
* ``adu``         Solver.reduce_noise_adu on raw camera counts (uint8, uint16 or float32, one to
                  three amplifier gains);
* ``host``        Solver.reduce_noise_host, page-locked host stack in and out;
* ``dropin``      reduceNoise(), the reference's Python call: a list of numpy frames in and out;
* ``batch``       Solver.batch_reduce_noise, many stacks with their own shape, alpha and mask;
* ``warm``        the learned warm start: E4M3 proposals, then the solve from them;
* ``propose``     the FP32 proposals of the same network;
* ``train``       one training step of the network (forward, backward, Adam);
* ``normalized``  reduce_noise_normalized, the single-pixel variant.

The frames are simulated on the GPU from the seed: filaments of point emitters through a Gaussian
point spread function, background, shot noise, and a camera with per-pixel gain and read noise.
"""
import math

import numpy
import torch
import torch.nn.functional as F

import ncs_b200
from ncs_b200.warmstart import DEFAULT_WEIGHTS, WarmStartNet

DEV = "cuda"
MOST_PX = 100 * 2048 * 2048


def listed():
    return [
        # one live region of interest while focusing: the smallest call, latency is all
        dict(name="roi64", kind="stack", T=1, H=64, W=64, alpha=0.2, max_iters=200, hot=0.0,
             per_frame=False),
        # one camera frame at a time, iteration cap of the demos
        dict(name="frame256", kind="stack", T=1, H=256, W=256, alpha=0.2, max_iters=15, hot=0.0,
             per_frame=False),
        # an ordinary acquisition: a few hundred frames of a cropped sensor
        dict(name="stack512", kind="stack", T=200, H=512, W=512, alpha=0.2, max_iters=20, hot=0.0,
             per_frame=False),
        # the whole sensor with hot pixels, to the stopping rule: the largest call
        dict(name="sensor2048", kind="stack", T=100, H=2048, W=2048, alpha=0.2, max_iters=200,
             hot=0.005, per_frame=False),
        # raw 16-bit counts of an odd crop straight from the camera's memory
        dict(name="raw_crop", kind="adu", T=60, H=411, W=301, alpha=0.2, max_iters=200, hot=0.005,
             dtype="uint16", levels=1),
        # a stack in page-locked host memory, denoised into page-locked host memory
        dict(name="host_stack", kind="host", T=100, H=512, W=512, alpha=0.2, max_iters=20, hot=0.0,
             per_frame=False),
        # the reference's own demo call: 50 small numpy frames through its Python entry
        dict(name="dropin50", kind="dropin", T=50, H=128, W=128, alpha=0.1, max_iters=200, hot=0.0),
        # regions of many experiments in one launch, each with its own alpha and optics
        dict(name="batch16", kind="batch", n=16, shapes=7, lo=32, hi=640, frames=48),
        # network proposals on the tensor cores, then the solve from them
        dict(name="warm512", kind="warm", T=50, H=512, W=512, alpha=0.2, max_iters=200, hot=0.005,
             per_frame=False),
        # proposals in FP32, the network's default precision
        dict(name="propose512", kind="propose", T=20, H=512, W=512, hot=0.005, per_frame=False),
        # one step of training the network at its default batch
        dict(name="train2048", kind="train", n=2048),
        # the single-pixel variant at its demos' cap of 15 iterations
        dict(name="normalized512", kind="normalized", T=20, H=512, W=512, hot=0.0,
             per_frame=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, most_px, most_t=200, lo=14, hi=2048):
    """A frame size over the whole range (odd sizes, oblong frames) and a frame count."""
    H = _log_int(rng, lo, hi)
    W = min(hi, max(lo, int(H * rng.uniform(0.5, 2.0))))
    T = _log_int(rng, 1, most_t)
    while T * H * W > most_px:
        T = max(1, T // 2)
        if T == 1 and H * W > most_px:
            H, W = max(lo, H // 2), max(lo, W // 2)
    return T, H, W


def draw(rng):
    kind = rng.choice(["stack", "stack", "stack", "adu", "host", "dropin", "batch", "warm",
                       "propose", "train", "normalized"])
    c = dict(kind=kind)
    if kind == "train":
        c.update(n=_log_int(rng, 64, 8192))
        return c
    if kind == "batch":
        c.update(n=_log_int(rng, 2, 32), shapes=rng.randrange(1 << 20), lo=14,
                 hi=_log_int(rng, 64, 900), frames=_log_int(rng, 1, 64))
        return c
    most = {"stack": MOST_PX // 4, "adu": 40 << 20, "host": 40 << 20, "dropin": 6 << 20,
            "warm": 16 << 20, "propose": 6 << 20, "normalized": 12 << 20}[kind]
    T, H, W = _shape(rng, most, most_t=60 if kind == "dropin" else 200)
    c.update(T=T, H=H, W=W, hot=rng.choice([0.0, 0.005]))
    if kind not in ("propose", "normalized"):
        c.update(alpha=round(rng.uniform(0.05, 0.5), 3), max_iters=rng.choice([15, 20, 200]))
    if kind == "adu":
        c.update(dtype=rng.choice(["uint16", "uint8", "float32"]), levels=rng.choice([1, 1, 2, 3]))
    elif kind != "dropin":
        c.update(per_frame=rng.choice([False, False, True]))
    return c


# ---- simulated frames ---------------------------------------------------------------------------

def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFFFFFF)
    return g


def _ideal(H, W, seed, bg=10.0, photons=100.0):
    """Filaments of emitters (one chain per 150 x 150 px) through a Gaussian PSF; integer counts
    per pixel and fixed-order sums, so the image depends on the seed alone."""
    g = _gen(seed, 1)
    n = max(1, int(round(H * W / 22500.0)))
    steps = 350
    u = torch.rand((n, 3), generator=g, device=DEV, dtype=torch.float64)
    turn = 0.14 * torch.randn((n, steps), generator=g, device=DEV, dtype=torch.float64)
    th = 2 * math.pi * u[:, :1] + torch.cumsum(turn, 1)
    x = u[:, 1:2] * W + 0.2 * torch.cumsum(torch.cos(th), 1)
    y = u[:, 2:3] * H + 0.2 * torch.cumsum(torch.sin(th), 1)
    xi, yi = x.floor().long(), y.floor().long()
    keep = (xi >= 0) & (xi < W) & (yi >= 0) & (yi < H)
    img = torch.bincount((yi * W + xi)[keep], minlength=H * W).reshape(1, 1, H, W).double()
    k = torch.exp(-0.5 * (torch.arange(-5, 6, device=DEV).double() / 1.05) ** 2)
    k = k / k.sum()
    img = F.pad(img, (5, 5, 5, 5))
    img = sum(k[i] * img[..., i:i + W] for i in range(11))
    img = sum(k[i] * img[..., i:i + H, :] for i in range(11))
    return (bg + photons * img[0, 0]).float()


def _camera(H, W, seed, hot, bits=16):
    """Per-pixel offset, gain and read variance."""
    g = _gen(seed, 2)

    def normal(mean, sd):
        return mean + sd * torch.randn((H, W), generator=g, device=DEV)
    offset, gain = (normal(100.0, 2.0), normal(2.0, 0.2)) if bits > 8 else (normal(10.0, 1.0),
                                                                           normal(0.5, 0.03))
    gain = gain.clamp_min(0.1)
    var = -60.0 * torch.log1p(-torch.rand((H, W), generator=g, device=DEV).clamp_max(0.999999))
    var = (var if bits > 8 else var / 60.0) + 0.05
    spot = torch.rand((H, W), generator=g, device=DEV) < hot
    return offset, gain, torch.where(spot, 50.0 * var, var)


def _photons(ideal, T, gain, var, seed):
    """Photo-electrons [T, H, W] (non-positive values become 1e-6), in chunks of frames."""
    H, W = ideal.shape
    g = _gen(seed, 3)
    out = torch.empty((T, H, W), device=DEV)
    sd = var.sqrt() / gain
    step = max(1, (1 << 26) // (H * W))
    for f in range(0, T, step):
        n = min(step, T - f)
        d = torch.poisson(ideal.expand(n, H, W).contiguous(), generator=g)
        d = d + sd * torch.randn((n, H, W), generator=g, device=DEV)
        out[f:f + n] = torch.where(d <= 0, torch.full_like(d, 1e-6), d)
    return out


def _frames(T, H, W, hot, per_frame, seed):
    """(photo-electrons [T, H, W], gamma [H, W] or [T, H, W])."""
    _, gain, var = _camera(H, W, seed, hot)
    images = _photons(_ideal(H, W, seed), T, gain, var, seed)
    gamma = (var / gain ** 2).contiguous()
    if per_frame:  # the amplifier drifts a little from frame to frame
        drift = 1.0 + 0.1 * torch.rand((T, 1, 1), generator=_gen(seed, 4), device=DEV)
        gamma = gamma * drift
    return images, gamma


def _mask(pixel=0.1, NA=1.4, wavelength=0.7):
    """1 - incoherent OTF of a circular pupil, centred, 16 x 16."""
    r = numpy.arange(-8, 8)
    k = numpy.hypot(*numpy.meshgrid(r, r)) / (16 * pixel) / (2 * NA / wavelength)
    c = numpy.clip(k, 0.0, 1.0)
    otf = (2 / numpy.pi) * (numpy.arccos(c) - c * numpy.sqrt(1 - c ** 2))
    return numpy.where(k < 1, 1 - otf, 1.0)


def _mask3(pixel=0.1, NA=2.8, wavelength=0.7):
    """The single-pixel variant's raised-cosine mask, centred, 3 x 3."""
    r = numpy.arange(-1.0, 2.0)
    k = numpy.hypot(*numpy.meshgrid(r, r)) / (3 * pixel)
    T = wavelength / 2 / NA / 1.4
    rc = 0.5 * (1 + numpy.cos(numpy.pi * T * k))
    rc[k > 1 / T] = 0
    return 1 - rc


def _raw(c, seed):
    """Raw counts [T, H, W] and the calibration maps of a camera with c["levels"] amplifiers."""
    T, H, W, L = c["T"], c["H"], c["W"], c["levels"]
    bits = 8 if c["dtype"] == "uint8" else 16
    offset, gain, var = _camera(H, W, seed, c["hot"], bits)
    phot = _photons(_ideal(H, W, seed), T, gain, var, seed)
    adu = phot * gain + offset
    if c["dtype"] != "float32":
        adu = adu.round().clamp(0, 255 if bits == 8 else 65535)
        adu = adu.to(torch.uint8) if bits == 8 else adu.to(torch.int32).to(torch.uint16)
    top = 255.0 if bits == 8 else 400.0
    levels = [top * (q + 1) / (L + 1) for q in range(L - 1)]
    gains = torch.stack([gain * (1.0 + 0.02 * q) for q in range(L)])
    variances = torch.stack([var * (1.0 + 0.1 * q) for q in range(L)])
    return adu, offset, gains, variances, levels


def _batch(c, seed):
    """The stacks of a batch: shapes, alphas and optics from c["shapes"], frames from the seed."""
    rng = numpy.random.default_rng(c["shapes"])
    stacks = []
    for i in range(c["n"]):
        H = int(round(math.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"])))))
        W = int(min(c["hi"], max(c["lo"], int(H * rng.uniform(0.5, 2.0)))))
        T = int(rng.integers(1, c["frames"] + 1))
        alpha, NA = float(rng.uniform(0.05, 0.5)), float(rng.choice([1.2, 1.4, 1.49]))
        wl = float(rng.choice([0.52, 0.6, 0.7]))
        images, gamma = _frames(T, H, W, 0.0, False, seed * 97 + i)
        stacks.append(dict(images=images, gamma=gamma, alpha=alpha, mask=_mask(0.1, NA, wl)))
    return stacks


def _tiles(c, seed):
    """Training tiles: network input [n, 2, 16, 16] and target [n, 1, 16, 16] in FP64.  The target
    is the correction to the noise-free tile in units of the tile's scale."""
    n = c["n"]
    side = 16 * int(math.ceil(math.sqrt(n)))
    ideal = _ideal(side, side, seed)
    _, gain, var = _camera(side, side, seed, 0.005)
    d = _photons(ideal, 1, gain, var, seed)[0]

    def cut(a):
        k = side // 16
        return a.reshape(k, 16, k, 16).permute(0, 2, 1, 3).reshape(-1, 256)[:n].double()
    d, g, u = cut(d), cut(var / gain ** 2), cut(ideal)
    s = d.std(1, unbiased=False, keepdim=True) + 1.0
    x = torch.stack([(d - d.mean(1, keepdim=True)) / s, torch.sqrt(d + g) / s], 1)
    return x.reshape(n, 2, 16, 16), ((u - d) / s).reshape(n, 1, 16, 16)


# ---- the calls ----------------------------------------------------------------------------------

def _solver(c):
    s = ncs_b200.Solver(alpha=c["alpha"], max_iters=c["max_iters"])
    s.set_otf_mask(_mask())
    return s


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("stack", "warm", "propose", "normalized"):
        images, gamma = _frames(c["T"], c["H"], c["W"], c["hot"], c["per_frame"], seed)
        st = dict(kind=kind, images=images, gamma=gamma)
        if kind in ("stack", "warm"):
            st["solver"] = _solver(c)
        if kind in ("warm", "propose"):
            st["net"] = WarmStartNet.load(device=DEV)
        if kind == "normalized":
            st["mask"] = _mask3()
        return st
    if kind == "adu":
        adu, offset, gain, var, levels = _raw(c, seed)
        return dict(kind=kind, solver=_solver(c), adu=adu, offset=offset, gain=gain, var=var,
                    levels=levels)
    if kind == "host":
        images, gamma = _frames(c["T"], c["H"], c["W"], c["hot"], c["per_frame"], seed)
        return dict(kind=kind, solver=_solver(c), images=images.cpu().pin_memory(),
                    gamma=gamma.cpu().pin_memory(),
                    out=torch.empty(images.shape, pin_memory=True))
    if kind == "dropin":
        images, gamma = _frames(c["T"], c["H"], c["W"], c["hot"], False, seed)
        images = images.cpu().numpy()
        return dict(kind=kind, images=[images[i].copy() for i in range(c["T"])],
                    gamma=gamma.cpu().numpy(), mask=_mask(), alpha=c["alpha"],
                    max_iters=c["max_iters"])
    if kind == "batch":
        s = ncs_b200.Solver(max_iters=200)
        outs = s.batch_set(_batch(c, seed))
        return dict(kind=kind, solver=s, outs=outs)
    x, t = _tiles(c, seed)
    return dict(kind=kind, net=WarmStartNet.load(device=DEV), x=x.float().contiguous(),
                t=t.float().contiguous())


def run(state):
    st, kind = state, state["kind"]
    if kind == "stack":
        return st["solver"].reduce_noise(st["images"], st["gamma"])
    if kind == "adu":
        return st["solver"].reduce_noise_adu(st["adu"], st["offset"], st["gain"], st["var"],
                                             levels=st["levels"])
    if kind == "host":
        return st["solver"].reduce_noise_host(st["images"], st["gamma"], out=st["out"])
    if kind == "dropin":
        return ncs_b200.reduceNoise(st["images"], st["gamma"], st["mask"], st["alpha"],
                                    max_iters=st["max_iters"])
    if kind == "batch":
        st["solver"].batch_reduce_noise()
        return st["outs"]
    if kind == "warm":
        u0, _ = st["net"].propose_stack_tc(st["images"], st["gamma"], fp8=True)
        out, _ = st["solver"].reduce_noise_from(st["images"], st["gamma"], u0, stats=False)
        return u0, out
    if kind == "propose":
        return st["net"].propose_stack(st["images"], st["gamma"])
    if kind == "normalized":
        return ncs_b200.reduce_noise_normalized(st["images"], st["gamma"], st["mask"])
    net = st["net"]
    loss, grad = net.loss_and_grad(st["x"], st["t"])
    net.adam_step(grad, lr=2e-4)
    return loss, grad, net.params


# ---- what a pass cannot do without --------------------------------------------------------------

_NET_MACS = 256 * 9 * (2 * 32 + 32 * 32 + 32 * 32 + 32)  # multiply-adds of one tile
# per tile: the start (a 16 x 16 transform pair, gradient), then five iterations of a transform
# pair, the history's products, one line-search trial and the update
_SOLVE_FLOPS = 14592 + 5 * 21248


def _axis(n):
    last, o, out = n + 2 - 16, 0, []
    while True:
        out.append(min(o, last))
        if o >= last:
            return out
        o += 14


def _n_tiles(T, H, W):
    return T * len(_axis(H)) * len(_axis(W))


def work(case):
    c, kind = case, case["kind"]
    if kind == "train":
        n = c["n"]
        first = 256 * 9 * 2 * 32  # no input gradient in the first layer
        return {"bytes": 4.0 * (n * 3 * 256 + 8 * 19393),
                "flops": 2.0 * n * (3 * _NET_MACS - first)}
    if kind == "batch":
        rng, b, f = numpy.random.default_rng(c["shapes"]), 0.0, 0.0
        for i in range(c["n"]):
            H = int(round(math.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"])))))
            W = int(min(c["hi"], max(c["lo"], int(H * rng.uniform(0.5, 2.0)))))
            T = int(rng.integers(1, c["frames"] + 1))
            rng.uniform(), rng.choice(3), rng.choice(3)
            b += 8.0 * T * H * W + 4.0 * H * W
            f += _n_tiles(T, H, W) * _SOLVE_FLOPS
        return {"bytes": b, "flops": f}
    T, H, W = c["T"], c["H"], c["W"]
    px, tiles = float(T * H * W), _n_tiles(T, H, W)
    maps = 4.0 * (px if c.get("per_frame") else H * W)
    if kind == "adu":
        size = {"uint8": 1, "uint16": 2, "float32": 4}[c["dtype"]]
        return {"bytes": px * (4 + size) + 4.0 * H * W * (1 + 2 * c["levels"]),
                "flops": tiles * _SOLVE_FLOPS}
    if kind == "propose":
        return {"bytes": 4 * px + maps + 1024.0 * tiles, "flops": 2.0 * tiles * _NET_MACS}
    if kind == "warm":
        return {"bytes": 8 * px + maps + 1024.0 * tiles,
                "flops": tiles * (2.0 * _NET_MACS + _SOLVE_FLOPS)}
    if kind == "normalized":  # 10 quasi-Newton iterations of 9 unknowns
        return {"bytes": 8 * px + maps, "flops": px * 10 * 800}
    return {"bytes": 8 * px + maps, "flops": tiles * _SOLVE_FLOPS}


# ---- the results in 64 bits -----------------------------------------------------------------------

def _optimum(d, g, mask, alpha):
    """Minimisers [N, 16, 16] of the tile cost
        sum u - (d + g) log(u + g) + alpha / 256 sum |fft2 u|^2 M^2
    by Newton steps, each solved by conjugate gradients with the Fourier-diagonal
    preconditioner 1 / (mean curvature + 2 alpha M^2)."""
    M2 = torch.as_tensor(numpy.fft.fftshift(mask).astype(numpy.float32), device=DEV).double() ** 2
    a2 = 2.0 * alpha * M2
    half = a2[:, :9].contiguous()

    def filt(x, h):
        return torch.fft.irfft2(torch.fft.rfft2(x) * h, s=(16, 16))

    def dot(x, y):
        return (x * y).sum((1, 2), keepdim=True)
    c, u = d + g, d.clone()
    for _ in range(14):
        A = u + g
        grad = 1.0 - c / A + filt(u, half)
        curv = c / A ** 2
        pre = 1.0 / (curv.mean((1, 2), keepdim=True) + half)
        p, r = torch.zeros_like(u), -grad
        z = filt(r, pre)
        q, rz = z, dot(r, z)
        for _ in range(40):
            Hq = curv * q + filt(q, half)
            a = rz / dot(q, Hq).clamp_min(1e-300)
            p, r = p + a * q, r - a * Hq
            z = filt(r, pre)
            new = dot(r, z)
            q, rz = z + (new / rz.clamp_min(1e-300)) * q, new
            if float(new.max()) < 1e-22:
                break
        # stay inside the logarithm's domain, and damp the first long steps
        ratio = (-p / A).amax((1, 2), keepdim=True)
        t = torch.where(ratio > 0.9, 0.9 / ratio, torch.ones_like(ratio))
        u = u + t * p
        if float((p.abs() / (1.0 + u.abs())).max()) < 1e-11:
            break
    return u


def _solve64(images, gamma, mask, alpha):
    """The stack of tile optima, segmented and stitched as the library does: 16 x 16 tiles every 14
    pixels over the frame with a 1-pixel edge halo, a pixel taken from the last tile that covers it."""
    T, H, W = images.shape
    idx, own = [], []
    for n in (H, W):
        o = torch.tensor(_axis(n), device=DEV)
        idx.append((o[:, None] + torch.arange(16, device=DEV)[None] - 1).clamp(0, n - 1))
        at = torch.searchsorted(o, torch.arange(n, device=DEV), right=True) - 1
        own.append((at, torch.arange(n, device=DEV) - o[at] + 1))
    (ri, ci), ((ti, tr), (tj, tc)) = idx, own
    tx, ty = ri.shape[0], ci.shape[0]

    def cut(a):
        b = a[:, ri.reshape(-1)][:, :, ci.reshape(-1)]
        return b.reshape(a.shape[0], tx, 16, ty, 16).permute(0, 1, 3, 2, 4).reshape(-1, 16, 16)
    out = torch.empty((T, H, W), dtype=torch.float64, device=DEV)
    step = max(1, 40000 // (tx * ty))
    for f in range(0, T, step):
        n = min(step, T - f)
        g = (gamma[f:f + n] if gamma.dim() == 3 else gamma.expand(n, H, W)).double()
        u = _optimum(cut(images[f:f + n].double()), cut(g), mask, alpha)
        u = u.reshape(n, tx, ty, 16, 16)
        out[f:f + n] = u[:, ti[:, None], tj[None], tr[:, None], tc[None]]
    return out


def _net64(x, params):
    """The network in FP64 on features x [n, 2, 16, 16]; params as one flat vector."""
    o = 0
    for cin, cout, relu in ((2, 32, True), (32, 32, True), (32, 32, True), (32, 1, False)):
        w = params[o:o + cin * 9 * cout].reshape(cin, 3, 3, cout).permute(3, 0, 1, 2)
        b = params[o + cin * 9 * cout:o + cin * 9 * cout + cout]
        o += cin * 9 * cout + cout
        # nine shifted products instead of a library convolution, which is slow in FP64
        xp = F.pad(x, (1, 1, 1, 1))
        y = b.view(1, -1, 1, 1)
        for k in range(9):
            win = xp[:, :, k // 3:k // 3 + 16, k % 3:k % 3 + 16]
            y = y + torch.einsum("nchw,oc->nohw", win, w[:, :, k // 3, k % 3])
        x = torch.relu(y) if relu else y
    return x


def _propose64(images, gamma, params):
    T, H, W = images.shape
    ri, ci = [(torch.tensor(_axis(n), device=DEV)[:, None] + torch.arange(16, device=DEV)[None]
               - 1).clamp(0, n - 1) for n in (H, W)]

    def cut(a):
        b = a[:, ri.reshape(-1)][:, :, ci.reshape(-1)]
        return b.reshape(a.shape[0], len(ri), 16, len(ci), 16).permute(0, 1, 3, 2, 4).reshape(
            -1, 256).double()
    out, step = [], max(1, 4000 // (len(ri) * len(ci)))
    for f in range(0, T, step):
        n = min(step, T - f)
        d = cut(images[f:f + n])
        g = cut(gamma[f:f + n] if gamma.dim() == 3 else gamma.expand(n, H, W))
        s = d.std(1, unbiased=False, keepdim=True) + 1.0
        x = torch.stack([(d - d.mean(1, keepdim=True)) / s,
                         torch.sqrt(d.clamp_min(0) + g.clamp_min(0)) / s], 1)
        y = torch.cat([_net64(p, params) for p in x.reshape(-1, 2, 16, 16).split(8192)])
        u = torch.maximum(d + s * y.reshape(-1, 256), 0.05 * (d + g).clamp_min(1e-3) - g)
        out.append(u.reshape(-1, 16, 16))
    return torch.cat(out)


def _train64(x, t, params, lr):
    """(loss, gradient, parameters after one Adam step from zero moments)."""
    p = params.clone().requires_grad_(True)
    total, n = 0.0, x.shape[0]
    for i in range(0, n, 1024):
        part = ((_net64(x[i:i + 1024], p) - t[i:i + 1024]) ** 2).sum() / (n * 256)
        part.backward()
        total += float(part.detach())
    g = p.grad
    return (torch.tensor([total], dtype=torch.float64), g,
            params - lr * g / (g.abs() + 1e-8))


def _normalized64(images, gamma, mask, alpha=1.0):
    """Per pixel: the minimiser over its 3 x 3 segment of
        (2 / 9) sum [u - c log(u + g)] + alpha sum |fft2(u) / 3 M|^2 / sum u,
    centre value; Newton steps on the 9 unknowns, one vector per unknown."""
    T, H, W = images.shape
    M2 = numpy.fft.ifftshift(numpy.asarray(mask, numpy.float32)).astype(float) ** 2
    ker = numpy.real(numpy.fft.ifft2(M2))
    Q = [[float(ker[(i // 3 - j // 3) % 3, (i % 3 - j % 3) % 3]) for j in range(9)]
         for i in range(9)]
    out = torch.empty((T, H, W), dtype=torch.float64, device=DEV)

    def segment(a):
        p = F.pad(a[None], (1, 1, 1, 1), mode="replicate")[0]
        return [p[:, i // 3:i // 3 + H, i % 3:i % 3 + W].reshape(-1) for i in range(9)]
    step = max(1, (1 << 20) // (H * W))
    for f in range(0, T, step):
        n = min(step, T - f)
        d = segment(images[f:f + n].double())
        g = segment((gamma[f:f + n] if gamma.dim() == 3 else gamma.expand(n, H, W)).double())
        c, u = [a + b for a, b in zip(d, g)], [a.clone() for a in d]
        for _ in range(30):
            S = sum(u)
            Qu = [sum(Q[i][j] * u[j] for j in range(9)) for i in range(9)]
            P = sum(a * b for a, b in zip(u, Qu))
            A = [a + b for a, b in zip(u, g)]
            grad = [2 / 9 * (1 - c[i] / A[i]) + alpha * (2 * Qu[i] / S - P / S ** 2)
                    for i in range(9)]
            L, tail = [[None] * 9 for _ in range(9)], 2 * P / S ** 3
            for i in range(9):  # Cholesky factor of the Hessian, column by column
                for j in range(i + 1):
                    h = alpha * (2 * Q[i][j] / S - 2 * (Qu[i] + Qu[j]) / S ** 2 + tail)
                    if i == j:
                        h = h + 2 / 9 * c[i] / A[i] ** 2
                    for k in range(j):
                        h = h - L[i][k] * L[j][k]
                    L[i][j] = h.clamp_min(1e-14).sqrt() if i == j else h / L[j][j]
            p = [None] * 9
            for i in range(9):
                p[i] = (-grad[i] - sum(L[i][k] * p[k] for k in range(i))) / L[i][i]
            for i in range(8, -1, -1):
                p[i] = (p[i] - sum(L[k][i] * p[k] for k in range(i + 1, 9))) / L[i][i]
            ratio = torch.stack([-b / a for a, b in zip(A, p)]).amax(0)
            t = torch.where(ratio > 0.9, 0.9 / ratio, torch.ones_like(ratio))
            u = [a + t * b for a, b in zip(u, p)]
            if max(float((b.abs() / (1 + a.abs())).max()) for a, b in zip(u, p)) < 1e-11:
                break
        out[f:f + n] = u[4].reshape(n, H, W)
    return torch.where(out < 0, torch.full_like(out, 1e-6), out)


def exact(case, seed):
    c, kind = case, case["kind"]
    with torch.no_grad():
        if kind == "train":
            x, t = _tiles(c, seed)
            x, t = x.float().double(), t.float().double()
            with torch.enable_grad():
                return _train64(x, t, _params(), 2e-4)
        if kind == "batch":
            return [_solve64(s["images"], s["gamma"], s["mask"], s["alpha"])
                    for s in _batch(c, seed)]
        if kind == "adu":
            adu, offset, gain, var, levels = _raw(c, seed)
            a = adu.to(torch.int32).double() if c["dtype"] == "uint16" else adu.double()
            at = sum((a >= float(numpy.float32(v))).long() for v in levels) if levels else \
                torch.zeros_like(a, dtype=torch.long)
            gn = gain.double().gather(0, at.reshape(-1, *offset.shape)) if levels else \
                gain.double().expand_as(a)
            vr = var.double().gather(0, at.reshape(-1, *offset.shape)) if levels else \
                var.double().expand_as(a)
            d = (a - offset.double()) / gn
            d = torch.where(d <= 0, torch.full_like(d, 1e-6), d)
            return _solve64(d, vr / gn ** 2, _mask(), c["alpha"])
        images, gamma = _frames(c["T"], c["H"], c["W"], c["hot"], c.get("per_frame", False), seed)
        if kind == "normalized":
            return _normalized64(images, gamma, _mask3())
        if kind == "propose":
            return _propose64(images, gamma, _params())
        if _n_tiles(c["T"], c["H"], c["W"]) > 1000000:  # over 20 seconds
            return None
        out = _solve64(images, gamma, _mask(), c["alpha"])
        if kind == "dropin":
            return [out[i] for i in range(c["T"])]
        if kind == "warm":
            return _propose64(images, gamma, _params()), out
        return out


def _params():
    return torch.as_tensor(numpy.load(DEFAULT_WEIGHTS).reshape(-1), device=DEV).double()
