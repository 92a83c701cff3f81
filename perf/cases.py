"""Performance cases of the imaging engine, its ILT gradient and its FNO surrogate.

Each case is one call that a program makes through the package's public entry
points, with the sizes of the repository's own workloads (single clips up to
the 256-clip batch of 1024^2 masks, the 2048^2 EUV clips, the 512^2 High-NA
surrogate, contact-array ILT) and ragged ones between them.

``prepare`` makes what a program has in hand before the call (an engine, device
inputs drawn from the seed, a plan or a network), ``run`` is one call, ``work``
is what the call cannot do without, ``exact`` is the same result in 64 bits
from plain numpy and torch.  Engines sample their source on a uniform lattice
(``source_points_per_axis``), which ``exact`` restates in a few lines.
"""
import math

import numpy as np
import torch

import highuvlith_b200 as HB
from highuvlith_b200 import ilt as hb_ilt
from highuvlith_b200.fno import FnoSurrogate

# Optical set-ups by name: wavelength (nm), NA, image-space index, inner and
# outer sigma of the (annular or conventional) fill, flare, central obscuration.
SETUPS = {
    # EUV scanner, conventional fill: the 1024^2 batch workload, ILT
    "euv": (13.5, 0.33, 1.0, 0.0, 0.5, 0.0, 0.0),
    # EUV with an annular fill at the edge of the pupil: the widest bands
    "euv_annular": (13.5, 0.33, 1.0, 0.7, 0.9, 0.0, 0.0),
    # High-NA EUV with its central obscuration: the surrogate's workload
    "high_na": (13.5, 0.55, 1.0, 0.3, 0.8, 0.0, 0.2),
    # ArF immersion with flare: narrow bands
    "arfi": (193.368, 1.35, 1.437, 0.6, 0.85, 0.02, 0.0),
    # F2 (157 nm) dry exposure: focus sweeps
    "f2": (157.63, 0.75, 1.0, 0.0, 0.7, 0.02, 0.0),
}
POINTS_PER_AXIS = 17


def listed():
    return [
        # one small clip: an interactive or scripted single exposure, where launches count
        dict(name="image_1x256_u8", kind="image", setup="euv", n=256, clips=1, kernels=20, dtype="u8", focus=0.0),
        # the batch workload: 256 Manhattan clips of 1024^2, 32 kernels
        dict(name="image_256x1024_u8", kind="image", setup="euv", n=1024, clips=256, kernels=32, dtype="u8", focus=0.0),
        # grey-level transmittance maps: images that train the surrogate and judge ILT iterates
        dict(name="image_27x512_f32", kind="image", setup="high_na", n=512, clips=27, kernels=48, dtype="f32",
             focus=0.0),
        # phase-shifting masks as complex maps, out of focus
        dict(name="image_7x512_c64", kind="image", setup="arfi", n=512, clips=7, kernels=30, dtype="c64", focus=40.0),
        # the largest clips: 2048^2 at full EUV band, 64 kernels
        dict(name="image_6x2048_u8", kind="image", setup="euv_annular", n=2048, clips=6, kernels=64, dtype="u8",
             focus=0.0),
        # a process window: one clip through 21 focus planes (planes already built)
        dict(name="focus_21x256", kind="focus", setup="f2", n=256, pixel=2.0, clips=1, kernels=20, planes=21,
             step=20.0),
        # layout clips as rectangles, exact spectra
        dict(name="rects_40x512", kind="rects", setup="euv", n=512, clips=40, kernels=30, rects=60),
        # ILT: cost and gradient of a full batch of masks, and of a few small ones
        dict(name="ilt_64x1024", kind="ilt", setup="euv", n=1024, clips=64, kernels=32),
        dict(name="ilt_3x256", kind="ilt", setup="euv", n=256, clips=3, kernels=20),
        # the surrogate: inference on a batch, and the gradients of a training step
        dict(name="fno_forward_16x512", kind="fno_forward", n=512, clips=16),
        dict(name="fno_backward_8x512", kind="fno_backward", n=512, clips=8, want_input=False),
        # clips of several sizes, sources and kernel budgets in one planned launch
        dict(name="plan_90_uneven", kind="plan", clips=90, top=1024),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["image", "image", "image", "focus", "rects", "ilt", "fno_forward", "fno_backward", "plan"])
    if kind == "image":
        n = rng.choice([256, 512, 1024, 2048])
        setup = rng.choice(["euv", "euv_annular", "high_na", "arfi"]) if n < 2048 else "euv_annular"
        dtype = rng.choice(["u8", "u8", "f32", "c64"])
        most = {256: 600, 512: 200, 1024: 60, 2048: 6}[n]
        return dict(kind=kind, setup=setup, n=n, clips=logint(1, most), kernels=rng.randint(8, 64), dtype=dtype,
                    focus=rng.choice([0.0, 0.0, round(rng.uniform(10.0, 60.0), 1)]))
    if kind == "focus":
        setup, n, pixel, step = rng.choice([("f2", 256, 2.0, 20.0), ("euv", 256, 1.0, 10.0), ("arfi", 512, 1.0, 15.0)])
        return dict(kind=kind, setup=setup, n=n, pixel=pixel, clips=logint(1, 9), kernels=rng.randint(8, 24),
                    planes=rng.randint(3, 21), step=step)
    if kind == "rects":
        return dict(kind=kind, setup=rng.choice(["euv", "arfi"]), n=rng.choice([256, 512, 1024]),
                    clips=logint(1, 60), kernels=rng.randint(8, 40), rects=logint(4, 120))
    if kind == "ilt":
        n = rng.choice([256, 512, 1024])
        return dict(kind=kind, setup=rng.choice(["euv", "arfi"]), n=n, clips=logint(1, 64 if n < 1024 else 40),
                    kernels=rng.randint(8, 32))
    if kind == "plan":
        return dict(kind=kind, clips=rng.randint(12, 90), top=rng.choice([512, 1024]))
    n = rng.choice([128, 256, 512])
    most = {128: 48, 256: 24, 512: 8}[n]
    c = dict(kind=kind, n=n, clips=logint(1, most))
    if kind == "fno_backward":
        c["want_input"] = rng.choice([False, True])
    return c


# ------------------------------------------------------------------ inputs
def _engine(setup, n, kernels, pixel=1.0):
    lam, na, index, s0, s1, flare, obscuration = SETUPS[setup]
    fill, par = ("annular", (s0, s1)) if s0 > 0 else ("conventional", (s1,))
    opt = (HB.OpticsConfig.euv(na, obscuration) if lam < 20 else
           HB.OpticsConfig(na, flare, index))
    return HB.SimulationEngine(HB.SourceConfig(lam, fill, par), opt, grid=HB.GridConfig(n, pixel),
                               max_kernels=kernels, source_points_per_axis=POINTS_PER_AXIS)


def _rasters(rng, n, clips):
    """Manhattan clips: clear rectangles of 10 to 80 pixels on a dark field."""
    count = max(3, int(0.5 * n * n / (45 * 45)))
    out = []
    for _ in range(clips):
        w = rng.integers(10, 81, (count, 2))
        xy = rng.integers(0, n - w + 1)
        out.append(np.concatenate([xy, w], axis=1).tolist())
    return HB.rasterize_rects(n, out)


def _maps(rng, n, clips, dtype):
    r = _rasters(rng, n, clips)
    if dtype == "u8":
        return r
    g = torch.Generator(device="cuda")
    g.manual_seed(int(rng.integers(1 << 40)))
    if dtype == "f32":  # grey levels between dark and clear, as ILT iterates have
        beta = 2.0 + 6.0 * torch.rand((clips, 1, 1), generator=g, device="cuda")
        return torch.sigmoid(beta * (r.float() - 0.5 + 0.15 * torch.randn(r.shape, generator=g, device="cuda")))
    # clear, or attenuated with a phase shift of 180 degrees, and phase errors
    t = torch.where(r > 0, torch.tensor(1.0 + 0j, device="cuda"), torch.tensor(-0.245 + 0j, device="cuda"))
    return (t * torch.exp(0.1j * torch.randn(r.shape, generator=g, device="cuda"))).to(torch.complex64)


def _rect_clips(rng, n, clips, count):
    out = []
    for _ in range(clips):
        w = rng.uniform(8.0, 60.0, (count, 2))
        c = rng.uniform(-0.4 * n, 0.4 * n, (count, 2))
        out.append([tuple(r) for r in np.concatenate([c, w], axis=1).tolist()])
    return out


def _targets(rng, n, clips):
    """Contact arrays (holes of 16 to 24 nm on a pitch of 32 to 48 nm)."""
    x = torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 - n / 2
    out = torch.empty((clips, n, n), device="cuda")
    for i in range(clips):
        size, pitch = rng.uniform(16.0, 24.0), rng.uniform(32.0, 48.0)
        axes = []
        for count in rng.integers(2, 9, 2):
            c = (torch.arange(int(count), device="cuda", dtype=torch.float64) - (int(count) - 1) / 2) * pitch
            edge = 0.5 * size - (x[:, None] - c[None, :]).abs() + 0.5
            axes.append(edge.clamp(0.0, 1.0).sum(1))
        out[i] = (axes[1][:, None] * axes[0][None, :]).float()
    g = torch.Generator(device="cuda")
    g.manual_seed(int(rng.integers(1 << 40)))
    theta = out - 0.5 + 0.2 * torch.randn(out.shape, generator=g, device="cuda")
    return theta, out


def _plan_groups(case):
    """(setup, n, kernel budget, clips) of the uneven batch's groups."""
    rng = np.random.default_rng(case["clips"])
    sizes = [n for n in (256, 512, 1024) if n <= case["top"]]
    kinds = [(s, n, k) for s in ("arfi", "euv") for n in sizes for k in (16, 40)]
    share = rng.multinomial(case["clips"], [1.0 / len(kinds)] * len(kinds))
    return [(s, n, k, int(c)) for (s, n, k), c in zip(kinds, share) if c]


ILT = hb_ilt.IltSettings(cost="resist", threshold=0.25, steepness=50.0, sigmoid_steepness=4.0, regularization=0.01,
                         tv_epsilon=0.01)


def prepare(case, seed):
    rng = np.random.default_rng([seed, 20])
    kind = case["kind"]
    if kind == "image":
        return dict(case=case, engine=_engine(case["setup"], case["n"], case["kernels"]),
                    x=_maps(rng, case["n"], case["clips"], case["dtype"]))
    if kind == "focus":
        z = [(i - (case["planes"] - 1) / 2) * case["step"] for i in range(case["planes"])]
        s = dict(case=case, engine=_engine(case["setup"], case["n"], case["kernels"], case["pixel"]), z=z,
                 x=_rasters(rng, case["n"], case["clips"]))
        s["engine"].compute_batch_through_focus(s["x"], z)  # the planes' kernels, kept by the engine
        return s
    if kind == "rects":
        return dict(case=case, engine=_engine(case["setup"], case["n"], case["kernels"]),
                    clips=_rect_clips(rng, case["n"], case["clips"], case["rects"]))
    if kind == "ilt":
        theta, target = _targets(rng, case["n"], case["clips"])
        return dict(case=case, engine=_engine(case["setup"], case["n"], case["kernels"]), theta=theta, target=target)
    if kind == "plan":
        groups = _plan_groups(case)
        engines = {(s, n): _engine(s, n, 40) for s, n, _, _ in groups}
        clips, out, store = [], [], []
        for s, n, k, c in groups:
            x = _rasters(rng, n, c)
            y = torch.empty((c, n, n), dtype=torch.float32, device="cuda")
            clips += [(engines[s, n], k, x[i], y[i]) for i in range(c)]
            out.append(y)
            store.append(x)
        return dict(case=case, plan=HB.UnevenPlan(clips), out=out, x=store, groups=groups)
    x = _maps(rng, case["n"], case["clips"], "f32")
    fno = FnoSurrogate(case["n"], 16, 4, seed=seed)
    s = dict(case=case, fno=fno, x=x)
    if kind == "fno_backward":  # images of the same scale as the engine's
        s["target"] = torch.nn.functional.avg_pool2d(x[:, None], 9, 1, 4)[:, 0] ** 2
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "image":
        # rasters are masks; grey-level and complex maps are transmittances
        return state["engine"].compute_batch(state["x"], focus_nm=case["focus"], pixel_transfer=case["dtype"] == "u8")
    if kind == "focus":
        return state["engine"].compute_batch_through_focus(state["x"], state["z"])
    if kind == "rects":
        return state["engine"].compute_batch_rects(state["clips"])
    if kind == "ilt":
        return hb_ilt.cost_and_gradient(state["engine"], state["theta"], state["target"], ILT)
    if kind == "plan":
        state["plan"].launch()
        return state["out"]
    if kind == "fno_forward":
        return state["fno"].forward(state["x"])
    loss, grads, dx = state["fno"].backward(state["x"], targets=state["target"], want_input_grad=case["want_input"])
    return [loss, grads] + ([dx] if dx is not None else [])


# ------------------------------------------------------------------ work
def _band(setup, n, pixel=1.0):
    lam, na, _, _, s1, _, _ = SETUPS[setup]
    return int(na / lam * (1 + s1) * n * pixel)


def _field_flops(setup, n, kernels, pixel=1.0):
    """K inverse transforms on the smallest grid that holds the intensity."""
    m = min(n, 4 * _band(setup, n, pixel) + 1)
    return kernels * 5.0 * m * m * math.log2(m * m)


def work(case):
    kind = case["kind"]
    if kind == "plan":
        groups = _plan_groups(case)
        return {"bytes": sum(c * 5.0 * n * n for _, n, _, c in groups),
                "flops": sum(c * _field_flops(s, n, k) for s, n, k, c in groups)}
    n, clips = case["n"], case["clips"]
    px = float(clips) * n * n
    if kind == "image":
        size = {"u8": 1, "f32": 4, "c64": 8}[case["dtype"]]
        return {"bytes": px * (size + 4), "flops": clips * _field_flops(case["setup"], n, case["kernels"])}
    if kind == "focus":
        return {"bytes": px * (1 + 4 * case["planes"]),
                "flops": clips * case["planes"] * _field_flops(case["setup"], n, case["kernels"], case["pixel"])}
    if kind == "rects":
        return {"bytes": px * 4, "flops": clips * _field_flops(case["setup"], n, case["kernels"])}
    if kind == "ilt":  # theta and target in, gradient out; fields, their adjoint
        return {"bytes": px * 12, "flops": clips * 3 * _field_flops(case["setup"], n, case["kernels"])}
    # lift, four layers of 64 x 64 channels, the projection 64 -> 128 -> 1; mode weights read once
    pointwise = px * 2 * (3 * 64 + 4 * 64 * 64 + 64 * 128 + 128)
    weights = 4.0 * 4 * 512 * 64 * 64 * 2
    if kind == "fno_forward":
        return {"bytes": px * 8 + weights, "flops": pointwise}
    return {"bytes": px * (12 if case["want_input"] else 8) + 2 * weights, "flops": 3 * pointwise}


# ------------------------------------------------------------------ exact
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _source(s0, s1):
    """Cell centres of the uniform lattice over the fill's bounding square
    (probed in steps of 1/32 sigma) that lie inside the fill, equal weights."""
    half = math.floor(s1 * 32 + 1e-9) / 32 + 1 / 32
    c = (np.arange(POINTS_PER_AXIS) + 0.5 - POINTS_PER_AXIS / 2) * (2 * half / POINTS_PER_AXIS)
    x, y = np.meshgrid(c, c)
    r = np.hypot(x, y).ravel()
    keep = (r >= s0) & (r <= s1)
    return x.ravel()[keep], y.ravel()[keep]


def _kernels(setup, n, budget, pixel, z):
    """Leading eigenfunctions of the transmission cross-coefficients, scaled by
    the root of their eigenvalue over the clear field: (orders, (K, S)), and flare."""
    lam, na, index, s0, s1, flare, obscuration = SETUPS[setup]
    sx, sy = _source(s0, s1)
    df = lam / (na * n * pixel)  # one order in units of the pupil radius
    r = (1 + np.hypot(sx, sy).max()) / df
    o = np.arange(-int(r), int(r) + 1)
    my, mx = (v.ravel() for v in np.meshgrid(o, o, indexing="ij"))
    keep = (mx * mx + my * my <= r * r * (1 + 1e-12)) & (abs(mx) <= n // 2) & (abs(my) <= n // 2)
    my, mx = my[keep], mx[keep]
    fx, fy = mx[:, None] * df + sx, my[:, None] * df + sy
    rho = np.hypot(fx, fy)
    open_ = (fx * fx + fy * fy <= 1.0) & ~(rho < obscuration)
    s2 = np.where(open_, (na * rho / index) ** 2, 0.0)
    phase = 2 * np.pi * index * z * s2 / ((1 + np.sqrt(1 - s2)) * lam)
    a = torch.from_numpy(np.where(open_, np.exp(1j * phase), 0.0) / math.sqrt(len(sx)))
    clear = float((a[(my == 0) & (mx == 0)].abs() ** 2).sum())
    a = a[:, (a != 0).any(0)].to(_dev())
    if a.shape[0] <= a.shape[1]:
        values, vectors = torch.linalg.eigh(a @ a.mH)
        values, vectors = values.flip(0), vectors.flip(1)
    else:
        values, vectors = torch.linalg.eigh(a.mH @ a)
        values, vectors = values.flip(0), vectors.flip(1)
        vectors = a @ (vectors / values.clamp_min(1e-300).sqrt())
    v = values.cpu().numpy()
    valid = int((v > 1e-12 * v[0]).sum())
    same = lambda i: i < valid and abs(v[i - 1] - v[i]) <= 1e-6 * max(abs(v[i - 1]), abs(v[i]))  # noqa: E731
    k = end = min(budget, valid)
    while 0 < end < valid and same(end):  # a cluster of equal values is kept or dropped whole
        end += 1
    if end <= budget:
        k = end
    else:
        while k > 0 and same(k):
            k -= 1
        k = k or end
    return (my, mx), (vectors[:, :k] * (values[:k] / clear).sqrt()).T.contiguous(), flare


def _image(spectrum, orders, kernels, flare):
    """Sum of |ifft2(kernel * spectrum)|^2, with uniform flare."""
    n = spectrum.shape[-1]
    img = torch.zeros((n, n), dtype=torch.float64, device=spectrum.device)
    my, mx = (torch.from_numpy(v % n).to(spectrum.device) for v in orders)
    part = spectrum[my, mx]
    for u in kernels:
        e = torch.zeros_like(spectrum)
        e[my, mx] = u * part
        e = torch.fft.ifft2(e)
        img += e.real ** 2 + e.imag ** 2
    return img * (1 - flare) + flare * img.mean() if flare > 0 else img


def _mask_spectrum(x, transfer):
    s = torch.fft.fft2(x.to(torch.complex128))
    if transfer:  # pixels are squares, not samples
        n = x.shape[-1]
        t = torch.from_numpy(np.sinc(np.fft.fftfreq(n))).to(x.device)
        s = s * t[:, None] * t[None, :]
    return s


def _rect_spectrum(rects, n):
    """Exact spectrum of the union of rectangles, from its cells."""
    r = np.asarray(rects)
    edges = [np.unique(np.concatenate([r[:, a] - r[:, a + 2] / 2, r[:, a] + r[:, a + 2] / 2])) for a in (0, 1)]
    cover = np.zeros((len(edges[1]) - 1, len(edges[0]) - 1))
    for x, y, w, h in r:
        i = [np.searchsorted(edges[a], (c - s / 2, c + s / 2)) for a, c, s in ((0, x, w), (1, y, h))]
        cover[i[1][0]:i[1][1], i[0][0]:i[0][1]] = 1.0
    m = np.fft.fftfreq(n, 1 / n)[:, None]
    axis = []
    for e in edges:
        a, b = e[:-1], e[1:]
        axis.append((b - a) * np.sinc(m * (b - a) / n) * np.exp(-1j * np.pi * m * (a + b) / n)
                    * np.exp(-1j * np.pi * m * (n - 1) / n))
    return torch.from_numpy(axis[1] @ cover @ axis[0].T).to(_dev())


def _ilt(theta, target, orders, kernels, flare):
    p = ILT
    theta = theta.double().requires_grad_(True)
    m = torch.sigmoid(p.sigmoid_steepness * theta)
    spectrum = torch.fft.fft2(m.to(torch.complex128))
    with torch.no_grad():
        img = _image(spectrum, orders, kernels, flare)
    img.requires_grad_(True)
    cost = ((torch.sigmoid(p.steepness * (p.dose * img - p.threshold)) - target.double()) ** 2).mean()
    cost.backward()
    with torch.no_grad():  # adjoint of the image, kernel by kernel
        n = m.shape[-1]
        g = img.grad * (1 - flare) + flare * img.grad.mean()
        my, mx = (torch.from_numpy(v % n).to(m.device) for v in orders)
        q = torch.zeros_like(spectrum)
        for u in kernels:
            e = torch.zeros_like(spectrum)
            e[my, mx] = u * spectrum[my, mx]
            q[my, mx] += u.conj() * torch.fft.fft2(g * torch.fft.ifft2(e))[my, mx]
        dm = 2 * torch.fft.ifft2(q).real
    dx, dy = torch.roll(m, -1, 1) - m, torch.roll(m, -1, 0) - m
    tv = p.regularization * (torch.sqrt(dx * dx + dy * dy + p.tv_epsilon ** 2) - p.tv_epsilon).mean()
    grad = torch.autograd.grad(tv + (m * dm).sum(), theta)[0]
    return float(cost) + float(tv), grad


def _fno(params, x, n, layers=4, modes=16, c=64, hidden=128):
    """The network in 64 bits: lift, four spectral layers, projection."""
    at = 0

    def take(*shape):
        nonlocal at
        size = int(np.prod(shape))
        at += size
        return params[at - size:at].reshape(shape)

    pos = torch.arange(n, dtype=torch.float64, device=x.device) / n
    wl, bl = take(c, 3), take(c)
    v = x[..., None] * wl[:, 0] + pos[None, None, :, None] * wl[:, 1] + pos[None, :, None, None] * wl[:, 2] + bl
    k = torch.arange(modes, dtype=torch.float64, device=x.device)
    ky = torch.cat([k, k - modes])
    ex = torch.exp(-2j * math.pi * torch.outer(k, pos))
    ey = torch.exp(-2j * math.pi * torch.outer(ky, pos))
    wx = torch.full((modes,), 2.0, dtype=torch.float64, device=x.device)
    wx[0] = 1.0
    for i in range(layers):
        r = torch.view_as_complex(take(2 * modes, modes, c, c, 2))
        w, b = take(c, c), take(c)
        f = torch.einsum("jy,bykc->bjkc", ey, torch.einsum("bysc,ks->bykc", v.to(torch.complex128), ex))
        y = torch.einsum("bjki,jkio->bjko", f, r) * wx[None, None, :, None]
        z = torch.einsum("bjko,jy->byko", y, ey.conj())
        s = torch.einsum("byko,ks->byso", z.real, ex.real) + torch.einsum("byko,ks->byso", z.imag, ex.imag)
        v = s / (n * n) + v @ w.T + b
        if i < layers - 1:
            v = torch.nn.functional.gelu(v)
    q1, b1, q2, b2 = take(hidden, c), take(hidden), take(hidden), take(1)
    return torch.nn.functional.gelu(v @ q1.T + b1) @ q2 + b2


def exact(case, seed):
    kind = case["kind"]
    state = prepare(case, seed)
    if kind in ("image", "focus"):
        pixel = case.get("pixel", 1.0)
        out = []
        for z in state.get("z", [case.get("focus", 0.0)]):
            optics = _kernels(case["setup"], case["n"], case["kernels"], pixel, z)
            transfer = kind == "focus" or case["dtype"] == "u8"
            out.append(torch.stack([_image(_mask_spectrum(x, transfer), *optics) for x in state["x"]]))
        return torch.stack(out) if kind == "focus" else out[0]
    if kind == "rects":
        optics = _kernels(case["setup"], case["n"], case["kernels"], 1.0, 0.0)
        return torch.stack([_image(_rect_spectrum(r, case["n"]), *optics) for r in state["clips"]])
    if kind == "ilt":
        optics = _kernels(case["setup"], case["n"], case["kernels"], 1.0, 0.0)
        both = [_ilt(t, g, *optics) for t, g in zip(state["theta"], state["target"])]
        return np.array([c for c, _ in both]), torch.stack([g for _, g in both])
    if kind == "plan":
        return [torch.stack([_image(_mask_spectrum(r, True), *_kernels(s, n, k, 1.0, 0.0)) for r in x])
                for (s, n, k, _), x in zip(state["groups"], state["x"])]
    params = torch.from_numpy(state["fno"].get_params()).double().to(_dev())
    if kind == "fno_forward":
        with torch.no_grad():
            return torch.cat([_fno(params, x[None].double(), case["n"]) for x in state["x"]])
    params.requires_grad_(True)
    loss, dx = 0.0, []
    for x, t in zip(state["x"], state["target"]):  # one sample at a time: the sums are the batch's
        x = x[None].double().requires_grad_(True)
        part = ((_fno(params, x, case["n"]) - t.double()) ** 2).sum() / state["x"].numel()
        part.backward()
        loss += float(part)
        dx.append(x.grad)
    return [loss, params.grad] + ([torch.cat(dx)] if case["want_input"] else [])
