"""Workloads of the deconvolution framework for timing and for comparing results.

Each case is one call that a user's program makes through the public entry
points: the convolution operator alone, the three solvers on it, the solvers
that build their operator themselves, tiled batches and PSF synthesis.  The
inputs are what such a program holds before the call (a measured stack, a PSF,
an operator built once); scenes are beads and filaments under Poisson noise,
PSFs are scalar widefield ones with a defocus phase and spherical aberration.
"""

import math

import numpy as np
import torch

import deconlib_b200.deconvolution as D
from deconlib_b200.batch import batched_tiled_rl, plan_uneven_tiles
from deconlib_b200.psf import pupil_to_psf

SPACING = (0.1, 0.085, 0.085)        # um per voxel (z, y, x)
SPACING_FINE = (0.05, 0.0425, 0.0425)
TILE_VOXELS = 2_400_000              # the largest padded grid that RL on a composed operator takes


def listed():
    return [
        # a patch around one bead, restored or blurred many thousands of times:
        # launches and latency only
        dict(name="conv_patch", kind="conv", nz=16, ny=32, nx=32, kz=9, ky=15, kx=15, precision="fp32"),
        # one frame of a camera, 2-D, with the lateral part of a PSF
        dict(name="conv_frame", kind="conv", nz=1, ny=512, nx=640, kz=1, ky=63, kx=63, precision="fp32"),
        # a stack cropped around a cell, so with extents that nobody rounds, and
        # a PSF cropped to its support: the operator in a caller's own solver
        dict(name="conv_stack", kind="conv", nz=47, ny=301, nx=243, kz=31, ky=63, kx=63, precision="fp32"),
        # the mixed-precision workload's volume: the operator with an FP16 OTF
        dict(name="conv_mixed", kind="conv", nz=128, ny=256, nx=256, kz=128, ky=256, kx=256,
             precision="mixed"),
        # the plain Richardson-Lucy workload as it is quoted: 50 iterations
        dict(name="rl_standard", kind="rl", nz=64, ny=128, nx=128, kz=64, ky=128, kx=128, iters=50),
        # a whole camera stack at once with a cropped PSF: the largest
        dict(name="rl_large", kind="rl", nz=150, ny=600, nx=700, kz=47, ky=95, kx=95, iters=10),
        # one tile through the tile solver: data coarser than the restored grid
        # by 1.5 laterally, PSF margins around it (generic operator chain)
        dict(name="rl_tile", kind="tile", nz=40, ny=96, nx=88, kz=31, ky=47, kx=47, zoom_z=1.0,
             zoom_xy=1.5, iters=10),
        # the Hessian-PDHG workload: one whole call from stack and PSF, 2x
        # sampling; a short run of the quoted solve
        dict(name="pdhg_hessian", kind="pdhg", nz=64, ny=128, nx=128, sampling=2.0, norm="L1",
             loss="poisson", iters=40),
        # total variation on an operator in hand, ragged extents, Gaussian data
        dict(name="pdhg_tv", kind="pdhg_op", nz=60, ny=210, nx=190, kz=25, ky=41, kx=41,
             reg="gradient", norm="L1_2", loss="gaussian", iters=15),
        # Poisson maximum likelihood by nonlinear CG, as many steps as it is run for
        dict(name="nlcg_plain", kind="nlcg", nz=64, ny=128, nx=128, kz=33, ky=65, kx=65, iters=8),
        # a volume in uneven overlapping tiles, all advanced by one graph
        dict(name="tiles_batch", kind="batch", nz=96, ny=384, nx=384, kz=32, ky=64, kx=64, core_z=48,
             core_xy=160, halo=16, iters=40),
        # the PSF of the PDHG workload from its pupil
        dict(name="psf_widefield", kind="psf", nz=128, ny=256, nx=256),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _volume(rng, z, xy):
    return dict(nz=_spread(rng, *z), ny=_spread(rng, *xy), nx=_spread(rng, *xy))


def _kernel(rng, c):
    return dict(kz=min(c["nz"], _spread(rng, 9, 65)), ky=_spread(rng, 15, 129), kx=_spread(rng, 15, 129))


def draw(rng):
    kind = rng.choice(["conv", "conv", "conv", "rl", "rl", "rl", "tile", "pdhg", "pdhg", "pdhg_op", "nlcg",
                       "batch", "psf"])
    if kind == "conv":
        c = _volume(rng, (12, 160), (32, 600))
        if rng.random() < 0.25:
            c["nz"] = 1
        c.update(_kernel(rng, c), precision="fp32")
        if c["nz"] > 1 and rng.random() < 0.25:
            # the canvases that have an FP16 OTF: an axial length of 64 or 256
            c.update(nz=rng.choice([rng.randint(24, 32), rng.randint(100, 128)]), precision="mixed")
            c["kz"] = 64 - c["nz"] + 1 if c["nz"] <= 32 else 256 - c["nz"] + 1
    elif kind == "rl":
        c = _volume(rng, (16, 150), (64, 560))
        c.update(_kernel(rng, c), iters=rng.randint(5, 10))
    elif kind == "tile":
        c = _volume(rng, (12, 64), (48, 160))
        c.update(kz=min(c["nz"], rng.randint(9, 33)), ky=rng.randint(15, 65), kx=rng.randint(15, 65),
                 zoom_z=rng.choice([1.0, 1.5, 2.0]), zoom_xy=rng.choice([1.0, 1.25, 1.5, 2.0]),
                 iters=rng.randint(5, 12))
        while math.prod(_tile_grids(c)[2]) > TILE_VOXELS:
            c.update(ny=max(24, c["ny"] * 7 // 8), nx=max(24, c["nx"] * 7 // 8), ky=max(15, c["ky"] * 7 // 8),
                     kx=max(15, c["kx"] * 7 // 8))
    elif kind == "pdhg":
        c = _volume(rng, (12, 64), (40, 160))
        c.update(sampling=rng.choice([1.0, 1.5, 2.0, 2.0]), norm=rng.choice(["L1", "L1_2"]),
                 loss=rng.choice(["poisson", "poisson", "gaussian"]), iters=rng.randint(10, 40))
    elif kind == "pdhg_op":
        c = _volume(rng, (12, 100), (48, 300))
        c.update(_kernel(rng, c), reg=rng.choice(["identity", "gradient", "hessian"]),
                 norm=rng.choice(["L1", "L1_2"]), loss=rng.choice(["poisson", "gaussian"]),
                 iters=rng.randint(8, 16))
    elif kind == "nlcg":
        c = _volume(rng, (16, 96), (64, 256))
        c.update(_kernel(rng, c), iters=rng.randint(4, 8))
    elif kind == "batch":
        c = dict(nz=rng.randint(48, 128), ny=rng.randint(256, 448), nx=rng.randint(256, 448),
                 kz=rng.randint(16, 40), ky=rng.randint(31, 80), kx=rng.randint(31, 80),
                 core_z=rng.choice([32, 48]), core_xy=rng.choice([96, 128, 160]),
                 halo=rng.randint(8, 24), iters=rng.randint(10, 40))
    else:
        smooth = [2 ** a * 3 ** b * 5 ** e for a in range(10) for b in range(3) for e in range(3)]
        lateral = [v for v in smooth if 96 <= v <= 512]
        c = dict(nz=_spread(rng, 9, 160), ny=rng.choice(lateral), nx=rng.choice(lateral))
    c["kind"] = kind
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * (int(seed) % 100003) + 17)


def _uniform(gen, lo, hi, n=1):
    return lo + (hi - lo) * torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)


def _pupil(ny, nx, spacing, seed):
    """Pupil (complex128) and axial frequencies of an NA 1.2-1.4 objective with
    up to half a radian of spherical aberration."""
    gen = _generator(seed)
    na, wl, ni = float(_uniform(gen, 1.2, 1.4)), 0.525, 1.515
    sph = float(_uniform(gen, -0.5, 0.5))
    f64 = dict(dtype=torch.float64, device="cuda")
    ky = torch.fft.fftfreq(ny, spacing[1], **f64)[:, None]
    kx = torch.fft.fftfreq(nx, spacing[2], **f64)[None, :]
    k = torch.sqrt(ky * ky + kx * kx)
    kmax = na / wl
    weight = ((kmax - k) * (max(ny * spacing[1], nx * spacing[2])) + 0.5).clamp(0.0, 1.0)
    rho = (k / kmax).clamp(0.0, 1.0)
    phase = sph * math.sqrt(5.0) * (6 * rho ** 4 - 6 * rho ** 2 + 1)
    kz = torch.sqrt(((ni / wl) ** 2 - k * k).clamp(min=0.0))
    return weight * torch.exp(1j * phase), kz


def _z_planes(nz, dz):
    return np.fft.fftfreq(nz) * nz * dz


def _psf(shape, spacing, seed):
    """Corner-origin widefield PSF, unit sum, float32."""
    nz, ny, nx = shape
    pupil, kz = _pupil(ny, nx, spacing, seed)
    out = torch.empty(shape, dtype=torch.float32, device="cuda")
    for i, z in enumerate(_z_planes(nz, spacing[0])):
        a = torch.fft.ifft2(pupil * torch.exp(2j * math.pi * kz * z))
        out[i] = (a.real ** 2 + a.imag ** 2).float()
    return out / out.sum(dtype=torch.float64).float()


def _scene(shape, seed):
    """Beads and filaments, amplitudes up to 1."""
    gen = _generator(seed + 1)
    t = torch.zeros(shape, dtype=torch.float32, device="cuda")
    ext = torch.tensor([s - 1 for s in shape], dtype=torch.float64, device="cuda")
    n = max(16, int(np.prod(shape)) // 20000)
    at = torch.rand(n, 3, generator=gen, device="cuda", dtype=torch.float64) * ext
    m = 12
    ends = torch.rand(2, m, 1, 3, generator=gen, device="cuda", dtype=torch.float64) * ext
    steps = torch.linspace(0, 1, 2 * max(shape), device="cuda", dtype=torch.float64)[None, :, None]
    lines = ends[0] + (ends[1] - ends[0]) * steps
    for pts, v in ((at, 1.0), (lines.reshape(-1, 3), 0.4)):
        z, y, x = pts.round().long().unbind(1)
        t[z, y, x] = v
    return t


def _blur64(x, psf):
    """Zero-boundary linear convolution with a corner-origin kernel, 64 bits."""
    f = [a + b + (a + b) % 2 for a, b in zip(x.shape, psf.shape)]
    return _apply64(x, _otf64(psf, f), f, False)


def _otf64(psf, f):
    big = torch.zeros(f, dtype=torch.float64, device="cuda")
    big[tuple(slice(0, s) for s in psf.shape)] = psf.double()
    for d, s in enumerate(psf.shape):
        # indices from ceil(s / 2) on are the negative offsets
        pos = (s + 1) // 2
        idx = torch.arange(f[d], device="cuda")
        src = torch.where(idx < pos, idx, torch.where(idx >= f[d] - (s - pos), idx - f[d] + s, f[d] - 1))
        big = big.index_select(d, src)
    return torch.fft.rfftn(big)


def _apply64(x, otf, f, adjoint):
    y = torch.fft.irfftn(torch.fft.rfftn(x.double(), s=f) * (otf.conj() if adjoint else otf), s=f)
    return y[tuple(slice(0, v) for v in x.shape)]


class _Conv64:
    def __init__(self, psf, n):
        self.psf = psf.double() / float(np.float32(psf.double().sum().item()))
        self.f = [a + b + (a + b) % 2 for a, b in zip(n, psf.shape)]
        self.otf = _otf64(self.psf, self.f)

    def forward(self, x):
        return _apply64(x, self.otf, self.f, False)

    def adjoint(self, y):
        return _apply64(y, self.otf, self.f, True)


def _area_weights(n_large, n_small):
    """Overlap of coarse pixel j with fine pixel i, in fine pixels."""
    r = n_large / n_small
    j = torch.arange(n_small, dtype=torch.float64, device="cuda")[:, None] * r
    i = torch.arange(n_large, dtype=torch.float64, device="cuda")[None, :]
    return (torch.minimum(j + r, i + 1) - torch.maximum(j, i)).clamp(min=0.0)


class _Area64:
    def __init__(self, large, small):
        self.w = [None if a == b else _area_weights(a, b) for a, b in zip(large, small)]

    def forward(self, x):
        for d, w in enumerate(self.w):
            if w is not None:
                x = torch.movedim(torch.tensordot(w, x, dims=([1], [d])), 0, d)
        return x

    def adjoint(self, y):
        for d, w in enumerate(self.w):
            if w is not None:
                y = torch.movedim(torch.tensordot(w, y, dims=([0], [d])), 0, d)
        return y


class _Crop64:
    def __init__(self, large, small, start):
        self.large = large
        self.at = tuple(slice(s, s + n) for s, n in zip(start, small))

    def forward(self, x):
        return x[self.at]

    def adjoint(self, y):
        out = torch.zeros(self.large, dtype=y.dtype, device=y.device)
        out[self.at] = y
        return out


class _Chain64:
    def __init__(self, *ops):
        self.ops = ops  # applied last to first

    def forward(self, x):
        for o in reversed(self.ops):
            x = o.forward(x)
        return x

    def adjoint(self, y):
        for o in self.ops:
            y = o.adjoint(y)
        return y


def _photons(blurred, peak, background, seed):
    b = blurred.clamp(min=0.0)
    b = b / b.max() * peak + background
    return torch.poisson(b, generator=_generator(seed + 2)).float()


def _stack(c, seed, shape=None, kshape=None, spacing=SPACING, peak=1000.0, background=10.0):
    """(observation on the grid of the PSF's samples, PSF)."""
    shape = shape or (c["nz"], c["ny"], c["nx"])
    psf = _psf(kshape or (c["kz"], c["ky"], c["kx"]), spacing, seed)
    return _photons(_blur64(_scene(shape, seed), psf), peak, background, seed), psf


def _tile_grids(c):
    """Visible and padded grids of a tile, and where the visible one starts."""
    data, zoom = (c["nz"], c["ny"], c["nx"]), (c["zoom_z"], c["zoom_xy"], c["zoom_xy"])
    k = (c["kz"], c["ky"], c["kx"])
    visible = tuple(max(1, round(d * z)) for d, z in zip(data, zoom))
    return data, visible, tuple(v + m - 1 for v, m in zip(visible, k)), tuple((m - 1) // 2 for m in k)


def _tile_data(c, seed):
    data, visible, padded, start = _tile_grids(c)
    psf = _psf((c["kz"], c["ky"], c["kx"]), SPACING, seed)
    fine = _blur64(_scene(padded, seed), psf)[tuple(slice(s, s + v) for s, v in zip(start, visible))]
    return _photons(_Area64(visible, data).forward(fine), 1000.0, 10.0, seed), psf


def _pdhg_data(c, seed):
    data = (c["nz"], c["ny"], c["nx"])
    fine = tuple(max(1, int(round(n * c["sampling"]))) for n in data)
    spacing = SPACING_FINE if c["sampling"] > 1 else SPACING
    psf = _psf(fine, spacing, seed)
    blurred = _Area64(fine, data).forward(_blur64(_scene(fine, seed), psf))
    return _photons(blurred, 500.0, 5.0, seed), psf, fine, spacing


def _batch_tiles(c):
    return plan_uneven_tiles((c["nz"], c["ny"], c["nx"]),
                             [(c["core_z"], 2 * c["core_z"]), (c["core_xy"], 2 * c["core_xy"]),
                              (c["core_xy"], 2 * c["core_xy"])], c["halo"], np.random.default_rng(5))


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = dict(case=case)
    if kind == "conv":
        shape, k = (c["nz"], c["ny"], c["nx"]), (c["kz"], c["ky"], c["kx"])
        obs, psf = _stack(c, seed)
        est = _scene(shape, seed) * 100.0 + 0.5
        if c["nz"] == 1 and c["kz"] == 1:
            shape, obs, est, psf = shape[1:], obs[0], est[0], psf[0]
        st.update(op=D.LinearFFTConvolver(psf, shape, precision=c["precision"]), x=est.contiguous(),
                  y=obs.contiguous())
    elif kind in ("rl", "nlcg", "pdhg_op"):
        obs, psf = _stack(c, seed)
        st.update(op=D.LinearFFTConvolver(psf, tuple(obs.shape)), y=obs)
    elif kind == "tile":
        y, psf = _tile_data(c, seed)
        st.update(y=y, model=D.make_forward_model(psf, tuple(y.shape), (c["zoom_z"], c["zoom_xy"], c["zoom_xy"])),
                  solve=D.richardson_lucy_solver(num_iter=c["iters"], background=10.0))
    elif kind == "pdhg":
        st["y"], st["psf"], _, st["spacing"] = _pdhg_data(c, seed)
    elif kind == "batch":
        st["y"], st["psf"] = _stack(c, seed)
        st["tiles"] = _batch_tiles(c)
        st["canvas"] = [D.static_fft_shape(t.shape, st["psf"].shape) for t in st["tiles"]]
    else:
        st["pupil"], st["kz"] = _pupil(c["ny"], c["nx"], SPACING_FINE, seed)
        st["z"] = _z_planes(c["nz"], SPACING_FINE[0])
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------


def _losses(values):
    return np.asarray(values, np.float32)


def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "conv":
        return {"blurred": st["op"].forward(st["x"]), "correlated": st["op"].adjoint(st["y"])}
    if kind == "rl":
        r = D.richardson_lucy_with_operator(st["y"], st["op"], num_iter=c["iters"], background=10.0)
        return {"restored": r.restored, "pred": r.pred, "loss": _losses(r.loss_history)}
    if kind == "tile":
        return {"restored": st["solve"](st["y"], st["model"])}
    if kind == "pdhg":
        r = D.solve_pdhg_mlx(st["y"], st["psf"], alpha=1e-3, norm=c["norm"], loss_type=c["loss"],
                             num_iter=c["iters"], background=5.0, spacing=st["spacing"], tol=0.0,
                             sampling_factors=c["sampling"] if c["sampling"] > 1 else None)
        return {"restored": r.restored, "loss": _losses(r.loss_history)}
    if kind == "pdhg_op":
        r = D.solve_pdhg_with_operator(st["y"], st["op"], alpha=1e-2, regularization=c["reg"],
                                       norm=c["norm"], loss_type=c["loss"], num_iter=c["iters"],
                                       background=10.0, tol=0.0)
        return {"restored": r.restored}
    if kind == "nlcg":
        r = D.nlcg_with_operator(st["y"], st["op"], num_iter=c["iters"], background=10.0, slack=0.0, tol=0.0)
        return {"restored": r.restored, "pred": r.pred, "loss": _losses(r.loss_history)}
    if kind == "batch":
        out, _, _ = batched_tiled_rl(st["y"], st["psf"], st["tiles"], c["iters"], background=10.0,
                                     fft_shapes=st["canvas"])
        return {"restored": out}
    return {"psf": pupil_to_psf(st["pupil"], st["kz"], st["z"])}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------


def _conv_work(n, k, otf_bytes=8):
    """(bytes, flops) of one convolution: signal in and out, the half OTF of
    the smallest wrap-free canvas once, two real transforms and the product."""
    f = [a + b - 1 for a, b in zip(n, k)]
    half = math.prod(f) / 2
    return (8.0 * math.prod(n) + otf_bytes * half,
            2 * 2.5 * math.prod(f) * math.log2(max(2, math.prod(f))) + 6 * half)


def work(case):
    c, kind = case, case["kind"]
    n = (c["nz"], c["ny"], c["nx"])
    vox = math.prod(n)
    k = (c.get("kz", 1), c.get("ky", 1), c.get("kx", 1))
    if kind == "conv":
        b, f = _conv_work(n, k, 4 if c["precision"] == "mixed" else 8)
        return {"bytes": 2 * b, "flops": 2 * f}
    if kind == "rl":  # set-up 2, an iteration 2 and the prediction 1; y, x and the sensitivity read besides
        b, f = _conv_work(n, k)
        return {"bytes": (2 * c["iters"] + 3) * b + c["iters"] * 12.0 * vox, "flops": (2 * c["iters"] + 3) * f}
    if kind == "tile":  # the loss of the first and last iteration costs a convolution each
        data, _, padded, _ = _tile_grids(c)
        b, f = _conv_work(padded, k)
        times = 2 * c["iters"] + 4
        return {"bytes": times * b + c["iters"] * (12.0 * vox + 12.0 * math.prod(padded)), "flops": times * f}
    if kind == "pdhg":  # x, x_prev, dual and its update, A x and data per iteration
        fine = tuple(max(1, int(round(v * c["sampling"]))) for v in n)
        b, f = _conv_work(fine, fine)
        nf, it = math.prod(fine), c["iters"]
        return {"bytes": (2 * it + 2) * b + it * (64.0 * nf + 16.0 * vox), "flops": (2 * it + 3) * f + 60.0 * nf * it}
    if kind == "pdhg_op":
        b, f = _conv_work(n, k)
        comp, it = {"identity": 1, "gradient": 3, "hessian": 6}[c["reg"]], c["iters"]
        return {"bytes": (2 * it + 1) * b + it * (8.0 * comp + 32.0) * vox, "flops": (2 * it + 1) * f}
    if kind == "nlcg":
        b, f = _conv_work(n, k)
        return {"bytes": (3 * c["iters"] + 4) * b + c["iters"] * 80.0 * vox, "flops": (3 * c["iters"] + 4) * f}
    if kind == "batch":
        tot = [0.0, 0.0]
        for t in _batch_tiles(c):
            b, f = _conv_work(t.shape, k)
            tot[0] += (2 * c["iters"] + 2) * b + c["iters"] * 12.0 * math.prod(t.shape)
            tot[1] += (2 * c["iters"] + 2) * f
        return {"bytes": tot[0], "flops": tot[1]}
    plane = c["ny"] * c["nx"]
    return {"bytes": 4.0 * vox + 24.0 * plane, "flops": 5.0 * vox * math.log2(plane) + 12.0 * vox}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------


def _divergence64(y, m):
    ys, ms = y.clamp(min=1e-6), m.clamp(min=1e-6)
    return float((y * torch.log(ys / ms) - (y - ms)).mean())


def _rl64(y, op, iters, background, every=10):
    x = op.adjoint((y - background).clamp(min=1e-6)).clamp(min=1e-6)
    sens = op.adjoint(torch.ones_like(y))
    active = sens > (sens.max() * 1e-6).clamp(min=1e-10)
    x = torch.where(active, x, 0.0)
    losses = []
    for k in range(iters):
        ratio = y / (op.forward(x) + background).clamp(min=1e-10)
        x = (x * torch.where(active, op.adjoint(ratio) / sens, 0.0)).clamp(min=1e-10)
        if k % every == 0 or k == iters - 1:
            losses.append(_divergence64(y, op.forward(x) + background))
    return x, op.forward(x) + background, losses


def _shift(x, d, by, edge):
    """x[i + by] along axis d, with the end value repeated (edge) or zero."""
    n = x.shape[d]
    i = torch.arange(n, device=x.device) + by
    out = x.index_select(d, i.clamp(0, n - 1))
    if not edge:
        keep = ((i >= 0) & (i < n)).double().reshape([-1 if a == d else 1 for a in range(x.dim())])
        out = out * keep
    return out


def _second(x, d):
    return _shift(x, d, -1, True) - 2 * x + _shift(x, d, 1, True)


def _central(x, d):
    return (_shift(x, d, 1, True) - _shift(x, d, -1, True)) / 2


def _central_t(x, d):
    n = x.shape[d]
    i = torch.arange(n, device=x.device).reshape([-1 if a == d else 1 for a in range(x.dim())])
    lo, hi = _shift(x, d, -1, False), _shift(x, d, 1, False)
    return (torch.where(i == 0, -x, lo) - torch.where(i == n - 1, -x, hi)) / 2


def _ahead(x, d):
    return _shift(x, d, 1, True) - x


def _ahead_t(x, d):
    n = x.shape[d]
    i = torch.arange(n, device=x.device).reshape([-1 if a == d else 1 for a in range(x.dim())])
    return torch.where(i == n - 1, 0.0, -x) + _shift(x, d, -1, False)


class _Reg64:
    def __init__(self, kind, r):
        s = math.sqrt(2.0)
        pairs = [(0, 1), (0, 2), (1, 2)]
        if kind == "identity":
            self.norm_sq, self.parts = 1.0, [(1.0, lambda x: x, lambda x: x)]
        elif kind == "gradient":
            self.norm_sq = 4.0 * (r * r + 2.0)
            self.parts = [(r if d == 0 else 1.0, lambda x, d=d: _ahead(x, d), lambda x, d=d: _ahead_t(x, d))
                          for d in range(3)]
        else:
            self.norm_sq = 16.0 * r ** 4 + 4.0 * r ** 2 + 34.0
            self.parts = [(r * r if d == 0 else 1.0, lambda x, d=d: _second(x, d), lambda x, d=d: _second(x, d))
                          for d in range(3)]
            self.parts += [(s * (r if a == 0 else 1.0), lambda x, a=a, b=b: _central(_central(x, a), b),
                            lambda x, a=a, b=b: _central_t(_central_t(x, b), a)) for a, b in pairs]

    def forward(self, x):
        return torch.stack([w * f(x) for w, f, _ in self.parts])

    def adjoint(self, y):
        return sum(w * t(y[i]) for i, (w, _, t) in enumerate(self.parts))


def _pdhg64(y, op, op_norm_sq, reg, x, c, alpha, background, want_loss):
    delta, eta = 0.99, 0.5
    step = 0.99 / math.sqrt(op_norm_sq + reg.norm_sq)
    tau = sigma = step
    theta = 1.0
    bar = x
    y1, y2 = torch.zeros_like(y), torch.zeros_like(reg.forward(x))
    ax, lx, losses = op.forward(x), reg.forward(x), []
    ax_bar, lx_bar = ax, lx
    d = y.clamp(min=0.0)
    for k in range(c["iters"]):
        v = y1 + sigma * ax_bar
        if c["loss"] == "poisson":
            cc = 1.0 - v - sigma * background
            z = 2.0 * sigma * d / (torch.sqrt(cc * cc + 4.0 * sigma * d) - cc + 1e-12)
            y1 = 1.0 - torch.where(d < 1e-6, cc.clamp(min=1e-6), z).clamp(min=1e-6)
        else:
            y1 = (v - sigma * (y - background)) / (1.0 + sigma)
        v = y2 + sigma * lx_bar
        if c["norm"] == "L1":
            y2 = v.clamp(-alpha, alpha)
        else:
            y2 = v / (torch.sqrt((v * v).sum(0, keepdim=True) + 1e-12) / alpha).clamp(min=1.0)
        new = (x - tau * (op.adjoint(y1) + reg.adjoint(y2))).clamp(min=0.0)
        ax_new, lx_new = op.forward(new), reg.forward(new)
        dx2 = float(((new - x) ** 2).sum())
        dk2 = float(((ax_new - ax) ** 2).sum() + ((lx_new - lx) ** 2).sum())
        cand = min(math.sqrt(1.0 + theta) * tau, delta * math.sqrt(dx2 / (2.0 * sigma * max(dk2, 1e-12))))
        tau_new = max(eta * cand if cand * sigma * dk2 > delta * dx2 else cand, step * 1e-4)
        theta = tau_new / tau
        sigma = min(max(sigma / max(theta, 0.1), step * 1e-4), step * 1e4)
        tau = tau_new
        ax_bar, lx_bar = ax_new + theta * (ax_new - ax), lx_new + theta * (lx_new - lx)
        x, ax, lx = new, ax_new, lx_new
        if want_loss and (k + 1) % 10 == 0:
            m = ax + background
            if c["loss"] == "poisson":
                fit = (y * torch.log((y + 1e-6) / m.clamp(min=1e-6)) - (y - m)).sum()
            else:
                fit = 0.5 * ((y - m) ** 2).sum()
            if c["norm"] == "L1":
                pen = lx.abs().sum()
            else:
                pen = torch.sqrt((lx * lx).sum(0) + 1e-12).sum()
            losses.append(float(fit + alpha * pen))
    return x, losses


def _norm_sq64(psf, n):
    """max |OTF|^2: the operator's norm bound; at zero frequency for a PSF."""
    p = psf.double()
    return (float(p.sum()) / float(np.float32(p.sum().item()))) ** 2


def _nlcg64(y, op, iters, background, every=10):
    s = torch.sqrt(op.adjoint((y - background).clamp(min=1e-6)).clamp(min=1e-6))
    eps = 1e-10

    def phi_of(m):
        return float((m - y * torch.log(m.clamp(min=eps))).sum())

    def minus_grad(s, m):
        return -2.0 * s * op.adjoint(1.0 - y / m.clamp(min=eps))

    m = op.forward(s * s) + background
    r = minus_grad(s, m)
    d, rr, losses = r, float((r * r).sum()), []
    for k in range(iters):
        for steepest in (False, True):
            d = r if steepest else d
            ksd, kdd, lam = op.forward(s * d), op.forward(d * d), 0.0
            for _ in range(3):
                ml = (m + 2.0 * lam * ksd + lam * lam * kdd).clamp(min=eps)
                kl, w = ksd + lam * kdd, 1.0 - y / ml
                d1 = 2.0 * float((kl * w).sum())
                d2 = 2.0 * float((kdd * w).sum()) + 4.0 * float((y * kl * kl / (ml * ml)).sum())
                lam -= d1 / d2
            m_new = m + 2.0 * lam * ksd + lam * lam * kdd
            if phi_of(m_new) < phi_of(m):
                break
        else:
            return None  # no step of this start lowers the objective
        s, m = s + lam * d, m_new
        r = minus_grad(s, m)
        rr_new = float((r * r).sum())
        d, rr = r + (rr_new / rr) * d, rr_new
        if k % every == 0 or k == iters - 1:
            losses.append(_divergence64(y, m))
    return s * s, op.forward(s * s) + background, losses


def exact(case, seed):
    c, kind = case, case["kind"]
    n = (c["nz"], c["ny"], c["nx"])
    if kind == "conv":
        obs, psf = _stack(c, seed)
        op = _Conv64(psf, n)
        out = {"blurred": op.forward(_scene(n, seed) * 100.0 + 0.5), "correlated": op.adjoint(obs)}
        return {k: v[0] if n[0] == 1 and c["kz"] == 1 else v for k, v in out.items()}
    if kind in ("rl", "nlcg"):
        obs, psf = _stack(c, seed)
        got = (_rl64 if kind == "rl" else _nlcg64)(obs.double(), _Conv64(psf, n), c["iters"], 10.0)
        return None if got is None else {"restored": got[0], "pred": got[1], "loss": np.asarray(got[2])}
    if kind == "tile":
        data, visible, padded, start = _tile_grids(c)
        y, psf = _tile_data(c, seed)
        crop = _Crop64(padded, visible, start)
        x, _, _ = _rl64(y.double(), _Chain64(_Area64(visible, data), crop, _Conv64(psf, padded)), c["iters"], 10.0)
        return {"restored": crop.forward(x)}
    if kind == "pdhg":
        y, psf, fine, spacing = _pdhg_data(c, seed)
        y = y.double()
        area = _Area64(fine, n)
        op = _Chain64(area, _Conv64(psf, fine))
        norm_sq = _norm_sq64(psf, fine) * (c["sampling"] ** 3 if c["sampling"] > 1 else 1.0)
        x0 = (op.adjoint(y) if c["sampling"] > 1 else y).clamp(min=0.0)
        reg = _Reg64("hessian", (spacing[1] + spacing[2]) / 2.0 / spacing[0])
        x, losses = _pdhg64(y, op, norm_sq, reg, x0, c, 1e-3, 5.0, True)
        return {"restored": x, "loss": np.asarray(losses)}
    if kind == "pdhg_op":
        obs, psf = _stack(c, seed)
        x0 = torch.full(n, 0.01, dtype=torch.float64, device="cuda")
        x, _ = _pdhg64(obs.double(), _Conv64(psf, n), _norm_sq64(psf, n), _Reg64(c["reg"], 1.0), x0, c, 1e-2,
                       10.0, False)
        return {"restored": x}
    if kind == "batch":
        obs, psf = _stack(c, seed)
        out = torch.empty(n, dtype=torch.float64, device="cuda")
        for t in _batch_tiles(c):
            x, _, _ = _rl64(obs[t.read].double(), _Conv64(psf, t.shape), c["iters"], 10.0)
            out[t.write] = x[t.crop]
        return {"restored": out}
    pupil, kz = _pupil(c["ny"], c["nx"], SPACING_FINE, seed)
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    for i, z in enumerate(_z_planes(c["nz"], SPACING_FINE[0])):
        a = torch.fft.ifft2(pupil * torch.exp(2j * math.pi * kz * z))
        out[i] = a.real ** 2 + a.imag ** 2
    return {"psf": out / out.sum()}
