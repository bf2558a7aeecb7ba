"""Cases that the performance of the CG-SENSE library is measured on.

Each case is one call (or one training step) of the package's public entry
points, at sizes of the benchmark configurations (``synth.WORKLOADS``), of the
tests, or generic ones between and around them.  All inputs are made from the
seed: coil maps, k-space samples of a cloud of Gaussian blobs seen through the
coils plus noise, a wave-CAIPI scan whose wave is slightly off its nominal
parameters, density weights and breathing bins.

``exact`` restates every path in 64 bits with plain torch: the Kaiser-Bessel
taps with the reference's float distances (Reco.h:218-242, Reco.cpp:698-806),
gridding, full transforms, the CG loop (Reco.cpp:175-321), and torch's own
autograd for the gradients.
"""
import importlib
import math

import numpy as np
import torch

cgs = importlib.import_module("4d_lung_gb300")
synth = importlib.import_module("4d_lung_gb300.synth")
ag = importlib.import_module("4d_lung_gb300.autograd")

ADJ_SCALE = 1e-3          # the library's default rescale of the adjoint (Reco.cpp:482)

# A case: op, image and grid, coils (ch), undersampling (ry, rz), samples per
# readout (nread), wave excursion and cycles, bins (breathing bins; 0: one bin
# of a share `gate` of the readouts), iterations, kernel width.


def _case(name, op, img, grid, ch, bins=0, iters=0, gate=1.0, ry=2, rz=2, wave=4.0, cyc=7, width=4.0, nread=0):
    c = {"op": op, "ix": img[0], "iy": img[1], "iz": img[2], "gx": grid[0], "gy": grid[1], "gz": grid[2], "ch": ch,
         "bins": bins, "iters": iters, "gate": gate, "ry": ry, "rz": rz, "wave": wave, "cyc": cyc, "width": width,
         "nread": nread or 4 * img[0]}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest reconstruction a user runs (the package's smoke size), host
        # arrays in and out through the drop-in call: latency and launches
        _case("solve_host_small", "solve_host", (16, 16, 12), (32, 32, 24), 4, iters=8, wave=2.0, nread=32),
        # the two NUFFT directions at the 64^3, 8-coil configuration, one gate
        _case("nufft_forward", "forward", (64, 64, 64), (128, 128, 128), 8),
        _case("nufft_adjoint", "adjoint", (64, 64, 64), (128, 128, 128), 8),
        # one application of the normal operator to one gate of the
        # 128 x 128 x 96, 12-coil scan: a user's own iteration
        _case("apply_one_gate", "apply", (128, 128, 96), (256, 256, 192), 12, gate=0.07, wave=5.0, cyc=8),
        # odd image sizes, an odd coil count, less than two-fold oversampling
        _case("apply_ragged", "apply", (75, 91, 49), (128, 176, 96), 5, bins=2, wave=3.0, nread=301),
        # the precision form (compensated spreading), 160 x 160 x 112, 16 coils
        _case("apply_compensated", "apply_compensated", (160, 160, 112), (320, 320, 224), 16, gate=0.25, ry=3, rz=2,
              wave=6.0, cyc=9),
        # the whole 4-D reconstruction: 16 breathing bins, 15 iterations
        _case("solve_4d", "solve", (128, 128, 96), (256, 256, 192), 12, bins=16, iters=15, wave=5.0, cyc=8),
        # four gates with the Toeplitz-embedded operator
        _case("solve_4d_toeplitz", "solve_toeplitz", (128, 128, 96), (256, 256, 192), 12, bins=4, iters=10, wave=5.0,
              cyc=8),
        # the data-consistency loss with its gradients in image and coordinates
        _case("loss_gradients", "loss", (128, 128, 96), (256, 256, 192), 12, wave=5.0, cyc=8),
        # one step of trajectory self-calibration: new coordinates each step
        _case("calibration_step", "calibrate", (64, 64, 64), (128, 128, 128), 8),
        # unrolled CG over four bins, differentiated with respect to the wave
        _case("unrolled_cg", "unrolled", (64, 64, 64), (128, 128, 128), 8, bins=4, iters=3),
        # iterative density weights of every bin of a scan
        _case("density_weights", "density", (128, 128, 96), (256, 256, 192), 12, bins=16, iters=10, wave=5.0,
              cyc=8),
    ]


_GRIDS = (32, 40, 48, 64, 80, 96, 128, 160, 192, 224, 256, 320)


def draw(rng):
    op = rng.choice(("solve_host", "forward", "adjoint", "apply", "apply_compensated", "solve", "solve_toeplitz",
                     "loss", "calibrate", "unrolled", "density"))
    while True:
        side = math.exp(rng.uniform(math.log(32), math.log(300)))
        grid = tuple(min(_GRIDS, key=lambda g: abs(math.log(g / (side * rng.uniform(0.7, 1.3))))) for _ in range(3))
        if rng.random() < 0.5 or op == "solve_toeplitz":
            img = tuple(g // 2 for g in grid)
        else:
            img = tuple(max(8, int(g * rng.uniform(0.4, 0.75))) for g in grid)
        ch = rng.randint(1, 16)
        bins = rng.choice((0, 0, 2, 3, 5, 8))
        if op in ("solve_host", "forward", "adjoint", "loss", "calibrate"):
            bins = 0
        iters = {"density": rng.randint(4, 12), "unrolled": rng.randint(2, 4)}.get(op, rng.randint(3, 12))
        if op in ("forward", "adjoint", "apply", "apply_compensated", "loss", "calibrate"):
            iters = 0
        c = _case("", op, img, grid, ch, bins=bins, iters=iters, gate=round(math.exp(rng.uniform(math.log(0.05), 0.0)), 3),
                  ry=rng.choice((1, 2, 3)), rz=rng.choice((1, 2)), wave=round(rng.uniform(1.0, 6.0), 2),
                  cyc=rng.randint(4, 10), width=rng.choice((4.0, 4.25)), nread=rng.randint(2 * img[0], 4 * img[0]))
        w = work(c)
        cells = grid[0] * grid[1] * grid[2] * ch * max(1, bins)
        limit = 4e8 if op != "unrolled" else 5e7
        if op == "solve_toeplitz" and max(grid) > 256:
            continue
        if 3e6 < w["flops"] < 2e12 and cells < limit and _samples(c) * ch < (4e7 if op != "unrolled" else 4e6):
            return c


# -- geometry ------------------------------------------------------------------

class _Workload(synth.Workload):
    """Any number of samples per readout (Workload's is a multiple of the image size)."""

    @property
    def n_read(self):
        return self.extra["n_read"]


def _workload(c):
    return _Workload("case", (c["ix"], c["iy"], c["iz"]), (c["gx"], c["gy"], c["gz"]), c["ch"], (c["ry"], c["rz"]), 1,
                     1, c["wave"], c["cyc"], max(1, c["bins"]), c["iters"], extra={"n_read": c["nread"]})


class _Scan:
    """What a case's scan consists of: trajectory, bins, density weights."""

    def __init__(self, c, seed):
        self.w = _workload(c)
        rng = np.random.default_rng(seed)
        lines = synth.readout_lines(self.w)
        if c["gate"] < 1.0 and not c["bins"]:
            keep = max(4, int(round(c["gate"] * len(lines))))
            lines = lines[np.sort(rng.permutation(len(lines))[:keep])]
        self.lines = lines
        self.wave = synth.perturbed_wave(self.w, 0.05, seed)
        self.k = synth.wave_trajectory(self.w, self.wave, lines)
        self.bins = None
        if c["bins"]:
            rb = synth.breathing_bins(len(lines), c["bins"], seed=seed % 1000)
            self.bins = synth.bin_samples(rb, self.w.n_read)
        self.dcf = synth.radial_dcf(self.k, self.w.grid)


def _samples(c):
    n = len(synth.readout_lines(_workload(c)))
    if c["gate"] < 1.0 and not c["bins"]:
        n = max(4, int(round(c["gate"] * n)))
    return n * c["nread"]


def _beta(c):
    """Beatty's shape parameter for the case's width and two-fold oversampling."""
    return float(math.pi * math.sqrt(c["width"] ** 2 / 4.0 * 1.5 ** 2 - 0.8))


def _axes(c, dev):
    return [torch.linspace(-1 + 1.0 / n, 1 - 1.0 / n, n, device=dev, dtype=torch.float64)
            for n in (c["ix"], c["iy"], c["iz"])]


def _maps(c, dev, gen):
    """Gaussian coil profiles on a ring with smooth phases, sum of squares 1."""
    X, Y, Z = torch.meshgrid(*[a.float() for a in _axes(c, dev)], indexing="ij")
    n = c["ch"]
    ph = torch.rand(n, generator=gen, device=dev) * 2 * math.pi
    maps = torch.empty((n,) + X.shape, dtype=torch.complex64, device=dev)
    for i in range(n):
        a = 2 * math.pi * i / n
        cx, cy, cz = 1.3 * math.cos(a), 1.3 * math.sin(a), (0.5 * ((i % 2) * 2 - 1) if n > 4 else 0.0)
        g = torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2 + (Z - cz) ** 2) / 1.28)
        maps[i] = torch.polar(g, ph[i] + 0.5 * (X * math.cos(a) + Y * math.sin(a)))
    maps /= maps.abs().square().sum(0).sqrt()
    return maps


_BLOBS = 24


def _blobs(c, dev, gen):
    """Positions (unit box), widths (voxels) and complex weights of the object."""
    pos = torch.rand((_BLOBS, 3), generator=gen, device=dev, dtype=torch.float64) * 1.2 - 0.6
    wid = 0.6 + 2.4 * torch.rand(_BLOBS, generator=gen, device=dev, dtype=torch.float64)
    amp = torch.polar(0.2 + torch.rand(_BLOBS, generator=gen, device=dev, dtype=torch.float64),
                      2 * math.pi * torch.rand(_BLOBS, generator=gen, device=dev, dtype=torch.float64))
    return pos, wid, amp


def _image(c, dev, gen):
    pos, wid, amp = _blobs(c, dev, gen)
    ax = _axes(c, dev)
    n = (c["ix"], c["iy"], c["iz"])
    f = [torch.exp(-(((ax[a][None, :] - pos[:, a:a + 1]) * n[a] / 2) ** 2) / (2 * wid[:, None] ** 2)) for a in range(3)]
    return torch.einsum("b,bx,by,bz->xyz", amp, *[t.to(torch.complex128) for t in f]).to(torch.complex64).contiguous()


def _data(c, k, dev, gen):
    """Samples [coil][sample] of the blobs seen through the coils at their
    centres, plus complex noise at SNR 30."""
    pos, wid, amp = _blobs(c, dev, gen)
    G = torch.tensor([c["gx"], c["gy"], c["gz"]], dtype=torch.float64, device=dev)
    n = torch.tensor([c["ix"], c["iy"], c["iz"]], dtype=torch.float64, device=dev)
    nu = (k * (G - 1) - G / 2) / G                       # cycles per voxel
    ang = 2 * math.pi * torch.arange(c["ch"], device=dev, dtype=torch.float64) / c["ch"]
    ctr = torch.stack([1.3 * torch.cos(ang), 1.3 * torch.sin(ang), torch.zeros_like(ang)], -1)
    sens = torch.polar(torch.exp(-((pos[None] - ctr[:, None]) ** 2).sum(-1) / 1.28), ang[:, None] + pos[None, :, 0])
    a = (sens * amp[None] * (2 * math.pi) ** 1.5 * wid[None] ** 3).to(torch.complex64)
    out = torch.empty((c["ch"], k.shape[0]), dtype=torch.complex64, device=dev)
    for s in range(0, k.shape[0], 1 << 19):
        q = nu[s:s + (1 << 19)]
        phase = -2 * math.pi * (q @ (pos * n / 2).T)
        mag = torch.exp(-2 * math.pi ** 2 * (q * q).sum(-1, keepdim=True) * wid[None] ** 2)
        out[:, s:s + (1 << 19)] = a @ torch.polar(mag, phase).to(torch.complex64).T
    rms = out.abs().square().mean().sqrt()
    noise = torch.randn(out.shape, generator=gen, device=dev, dtype=torch.complex64)
    return out + noise * (rms / 30.0)


def _inputs(c, seed):
    """Everything a case is made from, and nothing of the library's."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    s = _Scan(c, seed)
    d = {"scan": s, "dev": dev}
    op = c["op"]
    nb = max(1, c["bins"])
    img = (c["ix"], c["iy"], c["iz"])
    if op != "density":
        d["maps"] = _maps(c, dev, gen)
    if op in ("apply", "apply_compensated"):
        d["x"] = torch.stack([_image(c, dev, gen) for _ in range(nb)])
    elif op == "forward":
        d["x"] = d["maps"] * _image(c, dev, gen)[None]
    elif op in ("loss", "calibrate"):
        d["x"] = _image(c, dev, gen)
    if op in ("adjoint", "loss", "calibrate", "unrolled", "solve", "solve_host", "solve_toeplitz"):
        d["y"] = _data(c, torch.from_numpy(s.k).to(dev), dev, gen)
    if op == "unrolled":
        d["v"] = torch.stack([_image(c, dev, gen) for _ in range(nb)]).reshape(nb, -1)
    if op in ("calibrate", "unrolled"):
        d["theta"] = torch.tensor(s.wave.vector(), dtype=torch.float64, device=dev)
    return d


# -- the framework's calls -------------------------------------------------------

_STREAM = None


def _stream():
    """One stream for every context, as a program with one torch stream has."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def prepare(case, seed):
    c = dict(case)
    d = _inputs(c, seed)
    s = d["scan"]
    op = c["op"]
    img = (c["ix"], c["iy"], c["iz"])
    nb = max(1, c["bins"])
    r = cgs.Reco(img, (c["gx"], c["gy"], c["gz"]), c["ch"], kb_w=c["width"], kb_b=_beta(c))
    r.set_stream(_stream().cuda_stream)
    r.set_trajectory(s.k)
    if s.bins is not None:
        r.set_bins(s.bins)
    r.set_dcf(s.dcf)
    torch.cuda.synchronize()
    if op != "density":
        r.set_smaps_tensor(d["maps"])
    if op == "apply_compensated":
        r.set_precision(True)
    if op == "solve_toeplitz":
        r.set_toeplitz(1)
    st = {"op": op, "reco": r, "iters": c["iters"]}
    dev = d["dev"]
    if op == "solve_host":
        st["y"] = d["y"].cpu().numpy()
    elif op == "forward":
        st["x"], st["out"] = d["x"], torch.empty((c["ch"], r.ns), dtype=torch.complex64, device=dev)
    elif op == "adjoint":
        st["y"], st["out"] = d["y"], torch.empty((c["ch"],) + img, dtype=torch.complex64, device=dev)
    elif op in ("apply", "apply_compensated"):
        st["x"], st["out"] = d["x"], torch.empty_like(d["x"])
    elif op in ("solve", "solve_toeplitz"):
        st["y"], st["out"] = d["y"], torch.empty((nb,) + img, dtype=torch.complex64, device=dev)
    elif op == "loss":
        st["y"] = d["y"]
        st["x"] = d["x"].clone().requires_grad_(True)
        st["k"] = torch.from_numpy(s.k).to(dev).requires_grad_(True)
    elif op == "calibrate":
        st["y"], st["x"] = d["y"], d["x"]
        st["theta"] = d["theta"].clone().requires_grad_(True)
        st["w"], st["lines"] = s.w, s.lines
    elif op == "unrolled":
        st["y"], st["v"] = d["y"], d["v"]
        st["theta"] = d["theta"].clone().requires_grad_(True)
        st["w"], st["lines"] = s.w, s.lines
    torch.cuda.synchronize()
    return st


def run(state):
    op, r = state["op"], state["reco"]
    if op == "solve_host":
        x, res, it = r.cg_sense(state["y"], 0.0, state["iters"])
        return {"x": x, "residuals": res, "iterations": it}
    if op == "forward":
        r.nufft_fwd_tensor(state["x"], state["out"])
        return state["out"]
    if op == "adjoint":
        r.nufft_adj_tensor(state["y"], state["out"])
        return state["out"]
    if op in ("apply", "apply_compensated"):
        r.apply_ehde_tensor(state["x"], state["out"], 0, state["x"].shape[0])
        return state["out"]
    if op in ("solve", "solve_toeplitz"):
        res, it = r.cg_sense_batched_tensor(state["y"], state["out"], 0.0, state["iters"])
        return {"x": state["out"], "residuals": res, "iterations": it}
    if op == "density":
        return r.pipe_menon_dcf(state["iters"])
    with torch.cuda.stream(_stream()):
        if op == "loss":
            state["x"].grad = state["k"].grad = None
            loss = ag.dc_loss(r, state["x"], state["k"], state["y"])
            loss.backward()
            return {"loss": loss.detach(), "grad_x": state["x"].grad, "grad_k": state["k"].grad}
        state["theta"].grad = None
        k = ag.wave_trajectory_torch(state["w"], state["theta"], state["lines"])
        k.retain_grad()
        if op == "calibrate":
            loss = ag.dc_loss(r, state["x"], k, state["y"])
            loss.backward()
            return {"loss": loss.detach(), "grad_k": k.grad, "grad_theta": state["theta"].grad}
        x = ag.cg_unrolled(r, k, state["y"], state["iters"])
        x.backward(state["v"])
        return {"x": x.detach(), "grad_k": k.grad, "grad_theta": state["theta"].grad}


def work(case):
    c = dict(case)
    op, ch, nb, it = c["op"], c["ch"], max(1, c["bins"]), c["iters"]
    ni, m = c["ix"] * c["iy"] * c["iz"], _samples(c)
    gx, gy, gz = c["gx"], c["gy"], c["gz"]
    # the pruned transform's three passes, and the taps of one direction
    fft = 5.0 * (c["ix"] * c["iy"] * gz * math.log2(gz) + c["ix"] * gz * gy * math.log2(gy) + gy * gz * gx * math.log2(gx))
    taps = 4.0 * 4 ** 3 * m                      # all bins' samples, one coil
    image, maps, coords, samples = 8.0 * ni, 8.0 * ni * ch, 28.0 * m, 8.0 * m * ch
    half = ch * (nb * fft + taps)                # one direction, all bins
    if op == "density":
        return {"bytes": 24.0 * m + 4.0 * m, "flops": it * 2 * taps}
    if op in ("forward", "adjoint"):
        return {"bytes": maps + coords + samples, "flops": half}
    if op in ("apply", "apply_compensated"):
        return {"bytes": 2 * nb * image + maps + coords, "flops": 2 * half}
    if op in ("solve", "solve_host"):
        return {"bytes": samples + nb * image + maps + coords, "flops": (2 * it + 1) * half}
    if op == "solve_toeplitz":
        return {"bytes": samples + nb * image + maps + coords, "flops": (2 * it * nb * fft * ch) + half}
    if op == "loss":
        return {"bytes": 2 * image + maps + coords + samples + 24.0 * m, "flops": 2 * half + 3 * ch * taps}
    if op == "calibrate":
        return {"bytes": image + maps + coords + samples + 24.0 * m, "flops": half + 3 * ch * taps}
    return {"bytes": samples + 2 * nb * image + maps + coords + 24.0 * m,
            "flops": (2 * it + 1) * half + (6 * it + 2) * half + 3 * (2 * it + 1) * ch * taps}


# -- the same in 64 bits ---------------------------------------------------------

def _taps(c, k, dev):
    """Per sample: 125 flat grid indices and weights (0 where there is no tap)."""
    G = (c["gx"], c["gy"], c["gz"])
    w, b = np.float32(c["width"]), float(np.float32(_beta(c)))
    ws, gs = [], []
    peak = 1.0
    for a in range(3):
        N = G[a]
        dk = np.float32(1.0 / float(np.float32(N - 1)))
        scale = float(np.float32(np.float32(np.float32(100.0) * w) * dk))
        ka = k[:, a:a + 1]
        near = (ka.detach() * (N - 1) + 0.5).to(torch.int64).clamp(0, N - 1)
        g = near + torch.arange(-2, 3, device=dev)[None]
        inside = (g >= 0) & (g <= N - 1)
        gpos = (g.to(torch.float32) * float(dk)).to(torch.float64)
        # float distance; its derivative is that of |k - g dk|
        d64 = (ka - gpos).abs()
        d = d64 + (d64.detach().to(torch.float32).to(torch.float64) - d64.detach())
        half = float(np.float32(np.float32(float(w) / 2.0) * dk))
        inside &= ~(d.detach() > half)
        wdk = float(np.float32(w * dk))
        q = 2.0 * d / wdk
        q = q + ((q.detach().to(torch.float32)).to(torch.float64) - q.detach())
        s2 = torch.where(inside, 1.0 - q * q, torch.ones_like(q)).clamp_min(1e-30)
        val = torch.special.i0(b * torch.sqrt(s2)) / scale
        ws.append(torch.where(inside, val, torch.zeros_like(val)))
        gs.append(g.clamp(0, N - 1))
        peak *= float(torch.special.i0(torch.tensor(b, dtype=torch.float64))) / scale
    wt = (ws[0][:, :, None, None] * ws[1][:, None, :, None] * ws[2][:, None, None, :]).reshape(k.shape[0], 125)
    idx = ((gs[0][:, :, None, None] * G[1] + gs[1][:, None, :, None]) * G[2] + gs[2][:, None, None, :]).reshape(-1, 125)
    wt = torch.where(wt.detach() > peak * 1e-7, wt, torch.zeros_like(wt))
    return idx, wt


def _apod(c, dev):
    """1 / transform of the sampled kernel, per image axis (Reco.cpp:560-601)."""
    out = []
    for a, (I, N) in enumerate(((c["ix"], c["gx"]), (c["iy"], c["gy"]), (c["iz"], c["gz"]))):
        n = torch.arange(N, dtype=torch.float64, device=dev) - N // 2
        dist = n.abs() / (N - 1)
        dk = 1.0 / (N - 1)
        q = 2 * dist / (c["width"] * dk)
        f = torch.where(q <= 1.0, torch.special.i0(_beta(c) * torch.sqrt((1 - q * q).clamp_min(0.0)))
                        / (100.0 * c["width"] * dk), torch.zeros_like(q))
        g = torch.arange(I, dtype=torch.float64, device=dev) + (N - I) // 2 - N // 2
        out.append(1.0 / (f[None] * torch.cos(2 * math.pi * g[:, None] * n[None] / N)).sum(1))
    return out[0][:, None, None] * out[1][None, :, None] * out[2][None, None, :]


class _Exact:
    def __init__(self, c, dev):
        self.c, self.dev = c, dev
        self.G, self.I = (c["gx"], c["gy"], c["gz"]), (c["ix"], c["iy"], c["iz"])
        self.lo = [(g - i) // 2 for g, i in zip(self.G, self.I)]
        self.apod = _apod(c, dev)
        self.scale = ADJ_SCALE / math.sqrt(self.G[0] * self.G[1] * self.G[2])
        self.sign = [1.0 - 2.0 * (torch.arange(g, device=dev) % 2).to(torch.float64) for g in self.G]

    def _pass(self, x, axis, fwd):
        sh = [1, 1, 1]
        sh[axis] = -1
        x = x * self.sign[axis].reshape(sh)
        x = torch.fft.fft(x, dim=axis) if fwd else torch.fft.ifft(x, dim=axis, norm="forward")
        return x * self.sign[axis].reshape(sh)

    def to_grid(self, x):
        """Deapodised image -> its centred transform on the grid."""
        x = x * self.apod
        for a in (2, 1, 0):
            pad = [0] * 6
            pad[2 * (2 - a)], pad[2 * (2 - a) + 1] = self.lo[a], self.G[a] - self.I[a] - self.lo[a]
            x = self._pass(torch.nn.functional.pad(x, pad), a, True)
        return x

    def from_grid(self, g):
        for a in (0, 1, 2):
            g = self._pass(g, a, False).narrow(a, self.lo[a], self.I[a])
        return g * self.apod

    _CHUNK = 1 << 18

    def interp(self, g, idx, wt):
        g = g.reshape(-1)
        return torch.cat([(g[idx[s:s + self._CHUNK]] * wt[s:s + self._CHUNK]).sum(1)
                          for s in range(0, idx.shape[0], self._CHUNK)])

    def spread(self, v, idx, wt):
        n = self.G[0] * self.G[1] * self.G[2]
        g = torch.zeros(n, 2, dtype=torch.float64, device=self.dev)
        for s in range(0, idx.shape[0], self._CHUNK):
            p = torch.view_as_real(v[s:s + self._CHUNK, None] * wt[s:s + self._CHUNK]).reshape(-1, 2)
            g = g.index_add(0, idx[s:s + self._CHUNK].reshape(-1), p)
        return torch.view_as_complex(g).reshape(self.G)

    def forward(self, x, idx, wt):
        return self.interp(self.to_grid(x), idx, wt)

    def adjoint(self, v, idx, wt, scale=None):
        return self.from_grid(self.spread(v, idx, wt)) * (self.scale if scale is None else scale)

    def normal(self, x, maps, idx, wt, D):
        q = 0
        for m in maps:
            m = m.to(torch.complex128)
            q = q + m.conj() * self.adjoint(D * self.forward(m * x, idx, wt), idx, wt)
        return q

    def rhs(self, y, maps, idx, wt, D):
        return sum(m.to(torch.complex128).conj() * self.adjoint(D * v.to(torch.complex128), idx, wt)
                   for m, v in zip(maps, y))


def _cg(A, b, iters):
    """The reference's loop (Reco.cpp:232-309): complex step, residual |r|."""
    x, r, p = torch.zeros_like(b), b, b
    rr = (r.conj() * r).sum()
    res = []
    for _ in range(iters):
        q = A(p)
        alpha = rr / (p.conj() * q).sum()
        x = x + alpha * p
        r = r - alpha * q
        new = (r.conj() * r).sum()
        p = r + (new / rr) * p
        rr = new
        res.append(rr.real.sqrt())
    return x, torch.stack(res)


def _psf_normal(c, k, D, maps, ex):
    """x -> the exact normal operator, by circular convolution with the exact
    point-spread function (a wide-kernel transform of type 1 in 64 bits)."""
    dev = ex.dev
    W, I = 14, ex.I
    nf = [2 * (2 * i) for i in I]                       # two-fold oversampling of the 2 I positions
    beta = math.pi * math.sqrt(W * W / 4.0 * 1.5 ** 2 - 0.8)
    G = torch.tensor(ex.G, dtype=torch.float64, device=dev)
    nu = (k * (G - 1) - G / 2) / G                      # cycles per voxel
    fine = torch.zeros(nf[0] * nf[1] * nf[2], dtype=torch.float64, device=dev)
    step = 1 << 13
    for s in range(0, k.shape[0], step):
        ks, gs = [], []
        for a in range(3):
            u = (nu[s:s + step, a] - torch.floor(nu[s:s + step, a])) * nf[a]
            g = torch.ceil(u - W / 2).to(torch.int64)[:, None] + torch.arange(W, device=dev)[None]
            t = 2 * (g.to(torch.float64) - u[:, None]) / W
            ks.append(torch.special.i0(beta * torch.sqrt((1 - t * t).clamp_min(0.0))) / math.exp(beta))
            gs.append(g % nf[a])
        w = (ks[0] * D[s:s + step, None])[:, :, None, None] * ks[1][:, None, :, None] * ks[2][:, None, None, :]
        i = (gs[0][:, :, None, None] * nf[1] + gs[1][:, None, :, None]) * nf[2] + gs[2][:, None, None, :]
        fine.index_add_(0, i.reshape(-1), w.reshape(-1))
    # T(d) = sum_s D_s exp(2 pi i nu_s . d), d in [-I, I)
    T = torch.fft.ifftn(fine.reshape(nf).to(torch.complex128), norm="forward")
    for a in range(3):
        d = torch.arange(-I[a], I[a], device=dev)
        xi = d.to(torch.float64) / nf[a]
        z = torch.sqrt(torch.complex(beta ** 2 - (math.pi * W * xi) ** 2, torch.zeros_like(xi)))
        ft = (W * torch.sinh(z) / z).real / math.exp(beta)
        sh = [1, 1, 1]
        sh[a] = -1
        T = T.index_select(a, d % nf[a]) / ft.reshape(sh)
    P = torch.fft.fftn(torch.fft.ifftshift(T, dim=(0, 1, 2)))

    def A(x):
        q = 0
        for m in maps:
            m = m.to(torch.complex128)
            v = torch.fft.fftn(m * x, s=[2 * i for i in I])
            q = q + m.conj() * torch.fft.ifftn(v * P)[:I[0], :I[1], :I[2]]
        return q * ex.scale
    return A


def exact(case, seed):
    c = dict(case)
    op = c["op"]
    w = work(c)
    if w["flops"] > 6e12 or (op == "unrolled" and w["flops"] > 2e11):
        return None                                     # minutes in 64 bits
    d = _inputs(c, seed)
    s, dev = d["scan"], d["dev"]
    ex = _Exact(c, dev)
    D_all = torch.from_numpy(s.dcf).to(dev).to(torch.float64)
    bins = [torch.from_numpy(np.asarray(b)).to(dev) for b in s.bins] if s.bins is not None else None
    if op in ("calibrate", "unrolled"):
        # the wave of the case as a function of its six parameters, in 64 bits
        theta = d["theta"].clone().requires_grad_(True)
        k = _wave(s, theta, dev)
        k.retain_grad()
    else:
        k = torch.from_numpy(s.k).to(dev)
    maps = d.get("maps")
    nb = max(1, c["bins"])
    per_bin = bins if bins is not None else [torch.arange(k.shape[0], device=dev)]

    if op == "density":
        n = ex.G[0] * ex.G[1] * ex.G[2]
        out = torch.zeros(k.shape[0], dtype=torch.float64, device=dev)
        for sel in per_bin:
            idx, wt = _taps(c, k[sel], dev)
            wv = torch.ones(len(sel), dtype=torch.float64, device=dev)
            for _ in range(c["iters"]):
                g = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, idx.reshape(-1), (wt * wv[:, None]).reshape(-1))
                u = (g[idx] * wt).sum(1)
                wv = torch.where(u > 0, wv / u, torch.zeros_like(u))
            out[sel] = wv / wv.max()
        return out.cpu().numpy()
    if op in ("forward", "adjoint"):
        idx, wt = _taps(c, k, dev)
        if op == "forward":
            return torch.stack([ex.forward(x.to(torch.complex128), idx, wt) for x in d["x"]])
        return torch.stack([ex.adjoint(y.to(torch.complex128), idx, wt) for y in d["y"]])
    if op in ("apply", "apply_compensated"):
        out = []
        for b, sel in enumerate(per_bin):
            idx, wt = _taps(c, k[sel], dev)
            out.append(ex.normal(d["x"][b].to(torch.complex128), maps, idx, wt, D_all[sel]))
        return torch.stack(out)
    if op in ("solve", "solve_host", "solve_toeplitz"):
        xs, rs = [], []
        for sel in per_bin:
            idx, wt = _taps(c, k[sel], dev)
            b = ex.rhs(d["y"][:, sel], maps, idx, wt, D_all[sel])
            if op == "solve_toeplitz":
                A = _psf_normal(c, k[sel], D_all[sel], maps, ex)
            else:
                def A(p, idx=idx, wt=wt, D=D_all[sel]):
                    return ex.normal(p, maps, idx, wt, D)
            x, res = _cg(A, b, c["iters"])
            xs.append(x)
            rs.append(res)
        if op == "solve_host":
            return {"x": xs[0].cpu().numpy(), "residuals": rs[0].cpu().numpy(), "iterations": None}
        return {"x": torch.stack(xs), "residuals": torch.stack(rs).cpu().numpy(), "iterations": None}
    if op in ("loss", "calibrate"):
        x = d["x"].to(torch.complex128).requires_grad_(op == "loss")
        kk = k if op == "calibrate" else k.clone().requires_grad_(True)
        # coil by coil and chunk by chunk, so that the tape stays small
        gk = torch.zeros_like(kk)
        total = torch.zeros((), dtype=torch.float64, device=dev)
        gx = torch.zeros_like(x.detach())
        for m, y in zip(maps, d["y"]):
            m, y = m.to(torch.complex128), y.to(torch.complex128)
            g = ex.to_grid(m * x.detach()).requires_grad_(True)
            gg = torch.zeros_like(g)
            for a in range(0, kk.shape[0], ex._CHUNK):
                kc = kk.detach()[a:a + ex._CHUNK].clone().requires_grad_(True)
                idx, wt = _taps(c, kc, dev)
                rr = (g.reshape(-1)[idx] * wt).sum(1) - y[a:a + ex._CHUNK]
                part = 0.5 * (D_all[a:a + ex._CHUNK] * (rr.real ** 2 + rr.imag ** 2)).sum()
                ga, ka = torch.autograd.grad(part, (g, kc))
                gg += ga
                gk[a:a + ex._CHUNK] = gk[a:a + ex._CHUNK] + ka
                total = total + part.detach()
            if op == "loss":
                gx = gx + m.conj() * ex.from_grid(gg)
        if op == "loss":
            return {"loss": total, "grad_x": gx, "grad_k": gk}
        k.backward(gk.detach())
        return {"loss": total, "grad_k": gk.detach(), "grad_theta": theta.grad}
    # unrolled CG, differentiated by torch
    from torch.utils.checkpoint import checkpoint
    xs = []
    for b, sel in enumerate(per_bin):
        kb = k[sel]
        y = d["y"][:, sel]

        def adj(v, kb):
            i, t = _taps(c, kb, dev)
            return ex.adjoint(v, i, t)

        def nrm(mp, kb, D):
            i, t = _taps(c, kb, dev)
            return ex.adjoint(D * ex.forward(mp, i, t), i, t)

        rhs = sum(m.to(torch.complex128).conj() * checkpoint(adj, D_all[sel] * v.to(torch.complex128), kb, use_reentrant=False)
                  for m, v in zip(maps, y))

        def A(p):
            return sum(m.to(torch.complex128).conj()
                       * checkpoint(nrm, m.to(torch.complex128) * p, kb, D_all[sel], use_reentrant=False) for m in maps)
        x, r, p = torch.zeros_like(rhs), rhs, rhs
        rr = (r.conj() * r).sum().real
        for _ in range(c["iters"]):
            q = A(p)
            alpha = rr / (p.conj() * q).sum()
            x = x + alpha * p
            r = r - alpha * q
            new = (r.conj() * r).sum().real
            p = r + (new / rr) * p
            rr = new
        x.reshape(-1).backward(d["v"][b].to(torch.complex128), retain_graph=True)
        xs.append(x.detach().reshape(-1))
    return {"x": torch.stack(xs), "grad_k": k.grad, "grad_theta": theta.grad}


def _wave(s, theta, dev):
    """The parametric wave-CAIPI readouts: x linear, y and z sinusoids around
    the base lines, coordinates in [0, 1]."""
    w = s.w
    G, I, n = w.grid, w.img, w.n_read
    i = torch.arange(n, dtype=torch.float64, device=dev)
    t, om = i / n, 2 * math.pi * w.wave_cycles
    ln = torch.from_numpy(np.asarray(s.lines)).to(dev).to(torch.float64)
    ux = G[0] / 2 + (i - n / 2) * G[0] / n
    uy = G[1] / 2 + (ln[:, :1] - I[1] / 2) * G[1] / I[1] + (theta[0] * torch.sin(om * (t - theta[4]) + theta[2]))[None]
    uz = G[2] / 2 + (ln[:, 1:] - I[2] / 2) * G[2] / I[2] + (theta[1] * torch.cos(om * (t - theta[5]) + theta[3]))[None]
    kx = (ux / (G[0] - 1))[None].expand(len(ln), n)
    return torch.stack([kx, uy / (G[1] - 1), uz / (G[2] - 1)], -1).reshape(-1, 3)
