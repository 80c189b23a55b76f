"""Cases of the NUFFT backend that are timed: what programs use it for.

A case is a plain dict: ``kind`` names the call, the other entries its sizes.
The listed cases are the repository's own workloads (its benchmark
configurations and served request templates) and two generic 3D ones with odd
sizes, few coils and a loose tolerance; ``draw`` spreads the same calls over
the ranges that those stand for.  Inputs are synthetic: ellipse phantoms,
smooth coil maps, noisy k-space, trajectories turned by an angle of the seed.

``exact`` evaluates the same sums in double precision with plain torch: a
NUFFT of its own (kernel of 10 cells on a twice oversampled double grid, whose
error is about 1e-9), without this repository's code.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__

DEV = "cuda"


# ------------------------------------------------------------------ the cases
# n0, n1, n2: the image axes (n2 = 0: a 2D image)
def _shape(case):
    return tuple(n for n in (case["n0"], case["n1"], case["n2"]) if n)


def listed():
    return [
        # one image, one coil: a radial scan gridded there and back (latency)
        {"name": "radial2d_1coil", "kind": "op_adj", "n0": 256, "n1": 256, "n2": 0, "traj": "radial",
         "shots": 100, "ns": 500, "coils": 1, "sense": False, "density": False, "eps": 1e-6},
        # one gradient of an iterative SENSE reconstruction, 2D radial
        {"name": "radial2d_dc_16coils", "kind": "dc", "n0": 256, "n1": 256, "n2": 0, "traj": "radial",
         "shots": 256, "ns": 512, "coils": 16, "sense": True, "density": False, "eps": 1e-6},
        # density-compensated spiral there and back, a larger image
        {"name": "spiral2d_384_16coils", "kind": "op_adj", "n0": 384, "n1": 384, "n2": 0, "traj": "spiral",
         "shots": 32, "ns": 4096, "coils": 16, "sense": True, "density": True, "eps": 1e-6},
        # trajectory learning: forward and backward for image and trajectory
        {"name": "spiral2d_train_8coils", "kind": "train", "n0": 256, "n1": 256, "n2": 0, "traj": "spiral",
         "shots": 64, "ns": 2048, "coils": 8, "sense": True, "density": False, "eps": 1e-6},
        # 3D multi-coil radial: the headline configuration
        {"name": "koosh3d_16coils", "kind": "op_adj", "n0": 128, "n1": 128, "n2": 128, "traj": "koosh",
         "shots": 4096, "ns": 512, "coils": 16, "sense": True, "density": True, "eps": 1e-6},
        # one gradient of a 3D SENSE reconstruction
        {"name": "koosh3d_dc_8coils", "kind": "dc", "n0": 128, "n1": 128, "n2": 128, "traj": "koosh",
         "shots": 2048, "ns": 512, "coils": 8, "sense": True, "density": False, "eps": 1e-6},
        # odd, uneven axes without coil maps, few coils
        {"name": "stack3d_odd_3coils", "kind": "op_adj", "n0": 97, "n1": 110, "n2": 75, "traj": "stack",
         "shots": 1201, "ns": 257, "coils": 3, "sense": False, "density": True, "eps": 1e-6},
        # preview quality: a narrower kernel
        {"name": "koosh3d_eps1e-4", "kind": "op_adj", "n0": 96, "n1": 96, "n2": 96, "traj": "koosh",
         "shots": 2048, "ns": 384, "coils": 8, "sense": True, "density": True, "eps": 1e-4},
        # Toeplitz form of A^H A, 3D
        {"name": "gram3d_16coils", "kind": "gram", "n0": 128, "n1": 128, "n2": 128, "traj": "koosh",
         "shots": 2048, "ns": 512, "coils": 16, "sense": True, "density": False, "eps": 1e-6},
        # density estimation of a new 3D trajectory: plan, sort, iterations
        {"name": "pipe3d", "kind": "pipe", "n0": 128, "n1": 128, "n2": 128, "traj": "koosh",
         "shots": 4096, "ns": 512, "coils": 1, "sense": False, "density": False, "eps": 1e-6},
        # stack of stars: 64 planes of 16 coils on one 2D trajectory
        {"name": "stacked_64planes_16coils", "kind": "stacked", "n0": 256, "n1": 256, "n2": 64, "traj": "radial",
         "shots": 256, "ns": 512, "coils": 16, "sense": True, "density": True, "eps": 1e-6},
        # off-resonance corrected spiral, 30 time segments
        {"name": "offres2d_16coils", "kind": "offres", "n0": 256, "n1": 256, "n2": 0, "traj": "spiral",
         "shots": 48, "ns": 4096, "coils": 16, "sense": True, "density": True, "eps": 1e-6,
         "segments": 30},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["op_adj2", "dc2", "train", "op_adj3", "op_adj3", "dc3", "gram", "pipe", "stacked",
                       "offres"])
    c = {"kind": kind.rstrip("23"), "eps": 1e-6, "density": rng.random() < 0.5, "sense": True}
    if kind in ("op_adj2", "dc2", "train", "stacked", "offres"):
        n0 = rng.choice([128, 192, 256, 256, 320, 384, rng.randint(100, 384)])
        n1 = n0 if rng.random() < 0.6 else rng.randint(100, 384)
        s = [n0, n1, 0]
        c["traj"] = rng.choice(["radial", "spiral"])
        c["shots"] = _log(rng, 64, 256) if c["traj"] == "radial" else _log(rng, 16, 64)
        c["ns"] = _log(rng, 256, 1024) if c["traj"] == "radial" else _log(rng, 1024, 4096)
        c["coils"] = rng.choice([1, 4, 8, 16, 32, rng.randint(1, 32)])
        if kind == "op_adj2":
            c["eps"] = rng.choice([1e-6, 1e-6, 1e-4])
            c["sense"] = c["coils"] > 1 and rng.random() < 0.7
        if kind == "train":
            c["coils"] = rng.choice([4, 8, rng.randint(2, 16)])
            c["density"] = False
        if kind == "stacked":
            s = [min(n0, 256), min(n1, 256), _log(rng, 8, 64)]
            c["coils"] = _log(rng, 2, 16)
            c["shots"], c["ns"] = min(c["shots"], 256), min(c["ns"], 512 if c["traj"] == "radial" else 2048)
        if kind == "offres":
            c["traj"], c["segments"] = "spiral", rng.randint(5, 30)
            s = [min(n0, 256), min(n1, 256), 0]
            c["shots"], c["ns"] = _log(rng, 16, 48), _log(rng, 1024, 4096)
            c["coils"] = _log(rng, 2, 16)
    else:
        s = [rng.choice([64, 96, 128, 128, rng.randint(48, 128)]) for _ in range(3)]
        s = [s[0]] * 3 if rng.random() < 0.5 else s
        c["traj"] = rng.choice(["koosh", "koosh", "stack"])
        c["shots"], c["ns"] = _log(rng, 512, 4096), _log(rng, 200, 512)
        c["coils"] = rng.choice([1, 4, 8, 16, rng.randint(1, 16)])
        if kind == "op_adj3":
            c["eps"] = rng.choice([1e-6, 1e-6, 1e-4])
            c["sense"] = c["coils"] > 1 and rng.random() < 0.7
        if kind == "pipe":
            c["coils"], c["density"], c["sense"] = 1, False, False
    c["n0"], c["n1"], c["n2"] = s
    return c


# ------------------------------------------------------------------ inputs
def _turn2(t, a):
    r = np.array([[math.cos(a), -math.sin(a)], [math.sin(a), math.cos(a)]])
    return t @ r.T


def _trajectory(case, seed):
    """(M, d) float32 in [-0.5, 0.5]: the case's trajectory, turned by the seed."""
    kind, shots, ns = case["traj"], case["shots"], case["ns"]
    rng = np.random.default_rng(seed + 17)
    turn = rng.uniform(0, 2 * math.pi)
    i = np.arange(shots)[:, None]
    if kind == "radial":  # full spokes out of the centre
        a = turn + 2 * math.pi * i / shots
        r = 0.5 * np.linspace(0, 1, ns)[None]
        t = np.stack([r * np.cos(a), r * np.sin(a)], -1)
    elif kind == "spiral":  # one revolution, radius growing with its square
        th = 2 * math.pi * np.linspace(0, 1, ns)[None]
        r = 0.5 * (th / (2 * math.pi)) ** 2
        a = turn + 2 * math.pi * i / shots + th
        t = np.stack([r * np.cos(a), r * np.sin(a)], -1)
    elif kind == "koosh":  # centre-out spokes on a Fibonacci sphere
        z = np.linspace(-1, 1, shots)[:, None]
        a = turn + math.pi * (3 - math.sqrt(5)) * i
        q = np.sqrt(1 - z * z)
        r = 0.5 * np.linspace(0, 1, ns)[None]
        t = np.stack([r * q * np.cos(a), r * q * np.sin(a), r * z], -1)
    else:  # full diameters in planes turned about the first axis
        planes = max(1, int(math.sqrt(shots)))
        p, s = i // -(-shots // planes), i % -(-shots // planes)
        a = turn + math.pi * s / -(-shots // planes)
        b = math.pi * p / planes
        r = np.linspace(-0.5, 0.4999, ns)[None]
        t = np.stack([r * np.cos(a), r * np.sin(a) * np.cos(b), r * np.sin(a) * np.sin(b)], -1)
    return t.reshape(-1, t.shape[-1]).astype(np.float32)


def _axes(shape):
    return torch.meshgrid(*[torch.linspace(-1, 1, n, device=DEV, dtype=torch.float32) for n in shape],
                          indexing="ij")


def _phantom(shape, seed):
    """Twenty random ellipses with complex amplitudes, and 1 % noise."""
    rng = np.random.default_rng(seed)
    ax = _axes(shape)
    img = torch.zeros(tuple(shape), dtype=torch.complex64, device=DEV)
    for _ in range(20):
        c, h = rng.uniform(-0.6, 0.6, len(shape)), rng.uniform(0.05, 0.5, len(shape))
        inside = sum(((x - float(cc)) / float(hh)) ** 2 for x, cc, hh in zip(ax, c, h)) <= 1
        a = rng.uniform(0.1, 1.0) * np.exp(2j * math.pi * rng.random())
        img += inside * complex(a)
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    return img + 0.01 * torch.randn(tuple(shape), dtype=torch.complex64, device=DEV, generator=g)


def _maps(shape, coils, seed):
    """Gaussian magnitudes around the object with linear phases, sum of squares 1."""
    rng = np.random.default_rng(seed + 2)
    ax = _axes(shape)
    out = torch.empty((coils, *shape), dtype=torch.complex64, device=DEV)
    for c in range(coils):
        v = rng.standard_normal(len(shape))
        v *= 0.8 / np.linalg.norm(v)
        d2 = sum((x - float(q)) ** 2 for x, q in zip(ax, v))
        ph = sum(x * float(q) for x, q in zip(ax, rng.uniform(-1.5, 1.5, len(shape))))
        out[c] = torch.polar(torch.exp(-d2 / 0.72), ph + float(rng.uniform(0, 2 * math.pi)))
    return out / torch.sqrt((out.abs() ** 2).sum(0, keepdim=True))


def _inputs(case, seed):
    """Every array that a program has in hand, on the GPU, from the seed."""
    shape, C = _shape(case), case["coils"]
    k = _trajectory(case, seed)
    M = k.shape[0]
    kd = torch.from_numpy(k).to(DEV)
    v = {"k": k}
    r = torch.linalg.vector_norm(kd, dim=1)
    # radial and spiral samples thin out with the radius: ramp weights
    v["density"] = (r ** (kd.shape[1] - 1) + 1e-3).contiguous() if case["density"] else None
    v["smaps"] = _maps(shape, C, seed) if case["sense"] else None
    if case["kind"] == "pipe":
        v["kd"] = kd
        return v
    img = _phantom(shape, seed)
    if not case["sense"]:
        img = img[None] * _maps(shape, C, seed) if C > 1 else img[None]
    v["img"] = img.contiguous()
    if case["kind"] != "gram":  # k-space: decays from the centre, with noise
        planes = shape[2] if case["kind"] == "stacked" else 1
        g = torch.Generator(device=DEV).manual_seed(seed + 3)
        y = torch.randn((1, C, planes * M), dtype=torch.complex64, device=DEV, generator=g)
        v["ksp"] = (y * (0.02 + torch.exp(-12 * r)).repeat(planes)).contiguous()
    if case["kind"] == "offres":  # time segmentation of a smooth +-120 Hz field
        NK, L, T = case["ns"], case["segments"], 0.0123
        ax = _axes(shape)
        field = 2 * math.pi * 120 * torch.sin(2.1 * ax[0] + seed) * torch.cos(1.7 * ax[1])
        t, tl = np.linspace(0, T, NK), np.linspace(0, T, L)
        B = np.maximum(0.0, 1 - np.abs(t[:, None] - tl[None]) / (tl[1] - tl[0]))
        v["B"] = B.astype(np.complex64)
        v["C"] = torch.polar(torch.ones((), device=DEV), field[None] * torch.tensor(
            tl, device=DEV, dtype=torch.float32).reshape(-1, 1, 1)).contiguous()
    return v


def prepare(case, seed):
    pkg = __graft_entry__.import_package()
    v = _inputs(case, seed)
    shape, C = _shape(case), case["coils"]
    st = {"case": case, **v}
    if case["kind"] == "pipe":
        st["cls"] = pkg.MRIGB300
        return st
    if case["kind"] == "stacked":
        st["op"] = pkg.MRIStackedGB300(v["k"], shape, smaps=v["smaps"], n_coils=C, z_index=None,
                                       density=v["density"] if v["density"] is not None else False,
                                       eps=case["eps"])
        return st
    op = pkg.MRIGB300(v["k"], shape, density=v["density"] if v["density"] is not None else False, n_coils=C,
                      smaps=v["smaps"], squeeze_dims=False, eps=case["eps"])
    if case["kind"] == "offres":
        op = pkg.MRIFourierCorrectedGB300(op, interpolator=(v["B"], v["C"]))
    if case["kind"] == "train":
        op = op.make_autograd(wrt_data=True, wrt_traj=True)
    if case["kind"] == "gram":
        op.compute_toeplitz_kernel()
    st["op"] = op
    st["x"] = v["img"].reshape(1, 1 if case["sense"] else C, *shape)
    return st


def run(st):
    case, op = st["case"], st.get("op")
    kind = case["kind"]
    if kind == "pipe":
        return st["cls"].pipe(st["kd"], _shape(case), max_iter=10)
    if kind == "stacked":
        return [op.op(st["img"][None]), op.adj_op(st["ksp"])]
    if kind in ("op_adj", "offres"):
        return [op.op(st["x"]), op.adj_op(st["ksp"])]
    if kind == "dc":
        return op.data_consistency(st["x"], st["ksp"])
    if kind == "gram":
        return op.gram_op(st["x"])
    x = st["x"].clone().requires_grad_(True)
    op.samples.grad = None
    y = op.op(x)
    loss = torch.sum(torch.abs(y - st["ksp"]) ** 2)
    loss.backward()
    return [y.detach(), x.grad, op.samples.grad]


# ------------------------------------------------------------------ the work
def work(case):
    """Each input and output once; kernel footprints and transforms of the
    twice oversampled grid."""
    shape, C = _shape(case), case["coils"]
    kind = case["kind"]
    planes = shape[2] if kind == "stacked" else 1
    grid = shape[:2] if kind == "stacked" else shape
    d, M = len(grid), case["shots"] * case["ns"]
    N = math.prod(shape)
    w = math.ceil(-math.log10(case["eps"] / 10))
    G = 2 ** d * math.prod(grid)
    T = C * planes * case.get("segments", 1)  # transforms of one direction
    fft = 5 * G * math.log2(G)
    foot = 4 * w ** d * M
    img, maps, ksp = 8 * N * (1 if case["sense"] else C), 8 * N * C if case["sense"] else 0, 8 * C * planes * M
    pts = 4 * d * M
    dens = 4 * M if case["density"] else 0
    if kind == "pipe":
        return {"bytes": pts + 4 * M, "flops": 20 * 4 * w ** d * M}
    if kind == "gram":
        return {"bytes": 2 * img + maps + 4 * G, "flops": C * 2 * fft}
    if kind == "dc":
        return {"bytes": 2 * img + maps + ksp + pts, "flops": C * 2 * (foot + fft)}
    if kind == "train":
        return {"bytes": 2 * img + maps + 2 * ksp + 2 * pts, "flops": C * (3 * fft + (2 + 2 * d) * foot)}
    extra = 8 * case["ns"] * case["segments"] + 8 * N * case["segments"] if kind == "offres" else 0
    return {"bytes": 2 * img + maps + 2 * ksp + pts + dens + extra, "flops": 2 * T * (foot + fft)}


# ------------------------------------------------------------------ in 64 bits
class _Nufft64:
    """sum_n x_n e^{-i k.n} and its adjoint over integer modes
    n = -(N // 2) .. N - N // 2 - 1, in double precision."""

    W = 10

    def __init__(self, k, shape):
        self.shape, self.d = tuple(shape), len(shape)
        self.nf = [max(2 * n + n % 2, 2 * self.W + 2) for n in shape]
        self.beta = 2.3 * self.W
        self.k = k.to(DEV, torch.float64)
        z, wt = np.polynomial.legendre.leggauss(120)
        self.dec = []
        for n, f in zip(self.shape, self.nf):
            m = np.arange(n) - n // 2
            ph = np.exp(self.beta * (np.sqrt(1 - z * z) - 1)) * wt * self.W / 2
            hat = (ph[None] * np.cos(2 * math.pi * m[:, None] * z[None] * (self.W / 2) / f)).sum(1)
            self.dec.append(torch.tensor(1 / hat, device=DEV))
        self.modes = [torch.arange(n, device=DEV).sub(n // 2) % f for n, f in zip(self.shape, self.nf)]

    def _axis(self, u, nf):
        i0 = torch.ceil(u - self.W / 2)
        t = torch.arange(self.W, device=DEV, dtype=torch.float64)
        x = (i0[:, None] + t - u[:, None]) * (2 / self.W)
        w = torch.exp(self.beta * (torch.sqrt(torch.clamp(1 - x * x, min=0)) - 1)) * (x.abs() < 1)
        return (i0[:, None] + t).long() % nf, w

    def _chunks(self):
        step = 1 << 19 if self.d == 3 else 1 << 18
        for a in range(0, self.k.shape[0], step):
            k = self.k[a:a + step]
            yield a, k.shape[0], [self._axis(k[:, j] * (self.nf[j] / (2 * math.pi)), self.nf[j])
                                  for j in range(self.d)]

    def _pairs(self, ax):
        """(row index, row weight) of every offset of all axes but the last."""
        for t0 in range(self.W):
            i0, w0 = ax[0][0][:, t0], ax[0][1][:, t0]
            if self.d == 2:
                yield i0, w0
                continue
            for t1 in range(self.W):
                yield i0 * self.nf[1] + ax[1][0][:, t1], w0 * ax[1][1][:, t1]

    def _place(self):
        return torch.meshgrid(*self.modes, indexing="ij")

    def type2(self, x):
        """(T, *shape) -> (T, M)"""
        T = x.shape[0]
        out = torch.zeros((T, self.k.shape[0]), dtype=torch.complex128, device=DEV)
        for t in range(T):
            v = x[t].to(torch.complex128)
            for j in range(self.d):
                v = v * self.dec[j].reshape([-1 if q == j else 1 for q in range(self.d)])
            g = torch.zeros(self.nf, dtype=torch.complex128, device=DEV)
            g[self._place()] = v
            g = torch.fft.fftn(g).reshape(-1, self.nf[-1])
            flat = torch.view_as_real(g.reshape(-1))
            for a, n, ax in self._chunks():
                acc = torch.zeros((n, 2), dtype=torch.float64, device=DEV)
                last, wl = ax[-1]
                for row, wr in self._pairs(ax):
                    vals = flat[(row[:, None] * self.nf[-1] + last).reshape(-1)].reshape(n, self.W, 2)
                    acc += wr[:, None] * torch.einsum("mtc,mt->mc", vals, wl)
                out[t, a:a + n] = torch.view_as_complex(acc)
        return out

    def type1(self, y):
        """(T, M) -> (T, *shape), the adjoint of type2"""
        T = y.shape[0]
        out = torch.empty((T, *self.shape), dtype=torch.complex128, device=DEV)
        for t in range(T):
            g = torch.zeros((math.prod(self.nf), 2), dtype=torch.float64, device=DEV)
            for a, n, ax in self._chunks():
                v = torch.view_as_real(y[t, a:a + n].to(torch.complex128).contiguous())
                last, wl = ax[-1]
                for row, wr in self._pairs(ax):
                    idx = (row[:, None] * self.nf[-1] + last).reshape(-1)
                    g.index_add_(0, idx, ((wr[:, None] * wl)[:, :, None] * v[:, None]).reshape(-1, 2))
            g = torch.fft.ifftn(torch.view_as_complex(g).reshape(self.nf)) * math.prod(self.nf)
            v = g[self._place()]
            for j in range(self.d):
                v = v * self.dec[j].reshape([-1 if q == j else 1 for q in range(self.d)])
            out[t] = v
        return out


def _footprint(k, n, w, beta):
    """Cells and weights of the interpolation kernel on an n-cell axis."""
    u = (k * (n / (2 * math.pi))) % n
    i0 = torch.ceil(u - w / 2)
    t = torch.arange(w, device=DEV, dtype=torch.float64)
    x = (i0[:, None] + t - u[:, None]) * (2 / w)
    v = torch.exp(beta * (torch.sqrt(torch.clamp(1 - x * x, min=0)) - 1)) * (x.abs() < 1)
    return (i0[:, None] + t).long() % n, v


def _pipe64(k, shape, iters):
    w = 7
    ax = [_footprint(k[:, j], n, w, 2.3 * w) for j, n in enumerate(shape)]
    M, scale = k.shape[0], 1.0 / (math.prod(shape) * 2 ** len(shape))
    wts = torch.ones(M, dtype=torch.float64, device=DEV)
    for _ in range(iters):
        g = torch.zeros(math.prod(shape), dtype=torch.float64, device=DEV)
        for t0 in range(w):
            for t1 in range(w):
                row = (ax[0][0][:, t0] * shape[1] + ax[1][0][:, t1])[:, None] * shape[2] + ax[2][0]
                f = (ax[0][1][:, t0] * ax[1][1][:, t1])[:, None] * ax[2][1]
                g.index_add_(0, row.reshape(-1), (f * wts[:, None]).reshape(-1))
        v = torch.zeros(M, dtype=torch.float64, device=DEV)
        for t0 in range(w):
            for t1 in range(w):
                row = (ax[0][0][:, t0] * shape[1] + ax[1][0][:, t1])[:, None] * shape[2] + ax[2][0]
                f = (ax[0][1][:, t0] * ax[1][1][:, t1])[:, None] * ax[2][1]
                v += (f * g[row]).sum(1)
        wts = wts / (scale * v).abs()
    return wts


def exact(case, seed):
    kind, shape, C = case["kind"], _shape(case), case["coils"]
    d = 2 if kind == "stacked" else len(shape)
    M = case["shots"] * case["ns"]
    T = C * case.get("segments", 1) * (shape[2] if kind == "stacked" else 1)
    calls = 2 + d if kind == "train" else 2
    if calls * T * (M * 10.0 ** d + 10.0 * 2 ** d * math.prod(shape[:d])) > 4.5e10:
        return None  # over about 20 seconds
    v = _inputs(case, seed)
    k = torch.from_numpy(v["k"]).to(DEV)
    # the trajectory as the operator receives it: float32 radians
    k = (k * 2 * math.pi).to(torch.float32).to(torch.float64)
    f = _Nufft64(k, shape[:d])
    nrm = 1.0 / math.sqrt(math.prod(shape) * 2 ** len(shape))
    s = None if v["smaps"] is None else v["smaps"].to(torch.complex128)
    if kind == "pipe":
        w = _pipe64(k, shape, 10).to(torch.complex128)
        y = f.type2(torch.ones((1, *shape), dtype=torch.complex128, device=DEV)) * nrm
        r = f.type1(w[None] * y) * nrm
        return (w / r.abs().mean()).abs()
    img = v["img"].to(torch.complex128)
    if kind == "gram":
        out = torch.zeros(tuple(shape), dtype=torch.complex128, device=DEV)
        for c in range(C):
            out += s[c].conj() * f.type1(f.type2((s[c] * img)[None]))[0]
        return (out * nrm ** 2).reshape(1, 1, *shape)
    y = v["ksp"].to(torch.complex128)
    w = torch.ones(M, device=DEV, dtype=torch.float64) if v["density"] is None else v["density"].to(torch.float64)
    if kind == "stacked":
        Z, root = shape[2], 1 / math.sqrt(2 * shape[2])
        img = img.reshape(shape) if s is not None else img
        fwd = torch.empty((1, C, Z * M), dtype=torch.complex128, device=DEV)
        adj = torch.zeros(tuple(shape), dtype=torch.complex128, device=DEV)
        n2 = 1.0 / math.sqrt(math.prod(shape[:2]) * 4)
        for c in range(C):
            p = torch.fft.fftshift(torch.fft.fft(torch.fft.ifftshift(s[c] * img, dim=2), dim=2), dim=2) * root
            fwd[0, c] = (f.type2(p.permute(2, 0, 1).contiguous()) * n2).reshape(-1)
            q = (f.type1(y[0, c].reshape(Z, M) * w) * n2).permute(1, 2, 0)
            q = torch.fft.fftshift(torch.fft.ifft(torch.fft.ifftshift(q, dim=2), dim=2), dim=2) * (Z * root)
            adj += s[c].conj() * q
        return [fwd, adj.reshape(1, *shape)]
    src = s * img if s is not None else img  # (C, *shape)
    if kind == "offres":
        B, L = torch.from_numpy(v["B"]).to(DEV, torch.complex128), v["C"].to(torch.complex128)
        fwd = torch.zeros((1, C, M), dtype=torch.complex128, device=DEV)
        adj = torch.zeros(tuple(shape), dtype=torch.complex128, device=DEV)
        for i in range(case["segments"]):
            b = B[:, i].repeat(case["shots"])
            fwd[0] += b * f.type2(L[i] * src) * nrm
            adj += ((L[i] * s).conj() * f.type1(b.conj() * w * y[0])).sum(0) * nrm
        return [fwd, adj.reshape(1, 1, *shape)]
    ax = f.type2(src) * nrm
    if kind == "op_adj":
        z = f.type1(y[0] * w) * nrm
        z = (s.conj() * z).sum(0)[None] if s is not None else z
        return [ax[None], z[None]]
    r = (ax - y[0]) * (w if kind == "dc" else 2)
    z = f.type1(r) * nrm
    z = ((s.conj() * z).sum(0)[None] if s is not None else z)[None]
    if kind == "dc":
        return z
    g = torch.empty((M, d), dtype=torch.float64, device=DEV)
    for j in range(d):
        n = torch.arange(shape[j], device=DEV) - shape[j] // 2
        n = n.to(torch.float64).reshape([-1 if q == j else 1 for q in range(d)])
        g[:, j] = (r.conj() * (-1j) * f.type2(src * n) * nrm).real.sum(0)
    return [ax[None], z, g]
