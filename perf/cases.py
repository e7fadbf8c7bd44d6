"""Performance cases of the registration library: what a registration program has it do.

Each case names the work (``kind``), the grid (``nx``, ``ny``, ``nz`` voxels, x fastest) and the
options of one call sequence through the public classes; ``prepare`` makes what such a program holds
before the call, ``run`` is one pass, ``exact`` the same result in 64-bit torch arithmetic.

Kinds:
  fluid     the fluid operator K = L^-1 (or L) on a vector field: DiffOperB200
  greedy    a greedy-fluid registration from the identity at one scale level: GreedyIteratorB200.Run
  ldmm      an LDMM relaxation iteration from running velocities: LDMMIteratorB200.Run
  adshoot   an adjoint geodesic-shooting iteration from a running momentum: LDMMAdShootingIteratorB200
  atlas     greedy atlas building over subjects on grids of their own: GreedyAtlasBuilderB200
  predict   the learned warm start's inference on a pair: WarmStartPredictor
  train     one training step of the warm-start network: WarmStartNet.train_step
"""
import math
import os

import numpy as np
import torch

from atlaswerks_b200 import warmstart
from atlaswerks_b200.atlas import GreedyAtlasBuilderB200, GreedyAtlasParam
from atlaswerks_b200.greedy import (DiffOperB200, DiffOperParam, GreedyDeformationDataB200,
                                    GreedyIteratorB200, GreedyIteratorParam)
from atlaswerks_b200.ldmm import LDMMDeformationDataB200, LDMMIteratorB200, LDMMIteratorParam
from atlaswerks_b200.shooting import LDMMAdShootingIteratorB200, LDMMShootingDefDataB200

ALPHA, BETA, GAMMA = 0.01, 0.01, 0.001  # the DiffOperParam defaults
MAX_PERT = 0.5
LDMM_SIGMA, LDMM_STEP = 1.0, 0.01
SHOOT_SIGMA, SHOOT_STEP = 1.0, 0.0002
ATLAS_AXES = (96, 112, 128, 144, 160)


def listed():
    return [
        # the smallest call: the operator on the coarse level of a small image pyramid
        {"name": "fluid_28x20x24", "kind": "fluid", "nx": 28, "ny": 20, "nz": 24, "inverse": True, "spacing": 1.0},
        # a pyramid's coarsest level (n/4 of 128): short launches, many iterations
        {"name": "greedy_32", "kind": "greedy", "nx": 32, "ny": 32, "nz": 32, "iters": 20, "hinv": False,
         "fast": False, "spacing": 1.0},
        # the finest level of the three-level 128^3 registration, the benchmark's grid
        {"name": "greedy_128", "kind": "greedy", "nx": 128, "ny": 128, "nz": 128, "iters": 10, "hinv": False,
         "fast": False, "spacing": 1.0},
        # a subject of the uneven-grid atlas registered on its own grid, writing the inverse field too
        {"name": "greedy_96x112x144_hinv", "kind": "greedy", "nx": 96, "ny": 112, "nz": 144, "iters": 6,
         "hinv": True, "fast": False, "spacing": 1.25},
        # a head at about one millimetre, with the float interpolation option
        {"name": "greedy_180x216x180_fast", "kind": "greedy", "nx": 180, "ny": 216, "nz": 180, "iters": 4,
         "hinv": False, "fast": True, "spacing": 1.0},
        # a wide volume, whose slabs are larger than one block's shared memory
        {"name": "fluid_256x256x160", "kind": "fluid", "nx": 256, "ny": 256, "nz": 160, "inverse": True,
         "spacing": 0.75},
        # LDMM relaxation at the benchmark's grid and time steps, the splatting gradient
        {"name": "ldmm_128_T10", "kind": "ldmm", "nx": 128, "ny": 128, "nz": 128, "T": 10, "orig": False,
         "spacing": 1.0},
        # LDMM with the Jacobian-transport gradient (the default of the original program), a ragged grid
        {"name": "ldmm_orig_100x90x75_T5", "kind": "ldmm", "nx": 100, "ny": 90, "nz": 75, "T": 5, "orig": True,
         "spacing": 1.5},
        # geodesic shooting with the adjoint gradient at the benchmark's grid
        {"name": "adshoot_128_T5", "kind": "adshoot", "nx": 128, "ny": 128, "nz": 128, "T": 5, "spacing": 1.0},
        # an atlas of subjects on uneven grids, the mean renewed every second iteration
        {"name": "atlas_128_6", "kind": "atlas", "nx": 128, "ny": 128, "nz": 128, "subjects": 6, "iters": 4,
         "period": 2},
        # a pair's warm start: the network at half the pair's grid
        {"name": "predict_128", "kind": "predict", "nx": 128, "ny": 128, "nz": 128},
        # training on downsampled pairs, one pair a step
        {"name": "train_64", "kind": "train", "nx": 64, "ny": 64, "nz": 64},
    ]


def _axis(rng, lo, hi):
    """An axis length, even over its logarithm: half of them multiples of 8, a quarter even, a quarter any."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    u = rng.random()
    m = 8 if u < 0.5 else (2 if u < 0.75 else 1)
    return max(lo, min(hi, (n + m // 2) // m * m))


def _grid(rng, lo, hi, voxels):
    while True:
        nx, ny, nz = (_axis(rng, lo, hi) for _ in range(3))
        if nx * ny * nz <= voxels:
            return {"nx": nx, "ny": ny, "nz": nz}


def draw(rng):
    kind = rng.choice(["fluid", "greedy", "greedy", "greedy", "ldmm", "ldmm", "adshoot", "atlas", "predict", "train"])
    spacing = rng.choice([1.0, 0.75, 1.25, 1.5])
    if kind == "fluid":
        return {"kind": kind, **_grid(rng, 16, 288, 10_000_000), "inverse": rng.random() < 0.8, "spacing": spacing}
    if kind == "greedy":
        return {"kind": kind, **_grid(rng, 16, 216, 7_000_000), "iters": rng.randint(2, 4), "hinv": rng.random() < 0.3,
                "fast": rng.random() < 0.25, "spacing": spacing}
    if kind == "ldmm":
        return {"kind": kind, **_grid(rng, 16, 144, 2_100_000), "T": rng.randint(3, 10), "orig": rng.random() < 0.5,
                "spacing": spacing}
    if kind == "adshoot":
        return {"kind": kind, **_grid(rng, 16, 144, 2_100_000), "T": rng.randint(2, 5), "spacing": spacing}
    if kind == "atlas":
        return {"kind": kind, **_grid(rng, 48, 144, 2_100_000), "subjects": rng.randint(2, 6), "iters": rng.randint(2, 4),
                "period": rng.randint(1, 2)}
    lo, hi = (4, 16) if kind == "predict" else (4, 8)
    f = 16 if kind == "predict" else 8  # the network's axes are multiples of 8, its pairs twice as long
    while True:
        n = [rng.randint(lo // 2 if f == 16 else lo, hi // (2 if f == 16 else 1)) * f for _ in range(3)]
        if n[0] * n[1] * n[2] <= (2_100_000 if f == 16 else 262_144):
            return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2]}


# ---- inputs ------------------------------------------------------------------
def _shape(c):
    return (c["nz"], c["ny"], c["nx"])


def _coords(shape):
    return torch.meshgrid(*(torch.arange(n, device="cuda", dtype=torch.float64) for n in shape), indexing="ij")


def _smooth(shape, gen, umax, sigma=8.0, comps=3):
    """Gaussian-filtered white noise, scaled to a largest vector of umax voxels."""
    w = torch.randn((comps,) + tuple(shape), generator=gen, device="cuda")
    k = [torch.fft.fftfreq(shape[0], device="cuda")[:, None, None], torch.fft.fftfreq(shape[1], device="cuda")[None, :, None],
         torch.fft.rfftfreq(shape[2], device="cuda")[None, None, :]]
    g = torch.exp(-2.0 * (math.pi * sigma) ** 2 * (k[0] ** 2 + k[1] ** 2 + k[2] ** 2))
    u = torch.fft.irfftn(torch.fft.rfftn(w, dim=(1, 2, 3)) * g, s=tuple(shape), dim=(1, 2, 3))
    return u * (umax / u.square().sum(0).sqrt().max())


def _blobs(shape, gen, count, at=None):
    """Gaussian blobs of sigma 4 to 10 voxels (in a grid of 64; larger and smaller in proportion), clipped to [0, 1];
    at: positions (z, y, x) in voxels to sample them at, the voxels themselves without it."""
    z, y, x = at if at is not None else _coords(shape)
    r = torch.rand((count, 5), generator=gen, device="cuda", dtype=torch.float64).cpu().numpy()
    scale = min(shape) / 64.0
    img = torch.zeros_like(z)
    for cz, cy, cx, s, a in r:
        s = (4.0 + 6.0 * s) * max(scale, 0.3)
        c = [(0.15 + 0.7 * q) * (n - 1) for q, n in zip((cz, cy, cx), shape)]
        img += (0.3 + 0.7 * a) * torch.exp(-((z - c[0]) ** 2 + (y - c[1]) ** 2 + (x - c[2]) ** 2) / (2 * s * s))
    return img.clamp_(0.0, 1.0)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _pair(shape, seed, umax=3.0, noise=0.02):
    """(I0, I1): blobs, and the blobs seen through a smooth displacement with a little noise."""
    gen = _gen(seed)
    u = _smooth(shape, gen, umax).double()
    z, y, x = _coords(shape)
    state = gen.get_state()
    I0 = _blobs(shape, gen, 8)
    gen.set_state(state)
    I1 = _blobs(shape, gen, 8, (z + u[2], y + u[1], x + u[0]))
    n = torch.randn((2,) + tuple(shape), generator=gen, device="cuda")
    return (I0.float() + noise * n[0]).contiguous(), (I1.float() + noise * n[1]).contiguous(), u.float().contiguous()


def _spacing(c):
    # not the same along the three axes, as a scanner's slices are not
    s = c.get("spacing", 1.0)
    return (s, s, 1.0 if s == 1.0 else 1.25 * s)


def _force(c, seed):
    """A registration's body force grad(I0) (I1 - I0)."""
    I0, I1, _ = _pair(_shape(c), seed)
    return (_gradient(I0.double(), _spacing(c)) * (I1 - I0)).float().contiguous()


def _velocities(c, seed):
    gen = _gen(seed + 500)
    return torch.stack([_smooth(_shape(c), gen, 0.4) for _ in range(c["T"])]).contiguous()


def _momentum(c, seed, I0):
    """A momentum whose initial velocity K(grad(I0) alpha0) is at most 0.4 voxel."""
    a = _smooth(_shape(c), _gen(seed + 700), 1.0, comps=1)[0].double()
    v = _K(_gradient(I0.double(), _spacing(c)) * a, _spacing(c))
    return (a * (0.4 / v.square().sum(0).sqrt().max())).float().contiguous()


def _atlas_inputs(c, seed):
    rng = np.random.default_rng(int(seed) + 9)
    gen = _gen(seed)
    state = gen.get_state()
    images = []
    for i in range(c["subjects"]):
        shape = tuple(int(v) for v in rng.choice(ATLAS_AXES, 3))
        u = _smooth(shape, _gen(31 * seed + i), 5.0).double()
        z, y, x = _coords(shape)
        gen.set_state(state)
        img = _blobs(shape, gen, 24, (z + u[2], y + u[1], x + u[0])) * float(rng.uniform(0.9, 1.1))
        images.append(img.float().contiguous())
    return images


def _net_shape(c):
    return tuple(n // 2 for n in _shape(c)) if c["kind"] == "predict" else _shape(c)


def _load_trained(net):
    """The committed weights for 128^3 pairs (convolutions: any grid of the network's takes them)."""
    warmstart.load_weights(net, os.path.join(os.path.dirname(warmstart.__file__), "data", warmstart.TRAINED[128][0]))


# ---- the cases ---------------------------------------------------------------
def prepare(c, seed):
    kind, shape, size = c["kind"], _shape(c), (c["nx"], c["ny"], c["nz"])
    sp = _spacing(c)
    op = DiffOperParam(ALPHA, BETA, GAMMA)
    if kind == "fluid":
        K = DiffOperB200()
        K.SetSize(size, sp, op)
        f = _force(c, seed)
        return {"c": c, "K": K, "f": f, "v": torch.empty_like(f)}
    if kind == "greedy":
        I0, I1, _ = _pair(shape, seed)
        it = GreedyIteratorB200(size, spacing=sp)
        it.SetScaleLevel(size, sp, GreedyIteratorParam(op, MAX_PERT))
        if c["fast"]:
            it.SetFastInterpolation(True)
        return {"c": c, "it": it, "data": GreedyDeformationDataB200(I0, I1, sp, c["hinv"])}
    if kind == "ldmm":
        I0, I1, _ = _pair(shape, seed)
        it = LDMMIteratorB200(size, spacing=sp, n_time_steps=c["T"])
        it.SetUseOrigGradientCalc(c["orig"])
        it.SetScaleLevel(size, sp, LDMMIteratorParam(op, LDMM_SIGMA, LDMM_STEP, False))
        return {"c": c, "it": it, "data": LDMMDeformationDataB200(I0, I1, c["T"], sp), "V": _velocities(c, seed)}
    if kind == "adshoot":
        I0, I1, _ = _pair(shape, seed)
        it = LDMMAdShootingIteratorB200(size, spacing=sp, n_time_steps=c["T"])
        it.SetScaleLevel(size, sp, LDMMIteratorParam(op, SHOOT_SIGMA, SHOOT_STEP, False))
        data = LDMMShootingDefDataB200(I0, I1, sp)
        it.Iterate(data)  # the handle's buffers, as after a registration's first iteration
        return {"c": c, "it": it, "data": data, "alpha0": _momentum(c, seed, I0)}
    if kind == "atlas":
        p = GreedyAtlasParam(op, MAX_PERT, c["iters"], c["period"])
        z, y, x = _coords(shape)
        return {"c": c, "builder": GreedyAtlasBuilderB200(_atlas_inputs(c, seed), size, p),
                "id": torch.stack([x, y, z]).float().contiguous()}
    net = warmstart.WarmStartNet(_net_shape(c), seed=3)
    if kind == "predict":
        _load_trained(net)
        I0, I1, _ = _pair(shape, seed)
        return {"c": c, "net": net, "predictor": warmstart.WarmStartPredictor(net, shape), "I0": I0, "I1": I1}
    I0, I1, u = _pair(shape, seed)
    return {"c": c, "net": net, "I0": I0, "I1": I1, "target": u}


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind == "fluid":
        # the operator works in place, and the force is kept
        state["v"].copy_(state["f"])
        K = state["K"]
        return K.ApplyInverseOperator(state["v"]) if c["inverse"] else K.ApplyOperator(state["v"])
    if kind == "greedy":
        data = state["data"]
        data.SetToIdentity()
        state["it"].Run(data, c["iters"], update_first=True)
        return [data.Def1To0(), data.Def0To1()] if c["hinv"] else [data.Def1To0()]
    if kind == "ldmm":
        state["data"].V.copy_(state["V"])
        state["it"].Run(state["data"], 1)
        return state["data"].V
    if kind == "adshoot":
        data = state["data"]
        data.Alpha0.copy_(state["alpha0"])
        state["it"].Iterate(data)
        return [data.Alpha0, data.GetDef0To1(), data.GetDef1To0()]
    if kind == "atlas":
        b = state["builder"]
        for i in range(c["subjects"]):
            b.GetDeformationField(i).copy_(state["id"])
        mean = b.BuildAtlas()
        # copies: the builder's own tensors are views of its handle's memory, which goes with it
        return [mean.clone()] + [b.GetDeformationField(i).clone() for i in range(c["subjects"])]
    net = state["net"]
    if kind == "predict":
        h = state["predictor"](state["I0"], state["I1"])
        return {"h": h, "displacement": net.out}
    loss = net.train_step(state["I0"], state["I1"], state["target"])
    return {"loss": loss, "w": net.gw, "b": net.gb}


def _conv_flops(shape):
    v = shape[0] * shape[1] * shape[2]
    level = {"e0": 0, "e1": 1, "e2": 2, "e3": 3, "d2": 2, "d1": 1, "d0": 0, "he": 0}
    return sum(2.0 * (v / 8 ** level[n[:2]]) * ci * co * t for n, ci, co, t in warmstart.LAYERS)


def work(c):
    """Bytes: each field and image that an iteration's stages exchange, once in and once out (float32; the
    half spectrum counted as the field's own 12 bytes a voxel, twice, where a transform is part of the pass)."""
    n = float(c["nx"] * c["ny"] * c["nz"])
    kind = c["kind"]
    if kind == "fluid":
        return {"bytes": 24.0 * n, "flops": 0.0}
    if kind == "greedy":  # images 8, h in and out 24, spectrum out, in and out, in 48; h^-1 in and out 24
        return {"bytes": (80.0 + (24.0 if c["hinv"] else 0.0)) * n * c["iters"], "flops": 0.0}
    if kind == "ldmm":  # a time step: v in and out 24, two maps 48, image and residual 12, spectrum 48
        return {"bytes": 132.0 * n * c["T"], "flops": 0.0}
    if kind == "adshoot":  # a time step: two solves of 48 + 24, four maps 48, six images 24, splats 24
        return {"bytes": 240.0 * n * c["T"], "flops": 0.0}
    if kind == "atlas":
        return {"bytes": 80.0 * n * c["iters"] * c["subjects"], "flops": 0.0}
    f = _conv_flops(_net_shape(c))
    if kind == "predict":
        return {"bytes": 20.0 * n, "flops": f}
    return {"bytes": 20.0 * n + 16.0 * warmstart.n_parameters(), "flops": 3.0 * f}


def tolerance(c):
    """About four times the distance from the 64-bit result: 2e-7 for a transform, 1e-7 for fields and maps. The largest
    single difference is that of a voxel whose sample point crosses a cell's face."""
    kind = c["kind"]
    if kind == "fluid":
        return {"rel": 2e-6, "max": 5e-5}
    if kind in ("greedy", "atlas", "ldmm", "adshoot"):
        return {"rel": 1e-6, "max": 2e-4}
    # bf16 activations through 15 layers, and their gradients back
    return {"rel": 3e-2, "max": 0.5}


# ---- 64-bit references -------------------------------------------------------
def _f32(x):
    return float(np.float32(x))


def _K(f, sp, inverse=True):
    """L^-1 f (or L f), L = -alpha Lap - beta grad div + gamma with the operator's discrete symbols."""
    shape = f.shape[1:]
    F = torch.fft.rfftn(f, dim=(1, 2, 3))
    a, b, g = _f32(ALPHA), _f32(BETA), _f32(GAMMA)
    c, s = [], []
    for axis, (n, h) in enumerate(zip(shape[::-1], sp)):  # x, y, z
        m = n // 2 + 1 if axis == 0 else n
        w = 2.0 * math.pi * torch.arange(m, device="cuda", dtype=torch.float64) / n
        view = [1, 1, 1]
        view[2 - axis] = m
        c.append(((2.0 * torch.cos(w) - 2.0) / (h * h)).view(view))
        s.append((torch.sin(w) / h).view(view))
    lam = g - a * (c[0] + c[1] + c[2])
    L00, L11, L22 = lam - b * c[0], lam - b * c[1], lam - b * c[2]
    L10, L20, L21 = b * s[0] * s[1], b * s[0] * s[2], b * s[1] * s[2]
    if inverse:
        A, B, C = L11 * L22 - L21 * L21, L21 * L20 - L10 * L22, L10 * L21 - L11 * L20
        D, E, G = L00 * L22 - L20 * L20, L10 * L20 - L00 * L21, L00 * L11 - L10 * L10
        det = L00 * A + L10 * B + L20 * C
        out = [(A * F[0] + B * F[1] + C * F[2]) / det, (B * F[0] + D * F[1] + E * F[2]) / det,
               (C * F[0] + E * F[1] + G * F[2]) / det]
    else:
        out = [L00 * F[0] + L10 * F[1] + L20 * F[2], L10 * F[0] + L11 * F[1] + L21 * F[2],
               L20 * F[0] + L21 * F[1] + L22 * F[2]]
    return torch.fft.irfftn(torch.stack(out), s=shape, dim=(1, 2, 3))


def _gradient(a, sp):
    """Central differences, one-sided at the borders: x, y, z."""
    out = []
    for axis, h in zip((2, 1, 0), sp):
        n = a.shape[axis]
        g = torch.empty_like(a)
        g.narrow(axis, 1, n - 2).copy_((a.narrow(axis, 2, n - 2) - a.narrow(axis, 0, n - 2)) / (2.0 * h))
        g.narrow(axis, 0, 1).copy_((a.narrow(axis, 1, 1) - a.narrow(axis, 0, 1)) / h)
        g.narrow(axis, n - 1, 1).copy_((a.narrow(axis, n - 1, 1) - a.narrow(axis, n - 2, 1)) / h)
        out.append(g)
    return torch.stack(out)


def _corners(p, shape):
    """(weight, inside, flat index, corner coordinates) of the eight corners around positions p (x, y, z)."""
    f = torch.floor(p)
    t = p - f
    f = f.clamp(-2.0, 4096.0).long()
    n = shape[::-1]
    for k in range(8):
        d = (k & 1, k >> 1 & 1, k >> 2)
        w, ok, q = 1.0, True, []
        for a in range(3):
            i = f[a] + d[a]
            w = w * (t[a] if d[a] else 1.0 - t[a])
            ok = ok & (i >= 0) & (i < n[a])
            q.append(i)
        at = (q[2].clamp(0, n[2] - 1) * n[1] + q[1].clamp(0, n[1] - 1)) * n[0] + q[0].clamp(0, n[0] - 1)
        yield w, ok, at, q


def _sample(img, p):
    out = torch.zeros_like(p[0])
    for w, ok, at, _ in _corners(p, img.shape):
        out += torch.where(ok, w, 0.0) * img.reshape(-1)[at]
    return out


def _sample_field(h, p, identity):
    """A vector field at p; outside the volume the corner's own place (identity) or zero."""
    out = torch.zeros_like(p)
    for w, ok, at, q in _corners(p, h.shape[1:]):
        for a in range(3):
            out[a] += w * torch.where(ok, h[a].reshape(-1)[at], q[a].double() if identity else 0.0)
    return out


def _splat(img, h):
    out = torch.zeros(img.numel(), device="cuda", dtype=torch.float64)
    for w, ok, at, _ in _corners(h, img.shape):
        out.index_add_(0, at.reshape(-1), (torch.where(ok, w, 0.0) * img).reshape(-1))
    return out.view(img.shape)


def _identity(shape):
    z, y, x = _coords(shape)
    return torch.stack([x, y, z])


def _col(sp):
    return torch.tensor(sp, device="cuda", dtype=torch.float64).view(3, 1, 1, 1)


def _exact_greedy_step(I, target, h, eps, sp, point=None):
    J = _sample(I, h if point is None else point(h))
    v = _K(_gradient(J, sp) * (target - J), sp)
    if eps is None:
        eps = _f32(MAX_PERT) / v.square().sum(0).sqrt().max()
    return _sample_field(h, _identity(target.shape) + eps * v / _col(sp), True), v, eps


def _exact_greedy(c, seed):
    shape, sp = _shape(c), _spacing(c)
    I0, I1, _ = (t.double() for t in _pair(shape, seed))
    h, hinv, eps = _identity(shape), _identity(shape), None
    for _ in range(c["iters"]):
        h, v, eps = _exact_greedy_step(I0, I1, h, eps, sp)
        if c["hinv"]:
            hinv = hinv - _sample_field(eps * v, hinv, False) / _col(sp)
    return [h, hinv] if c["hinv"] else [h]


def _exact_ldmm(c, seed):
    shape, sp, T = _shape(c), _spacing(c), c["T"]
    I0, I1, _ = (t.double() for t in _pair(shape, seed))
    V = _velocities(c, seed).double()
    eps, sg = _f32(LDMM_STEP), _f32(LDMM_SIGMA)
    vfac, ufac, ident, s = 1.0 - 2.0 * eps, 2.0 * eps / (sg * sg), _identity(shape), _col(sp)
    h = ident
    if not c["orig"]:
        J = []
        for t in range(T):
            h = _sample_field(h, ident - V[t] / s, True)
            J.append(_sample(I0, h))
        diff, h = J[-1] - I1, ident
        for t in range(T - 1, -1, -1):
            h = h - _sample_field(V[t], h, False) / s
            G = J[t - 1] if t else I0
            V[t] = vfac * V[t] + ufac * _K(_gradient(G, sp) * _splat(diff, h), sp)
        return V
    JT, JD = [None] * T, [None] * T
    for t in range(T - 1, -1, -1):
        p = ident + V[t] / s
        h = _sample_field(h, p, True)
        JT[t] = _sample(I1, h)
        g = [_gradient(ident[a] * sp[a] + V[t][a], sp) for a in range(3)]
        det = (g[0][0] * (g[1][1] * g[2][2] - g[1][2] * g[2][1]) - g[0][1] * (g[1][0] * g[2][2] - g[1][2] * g[2][0])
               + g[0][2] * (g[1][0] * g[2][1] - g[1][1] * g[2][0]))
        JD[t] = det if t == T - 1 else _sample(JD[t + 1], p) * det
    h, S = ident, I0
    for t in range(T):
        V[t] = vfac * V[t] + ufac * _K(_gradient(S, sp) * ((S - JT[t]) * JD[t]), sp)
        h = _sample_field(h, ident - V[t] / s, True)
        S = _sample(I0, h)
    return V


def _exact_adshoot(c, seed):
    shape, sp, T = _shape(c), _spacing(c), c["T"]
    I0f, I1, _ = _pair(shape, seed)
    I0, I1, a0 = I0f.double(), I1.double(), _momentum(c, seed, I0f).double()
    ident, s = _identity(shape), _col(sp)
    p0, p1, V, A, I = [ident], [ident], [], [a0], [I0]
    for t in range(T):
        V.append(-_K(_gradient(I[t], sp) * A[t], sp))
        p0.append(p0[t] + _sample_field(V[t], p0[t], False) / s)
        p1.append(_sample_field(p1[t], ident - V[t] / s, True))
        A.append(_splat(a0, p0[-1]))
        I.append(_sample(I0, p1[-1]))
    IHat = (I1 - I[T]) / (_f32(SHOOT_SIGMA) ** 2)
    ITil, aTil = _splat(IHat, p1[T]), torch.zeros_like(I0)
    for t in range(T, 0, -1):
        gI = _gradient(I[t], sp)
        vh = _K(_gradient(_sample(aTil, p1[t]), sp) * A[t] - gI * _splat(ITil, p0[t]), sp)
        div = sum(_gradient(vh[a] * A[t], sp)[a] for a in range(3))
        aTil = aTil - _sample((gI * vh).sum(0), p0[t])
        ITil = ITil + _splat(div, p1[t])
    a = a0 - _f32(SHOOT_STEP) * (-(_gradient(I0, sp) * V[0]).sum(0) - aTil)
    return [a, p0[1], p1[1]]


def _exact_atlas(c, seed):
    shape, sp = _shape(c), (1.0, 1.0, 1.0)
    images = [i.double() for i in _atlas_inputs(c, seed)]
    w = _f32(1.0 / len(images))

    def point(img):
        r = torch.tensor([m / n for m, n in zip(img.shape[::-1], shape[::-1])], device="cuda", dtype=torch.float64)
        return lambda h: (h + 0.5) * r.view(3, 1, 1, 1) - 0.5

    h, eps = [_identity(shape) for _ in images], [None] * len(images)
    mean = sum(w * _sample(i, point(i)(q)) for i, q in zip(images, h))
    for k in range(c["iters"]):
        for j, img in enumerate(images):
            h[j], _, eps[j] = _exact_greedy_step(img, mean, h[j], eps[j], sp, point(img))
        if (k + 1) % c["period"] == 0:
            mean = sum(w * _sample(i, point(i)(q)) for i, q in zip(images, h))
    return [mean] + h


def _exact_forward(net, I0, I1, params):
    """The network with its bf16 weights and 64-bit activations; returns the head's [16, D, H, W]."""
    F = torch.nn.functional

    def conv(name, x, relu=True):
        w, b = params[name]
        y = F.conv3d(x, w, b, padding=1 if w.shape[2] == 3 else 0)
        return torch.relu(y) if relu else y

    def up(x):
        return F.interpolate(x, scale_factor=2, mode="nearest")

    x = torch.zeros((1, 16) + tuple(I0.shape), device="cuda", dtype=torch.float64)
    x[0, 0], x[0, 1] = I0, I1
    e0 = conv("e0b", conv("e0a", x))
    e1 = conv("e1b", conv("e1a", F.avg_pool3d(e0, 2)))
    e2 = conv("e2b", conv("e2a", F.avg_pool3d(e1, 2)))
    e3 = conv("e3b", conv("e3a", F.avg_pool3d(e2, 2)))
    d2 = conv("d2b", conv("d2a", torch.cat([up(e3), e2], 1)))
    d1 = conv("d1b", conv("d1a", torch.cat([up(d2), e1], 1)))
    d0 = conv("d0b", conv("d0a", torch.cat([up(d1), e0], 1)))
    return conv("head", d0, False)[0]


def _exact_params(net, grad):
    out = {}
    for name, ci, co, t in warmstart.LAYERS:
        k = 3 if t == 27 else 1
        w = net.w[name].bfloat16().double().view(co, k, k, k, ci).permute(0, 4, 1, 2, 3).contiguous()
        out[name] = (w.requires_grad_(grad), net.b[name].double().clone().requires_grad_(grad))
    return out


def _half(a):
    """A Gaussian of sigma 1 (two taps a side, weights renormalised at the borders), then the half-size grid's centres."""
    k = torch.exp(-0.5 * torch.arange(-2, 3, device="cuda", dtype=torch.float64) ** 2)
    for axis in range(3):
        n = a.shape[axis]
        num, den = torch.zeros_like(a), torch.zeros(n, device="cuda", dtype=torch.float64)
        for i, w in enumerate(k.tolist()):
            lo, hi = max(0, 2 - i), min(n, n + 2 - i)
            num.narrow(axis, lo, hi - lo).add_(a.narrow(axis, lo + i - 2, hi - lo), alpha=w)
            den[lo:hi] += w
        view = [1, 1, 1]
        view[axis] = n
        a = num / den.view(view)
    return torch.nn.functional.avg_pool3d(a[None, None], 2)[0, 0]


def _exact_net(c, seed):
    net = warmstart.WarmStartNet(_net_shape(c), seed=3)
    if c["kind"] == "predict":
        _load_trained(net)
        with torch.no_grad():
            I0, I1, _ = _pair(_shape(c), seed)
            u = _exact_forward(net, _half(I0.double()), _half(I1.double()), _exact_params(net, False))
        p = (_identity(_shape(c)) - 0.5) / 2.0  # the fine voxels' centres on the coarse grid
        lim = torch.tensor([n - 1.0 for n in u.shape[:0:-1]], device="cuda", dtype=torch.float64).view(3, 1, 1, 1)
        p = torch.minimum(p.clamp(min=0.0), lim)
        h = _identity(_shape(c)) + 2.0 * torch.stack([_sample(u[a], p) for a in range(3)])
        return {"h": h, "displacement": u.permute(1, 2, 3, 0).reshape(-1, 16)}
    with torch.enable_grad():
        params = _exact_params(net, True)
        I0, I1, u = (t.double() for t in _pair(_shape(c), seed))
        loss = (_exact_forward(net, I0, I1, params)[:3] - u).square().mean()
        loss.backward()
    gw = {n: w.grad.permute(0, 2, 3, 4, 1).reshape(w.shape[0], -1, w.shape[1]).contiguous() for n, (w, _) in params.items()}
    return {"loss": loss.detach().reshape(1), "w": gw, "b": {n: b.grad for n, (_, b) in params.items()}}


def exact(c, seed):
    kind = c["kind"]
    if kind == "fluid":
        return _K(_force(c, seed).double(), _spacing(c), c["inverse"])
    return {"greedy": _exact_greedy, "ldmm": _exact_ldmm, "adshoot": _exact_adshoot, "atlas": _exact_atlas,
            "predict": _exact_net, "train": _exact_net}[kind](c, seed)
