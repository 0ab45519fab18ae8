"""
The performance cases of this package: the calls that a segmentation program
makes, at the sizes and options of the repository's own configurations, tests
and benchmark.

Inputs are built on the GPU from the seed: an analytic helix (axis along array
axis 0) with additive Gaussian noise, its capacities, |grad I|^2 and the
squeezed quaternions of the helix frames, as the benchmark's configurations
define them.  Weightings stay in the lower part of the experiment's grid (and
lower still for isotropic TV and thin tubes): above it the relaxed labelling
of the noisier volumes collapses to zero and the outputs would be rounding
noise.
"""
from __future__ import annotations

import contextlib
import io
import math

import numpy as np
import torch

from miccai2016_gb300.adjust_directions import AdvancedAdjuster
from miccai2016_gb300.batched import BatchedCut
from miccai2016_gb300.continuous_cut_anisotropic_gpu import CmfCutQAnisotropicGpu
from miccai2016_gb300.gradient_vector_flow import GvfGpu, GvfParameters, time_step_for
from miccai2016_gb300.qfrangi_gpu import FeatureFilter, VesselnessCalculation
from miccai2016_gb300.serving import CutServer

ATV = (1.0, 10 ** -1.5, 10 ** -1.5)
TV = (1.0, 1.0, 1.0)
LARGEST = 256 ** 3 * 1000   # voxel-iterations of the largest cut


def listed():
    return [
        # the headline solve: one large volume, a fixed number of iterations, a residual every 30
        {"name": "cut-256", "kind": "cut", "d0": 256, "d1": 256, "d2": 256, "sigma": 1.0, "cut": "atv",
         "weighting": 10 ** -1.25, "decay": 10 ** 1.5, "iterations": 1000, "update": 30, "bound": -1.0, "aniso": False},
        # the plain 64^3 solve: launches and latency
        {"name": "cut-64", "kind": "cut", "d0": 64, "d1": 64, "d2": 64, "sigma": 1.5, "cut": "atv",
         "weighting": 10 ** -1.25, "decay": 10 ** 1.5, "iterations": 300, "update": 30, "bound": -1.0, "aniso": False},
        # the default CutParameters (residual after every iteration, stop at 1e-4) on an odd volume with
        # anisotropic voxels, isotropic TV: the second half of the experiment's loop
        {"name": "cut-tv-default", "kind": "cut", "d0": 97, "d1": 161, "d2": 203, "sigma": 0.7, "cut": "tv",
         "weighting": 0.05, "decay": 10.0, "iterations": 1000, "update": 1, "bound": 1e-4, "aniso": True},
        # supervised cut with per-voxel eigenvalues and a scalar TV weight
        {"name": "cut-seeded", "kind": "seeded", "d0": 80, "d1": 111, "d2": 130, "sigma": 0.8, "alpha": 0.1,
         "iterations": 200, "update": 10},
        # the (weighting, decay) grid search of one volume, anisotropic and isotropic at every grid point
        {"name": "grid-128", "kind": "grid", "d0": 128, "d1": 128, "d2": 128, "sigma": 1.5, "points": 16},
        # uneven volumes and noise levels cut together at one (weighting, decay)
        {"name": "ragged-8", "kind": "ragged", "volumes": 8, "weighting": 10 ** -1.25, "decay": 10 ** 1.5},
        # requests of uneven sizes handed to the server at once, from host memory and back
        {"name": "served-10", "kind": "served", "requests": 10, "low": 64, "high": 208},
        # vesselness at three scales, c from the image (the pipeline's first stage)
        {"name": "frangi-256", "kind": "frangi", "d0": 256, "d1": 256, "d2": 256, "sigma": 1.0, "low": 1.0,
         "high": 3.0, "scales": 3, "c": 0.0, "bright": True, "aniso": False},
        # dark tubes, a given c, anisotropic voxels, a small odd volume, wider kernels
        {"name": "frangi-small", "kind": "frangi", "d0": 45, "d1": 61, "d2": 83, "sigma": 0.3, "low": 2.0,
         "high": 6.0, "scales": 3, "c": 0.4, "bright": False, "aniso": True},
        # direction smoothing as the pipeline runs it
        {"name": "gvf-256", "kind": "gvf", "d0": 256, "d1": 256, "d2": 256, "mu": 0.2, "iterations": 100,
         "update": 10, "response": False, "normalize": False, "aniso": False},
        # with a response field, unit-length output, anisotropic voxels, the experiment's mu, odd sides
        {"name": "gvf-odd", "kind": "gvf", "d0": 75, "d1": 93, "d2": 110, "mu": 10 ** 0.5, "iterations": 300,
         "update": 30, "response": True, "normalize": True, "aniso": True},
        # sign adjustment of the vesselness directions, host arrays in and out
        {"name": "adjust-128", "kind": "adjust", "d0": 128, "d1": 128, "d2": 128},
    ]


def _side(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _shape(rng, low, high):
    return {"d0": _side(rng, low, high), "d1": _side(rng, low, high), "d2": _side(rng, low, high)}


def draw(rng):
    kind = rng.choice(["cut", "cut", "cut", "seeded", "grid", "ragged", "served", "frangi", "gvf", "adjust"])
    case = {"kind": kind}
    if kind == "cut":
        case.update(_shape(rng, 24, 288))
        n = case["d0"] * case["d1"] * case["d2"]
        update = rng.choice([1, 5, 7, 10, 30])
        stop = rng.random() < 0.4
        cut = rng.choice(["atv", "tv"])
        case.update(sigma=round(rng.uniform(0.3, 1.0), 2), cut=cut, weighting=0.03 if cut == "atv" else 0.01,
                    decay=10 ** 1.5, update=update, bound=1e-4 if stop else -1.0,
                    iterations=1000 if stop else min(int(LARGEST / n), rng.randint(100, 1000)),
                    aniso=rng.random() < 0.3)
    elif kind == "seeded":
        case.update(_shape(rng, 24, 160))
        case.update(sigma=round(rng.uniform(0.3, 1.2), 2), alpha=round(rng.uniform(0.05, 0.2), 3),
                    iterations=rng.randint(50, 300), update=rng.choice([5, 10, 30]))
    elif kind == "grid":
        case.update(_shape(rng, 48, 144))
        case.update(sigma=round(rng.uniform(0.5, 1.5), 2), points=rng.randint(2, 24))
    elif kind == "ragged":
        case.update(volumes=rng.randint(2, 16), weighting=10 ** -1.25, decay=10 ** 1.5)
    elif kind == "served":
        case.update(requests=rng.randint(2, 12), low=64, high=rng.randint(100, 208))
    elif kind == "frangi":
        case.update(_shape(rng, 20, 240))
        low = rng.choice([1.0, 1.5, 2.0])
        case.update(sigma=round(rng.uniform(0.2, 1.5), 2), low=low, high=low * rng.choice([2.0, 3.0]),
                    scales=rng.randint(1, 4), c=rng.choice([0.0, 0.4]), bright=rng.random() < 0.5,
                    aniso=rng.random() < 0.3)
    elif kind == "gvf":
        case.update(_shape(rng, 16, 256))
        case.update(mu=rng.choice([0.2, 10 ** 0.5]), iterations=rng.randint(20, 300), update=rng.choice([5, 10, 30]),
                    response=rng.random() < 0.5, normalize=rng.random() < 0.5, aniso=rng.random() < 0.3)
    else:
        case.update(_shape(rng, 40, 150))
    return case


# ---- inputs -------------------------------------------------------------------

def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _helix(shape, sigma, seed, radius=None, tube=None):
    """float64 CUDA tensors: the noisy image, the distance to the centreline and the unit tangent."""
    d0, d1, d2 = shape
    R = radius or 0.25 * min(d1, d2)
    r = tube or max(2.0, R / 5.0)
    a = 1.25 * R / (2 * math.pi)
    ax = [torch.arange(n, device="cuda", dtype=torch.float64) - (n - 1) / 2.0 for n in shape]
    z, y, x = ax[0].view(-1, 1, 1), ax[1].view(1, -1, 1), ax[2].view(1, 1, -1)
    rho = torch.sqrt(y * y + x * x)
    phi = torch.atan2(y, x)
    w = (z / a - phi) / (2 * math.pi)
    best = t_best = None
    for k in (torch.floor(w), torch.floor(w) + 1):
        t = phi + 2 * math.pi * k
        for _ in range(4):   # Newton on the distance's derivative
            s = t - phi
            g = a * (a * t - z) + R * rho * torch.sin(s)
            h = (a * a + R * rho * torch.cos(s)).clamp_min(0.5 * a * a)
            t = t - (g / h).clamp(-0.5, 0.5)
        d = (z - a * t) ** 2 + rho * rho + R * R - 2 * R * rho * torch.cos(t - phi)
        if best is None:
            best, t_best = d, t
        else:
            t_best = torch.where(d < best, t, t_best)
            best = torch.minimum(d, best)
    dist = best.clamp_min(0).sqrt()
    v = torch.stack([torch.full_like(t_best, a), R * torch.cos(t_best), -R * torch.sin(t_best)], -1)
    v /= math.hypot(a, R)
    img = (dist <= r).double() + sigma * torch.randn(shape, generator=_gen(seed, 1), device="cuda", dtype=torch.float64)
    return img, dist, v


def _squeeze(e0):
    """Squeezed quaternions (z-x-z Euler angles) of frames whose first column is the unit vector e0."""
    zero = torch.zeros_like(e0[..., 0])
    first = e0[..., 0].abs() > e0[..., 1].abs()
    e1 = torch.where(first[..., None], torch.stack([-e0[..., 2], zero, e0[..., 0]], -1),
                     torch.stack([zero, e0[..., 2], -e0[..., 1]], -1))
    e1 = e1 / e1.norm(dim=-1, keepdim=True).clamp_min(1e-300)
    e2 = torch.cross(e0, e1, dim=-1)
    m = lambda i, j: (e0, e1, e2)[j][..., i]
    half = lambda s: torch.sqrt(torch.clamp(s, min=0)) / 2
    w = half(1 + m(0, 0) + m(1, 1) + m(2, 2))
    x = torch.copysign(half(1 + m(0, 0) - m(1, 1) - m(2, 2)), m(2, 1) - m(1, 2))
    y = torch.copysign(half(1 - m(0, 0) + m(1, 1) - m(2, 2)), m(0, 2) - m(2, 0))
    z = torch.copysign(half(1 - m(0, 0) - m(1, 1) + m(2, 2)), m(1, 0) - m(0, 1))
    phi = torch.atan2(x * z + y * w, x * w - y * z)
    theta = torch.acos(torch.clamp(1 - 2 * (x * x + y * y), -1, 1))
    psi = torch.atan2(x * z - y * w, x * w + y * z)
    return torch.stack([phi, theta, psi], -1)


def _volume(shape, sigma, seed, radius=None, tube=None):
    """The cut inputs of one noisy helix volume, float32 CUDA tensors."""
    img, _, v = _helix(shape, sigma, seed, radius, tube)
    im = img.float().double()
    var = sigma * sigma
    norm = 1 / math.sqrt(2 * math.pi * var)
    pdf = lambda mean: torch.exp((im - mean) ** 2 / (-2 * var)) * norm
    ratio = torch.log((pdf(1) + 1e-9) / (pdf(0) + 1e-9)) / math.log((norm + 1e-9) / 1e-9)
    grad2 = sum(g ** 2 for g in torch.gradient(im))
    f = lambda t: t.float().contiguous()
    return {"img": f(im), "quats": f(_squeeze(v)), "cs": f(ratio.clamp_min(0)), "ct": f((-ratio).clamp_min(0)),
            "grad2": f(grad2)}


def _alpha(vol, weighting, decay):
    return weighting * torch.exp((-1.0 / decay ** 2) * vol["grad2"])


def _params(iterations, update, bound):
    p = CmfCutQAnisotropicGpu.CutParameters()
    p.num_iter, p.update, p.error_bound = iterations, update, bound
    return p


def _dims(case):
    return (case["d0"], case["d1"], case["d2"])


def _scaling(case):
    return (1.5, 0.7, 1.2) if case["aniso"] else (1.0, 1.0, 1.0)


def _cut_inputs(case, seed):
    vol = _volume(_dims(case), case["sigma"], seed)
    return vol, _alpha(vol, case["weighting"], case["decay"])


def _seeded_inputs(case, seed):
    """Seeds near the centreline (1) and far from it (2), eigenvalues drawn per voxel."""
    shape = _dims(case)
    _, dist, _ = _helix(shape, case["sigma"], seed)
    vol = _volume(shape, case["sigma"], seed)
    u = lambda salt, *s: torch.rand(s, generator=_gen(seed, salt), device="cuda", dtype=torch.float64)
    pick = u(2, *shape) < 0.02
    labels = torch.where(dist <= 1.5, 1, torch.where(dist > 8.0, 2, 0)) * pick
    eigs = torch.stack([torch.ones(shape, device="cuda", dtype=torch.float64), 0.02 + 0.2 * u(3, *shape),
                        0.02 + 0.2 * u(4, *shape)], -1)
    return vol, labels.to(torch.uint8), eigs


def _grid_inputs(case, seed):
    vol = _volume(_dims(case), case["sigma"], seed)
    g = np.random.RandomState(seed)
    pairs = [(float(_WEIGHTINGS[g.randint(11)]), float(_DECAYS[g.randint(17)])) for _ in range(case["points"])]
    return vol, [(w, d, eigs) for w, d in pairs for eigs in (ATV, TV)]


_WEIGHTINGS, _DECAYS = np.logspace(-2.5, -1.25, 11), np.logspace(-1, 3, 17)
_SHAPES = ((96, 96, 96), (128, 128, 192), (160, 160, 160), (224, 224, 160))


def _ragged_inputs(case, seed):
    g = np.random.RandomState(seed)
    vols = []
    for k in range(case["volumes"]):
        shape = _SHAPES[k % 4]
        vols.append(_volume(shape, float(g.uniform(0.1, 1.5)), seed * 100 + k,
                            radius=float(g.uniform(0.2, 0.3)) * min(shape), tube=float(g.uniform(2, 6))))
    return vols


def _served_inputs(case, seed):
    g = np.random.RandomState(seed)
    sides = np.random.RandomState(case["high"]).randint(case["low"], case["high"] + 1, size=(case["requests"], 3))
    out = []
    for k in range(case["requests"]):
        vol = _volume(tuple(int(s) for s in sides[k]), float(g.uniform(0.1, 1.0)), seed * 100 + k)
        out.append((vol, float(_WEIGHTINGS[g.randint(11)]), float(_DECAYS[g.randint(17)])))
    return out


def _gvf_inputs(case, seed):
    """Main directions times a vesselness-like weight, signs consistent near the helix only."""
    shape = _dims(case)
    _, dist, v = _helix(shape, 0.1, seed)
    sign = torch.where((torch.rand(shape, generator=_gen(seed, 5), device="cuda") < 0.5) & (dist > 4), -1.0, 1.0)
    noise = torch.randn(shape + (3,), generator=_gen(seed, 6), device="cuda", dtype=torch.float64)
    v = v + 0.3 * noise
    v = v / v.norm(dim=-1, keepdim=True)
    weight = torch.exp(-dist ** 2 / 18.0) + 0.05 * torch.rand(shape, generator=_gen(seed, 7), device="cuda")
    field = (v * (sign * weight)[..., None]).float().contiguous()
    return field, (weight.float().contiguous() if case["response"] else None)


def _smooth(t):
    """Three passes of a [1 2 1] / 4 filter along every axis."""
    for _ in range(3):
        for ax in range(3):
            t = (torch.roll(t, 1, ax) + 2 * t + torch.roll(t, -1, ax)) / 4
    return t


def _adjust_inputs(case, seed):
    """A vesselness-like response in [0, 1] (the tube over smoothed noise) and frames with random signs."""
    shape = _dims(case)
    _, dist, v = _helix(shape, 0.1, seed)
    noise = lambda salt: _smooth(torch.randn(shape, generator=_gen(seed, salt), device="cuda", dtype=torch.float64))
    resp = torch.exp(-dist ** 2 / 12.0) * (1 + 0.5 * noise(8)) + 0.4 * noise(9).clamp_min(0)
    resp = (resp - resp.min()) / (resp.max() - resp.min())
    rand = torch.stack([noise(10), noise(11), noise(12)], -1)
    rand = rand / rand.norm(dim=-1, keepdim=True).clamp_min(1e-9)
    e0 = v * torch.exp(-dist / 6.0)[..., None] + 0.6 * rand
    e0 = e0 / e0.norm(dim=-1, keepdim=True)
    sign = torch.where(torch.rand(shape, generator=_gen(seed, 13), device="cuda") < 0.5, -1.0, 1.0)
    return resp.float().cpu().numpy(), _squeeze(e0 * sign[..., None]).float().cpu().numpy()


def _vessel_params(case):
    p = VesselnessCalculation.Parameters()
    p.bright_objects = case["bright"]
    p.c = case["c"] or None
    p.scales = (case["low"], case["high"], case["scales"])
    return p


def _frangi_image(case, seed):
    img, _, _ = _helix(_dims(case), case["sigma"], seed)
    return (img if case["bright"] else 1.0 - img).float().contiguous()


def _gvf_params(case):
    p = GvfParameters()
    p.mu, p.tol, p.maxiter, p.callback = case["mu"], 0, case["iterations"], None
    p.update, p.normalize = case["update"], case["normalize"]
    return p


# ---- prepare and run ------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "cut":
        s["vol"], s["alpha"] = _cut_inputs(case, seed)
        s["cutter"] = CmfCutQAnisotropicGpu(_params(case["iterations"], case["update"], case["bound"]))
        s["eigs"] = ATV if case["cut"] == "atv" else TV
        del s["vol"]["grad2"]
    elif kind == "seeded":
        s["vol"], s["labels"], s["eigs"] = _seeded_inputs(case, seed)
        s["cutter"] = CmfCutQAnisotropicGpu(_params(case["iterations"], case["update"], -1.0))
    elif kind in ("grid", "ragged"):
        s["cut"] = BatchedCut(_params(3000, 30, 1e-4))
        if kind == "grid":
            vol, points = _grid_inputs(case, seed)
            vols = [vol]
            s["instances"] = [dict(volume=0, weighting=w, decay=d, eigs=e) for w, d, e in points]
        else:
            vols = _ragged_inputs(case, seed)
            s["instances"] = [dict(volume=k, weighting=case["weighting"], decay=case["decay"], eigs=ATV)
                              for k in range(len(vols))]
        s["volumes"] = [s["cut"].prepare_volume(v["img"], v["quats"], v["cs"], v["ct"], grad2=v["grad2"])
                        for v in vols]
    elif kind == "served":
        reqs = _served_inputs(case, seed)
        s["requests"] = [({k: t.cpu().pin_memory() for k, t in vol.items()}, w, d,
                          torch.empty(tuple(vol["img"].shape), dtype=torch.float32, pin_memory=True))
                         for vol, w, d in reqs]
        s["server"] = CutServer(workspace_bytes=12 << 30)
    elif kind == "frangi":
        s["img"] = _frangi_image(case, seed)
        s["filter"] = FeatureFilter(_vessel_params(case))
    elif kind == "gvf":
        s["field"], s["response"] = _gvf_inputs(case, seed)
        s["params"] = _gvf_params(case)
    else:
        s["response"], s["qeigs"] = _adjust_inputs(case, seed)
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "cut":
        v = s["vol"]
        return s["cutter"].execute(v["img"], v["quats"], s["eigs"], s["alpha"], v["cs"], v["ct"],
                                   scaling=_scaling(case), verbose=False)
    if kind == "seeded":
        v = s["vol"]
        return s["cutter"].execute(v["img"], v["quats"], s["eigs"], case["alpha"], v["cs"], v["ct"],
                                   labels=s["labels"], verbose=False)
    if kind in ("grid", "ragged"):
        return s["cut"].solve(s["volumes"], s["instances"])
    if kind == "served":
        server, todo = s["server"], list(enumerate(s["requests"]))
        left = len(todo)
        while left:
            while todo:
                tag, (inputs, w, d, u) = todo[0]
                if not server.admit(tag, inputs, w, d, ATV, u):
                    break
                todo.pop(0)
            server.step()
            left -= len(server.poll())
        return [u for _, _, _, u in s["requests"]]
    if kind == "frangi":
        val, quat, _ = s["filter"].execute_for(s["img"], None, voxel_size=_scaling(case))
        return {"vesselness": val, "quats": quat}
    if kind == "gvf":
        return GvfGpu(s["field"], s["params"], voxel_size=_scaling(case), response=s["response"]).execute()
    with contextlib.redirect_stdout(io.StringIO()):
        adjuster = AdvancedAdjuster((0.01, 0.3), s["qeigs"], s["response"], voxel_size=1)
        dirs = adjuster.execute(verbose=False)
    return {"dirs": dirs, "ridge": adjuster.ridge}


def work(case):
    """Inputs once, outputs once; operations per voxel and iteration as the method's formulas need them."""
    kind = case["kind"]
    n = case["d0"] * case["d1"] * case["d2"] if "d0" in case else 0
    cut = 75   # one max-flow iteration of one voxel
    if kind == "cut":
        its = case["iterations"] if case["bound"] < 0 else 150
        return {"bytes": 32 * n, "flops": cut * its * n}
    if kind == "seeded":
        return {"bytes": (4 + 12 + 24 + 8 + 1 + 4) * n, "flops": cut * case["iterations"] * n}
    if kind == "grid":
        return {"bytes": 28 * n + 4 * n * 2 * case["points"], "flops": cut * 250 * n * 2 * case["points"]}
    if kind == "ragged":
        n = sum(int(np.prod(_SHAPES[k % 4])) for k in range(case["volumes"]))
        return {"bytes": 32 * n, "flops": cut * 150 * n}
    if kind == "served":
        sides = np.random.RandomState(case["high"]).randint(case["low"], case["high"] + 1, size=(case["requests"], 3))
        n = int(sides.prod(axis=1).sum())
        return {"bytes": 32 * n, "flops": cut * 200 * n}
    if kind == "frangi":
        sigma = (case["low"] + case["high"]) / 2
        return {"bytes": 20 * n, "flops": case["scales"] * n * (30 * (8 * sigma + 1) + 500)}
    if kind == "gvf":
        return {"bytes": (24 + 4 * case["response"]) * n, "flops": 50 * case["iterations"] * n}
    return {"bytes": 32 * n, "flops": 1000 * n}


# ---- what the outputs are in 64 bits ---------------------------------------------

def _pad_diff(t, axis):
    """t[i + 1] - t[i] along axis, 0 at the last index."""
    out = torch.zeros_like(t)
    n = t.shape[axis]
    out.narrow(axis, 0, n - 1).copy_(t.narrow(axis, 1, n - 1) - t.narrow(axis, 0, n - 1))
    return out


def _rotation(quats):
    phi, theta, psi = quats.double().unbind(-1)
    pp, pm, th = (phi + psi) / 2, (phi - psi) / 2, theta / 2
    w, x = torch.cos(pp) * torch.cos(th), torch.cos(pm) * torch.sin(th)
    y, z = torch.sin(pm) * torch.sin(th), torch.sin(pp) * torch.cos(th)
    return [[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
            [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
            [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]]


def _cut64(vol, eigs, alpha, scaling, iterations, update, bound, labels=None):
    """The augmented-Lagrangian continuous max-flow with metric A = R diag(eigs) R^T; u in 64 bits."""
    cc, steps = 0.2, 0.11
    img, cs, ct = vol["img"].double(), vol["cs"].double(), vol["ct"].double()
    smin = min(scaling)
    rcc = 1 / (cc * smin ** 2)
    R = _rotation(vol["quats"])
    lam = [float(e) for e in eigs] if isinstance(eigs, tuple) else [e.contiguous() for e in eigs.unbind(-1)]
    A = {(i, j): sum(lam[k] * R[i][k] * R[j][k] for k in range(3)) for i in range(3) for j in range(i, 3)}
    I = {(i, j): sum(R[i][k] * R[j][k] / lam[k] for k in range(3)) for i in range(3) for j in range(i, 3)}
    del R
    s_off, t_off = 1.0, 0.0
    if labels is not None:
        s_off, t_off = ((labels & 2) == 0).double(), (labels & 1).double()
    u = img / (img.max() + float(np.finfo(np.float32).tiny))
    pt = torch.minimum(cs, ct)
    tmp = -u * rcc
    h = [torch.zeros_like(u) for _ in range(3)]
    sym = lambda M, i, j: M[(min(i, j), max(i, j))]
    for it in range(iterations):
        g = [_pad_diff(tmp, k).mul_(steps / scaling[k] * smin ** 2) for k in range(3)]
        for i in range(3):
            for j in range(3):
                h[i].addcmul_(sym(A, i, j), g[j])
        n2 = sum((1 if i == j else 2) * I[(i, j)] * h[i] * h[j] for i, j in I)
        norm = n2.clamp_min_(0).sqrt_()
        scale = torch.where(norm > alpha, alpha / norm, torch.ones_like(norm))
        div = torch.zeros_like(u)
        for k in range(3):
            h[k].mul_(scale)
            n = u.shape[k]
            part = h[k].narrow(k, 0, n - 1) / scaling[k]
            div.narrow(k, 0, n - 1).add_(part)
            div.narrow(k, 1, n - 1).sub_(part)
        ps = torch.minimum(cs, div + pt - rcc * (u - s_off))
        pt = torch.minimum(ct, -div + ps + rcc * (u - t_off))
        err = div - ps + pt
        u = u - err / rcc
        tmp = err - u * rcc
        if it % update == 0 and bound >= 0 and float(err.abs().mean()) / rcc < bound:
            break
    return u


def _gvf64(case, field, response):
    vs = _scaling(case)
    v = [c.contiguous() for c in field.double().unbind(-1)]
    r = response.double() if response is not None else v[0] ** 2 + v[1] ** 2 + v[2] ** 2
    mu, dt = case["mu"], float(time_step_for(vs, case["mu"], 3))

    def lap(c):
        out = torch.zeros_like(c)
        for k in range(3):
            n = c.shape[k]
            d = c.narrow(k, 1, n - 1) - c.narrow(k, 0, n - 1)
            f = 1 / vs[k] ** 2
            out.narrow(k, 0, n - 1).add_(d, alpha=f)
            out.narrow(k, 1, n - 1).sub_(d, alpha=f)
            out.narrow(k, 0, 1).add_(d.narrow(k, 0, 1), alpha=f)            # mirrored ends
            out.narrow(k, n - 1, 1).sub_(d.narrow(k, n - 2, 1), alpha=f)
        return out

    g = [torch.zeros_like(c) for c in v]
    for _ in range(case["iterations"]):
        g = [c - dt * (r * (c - w) - mu * lap(c)) for c, w in zip(g, v)]
    out = torch.stack(g, -1)
    if case["normalize"]:
        norm = out.norm(dim=-1, keepdim=True)
        out = torch.where(norm != 0, out / norm, out)
    return out


def _vesselness64(case, img):
    p = _vessel_params(case)
    vs = _scaling(case)
    img = img.double()
    best = torch.full_like(img, -float("inf"))

    def conv(t, sigma, order, axis):
        r = int(4 * sigma + 0.5)
        x = np.arange(-r, r + 1)
        g = np.exp(-0.5 * x ** 2 / sigma ** 2)
        g /= g.sum()
        taps = (g, g * -x / sigma ** 2, g * (x ** 2 - sigma ** 2) / sigma ** 4)[order] * sigma ** order
        n = t.shape[axis]
        out = torch.zeros_like(t)
        for j, w in zip(x, taps):
            m = np.abs(np.arange(n) - j) % max(2 * (n - 1), 1)
            m = np.where(m < n, m, 2 * (n - 1) - m)
            out.add_(t.index_select(axis, torch.from_numpy(m).cuda()), alpha=float(w))
        return out

    for scale in np.linspace(*p.scales):
        s = [scale / v for v in vs]
        z = [conv(img, s[0], o, 0) for o in range(3)]
        h = {}
        for key, (oz, oy, ox) in {"00": (2, 0, 0), "11": (0, 2, 0), "22": (0, 0, 2), "01": (1, 1, 0),
                                  "02": (1, 0, 1), "12": (0, 1, 1)}.items():
            h[key] = conv(conv(z[oz], s[1], oy, 1), s[2], ox, 2)
        del z
        q = (h["00"] + h["11"] + h["22"]) / 3
        for k in ("00", "11", "22"):
            h[k] -= q
        off = h["01"] ** 2 + h["02"] ** 2 + h["12"] ** 2
        w = torch.sqrt((h["00"] ** 2 + h["11"] ** 2 + h["22"] ** 2 + 2 * off) / 6)
        det = (h["00"] * (h["11"] * h["22"] - h["12"] ** 2) - h["01"] * (h["01"] * h["22"] - h["12"] * h["02"])
               + h["02"] * (h["01"] * h["12"] - h["11"] * h["02"]))
        angle = torch.acos((det / (2 * w ** 3)).clamp(-1, 1)) / 3
        del h, det, off
        l = torch.stack([q + 2 * w * torch.cos(angle + 2 * math.pi * k / 3) for k in range(3)])
        l = torch.gather(l, 0, l.abs().argsort(0))
        norm = l.norm(dim=0)
        c = p.c if p.c is not None else 0.5 * float(norm.max())
        l1, l2, l3 = l[0].abs(), *((l[1], l[2]) if p.bright_objects else (-l[1], -l[2]))
        valid = (l2 < 0) & (l3 < 0)
        l2, l3 = l2.abs(), l3.abs()
        tiny = float(np.finfo(np.float32).tiny)
        rb, ra = l1 / (torch.sqrt(l2 * l3) + tiny), l2 / (l3 + tiny)
        val = (1 - torch.exp(-0.5 * (ra / p.alpha) ** 2)) * torch.exp(-0.5 * (rb / p.beta) ** 2) \
            * (1 - torch.exp(-0.5 * (norm / c) ** 2))
        best = torch.maximum(best, torch.where(valid, val, torch.zeros_like(val)))
    return best


def exact(case, seed):
    kind = case["kind"]
    if kind == "cut":
        vol, alpha = _cut_inputs(case, seed)
        return _cut64(vol, ATV if case["cut"] == "atv" else TV, alpha.double(), _scaling(case), case["iterations"],
                      case["update"], case["bound"])
    if kind == "seeded":
        vol, labels, eigs = _seeded_inputs(case, seed)
        return _cut64(vol, eigs, case["alpha"], (1.0, 1.0, 1.0), case["iterations"], case["update"], -1.0, labels)
    one = lambda vol, w, d, eigs: _cut64(vol, eigs, w * torch.exp(vol["grad2"].double() / -d ** 2), (1.0, 1.0, 1.0),
                                         3000, 30, 1e-4)
    if kind == "grid":
        vol, points = _grid_inputs(case, seed)
        return [one(vol, w, d, e) for w, d, e in points]
    if kind == "ragged":
        return [one(v, case["weighting"], case["decay"], ATV) for v in _ragged_inputs(case, seed)]
    if kind == "served":
        return [one(v, w, d, ATV) for v, w, d in _served_inputs(case, seed)]
    if kind == "frangi":
        return {"vesselness": _vesselness64(case, _frangi_image(case, seed)), "quats": None}
    if kind == "gvf":
        return _gvf64(case, *_gvf_inputs(case, seed))
    return None   # the sign adjustment decides signs along a spanning tree: no 64-bit counterpart
