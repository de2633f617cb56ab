"""What a program that uses this package has it do, as cases that can be timed and compared.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs on the GPU, and the solver and plan (or operator) a program keeps
    run(state)           one pass through the package's public entry points, and its outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the same outputs in 64 bits, from plain torch

Kinds: `pair` (one frame pair, TVL13DOpticalFlow.compute), `batch` (pairs of any sizes,
compute_batch), `patient` (one direction of a cine sequence, processor.process_sequence), `plain`
(the per-operator form that a program written against the reference's module runs), `masks` and
`chains` (mask propagation through flows), `train` (the differentiable warp, forward and backward),
`resample` (a raw cine MRI to the flow grid), `median` (the flow post-filter). Solver parameters are
the default configuration (3 levels, 300 iterations a warp, cubic, MIRROR, anisotropic, blurred).
"""
import math

import torch
import torch.nn.functional as F

from singleventriclesegmentation_b200 import opticalFlow
from singleventriclesegmentation_b200.flow_utils import apply_median_filter
from singleventriclesegmentation_b200.preprocessing import resample_patient
from singleventriclesegmentation_b200.processor import process_sequence
from singleventriclesegmentation_b200.tvl13d import TVL13DOpticalFlow
from singleventriclesegmentation_b200.warping import Warp, propagate, propagate_batched
from singleventriclesegmentation_b200.warpingOps import warp

SCALES, ITERS = 3, 300
MATCHING, TV, SIGMA, TAU, GAMMA, ALPHA, BETA = 1.0, 0.025, 0.5, 0.5, 1.0, 5.0, 0.5
CUBIC, MIRROR = "CUBIC_HERMITESPLINE", "MIRROR"


def listed():
    return [
        # the smallest solve: a cropped volume with odd sizes, every field in FP32 (the default
        # storage); launch latency counts, every level is a fraction of the GPU
        {"name": "pair_small_f32", "kind": "pair", "sizes": "35x41x47", "storage": "f32", "warps": 15},
        # one 80^3 pair alone, the drop-in call with its default storage
        {"name": "pair_80_f32", "kind": "pair", "sizes": "80x80x80", "storage": "f32", "warps": 15},
        # the same pair in the mixed-precision mode that the benchmark uses (its latency workload)
        {"name": "pair_80_f16flow32", "kind": "pair", "sizes": "80x80x80", "storage": "f16-flow32", "warps": 15},
        # one direction of a patient from t = 0 to t = 12 (12 pairs), with the median post-filter
        {"name": "patient_80_f16flow32", "kind": "patient", "sizes": "80x80x80", "frames": 13, "storage": "f16-flow32",
         "warps": 15},
        # a batch of uneven, partly odd sizes in one graph, as a serving loop forms it
        {"name": "uneven_bf16flow32", "kind": "batch", "storage": "bf16-flow32", "warps": 15,
         "sizes": "64x80x96,40x48x40,120x104x128,72x88x56,48x65x81,96x112x72,57x40x63,80x80x80"},
        # all 68 pairs of a 35-frame sequence at once, with fewer warps than the default: a
        # preview, and the largest device-filling launches
        {"name": "sequence_68x80_f16flow32", "kind": "batch", "storage": "f16-flow32", "warps": 2,
         "sizes": ",".join(["80x80x80"] * 68)},
        # a program written against the reference's operators, unchanged, on the drop-in module
        {"name": "plain_80_f32", "kind": "plain", "sizes": "80x80x80", "warps": 1, "iters": 30},
        # both end masks of a patient carried through 12 flows each way
        {"name": "masks_80", "kind": "masks", "sizes": "80x80x80", "steps": 12},
        # eight structures carried through their flows at once, at an uncommon size
        {"name": "chains_8x96", "kind": "chains", "sizes": "91x112x105", "count": 8, "steps": 12},
        # the warp inside a training loss: forward, and gradients to the image and the flow
        {"name": "train_80", "kind": "train", "sizes": "80x80x80"},
        # a raw short-axis cine MRI, 25 frames, with its two segmentations, to 80^3 and 35 frames
        {"name": "resample_16x160x25", "kind": "resample", "sizes": "16x160x160", "frames": 25, "to": 80},
        # the flow post-filter by itself
        {"name": "median_80", "kind": "median", "sizes": "80x80x80", "window": 3},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, lo, hi):
    return "x".join(str(_size(rng, lo, hi)) for _ in range(3))


def draw(rng):
    kind = rng.choice(["pair", "pair", "batch", "batch", "patient", "plain", "masks", "chains", "train", "resample",
                       "median"])
    half = ["f16-flow32", "bf16-flow32"]
    if kind == "pair":
        return {"kind": kind, "sizes": _sizes(rng, 24, 112), "storage": rng.choice(["f32"] + half),
                "warps": rng.choice([5, 10, 15])}
    if kind == "batch":
        n = _size(rng, 2, 60)
        top = min(128, int(128 * (8 / max(n, 8)) ** (1 / 3)))
        same = rng.random() < 0.5
        one = _sizes(rng, 40, top)
        return {"kind": kind, "storage": rng.choice(["f32"] + half + half), "warps": rng.choice([1, 2, 3]),
                "sizes": ",".join(one if same else _sizes(rng, 40, top) for _ in range(n))}
    if kind == "patient":
        return {"kind": kind, "sizes": _sizes(rng, 40, 88), "frames": rng.randint(4, 13), "storage": rng.choice(half),
                "warps": rng.choice([3, 5, 8])}
    if kind == "plain":
        return {"kind": kind, "sizes": _sizes(rng, 32, 96), "warps": 1, "iters": rng.randint(10, 40)}
    if kind == "masks":
        return {"kind": kind, "sizes": _sizes(rng, 32, 128), "steps": rng.randint(4, 20)}
    if kind == "chains":
        return {"kind": kind, "sizes": _sizes(rng, 32, 128), "count": rng.randint(2, 16), "steps": rng.randint(2, 12)}
    if kind == "train":
        return {"kind": kind, "sizes": _sizes(rng, 32, 128)}
    if kind == "resample":
        plane = _size(rng, 96, 192)
        return {"kind": kind, "sizes": "%dx%dx%d" % (rng.randint(8, 24), plane, plane + rng.randint(0, 9)),
                "frames": rng.randint(15, 35), "to": rng.choice([64, 80, 81, 96])}
    return {"kind": kind, "sizes": _sizes(rng, 32, 128), "window": rng.choice([3, 3, 5])}


# ------------------------------------------------------------------------------------ inputs
def _dims(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _frames(g, dims, count, noise=0.01):
    """`count` frames of one beating volume: 40 Gaussian blobs, clipped to [0, 1], whose centres
    move by up to 3 voxels over the cycle, plus noise."""
    size = torch.tensor(dims, device="cuda", dtype=torch.float64)
    scale = (dims[0] * dims[1] * dims[2]) ** (1 / 3) / 80
    centre, width = _uniform(g, 0, 1, 40, 3) * size, _uniform(g, 3, 10, 40) * scale
    height, move, phase = _uniform(g, 0.2, 1, 40), _uniform(g, -3, 3, 3), _uniform(g, -0.6, 0.6, 40, 1)
    frames = []
    for t in range(count):
        at = centre + move * torch.sin(2 * math.pi * t / 35 + phase)
        ez, ey, ex = (torch.exp(-(torch.arange(n, device="cuda", dtype=torch.float64) - at[:, a:a + 1]) ** 2
                                / (2 * width[:, None] ** 2)) for a, n in enumerate(dims))
        plane = (ey[:, :, None] * ex[:, None, :]).reshape(40, -1)
        volume = ((ez * height[:, None]).T @ plane).reshape(dims).clamp(0, 1)
        volume += noise * torch.randn(*dims, generator=g, device="cuda", dtype=torch.float64)
        frames.append(volume.float())
    return frames


def _flow(g, dims, top=3.0):
    """A smooth displacement [Z, Y, X, 3] of up to `top` voxels."""
    z, y, x = (torch.arange(n, device="cuda", dtype=torch.float64) / n for n in dims)
    u = torch.zeros(*dims, 3, device="cuda", dtype=torch.float64)
    for c in range(3):
        k, phase, a = _uniform(g, 0.3, 1.5, 4, 3), _uniform(g, 0, 2 * math.pi, 4), _uniform(g, 0.5, 1, 4)
        for i in range(4):
            u[..., c] += a[i] * torch.sin(2 * math.pi * (k[i, 0] * z[:, None, None] + k[i, 1] * y[:, None] + k[i, 2] * x)
                                          + phase[i])
    return (u * (top / u.abs().max())).float().contiguous()


def _ellipsoid(g, dims):
    """A binary mask [Z, Y, X] of about a third of each axis, near the middle."""
    r = 0
    for a, n in enumerate(dims):
        at, half = _uniform(g, 0.4, 0.6, 1) * n, _uniform(g, 0.13, 0.2, 1) * n
        e = ((torch.arange(n, device="cuda", dtype=torch.float64) - at) / half) ** 2
        r = r + e.reshape([-1 if i == a else 1 for i in range(3)])
    return (r <= 1).float()


def _solver(case, storage):
    return TVL13DOpticalFlow(SCALES, case["warps"], case.get("iters", ITERS), MATCHING, TV, 2, (SIGMA, TAU, 0.25, GAMMA),
                             True, (ALPHA, BETA), True, 1.0, CUBIC, MIRROR, "numDofs", (1, 1, 1),
                             torch.device("cuda", torch.cuda.current_device()), storage=storage)


def _inputs(case, seed):
    g, kind, dims = _generator(seed), case["kind"], _dims(case)
    one = dims[0]
    if kind in ("pair", "plain"):
        a, b = _frames(g, one, 2)
        return {"I0": b, "I1": a}
    if kind == "batch":
        if len(set(dims)) == 1:  # consecutive frames of one sequence, forward and backward
            f = _frames(g, one, (len(dims) + 3) // 2)
            pairs = [(t + 1, t) for t in range(len(f) - 1)] + [(t, t + 1) for t in range(len(f) - 1)]
            pairs = pairs[:len(dims)]
            return {"I0": [f[i] for i, _ in pairs], "I1": [f[j] for _, j in pairs]}
        f = [_frames(g, d, 2) for d in dims]
        return {"I0": [b for _, b in f], "I1": [a for a, _ in f]}
    if kind == "patient":
        return {"img": torch.stack(_frames(g, one, case["frames"]))}
    if kind == "masks":
        return {"first": _ellipsoid(g, one)[None, None], "last": _ellipsoid(g, one)[None, None],
                "forward": torch.stack([_flow(g, one) for _ in range(case["steps"])]),
                "backward": torch.stack([_flow(g, one) for _ in range(case["steps"])])}
    if kind == "chains":
        return {"masks": torch.stack([_ellipsoid(g, one)[None] for _ in range(case["count"])]),
                "flows": torch.stack([torch.stack([_flow(g, one) for _ in range(case["count"])])
                                      for _ in range(case["steps"])])}
    if kind == "train":
        return {"image": _frames(g, one, 1)[0], "flow": _flow(g, one),
                "grad": torch.randn(*one, generator=g, device="cuda")}
    if kind == "resample":
        img = torch.stack(_frames(g, one, case["frames"]), dim=-1).contiguous()
        return {"img": img, "dia": _ellipsoid(g, one), "sys": _ellipsoid(g, one)}
    flow = _flow(g, one)
    return {"flow": flow + 0.05 * torch.randn(flow.shape, generator=g, device="cuda")}


def prepare(case, seed):
    state = _inputs(case, seed)
    kind, dims = case["kind"], _dims(case)
    state["kind"] = kind
    if kind in ("pair", "batch"):
        state["solver"] = _solver(case, case["storage"])
        state["solver"].plan_for(dims)
    elif kind == "patient":
        state["solver"] = _solver(case, case["storage"])
        state["frames"] = case["frames"]
    elif kind == "plain":
        state["solver"] = _solver(case, "f32")
        state["u"] = torch.zeros(dims[0] + (3,), device="cuda")
        state["p"] = torch.zeros(dims[0] + (3, 3), device="cuda")
    elif kind in ("masks", "chains"):
        state["warp"] = Warp(CUBIC, MIRROR, "numDofs", (1, 1, 1))
    elif kind == "train":
        mesh = opticalFlow.MeshInfo3D(*dims[0], *(n - 1 for n in dims[0]))
        state["op"] = opticalFlow.Warping3D(mesh, opticalFlow.INTERPOLATE_CUBIC_HERMITESPLINE,
                                            opticalFlow.BOUNDARY_MIRROR)
        state["image"].requires_grad_()
        state["flow"].requires_grad_()
    elif kind == "resample":
        state["to"] = case["to"]
    else:
        state["window"] = case["window"]
    return state


def run(state):
    kind = state["kind"]
    if kind == "pair":
        return state["solver"].compute(state["I0"], state["I1"])
    if kind == "batch":
        us = state["solver"].compute_batch(state["I0"], state["I1"])
        return torch.stack(us) if len(us) > 60 else us
    if kind == "patient":
        return process_sequence(state["img"], 0, state["frames"] - 1, "forward", state["solver"])
    if kind == "plain":
        return state["solver"].compute_unfused(state["I0"], state["I1"], state["u"], state["p"])
    if kind == "masks":
        return propagate(state["warp"], state["first"], state["last"], state["forward"], state["backward"])
    if kind == "chains":
        return propagate_batched(state["warp"], state["masks"], state["flows"])
    if kind == "train":
        out = warp(state["image"], state["flow"], state["op"])
        return (out.detach(),) + torch.autograd.grad(out, (state["image"], state["flow"]), state["grad"])
    if kind == "resample":
        n = state["to"]
        return resample_patient(state["img"], state["dia"], state["sys"], (n, n, n), 35)[:3]
    return apply_median_filter(state["flow"], state["window"])


# -------------------------------------------------------------------------------------- work
def _levels(dims):
    """Sizes of the pyramid's levels, finest first."""
    out = [tuple(dims)]
    for _ in range(1, SCALES):
        out.append(tuple((n + 1) // 2 for n in out[-1]))
    return out


def _voxels(dims):
    return dims[0] * dims[1] * dims[2]


def work(case):
    kind, dims = case["kind"], _dims(case)
    n = _voxels(dims[0])
    if kind in ("pair", "batch", "patient", "plain"):
        # an iteration reads u 3, p 9, D 6, rho_c 1, warped gradient 3 and writes u 3, p 9 at each
        # voxel (u in 4 bytes); the linearisation moves 12 values, the preparation of a level 10
        field = 4 if case.get("storage", "f32") == "f32" else 2
        pairs = dims * (case["frames"] - 1) if kind == "patient" else dims
        voxels = sum(_voxels(level) for d in pairs for level in _levels(d))
        iters = case["warps"] * case.get("iters", ITERS)
        return {"bytes": voxels * (iters * (6 * 4 + 28 * field) + case["warps"] * 48 + 40),
                "flops": voxels * iters * 225.0}
    if kind == "masks":
        return {"bytes": 2 * case["steps"] * n * 20, "flops": 2 * case["steps"] * n * 21 * 14.0}
    if kind == "chains":
        return {"bytes": case["count"] * case["steps"] * n * 20,
                "flops": case["count"] * case["steps"] * n * 21 * 14.0}
    if kind == "train":
        # forward: image, flow, output; backward: image, flow, output's gradient, both gradients
        return {"bytes": n * (20 + 36), "flops": n * (21 * 14 + 64 * 4.0)}
    if kind == "resample":
        m = case["to"] ** 3
        return {"bytes": 4 * (n * (case["frames"] + 2) + m * (35 + 2)), "flops": m * (case["frames"] + 2) * 24.0}
    return {"bytes": n * 24, "flops": n * 3 * case["window"] ** 3 * 4.0}


# --------------------------------------------------------------------------- 64-bit outputs
def _fold(i, n):
    i = torch.where(i < 0, -i - 1, i)
    return torch.where(i > n - 1, 2 * n - 1 - i, i).clamp(0, n - 1)


def _cubic_weights(w):
    w2, w3 = w * w, w * w * w
    return [-w3 / 2 + w2 - w / 2, 1.5 * w3 - 2.5 * w2 + 1, -1.5 * w3 + 2 * w2 + w / 2, w3 / 2 - w2 / 2]


def _sample(fields, cz, cy, cx):
    """Tricubic values of `fields` [C, Z, Y, X] at the given voxel coordinates."""
    nz, ny, nx = fields.shape[1:]
    fz, fy, fx = cz.floor(), cy.floor(), cx.floor()
    Wz, Wy, Wx = _cubic_weights(cz - fz), _cubic_weights(cy - fy), _cubic_weights(cx - fx)
    iz, iy, ix = ([_fold(f.long() + d - 1, n) for d in range(4)] for f, n in ((fz, nz), (fy, ny), (fx, nx)))
    flat, out = fields.reshape(len(fields), -1), 0
    for a in range(4):
        for b in range(4):
            for c in range(4):
                out = out + Wz[a] * Wy[b] * Wx[c] * flat[:, (iz[a] * ny + iy[b]) * nx + ix[c]]
    return out


def _grid(dims):
    return torch.meshgrid(*(torch.arange(n, device="cuda", dtype=torch.float64) for n in dims), indexing="ij")


def _warped(fields, u):
    z, y, x = _grid(fields.shape[1:])
    return _sample(fields, z + u[2], y + u[1], x + u[0])


def _resized(fields, dims, cubic=True):
    """`fields` [C, Z, Y, X] at the nodes of a mesh of `dims` nodes over the same extent."""
    for axis, n in enumerate(dims, 1):
        m = fields.shape[axis]
        at = torch.arange(n, device="cuda", dtype=torch.float64) * (m - 1) / (n - 1)
        low = at.floor()
        W = _cubic_weights(at - low) if cubic else [None, 1 - (at - low), at - low]
        shape, out = [-1 if a == axis else 1 for a in range(4)], 0
        for d, w in enumerate(W):
            if w is not None:
                out = out + w.reshape(shape) * fields.index_select(axis, _fold(low.long() + d - 1, m))
        fields = out
    return fields


def _along(axis, lo, hi):
    return (Ellipsis,) + tuple(slice(lo, hi) if a == axis else slice(None) for a in range(3))


def _gradient(f):
    """Central differences [..., C, 3 (x, y, z), Z, Y, X] of [..., C, Z, Y, X], zero on the faces."""
    g = torch.zeros(f.shape[:-3] + (3,) + f.shape[-3:], device=f.device, dtype=f.dtype)
    for d, axis in enumerate((2, 1, 0)):
        n = f.shape[-3 + axis]
        g[(Ellipsis, d) + _along(axis, 1, n - 1)[1:]] = (f[_along(axis, 2, n)] - f[_along(axis, 0, n - 2)]) / 2
    return g


def _divergence(q):
    """The adjoint of _gradient: [C, 3, Z, Y, X] -> [C, Z, Y, X]."""
    out = torch.zeros_like(q[:, 0])
    for d, axis in enumerate((2, 1, 0)):
        n, f = q.shape[-3 + axis], q[:, d]
        out[_along(axis, 2, n)] += f[_along(axis, 1, n - 1)] / 2
        out[_along(axis, 0, n - 2)] -= f[_along(axis, 1, n - 1)] / 2
    return out


def _blurred(f):
    t = torch.linspace(-3, 3, 5)  # the reference's taps: linspace(-ks // 2, ks // 2 + 1, ks), ks = 5, sigma = 1
    k = torch.exp(-t ** 2 / 2)
    k = k / k.sum()
    k3 = torch.einsum("i,j,k->ijk", k, k, k)
    k3 = (k3 / k3.sum()).double().cuda()
    return F.conv3d(f[None, None], k3[None, None], padding=2)[0, 0]


def _solved(I0, I1, warps, iters):
    """(u [3, Z, Y, X], p [3, 3, Z, Y, X]) of one pair by the primal-dual scheme in 64 bits."""
    levels = _levels(I0.shape)
    images = [torch.stack([_blurred(I0.double()), _blurred(I1.double())])]
    for dims in levels[1:]:
        images.append(_resized(images[-1], dims))
    u = torch.zeros((3,) + levels[-1], device="cuda", dtype=torch.float64)
    p = torch.zeros((3, 3) + levels[-1], device="cuda", dtype=torch.float64)
    for k in range(SCALES - 1, -1, -1):
        a, b = images[k]
        if k < SCALES - 1:
            grow = torch.tensor([(levels[k][d] - 1) / (levels[k + 1][d] - 1) for d in (2, 1, 0)], device="cuda",
                                dtype=torch.float64)
            u = _resized(u, levels[k]) * grow[:, None, None, None]
            p = _resized(p.reshape((9,) + levels[k + 1]), levels[k]).reshape((3, 3) + levels[k])
        g = _gradient(b)
        norm = g.square().sum(0).sqrt()
        n = torch.where(norm > 0, g / norm, 0.0)
        s = torch.where(norm > 0, torch.exp(-ALPHA * norm ** BETA), 0.0)
        zero = torch.zeros_like(s)
        steep = n[2] > 0.5
        t = torch.stack([torch.where(steep, n[2], n[1]), torch.where(steep, zero, -n[0]), torch.where(steep, -n[0], zero)])
        D = s * n[:, None] * n[None] + t[:, None] * t[None]
        both = torch.cat([b[None], g])
        for _ in range(warps):
            w = _warped(both, u)
            gw, rc = w[1:], w[0] - (u * w[1:]).sum(0) - a
            g2 = gw.square().sum(0)
            tau, sigma = TAU, SIGMA
            for _ in range(iters):
                e = _gradient(u)
                p = p + sigma * (D[None, :, 0] * e[:, None, 0] + D[None, :, 1] * e[:, None, 1] + D[None, :, 2] * e[:, None, 2])
                p = p / (p.square().sum(1, keepdim=True).sqrt() / TV).clamp(min=1)
                q = D[None, :, 0] * p[:, None, 0] + D[None, :, 1] * p[:, None, 1] + D[None, :, 2] * p[:, None, 2]
                rho, most = rc + (u * gw).sum(0), tau * MATCHING
                step = torch.where(g2 >= 1e-10, -rho / g2, 0.0)
                step = torch.where(rho < -most * g2, most, torch.where(rho > most * g2, -most, step))
                u = u - tau * _divergence(q) + step * gw
                theta = 1 / math.sqrt(1 + 2 * GAMMA * tau)
                tau, sigma = tau * theta, sigma / theta
    return u, p


def _median(f, window):
    """Median of the window around each voxel of [C, Z, Y, X]."""
    r = window // 2
    for axis in (1, 2, 3):
        n = f.shape[axis]
        f = f.index_select(axis, _fold(torch.arange(-r, n + r, device="cuda"), n))
    f = f.unfold(1, window, 1).unfold(2, window, 1).unfold(3, window, 1)
    return torch.stack([plane.reshape(plane.shape[:3] + (-1,)).median(-1).values for plane in f.unbind(1)], 1)


def exact(case, seed):
    kind, dims = case["kind"], _dims(case)
    if kind in ("pair", "batch", "patient", "plain"):
        pairs = dims * (case["frames"] - 1) if kind == "patient" else dims
        iters = case["warps"] * case.get("iters", ITERS)
        if sum(iters * (SCALES * 5e-4 + 1.2e-9 * _voxels(d)) for d in pairs) > 12:  # seconds, about
            return None
        state = _inputs(case, seed)
        if kind == "patient":
            state["I0"], state["I1"] = list(state["img"][1:]), list(state["img"][:-1])
        if kind != "batch" and kind != "patient":
            u, p = _solved(state["I0"], state["I1"], case["warps"], case.get("iters", ITERS))
            # p is not unique where the tensor is degenerate: a long solve says little about it
            return u.permute(1, 2, 3, 0), p.permute(2, 3, 4, 0, 1) if kind == "plain" else None
        us = [_solved(a, b, case["warps"], ITERS)[0] for a, b in zip(state["I0"], state["I1"])]
        if kind == "patient":
            return torch.stack([_median(u, 3).permute(0, 3, 2, 1) for u in us])
        us = [u.permute(1, 2, 3, 0) for u in us]
        return torch.stack(us) if len(us) > 60 else us
    state = _inputs(case, seed)
    if kind == "masks":
        return None  # ones and zeros: a voxel on the threshold may be either
    if kind == "chains":
        out = [state["masks"].double()]
        for flows in state["flows"].double():
            out.append(torch.stack([_warped(m, f.permute(3, 0, 1, 2)) for m, f in zip(out[-1], flows)]))
        return torch.stack(out)
    if kind == "train":
        image, flow = state["image"].double().requires_grad_(), state["flow"].double().requires_grad_()
        out = _warped(image[None], flow.permute(3, 0, 1, 2))[0]
        return (out.detach(),) + torch.autograd.grad(out, (image, flow), state["grad"].double())
    if kind == "resample":
        n = case["to"]
        img = _resized(state["img"].double().permute(3, 0, 1, 2), (n, n, n), cubic=False).permute(1, 2, 3, 0)
        return F.pad(img, [0, 35 - case["frames"]]), None, None  # the masks are rounded: a half may go either way
    return _median(state["flow"].double().permute(3, 0, 1, 2), case["window"]).permute(1, 2, 3, 0)
