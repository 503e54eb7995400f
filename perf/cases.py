"""The work a user of this package has it do, as measurable cases.

A case is a dict of plain values: ``op`` (which entry point), the volume's
``nx ny nz``, the radii, ``slices``, the precision, the noise mode and the
number of iterations. ``prepare`` builds what a program holds before the call
(volumes on the device, a configured handle), ``run`` makes one pass through the
public entry points, ``work`` counts the bytes and operations a pass cannot do
without and ``exact`` restates the method in 64-bit torch.

Volumes are two-phase grain images with blurred noise and rings, quantised to
16 bits, as a tomography scan is delivered.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import microtomodenoise_b200 as inlm
from microtomodenoise_b200 import DenoiseParameters, IterativeNLM_GPU, NoiseLevel, proposal

CUTOFF = -3.56648  # the weight's cutoff, a constant of the method
MAX_WORK = 4 * 512 ** 3 * 514 * (2 * 33 + 20)  # operations of the largest listed case


def _case(name, op, nx, ny, nz, patch, search, precision="f32", mode="z-adaptive", iterations=4, slices=11):
    return {"name": name, "op": op, "nx": nx, "ny": ny, "nz": nz, "patch": patch, "search": search,
            "precision": precision, "mode": mode, "iterations": iterations, "slices": slices}


def listed():
    return [
        # a preview crop while a user picks radii: launches and host work count
        _case("job_preview", "job", 48, 40, 12, 2, 3, mode="global", iterations=2),
        # the README's small spheres volume, whole job
        _case("job_spheres_p1s5", "job", 128, 128, 64, 1, 5, mode="global"),
        # the program's default radii on a 256^3 stack, whole job
        _case("job_default_p1s10", "job", 256, 256, 256, 1, 10),
        # the benchmark's volume and radii, whole job: the largest
        _case("job_grains_p2s5", "job", 512, 512, 512, 2, 5),
        # a ragged region of interest at the large radii, one iteration at a
        # time with the caller's own sigma profile
        _case("steps_ragged_p3s7", "steps", 203, 187, 61, 3, 7, iterations=2),
        # a user-known sigma and a wider search, whole job
        _case("job_manual_p2s7", "job", 190, 190, 100, 2, 7, mode="manual", iterations=2),
        # the fused FP32 form on a ragged stack
        _case("steps_fused_p2s5", "steps", 255, 257, 96, 2, 5, precision="f32_fma", iterations=2),
        # the FP16-storage form, whole job
        _case("job_f16_p2s5", "job", 256, 256, 128, 2, 5, precision="f16"),
        # the learned search proposal on the FP16 form with its benchmark
        # schedule, whole job
        _case("learned_p2s5", "learned", 512, 512, 128, 2, 5, precision="f16"),
        # the noise estimator alone, one sigma per slice of a tall stack
        _case("noise_zadaptive", "noise", 512, 512, 256, 1, 5),
        # several small stacks of uneven size and mixed radii in one batch
        _case("batch_uneven", "batch", 150, 140, 90, 2, 5, mode="global"),
        # a host-resident stack filtered in z slabs
        _case("stream_p3s5", "stream", 230, 210, 150, 3, 5, iterations=2),
    ]


def draw(rng):
    """One more case of the listed ranges; sizes spread over their logarithm."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["job", "job", "job", "steps", "steps", "learned", "noise", "batch", "stream"])
    while True:
        c = {"op": op, "nx": size(36, 512), "ny": size(36, 512), "nz": size(12, 320)}
        c["patch"], c["search"] = rng.choice([(1, 3), (1, 5), (1, 10), (2, 3), (2, 5), (2, 7), (3, 3), (3, 5), (3, 7)])
        c["precision"] = rng.choice(["f32", "f32", "f32", "f32_fma", "f16"])
        c["mode"] = rng.choice(["z-adaptive", "z-adaptive", "global", "manual"])
        c["iterations"] = rng.choice([2, 4])
        c["slices"] = 11
        if op == "learned":
            c.update(patch=2, search=5, precision="f16", iterations=4, mode=rng.choice(["z-adaptive", "global"]))
        elif op == "noise":
            c["mode"] = rng.choice(["z-adaptive", "global"])
        elif op == "batch":
            c.update(precision="f32", mode="global", nx=min(c["nx"], 200), ny=min(c["ny"], 200), nz=min(c["nz"], 120))
        elif op == "stream":
            c.update(iterations=2, nz=max(c["nz"], 40))
        if work(c)["flops"] <= MAX_WORK:
            return c


# ---------------- inputs ----------------

def _blur(vol, sigma):
    r = max(1, int(3 * sigma + 0.5))
    k = torch.exp(-0.5 * (torch.arange(-r, r + 1, device=vol.device, dtype=torch.float32) / sigma) ** 2)
    k = k / k.sum()
    for ax in range(3):
        n = vol.shape[ax]
        idx = torch.arange(n, device=vol.device)
        acc = torch.zeros_like(vol)
        for j in range(-r, r + 1):
            acc.add_(vol.index_select(ax, (idx + j).clamp_(0, n - 1)), alpha=float(k[j + r]))
        vol = acc
    return vol


def _volume(shape, seed, noise=0.04):
    """Grains (0.7) in pores (0.3), blurred noise drifting along z, rings."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nz, ny, nx = shape
    grains = _blur(torch.randn(shape, generator=g, device="cuda"), 4.0)
    vol = torch.where(grains > grains.mean(), 0.7, 0.3)
    n = _blur(torch.randn(shape, generator=g, device="cuda"), 1.2)
    drift = torch.linspace(0.75, 1.25, nz, device="cuda")[:, None, None]
    vol = vol + n * (noise / n.std()) * drift
    y = torch.arange(ny, device="cuda", dtype=torch.float32)[:, None] - 0.5 * (ny - 1)
    x = torch.arange(nx, device="cuda", dtype=torch.float32)[None, :] - 0.5 * (nx - 1)
    vol = vol + 0.02 * torch.sin(2 * math.pi / 6.0 * torch.sqrt(x * x + y * y))
    return (torch.round(vol.clamp(0, 1) * 65535.0) / 65535.0).contiguous()


def _params(c, **kw):
    return DenoiseParameters(radius_patchspace=(c["patch"],) * 3, radius_searchspace=(c["search"],) * 3,
                             nslices=c["slices"], maxiterations=c["iterations"], noise_mode=c["mode"],
                             sigma=(0.09, 0.06), precision=c["precision"], n_samples=_n_samples(c),
                             noise_seed=7, **kw)


def _n_samples(c):
    return 100000 if c["nx"] * c["ny"] * c["nz"] > 1 << 18 else 4000


def _sigmas(c):
    """The caller's per-slice sigma of each iteration (op "steps")."""
    z = np.arange(c["nz"], dtype=np.float32)
    first = (0.10 + 0.02 * np.sin(0.05 * z)).astype(np.float32)
    return [first] + [(np.float32(0.8) * first).astype(np.float32)] * (c["iterations"] - 1)


def _batch(c):
    """The stacks of a batch: uneven sizes up to the case's, mixed radii."""
    out = []
    for i, (f, patch, search) in enumerate([(1.0, 2, 5), (0.8, 1, 7), (0.6, 3, 3), (0.5, 1, 3), (0.9, 1, 5), (0.7, 2, 3)]):
        out.append(dict(c, nx=max(24, int(c["nx"] * f)), ny=max(24, int(c["ny"] * (1.05 - 0.05 * i) * f)),
                        nz=max(12, int(c["nz"] * f)), patch=patch, search=search))
    return out


def prepare(case, seed):
    c = case
    shape = (c["nz"], c["ny"], c["nx"])
    st = {"case": c}
    if c["op"] == "batch":
        parts = _batch(c)
        st["raw"] = [_volume((p["nz"], p["ny"], p["nx"]), seed * 16 + i) for i, p in enumerate(parts)]
        st["out"] = [torch.empty_like(v) for v in st["raw"]]
        st["batch"] = inlm.Batch([v.shape for v in st["raw"]], [_params(p) for p in parts])
    elif c["op"] == "stream":
        st["raw"] = _volume(shape, seed).cpu().numpy()
        st["params"] = _params(c)
        st["out"] = np.empty(shape, np.float32)
    elif c["op"] == "noise":
        st["raw"] = _volume(shape, seed)
        st["params"] = _params(c)
        st["noise"] = NoiseLevel(_n_samples(c), 15, shape, seed=7)
    else:
        st["raw"] = _volume(shape, seed)
        st["out"] = torch.empty_like(st["raw"])
        st["handle"] = IterativeNLM_GPU()
        st["handle"].configure_device(shape, _params(c))
        if c["op"] == "learned":
            st["net"] = proposal.ProposalNet.load(proposal.default_weights((2, 2, 2), (5, 5, 5)))
            st["handle"].attach_proposal(st["net"], k=[112, 112, 112, 256], rel_mass=[0, 0, 0, 0.9],
                                         min_mass=0.0, tiles_x=4)
    torch.cuda.synchronize()
    return st


def run(state):
    c = state["case"]
    if c["op"] == "batch":
        state["batch"].run([v.data_ptr() for v in state["raw"]], [o.data_ptr() for o in state["out"]], on_device=True)
        return state["out"]
    if c["op"] == "stream":
        out, s0, s1, _ = inlm.stream_denoise(state["raw"], state["params"], slab_depth=64, out=state["out"])
        return {"out": out, "sigma0": s0, "sigma1": s1}
    if c["op"] == "noise":
        return state["noise"].get_noiselevel(state["raw"].data_ptr(), state["params"], on_device=True)
    g, raw, out = state["handle"], state["raw"], state["out"]
    if c["op"] == "steps":
        for it, sigma in enumerate(_sigmas(c), 1):
            g.set_sigma(sigma)
            g.Run_GaussianNoise_device(it, raw.data_ptr() if it == 1 else None)
        g.get_result_device(out.data_ptr())
        return out
    _, s0, s1 = g.denoise(raw.data_ptr(), on_device=True, out=out.data_ptr())
    return {"out": out, "sigma0": s0, "sigma1": s1}


# ---------------- the work of a pass ----------------

def _ball(r):
    """Points of the ellipsoid of radius r, (z, y, x) ascending, by the
    method's single-precision test (its rounding leaves some points out)."""
    f = np.float32

    def member(x, y, z):
        a, b, d = f(x) / f(max(r, 1)), f(y) / f(max(r, 1)), f(z) / f(max(r, 1))
        return f(f(a * a + b * b) + d * d) <= f(1)

    span = range(-r, r + 1)
    return [(z, y, x) for z in span for y in span for x in span if member(x, y, z)]


def _taps(r):
    return _ball(r)


def _offsets(c):
    return [o for o in _ball(c["search"]) if abs(o[0]) <= c["slices"] // 2 and o != (0, 0, 0)]


def work(case):
    c = case
    if c["op"] == "batch":
        parts = [dict(work(dict(p, op="job"))) for p in _batch(c)]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    vox = c["nx"] * c["ny"] * c["nz"]
    if c["op"] == "noise":
        return {"bytes": 4.0 * min(vox, _n_samples(c) * 225), "flops": 5.0 * _n_samples(c) * 225}
    per = len(_offsets(c)) * (2 * len(_taps(c["patch"])) + 20)
    if c["op"] == "learned":  # the lists' share of the offsets
        per *= (3 * 112 + 256) / (4.0 * len(_offsets(c)))
    return {"bytes": 8.0 * vox, "flops": float(vox) * c["iterations"] * per}


# ---------------- 64-bit restatement ----------------

def _weights(r):
    out = []
    for z, y, x in _taps(r):
        w = 1.0 / (2.0 * math.sqrt(z * z + y * y + x * x) + 1.0) ** 2
        out.append(w)
    if r == 1:
        return [1.0 / 7.0] * len(out)
    out[out.index(max(out))] = max(w for w in out if w < 1.0)  # the centre takes the largest other weight
    return [float("%g" % w) for w in out]


def _filter64(raw, prev, c, sigma):
    dev = raw.device
    pr, sr, zc = c["patch"], c["search"], min(c["slices"] // 2, c["search"])
    pad = (zc + pr, sr + pr, sr + pr)

    def padded(v):
        for ax in range(3):
            n, p = v.shape[ax], pad[ax]
            i = torch.arange(-p, n + p, device=dev)
            period = max(1, 2 * (n - 1))
            i = i.remainder(period)
            v = v.index_select(ax, torch.where(i >= n, period - i, i))
        return v

    nz, ny, nx = raw.shape
    rp, pp = padded(raw), padded(prev)
    m = (-1.0 / (torch.as_tensor(sigma, dtype=torch.float64, device=dev) ** 2))[:, None, None]
    taps, w = _taps(pr), _weights(pr)
    ez, ey, ex = nz + 2 * pr, ny + 2 * pr, nx + 2 * pr
    org = pp[zc:zc + ez, sr:sr + ey, sr:sr + ex]
    acc, wsum, wmax = (torch.zeros_like(raw) for _ in range(3))
    for dz, dy, dx in _offsets(c):
        d = pp[zc + dz:zc + dz + ez, sr + dy:sr + dy + ey, sr + dx:sr + dx + ex] - org
        d.mul_(d)
        dist = torch.zeros_like(raw)
        for (tz, ty, tx), wt in zip(taps, w):
            dist.add_(d[pr + tz:pr + tz + nz, pr + ty:pr + ty + ny, pr + tx:pr + tx + nx], alpha=wt)
        x = dist.mul_(m)
        q = (120 + 60 * x + 12 * x * x + x ** 3) / (120 - 60 * x + 12 * x * x - x ** 3)
        q = torch.where(x > CUTOFF, q, torch.zeros_like(q))
        z0, y0, x0 = pad[0] + dz, pad[1] + dy, pad[2] + dx
        acc.addcmul_(q, rp[z0:z0 + nz, y0:y0 + ny, x0:x0 + nx])
        wsum.add_(q)
        torch.maximum(wmax, q, out=wmax)
    return torch.where(wmax > 0, (acc + wmax * raw) / (wsum + wmax), raw)


def _samples(c):
    """Sample positions: the C library's rand() from the noise seed, sorted."""
    libc = ctypes.CDLL(None)
    libc.srand(7)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    pos = []
    for _ in range(_n_samples(c)):
        x, y = libc.rand() % (nx - 15), libc.rand() % (ny - 15)
        pos.append(((libc.rand() % nz) * ny + y) * nx + x)
    return torch.tensor(sorted(pos))


def _em64(v):
    """Two-cluster hard EM; mean + std of the cluster with the lower mean."""
    v = v[v != 0]
    if v.numel() == 0:
        return None
    lo, hi = v.min(), v.max()
    mean = torch.stack([lo + 0.25 * (hi - lo), hi - 0.25 * (hi - lo)])
    a = (v - mean[0]).abs() >= (v - mean[1]).abs()

    def moments(a, mean, means):
        n = torch.stack([(~a).sum(), a.sum()]).double()
        if means:
            s = torch.stack([v[~a].sum(), v[a].sum()])
            mean = torch.where(n > 0, s / n.clamp(min=1), mean)
        d = torch.stack([((v[~a] - mean[0]) ** 2).sum(), ((v[a] - mean[1]) ** 2).sum()])
        return mean, d / n.clamp(min=1)

    mean, var = moments(a, mean, True)
    for _ in range(1000):
        if not bool((var > 0).all()):
            break
        p = [torch.exp(-(v - mean[k]) ** 2 / (2 * var[k])) / torch.sqrt(2 * math.pi * var[k]) for k in (0, 1)]
        b = p[1] > p[0]
        changed = bool((b != a).any())
        a = b
        mean, var = moments(a, mean, True)
        if not changed:
            break
    k = 0 if bool(mean[0] <= mean[1]) or bool(var[1] <= 0) else 1
    return float(mean[k] + torch.sqrt(var[k]))


def _noise64(vol, c, pos):
    """Per-slice sigma of a 64-bit volume."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    o = torch.arange(15)
    patch = (o[:, None] * nx + o[None, :]).reshape(-1).to(vol.device)
    std = torch.cat([vol.reshape(-1)[(p[:, None].to(vol.device) + patch)].std(dim=1, unbiased=False)
                     for p in pos.split(8192)])
    if c["mode"] == "global":
        return np.full(nz, _em64(std))
    z = (pos // (nx * ny)).numpy()
    n, out = len(z), []
    for i in range(nz):
        first = min(int(np.searchsorted(z, i - 50, side="right")), n - 1)
        last = min(int(np.searchsorted(z, i + 50, side="right")), n - 1)
        s = _em64(std[first:last + 1])
        if s is None:
            return None
        out.append(s)
    return np.array(out)


def _exact_cost(c):
    """Seconds _filter64 takes, from the bytes its torch calls move."""
    per_call = max(6e-6, c["nx"] * c["ny"] * c["nz"] * 24 / 4e12)
    seconds = c["iterations"] * len(_offsets(c)) * (len(_taps(c["patch"])) + 24) * per_call
    if c["mode"] == "z-adaptive" and c["op"] != "steps":
        seconds += 2 * c["nz"] * 0.02
    return seconds


def exact(case, seed):
    c = case
    if c["op"] == "learned":  # its lists are a network's choice
        return None
    if c["op"] == "noise":
        return _noise64(_volume((c["nz"], c["ny"], c["nx"]), seed).double(), c, _samples(c)) if c["nz"] < 400 else None
    parts = _batch(c) if c["op"] == "batch" else [c]
    if sum(_exact_cost(p) for p in parts) > 15:
        return None
    outs = []
    for i, p in enumerate(parts):
        raw = _volume((p["nz"], p["ny"], p["nx"]), seed * 16 + i if c["op"] == "batch" else seed).double()
        cur = raw
        if c["op"] == "steps":
            for sigma in _sigmas(p):
                cur = _filter64(raw, cur, p, sigma)
            return cur
        if p["mode"] == "manual":
            s0, s1 = np.full(p["nz"], np.float32(0.09)), np.full(p["nz"], np.float32(0.06))
        else:
            pos = _samples(p)
            s0 = _noise64(raw, p, pos)
            if s0 is None:
                return None
        cur = _filter64(raw, raw, p, s0)
        if p["mode"] != "manual":
            s1 = _noise64(cur, p, pos)
            if s1 is None:
                return None
        for _ in range(p["iterations"] - 1):
            cur = _filter64(raw, cur, p, 0.5 * s0 + 0.5 * s1)
        outs.append(cur)
    if c["op"] == "batch":
        return outs
    return {"out": outs[0], "sigma0": s0, "sigma1": s1}
