"""The work a user of this engine has it do, as cases that can be timed and compared.

A case is one pass through the public entry points: states go in, some generations run, states come
out (or, for the screen proposer, rows go in and probabilities or gradients come out).  Device-resident
states go through the C ABI (include/lenia_gb300.h), as a C or Rust host uses it; host states through
``auto_gb300.Sim``.

Growth parameters: sigma >= 0.036 and dt <= 0.05 wherever a pass runs more than a few generations.  A
narrower or faster growth amplifies the last bit of one generation a thousandfold within sixty-four, so
that states after a pass would say nothing about the arithmetic.  A generation costs the same whatever
they are.
"""
import ctypes
import math

import numpy as np
import torch

import auto_gb300 as ag
from auto_gb300 import _lib, configs
from auto_gb300.program import Kernel, Seed, World
from auto_gb300.screen import Proposer, sample_params, worlds_for

SIDES = (32, 48, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 3072, 4096, 6144, 8192)


def listed():
    return [
        # a viewer's frame of the smallest configuration: host state in, one generation, host state out
        {"name": "frame_256", "kind": "frame", "w": 256, "h": 256},
        # one small world run on (the reference's own 256 x 256 case): launches and latency only
        {"name": "run_256", "kind": "run", "w": 256, "h": 256, "radius": 13.0, "shells": 1, "gens": 64},
        # a window's size rounded up to a grid the engine takes: not square, one side 3 * 2^k
        {"name": "run_1536x768", "kind": "run", "w": 1536, "h": 768, "radius": 13.0, "shells": 1, "gens": 64},
        # the large configuration: one 4096 x 4096 world, R = 52, three shells
        {"name": "run_4096", "kind": "run", "w": 4096, "h": 4096, "radius": 52.0, "shells": 3, "gens": 64},
        # the largest grid there is, and a number of generations that is no whole graph of 64
        {"name": "run_8192", "kind": "run", "w": 8192, "h": 8192, "radius": 13.0, "shells": 1, "gens": 20},
        # the headline: 384 worlds of seven sizes, streamed in and out every 64 generations
        {"name": "batched_384", "kind": "batch", "worlds": 384, "path": "fp32", "gens": 64},
        # labelling worlds for the screen: statistics, then 100 generations to the next checkpoint
        {"name": "screen_1024", "kind": "screen", "worlds": 1024, "side": 256, "gens": 100},
        # three channels, nine kernels
        {"name": "multichannel_1024", "kind": "multi", "w": 1024, "h": 1024, "channels": 3, "gens": 16},
        # SmoothLife on its default grid: two kernels, one channel
        {"name": "smoothlife_2048x1024", "kind": "smoothlife", "w": 2048, "h": 1024, "gens": 8},
        # the tensor-core path on mixed sizes
        {"name": "bf16x3_batched_24", "kind": "batch", "worlds": 24, "path": "bf16x3", "gens": 16},
        # the proposer's training: forward and backward of one minibatch
        {"name": "mlp_gradients_1000", "kind": "gradients", "rows": 1000},
        # the proposer's use: ranking candidates
        {"name": "mlp_predict_250k", "kind": "predict", "rows": 250001},
    ]


def draw(rng):
    kind = rng.choice(("frame", "run", "run", "run", "batch", "screen", "multi", "smoothlife", "gradients", "predict"))
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    side = lambda lo, hi: rng.choice([s for s in SIDES if lo <= s <= hi])  # noqa: E731
    if kind == "frame":
        return {"kind": kind, "w": side(64, 1024), "h": side(64, 1024)}
    if kind == "run":
        w = side(64, 8192)
        h = w if rng.random() < 0.5 else side(64, 8192)
        gens = rng.choice((1, 5, 20, 64, 64)) if w * h < 1 << 25 else rng.randint(1, 20)
        top = (min(w, h) - 1) // 2
        return {"kind": kind, "w": w, "h": h, "radius": float(rng.randint(min(6, top), min(40, top))),
                "shells": rng.randint(1, 3), "gens": gens}
    if kind == "batch":
        path = rng.choice(("fp32", "fp32", "bf16x3"))
        return {"kind": kind, "worlds": log(8, 384 if path == "fp32" else 48), "path": path,
                "gens": 64 if path == "fp32" else 16}
    if kind == "screen":
        return {"kind": kind, "worlds": log(32, 1024), "side": rng.choice((128, 192, 256)), "gens": rng.randint(20, 100)}
    if kind == "multi":
        return {"kind": kind, "w": side(96, 1024), "h": side(96, 1024), "channels": rng.randint(2, 3),
                "gens": rng.randint(2, 16)}
    if kind == "smoothlife":
        return {"kind": kind, "w": side(64, 2048), "h": side(64, 2048), "gens": rng.randint(2, 8)}
    if kind == "gradients":
        return {"kind": kind, "rows": log(64, 4096)}
    return {"kind": kind, "rows": log(1000, 500000)}


# ------------------------------------------------------------------ the worlds of a case

def _unit(i, j):
    return ag.program.unit_f(ag.program.rand3(i, j, 77))


def _worlds(case):
    kind = case["kind"]
    if kind in ("frame", "run"):
        w, h = case["w"], case["h"]
        if kind == "frame":
            return [ag.lenia(w, h, 13.0)]
        beta = [1.0, 0.5, 0.25][: case["shells"]]
        return [World(w, h, [Kernel(radius=case["radius"], beta=beta, mu=0.26, sigma=0.05)], dt=0.03)]
    if kind == "batch":
        out = configs.batched(case["worlds"])  # its sides and radii
        for i, w in enumerate(out):
            w.seed = Seed()
            w.dt = 0.02 + 0.02 * _unit(i, 0)
            w.kernels[0].mu = 0.2 + 0.15 * _unit(i, 1)
            w.kernels[0].sigma = 0.045 + 0.015 * _unit(i, 2)
        return out
    if kind == "screen":
        P = sample_params(case["worlds"], 5)
        P["sigma"] = (0.045 + 0.3 * (P["sigma"] - 0.01)).astype(np.float32)
        P["dt"] = (0.01 + 0.1 * (P["dt"] - 0.05)).astype(np.float32)
        out = worlds_for(P, case["side"])
        for w in out:
            w.seed = Seed()
        return out
    if kind == "multi":
        c, kernels = case["channels"], []
        for src in range(c):
            for dst in range(c):
                i = 100 + c * src + dst
                beta = [1.0] + [_unit(i, 1 + s) for s in range(ag.program.rand3(i, 0, 77) % 3)]
                kernels.append(Kernel(radius=float(10 + ag.program.rand3(i, 4, 77) % 21), beta=beta, src=src, dst=dst,
                                      mu=0.15 + 0.2 * _unit(i, 5), sigma=0.04 + 0.04 * _unit(i, 6), weight=1.0 / c))
        return [World(case["w"], case["h"], kernels, channels=c, dt=0.05)]
    w = ag.smoothlife(case["w"], case["h"])
    w.seed = Seed()
    return [w]


def _states(case, worlds, seed, device):
    """One flat float32 array: per world and channel a U[0,1] patch over half of each side, zeros around it."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    total = sum(w.channels * w.height * w.width for w in worlds)
    flat = torch.rand(total, generator=g, device=device)
    off = 0
    for w in worlds:
        n = w.channels * w.height * w.width
        a = flat[off:off + n].view(w.channels, w.height, w.width)
        y0, x0 = w.height // 4, w.width // 4
        a[:, :y0] = 0
        a[:, y0 + w.height // 2:] = 0
        a[:, :, :x0] = 0
        a[:, :, x0 + w.width // 2:] = 0
        off += n
    return flat


def _features(case, seed):
    g = torch.Generator()
    g.manual_seed(seed)
    x = torch.rand((case["rows"], 16), generator=g).numpy()
    y = (torch.rand((case["rows"], 3), generator=g) < 0.3).float().numpy()
    return x, y


def _params(seed, count):
    """A network as it is after some training: weights of the usual scale and biases that are not zero."""
    g = torch.Generator()
    g.manual_seed(seed + 1)
    p = torch.empty(count)
    for off, n, scale in ((0, 4096, 6 / 16), (4096, 256, 0.01), (4352, 65536, 6 / 256), (69888, 256, 0.01),
                          (70144, 768, 6 / 256), (70912, 3, 0.01)):
        p[off:off + n] = math.sqrt(scale) * (2 * torch.rand(n, generator=g) - 1)
    return p.numpy()


# ------------------------------------------------------------------ prepare and run

class _Engine:
    """A context over device-resident states, through the C ABI."""

    def __init__(self, worlds, path=_lib.PATH_FP32):
        self.L = _lib.load()
        self.ctx = ctypes.c_void_p()
        descs = (_lib.LeniaWorldDesc * len(worlds))(*[w.to_desc() for w in worlds])
        _lib.check(self.L.lenia_create(descs, len(worlds), path, ctypes.byref(self.ctx)))

    def __del__(self):
        if self.ctx:
            self.L.lenia_destroy(self.ctx)

    def call(self, name, *args):
        _lib.check(getattr(self.L, name)(self.ctx, *args), self.ctx)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("gradients", "predict"):
        mlp = Proposer(seed=1, max_batch=4096)
        mlp.set_params(_params(seed, mlp.nparam))
        x, y = _features(case, seed)
        return {"case": case, "mlp": mlp, "x": x, "y": y}
    worlds = _worlds(case)
    flat = _states(case, worlds, seed, "cuda")
    if kind == "frame":
        w = worlds[0]
        sim = ag.Sim(worlds)
        return {"case": case, "sim": sim, "in": flat.view(1, w.height, w.width).cpu().numpy()}
    if kind in ("batch", "screen"):
        sim = ag.Sim(worlds, path=case.get("path", "fp32"))
        a = torch.empty(flat.numel(), pin_memory=True)
        a.copy_(flat)
        out = torch.empty(flat.numel(), pin_memory=True)
        return {"case": case, "sim": sim, "in": a.numpy(), "out": out.numpy(), "pinned": (a, out)}
    torch.cuda.synchronize()
    return {"case": case, "engine": _Engine(worlds), "in": flat, "out": torch.empty_like(flat)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gradients":
        loss, g = state["mlp"].gradients(state["x"], state["y"])
        return {"loss": loss, "grads": g}
    if kind == "predict":
        return {"probs": state["mlp"].predict(state["x"])}
    if kind == "frame":
        sim = state["sim"]
        sim.write_state(0, state["in"])
        sim.step(1)
        return {"state": sim.read_state(0)}
    if kind in ("batch", "screen"):
        sim, got = state["sim"], {}
        sim.write_states_async(state["in"])
        if kind == "screen":
            got["stats"] = sim.stats()
        sim.step(case["gens"])
        sim.read_states_async(state["out"])
        sim.wait()
        got["states"] = state["out"]
        return got
    e, n = state["engine"], state["in"].numel()
    e.call("lenia_write_state_device", 0, state["in"].data_ptr(), n)
    e.call("lenia_step", case["gens"])
    e.call("lenia_read_state_device", 0, state["out"].data_ptr(), n)
    e.call("lenia_sync")
    return {"state": state["out"]}


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    if case["kind"] in ("gradients", "predict"):
        n, p = case["rows"], 70915
        macs = 16 * 256 + 256 * 256 + 256 * 3
        if case["kind"] == "predict":
            return {"bytes": 4 * (n * (16 + 3) + p), "flops": 2 * macs * n}
        return {"bytes": 4 * (n * (16 + 3) + 2 * p), "flops": 2 * n * (3 * macs - 16 * 256)}
    byts = flops = 0
    gens = case.get("gens", 1)
    for w in _worlds(case):
        cells = w.width * w.height
        fft = 2.5 * cells * math.log2(cells)  # a real 2-D transform
        byts += 8 * cells * w.channels + cells * len(w.kernels)
        flops += gens * (fft * (w.channels + len(w.kernels)) + cells * len(w.kernels) * 10)
    return {"bytes": byts, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits

def _core(q):
    inside = (q > 0) & (q < 1)
    s = torch.where(inside, q, torch.full_like(q, 0.5))
    return torch.where(inside, torch.exp(4 - 1 / (s * (1 - s))), torch.zeros_like(q))


def _spectrum(k, h, w, dev):
    y = torch.arange(h, device=dev, dtype=torch.float64)
    x = torch.arange(w, device=dev, dtype=torch.float64)
    r = torch.hypot(torch.minimum(y, h - y)[:, None], torch.minimum(x, w - x)[None, :])
    if k.shape == _lib.SHAPE_LENIA:
        b = torch.tensor([float(np.float32(v)) for v in k.beta] + [0.0], device=dev, dtype=torch.float64)
        n = len(k.beta)
        q = r / float(np.float32(k.radius)) * n
        shell = torch.clamp(q.floor(), 0, n)
        v = torch.where(q < n, b[shell.long()] * _core(q - shell), torch.zeros_like(q))
    elif k.shape == _lib.SHAPE_SL_INNER:
        v = torch.clamp(k.radius / 3 + 0.5 - r, 0, 1)
    else:
        v = torch.clamp(k.radius + 0.5 - r, 0, 1) * torch.clamp(r - k.radius / 3 + 0.5, 0, 1)
    return torch.fft.rfft2(v / v.sum()).real


def _f32(v):
    return float(np.float32(v))


def _exact_worlds(worlds, a, gens):
    """Worlds of one size and one rule, a [n, C, H, W] in 64 bits, `gens` generations on."""
    n, c, h, w = a.shape
    w0, dev = worlds[0], a.device
    col = lambda f: torch.tensor([[[_f32(f(x))]] for x in worlds], device=dev, dtype=torch.float64)  # noqa: E731
    spec = [torch.stack([_spectrum(x.kernels[k], h, w, dev) for x in worlds]) for k in range(len(w0.kernels))]
    dt = col(lambda x: x.dt)
    for _ in range(gens):
        f = torch.fft.rfft2(a)
        if w0.rule == _lib.RULE_SMOOTHLIFE:
            m, o = (torch.fft.irfft2(f[:, 0] * s, s=(h, w)) for s in spec)
            lg = lambda x, width: torch.sigmoid(x * (4 / width))  # noqa: E731
            t = lg(m - 0.5, 0.147)
            lo, hi = 0.278 * (1 - t) + 0.267 * t, 0.365 * (1 - t) + 0.445 * t
            target = lg(o - lo, 0.028) * (1 - lg(o - hi, 0.028))
            a = torch.clamp(a + 0.1 * (2 * target - 1)[:, None], 0, 1)
            continue
        growth = torch.zeros_like(a)
        for k, kern in enumerate(w0.kernels):
            u = torch.fft.irfft2(f[:, kern.src] * spec[k], s=(h, w))
            mu, sigma, weight = (col(lambda x: getattr(x.kernels[k], p)) for p in ("mu", "sigma", "weight"))
            growth[:, kern.dst] += weight * (2 * torch.exp(-((u - mu) ** 2) / (2 * sigma ** 2)) - 1)
        a = torch.clamp(a + dt[:, None] * growth, 0, 1)
    return a


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind in ("gradients", "predict"):
        x, y = (torch.from_numpy(v).to(dev).double() for v in _features(case, seed))
        p = torch.from_numpy(_params(seed, 70915)).to(dev).double().requires_grad_()
        w1, b1, w2 = p[:4096].view(256, 16), p[4096:4352], p[4352:69888].view(256, 256)
        b2, w3, b3 = p[69888:70144], p[70144:70912].view(3, 256), p[70912:]
        z = torch.relu(torch.relu(x @ w1.T + b1) @ w2.T + b2) @ w3.T + b3
        if kind == "predict":
            return {"probs": torch.sigmoid(z).detach()}
        loss = torch.nn.functional.binary_cross_entropy_with_logits(z, y)
        loss.backward()
        return {"loss": float(loss.detach()), "grads": p.grad}
    worlds = _worlds(case)
    flat = _states(case, worlds, seed, dev)
    parts, off = [], 0
    for w in worlds:
        n = w.channels * w.height * w.width
        parts.append(flat[off:off + n].view(w.channels, w.height, w.width))
        off += n
    out = torch.empty(flat.numel(), dtype=torch.float64, device=dev)
    views, off = [], 0
    for w in worlds:
        n = w.channels * w.height * w.width
        views.append(out[off:off + n].view(w.channels, w.height, w.width))
        off += n
    groups = {}
    for i, w in enumerate(worlds):
        groups.setdefault((w.width, w.height), []).append(i)
    for members in groups.values():
        most = max(1, (1 << 26) // parts[members[0]].numel())
        for at in range(0, len(members), most):
            some = members[at:at + most]
            a = _exact_worlds([worlds[i] for i in some], torch.stack([parts[i] for i in some]).double(), case.get("gens", 1))
            for i, v in zip(some, a):
                views[i].copy_(v)
    if kind == "frame":
        return {"state": out.view(1, case["h"], case["w"])}
    if kind != "screen":
        return {"states" if kind == "batch" else "state": out}
    stats = []
    for p in parts:  # mass and the circular mean of each axis, as the screen reads them
        s, (h, w) = p[0].double(), p.shape[1:]
        row = [s.sum()]
        for m, n in ((s.sum(0), w), (s.sum(1), h)):
            ang = torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n)
            c = torch.atan2((m * ang.sin()).sum(), (m * ang.cos()).sum()) / (2 * math.pi) * n
            row.append(torch.where(c < 0, c + n, c))
        stats.append(torch.stack(row))
    return {"stats": torch.stack(stats), "states": out}
