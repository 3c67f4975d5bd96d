"""Workloads of the engine, as a program that uses it calls them.

Kinds of call, each through the public entry points:

* ``step``: ``Model.step`` on host arrays, one tick of one grid (the loop of the
  reference's ``engine-cli rollout`` and of its web demo);
* ``rollout``: ``jc_rollout_device``, many projected ticks of one grid whose
  state is on the device;
* ``batch``: ``Batch.rollout`` on device buffers, many grids of several sizes
  and horizons, forward and rewind checkpoints in one call;
* ``serve``: ``Server.submit_device`` / ``wait_device``, forward, rewind and
  reconstruct requests together;
* ``solver``: ``jc_sw_run_device``, the shallow-water solver on many states.

Checkpoints are the synthetic seeded families of ``checkpoint.py`` (forward
family seed 0, reverse family seed 1: weights do not depend on the inputs' seed);
fields are 1 to 8 Gaussian drops of amplitude 0.02-0.15 and width 2-6 cells.
``exact`` restates the forward, the projections, the reconstruct rule and the
solver in float64 torch.
"""

import ctypes as C
import functools
import math
import random

import numpy as np
import torch

from jacobi2000_gb300 import engine
from jacobi2000_gb300.checkpoint import parse_config, synthetic_family, write_safetensors_bytes

FORWARD, REVERSE = 0, 1  # family seeds
KEEP = 0.02  # share of the space-time cells a reconstruct request knows
SWEEPS = 4
FLAGS = engine.PROJECT_MASS | engine.PROJECT_ENERGY
MIXED = 4  # distinct grids of a mixed batch or of a served load


def listed():
    return [
        # the smallest call there is: one interactive tick, latency and launches only
        {"name": "step_f32_32", "kind": "step", "bf16": False, "nx": 32, "ny": 32, "dim": 128, "layers": 4},
        # one tick of the model's own published grid in the precision form
        {"name": "step_bf16_64", "kind": "step", "bf16": True, "nx": 64, "ny": 64, "dim": 128, "layers": 4},
        # a plain FP32 rollout, one request at a time
        {"name": "rollout_f32_128", "kind": "rollout", "bf16": False, "nx": 128, "ny": 128, "dim": 128, "layers": 4,
         "ticks": 10},
        # a small ragged grid (token tiles and cell tiles overhang it on both sides)
        {"name": "rollout_bf16_100x60", "kind": "rollout", "bf16": True, "nx": 100, "ny": 60, "dim": 128, "layers": 4,
         "ticks": 20},
        # the largest grid of the served range, alone
        {"name": "rollout_bf16_256", "kind": "rollout", "bf16": True, "nx": 256, "ny": 256, "dim": 128, "layers": 4,
         "ticks": 10},
        # the wide model on the largest grid
        {"name": "rollout_bf16_256_wide", "kind": "rollout", "bf16": True, "nx": 256, "ny": 256, "dim": 256,
         "layers": 6, "ticks": 10},
        # FP32 rollouts of several grids at once (scoring a checkpoint at full precision)
        {"name": "batch_f32_mixed", "kind": "batch", "bf16": False, "count": 24, "lo": 32, "hi": 128, "rewind": False,
         "ticks": 8, "grids": 11},
        # the uniform batch: one grid size, every instance to the same horizon
        {"name": "batch_bf16_64x128", "kind": "batch", "bf16": True, "count": 64, "lo": 128, "hi": 128,
         "rewind": False, "ticks": 8, "grids": 0},
        # a heterogeneous batch: forward and rewind, sides 32-192, horizons of 1/4 to all of the ticks
        {"name": "batch_bf16_mixed", "kind": "batch", "bf16": True, "count": 64, "lo": 32, "hi": 192, "rewind": True,
         "ticks": 16, "grids": 5},
        # one reconstruct request on an idle server: a space-time volume, four Jacobi sweeps
        {"name": "reconstruct_bf16_96", "kind": "serve", "bf16": True, "count": 1, "lo": 96, "hi": 96, "tasks": "c",
         "ticks": 16, "grids": 0},
        # a served load of the three tasks, sides 32-256
        {"name": "serve_bf16_mixed", "kind": "serve", "bf16": True, "count": 48, "lo": 32, "hi": 256,
         "tasks": "frc", "ticks": 16, "grids": 3},
        # solver trajectories to score against, or to train on
        {"name": "solver_96x256", "kind": "solver", "nx": 256, "ny": 256, "count": 96, "steps": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "rollout", "rollout", "batch", "batch", "serve", "solver"])
    bf16 = rng.random() < 0.7

    def side(lo, hi):
        return max(lo, min(hi, 4 * _log(rng, lo / 4, hi / 4)))

    if kind == "step":
        return {"kind": kind, "bf16": bf16, "nx": side(32, 128), "ny": side(32, 128), "dim": 128, "layers": 4}
    if kind == "rollout":
        wide = rng.random() < 0.25
        hi = 256 if bf16 else 128
        return {"kind": kind, "bf16": bf16, "nx": side(32, hi), "ny": side(32, hi), "dim": 256 if wide else 128,
                "layers": 6 if wide else 4, "ticks": rng.randint(4, 10) if wide else rng.randint(4, 20)}
    if kind == "batch":
        lo = side(32, 96)
        return {"kind": kind, "bf16": bf16, "count": _log(rng, 2, 64 if bf16 else 24), "lo": lo,
                "hi": side(lo, 192 if bf16 else 128), "rewind": rng.random() < 0.5, "ticks": rng.randint(4, 12),
                "grids": rng.randint(0, 9999)}
    if kind == "serve":
        return {"kind": kind, "bf16": True, "count": _log(rng, 1, 32), "lo": 32, "hi": side(48, 256),
                "tasks": rng.choice(["f", "r", "c", "fr", "frc"]), "ticks": rng.randint(6, 14),
                "grids": rng.randint(0, 9999)}
    return {"kind": kind, "nx": _log(rng, 32, 256), "ny": _log(rng, 32, 256), "count": _log(rng, 2, 96),
            "steps": rng.randint(1, 16)}


# ---- checkpoints and inputs -----------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _stream():
    """The one stream a program issues its device work on."""
    return torch.cuda.Stream()


@functools.lru_cache(maxsize=None)
def _checkpoint(nx, ny, dim, layers, seed):
    tensors, config = synthetic_family(dim, layers, seed, [], rect=[(nx, ny)])[(nx, ny)]
    return tensors, config, parse_config(config, tensors)


@functools.lru_cache(maxsize=None)
def _packed(nx, ny, dim, layers, seed, bf16):
    """The pre-packed checkpoint a program keeps beside model.safetensors."""
    tensors, config, _ = _checkpoint(nx, ny, dim, layers, seed)
    with engine.Model.from_bytes(write_safetensors_bytes(tensors), config, engine.BF16 if bf16 else engine.FP32) as m:
        return m.pack()


def _model(nx, ny, dim, layers, seed, bf16):
    return engine.Model.from_packed(_packed(nx, ny, dim, layers, seed, bf16))


def _fields(cfg, count, gen):
    """Normalized states [count, 3, ny, nx] of 1 to 8 drops each, periodic images included."""
    dev = torch.device("cuda")
    ys = torch.arange(cfg.ny, device=dev, dtype=torch.float32)[None, :, None]
    xs = torch.arange(cfg.nx, device=dev, dtype=torch.float32)[None, None, :]
    h = torch.full((count, cfg.ny, cfg.nx), cfg.depth, device=dev)
    p = torch.rand((8, 5, count), generator=gen).to(dev)
    for d in range(8):
        cx, cy, amp, sigma = p[d, 0] * cfg.nx, p[d, 1] * cfg.ny, 0.02 + 0.13 * p[d, 2], 2 + 4 * p[d, 3]
        amp = amp * ((p[d, 4] < 0.6) if d else 1.0)
        inv = (0.5 / (sigma * sigma))[:, None, None]
        for ox in (-cfg.nx, 0, cfg.nx):
            for oy in (-cfg.ny, 0, cfg.ny):
                dx, dy = xs - (cx + ox)[:, None, None], ys - (cy + oy)[:, None, None]
                h += amp[:, None, None] * torch.exp(-(dx * dx + dy * dy) * inv)
    x = torch.zeros((count, 3, cfg.ny, cfg.nx), device=dev)
    x[:, 0] = (h - cfg.norm_depth - cfg.norm_mean[0]) / cfg.norm_std[0]
    x[:, 1] = -cfg.norm_mean[1] / cfg.norm_std[1]
    x[:, 2] = -cfg.norm_mean[2] / cfg.norm_std[2]
    return x


def _meta(cfg):
    f = np.float32
    return np.array([np.log(f(cfg.dx)), np.log(f(cfg.dt)), np.log(f(cfg.g)), np.log(f(cfg.depth)),
                     np.log(f(cfg.nu) + f(1e-6))], dtype=np.float32)


def _grids(case):
    """The grids of a batch or a served load: up to MIXED sizes in [lo, hi], the first of side hi."""
    rng = random.Random(case["grids"])
    lo, hi = case["lo"], case["hi"]
    if lo == hi:
        return [(lo, lo)]

    def one():
        return max(lo, min(hi, 4 * _log(rng, lo / 4, hi / 4)))

    return [(hi, hi)] + [(one(), one()) for _ in range(MIXED - 1)]


def _jobs(case):
    """(task, grid index, ticks) of every instance or request: f forward, r rewind, c reconstruct. The largest grid is
    one in eight."""
    rng = random.Random(case["grids"] + 1)
    n = len(_grids(case))
    tasks = case["tasks"] if case["kind"] == "serve" else ("fr" if case["rewind"] else "f")
    jobs = []
    for k in range(case["count"]):
        g = 0 if n == 1 or k % 8 == 0 else rng.randint(1, n - 1)
        task = tasks[k % len(tasks)]
        ticks = case["ticks"]
        if n > 1:
            ticks = rng.randint(max(1, ticks // 4), ticks)
        if task == "c" and n > 1:
            ticks = min(ticks, 8)
        jobs.append((task, g, ticks))
    return jobs


def _inputs(case, seed):
    """Every job's input on the GPU: the state, or for a reconstruct (values, known)."""
    gen = torch.Generator().manual_seed(seed)
    grids, jobs = _grids(case), _jobs(case)
    out = []
    for g, (nx, ny) in enumerate(grids):
        cfg = _checkpoint(nx, ny, 128, 4, FORWARD)[2]
        mine = [k for k, j in enumerate(jobs) if j[1] == g]
        fields = _fields(cfg, max(1, len(mine)), gen)
        out += [(k, fields[i]) for i, k in enumerate(mine)]
    out = [x for _, x in sorted(out, key=lambda p: p[0])]
    for k, (task, g, ticks) in enumerate(jobs):
        if task == "c":
            nx, ny = grids[g]
            known = (torch.rand((ticks + 1, ny, nx), generator=gen) < KEEP).to("cuda")
            vals = out[k][None] * torch.linspace(1.0, 0.7, ticks + 1, device="cuda")[:, None, None, None]
            out[k] = (torch.where(known[:, None], vals, torch.zeros_like(vals)).contiguous(),
                      known.to(torch.uint8).contiguous())
        else:
            out[k] = out[k].contiguous()
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solver":
        cfg = _checkpoint(32, 32, 128, 4, FORWARD)[2]
        p = engine.JcSwParams(case["nx"], case["ny"], cfg.dx, cfg.dt, cfg.g, cfg.depth, cfg.nu)
        lib = engine.load_library()
        engine._declare_eval(lib)
        s = {"case": case, "p": p, "lib": lib, "x0": _solver_states(case, seed), "stream": _stream()}
        s["x"] = torch.empty_like(s["x0"])
    elif kind in ("step", "rollout"):
        nx, ny = case["nx"], case["ny"]
        cfg = _checkpoint(nx, ny, case["dim"], case["layers"], FORWARD)[2]
        x = _fields(cfg, 1, torch.Generator().manual_seed(seed))[0]
        s = {"case": case, "model": _model(nx, ny, case["dim"], case["layers"], FORWARD, case["bf16"])}
        if kind == "step":  # the caller's state is a host array
            s.update(x=x.cpu().numpy(), meta=_meta(cfg))
        else:
            s.update(x=x, meta=torch.from_numpy(_meta(cfg)).cuda(), out=torch.empty_like(x),
                     lib=engine.load_library(), stream=_stream())
    else:
        grids, jobs = _grids(case), _jobs(case)
        tasks = {t for t, _, _ in jobs}
        fwd = [_model(nx, ny, 128, 4, FORWARD, case["bf16"]) for nx, ny in grids]
        rev = [_model(nx, ny, 128, 4, REVERSE, case["bf16"]) for nx, ny in grids] if tasks & set("rc") else []
        meta = torch.from_numpy(_meta(_checkpoint(*grids[0], 128, 4, FORWARD)[2])).cuda()
        x = _inputs(case, seed)
        shapes = [((t + 1,) if task == "c" else ()) + (3, grids[g][1], grids[g][0]) for task, g, t in jobs]
        ends = np.cumsum([int(np.prod(sh)) for sh in shapes])
        flat = torch.empty(int(ends[-1]), device="cuda")  # every result, one after another
        s = {"case": case, "jobs": jobs, "fwd": fwd, "rev": rev, "meta": meta, "x": x, "flat": flat}
        s["out"] = [flat[e - int(np.prod(sh)):e] for e, sh in zip(ends, shapes)]
        if kind == "batch":
            cells = sum(grids[g][0] * grids[g][1] for _, g, _ in jobs)
            s["batch"] = engine.Batch(fwd + rev, max_instances=len(jobs), max_cells=cells)
            s["stream"] = _stream()
            s["items"] = [(g + (len(fwd) if task == "r" else 0), x[k].data_ptr(), meta.data_ptr(), ticks, FLAGS,
                           s["out"][k].data_ptr()) for k, (task, g, ticks) in enumerate(jobs)]
        else:
            s["server"] = engine.Server(fwd, rev or None, max_active_cells=1 << 21)
    torch.cuda.synchronize()
    return s


def _solver_states(case, seed):
    cfg = _checkpoint(32, 32, 128, 4, FORWARD)[2]
    gen = torch.Generator().manual_seed(seed)
    n, ny, nx = case["count"], case["ny"], case["nx"]
    ys = torch.arange(ny, device="cuda", dtype=torch.float32)[None, :, None]
    xs = torch.arange(nx, device="cuda", dtype=torch.float32)[None, None, :]
    p = torch.rand((3, 6, n), generator=gen).cuda()[..., None, None]
    x = torch.zeros((n, 3, ny, nx), device="cuda")
    x[:, 0] = cfg.depth
    for d in range(3):
        r2 = (xs - p[d, 0] * nx) ** 2 + (ys - p[d, 1] * ny) ** 2
        bump = torch.exp(-r2 * (0.5 / (2 + 4 * p[d, 3]) ** 2))
        x[:, 0] += (0.02 + 0.13 * p[d, 2]) * bump
        x[:, 1] += 0.1 * (p[d, 4] - 0.5) * bump
        x[:, 2] += 0.1 * (p[d, 5] - 0.5) * bump
    return x


# ---- one pass -------------------------------------------------------------------------


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        return s["model"].step(s["x"], s["meta"])
    if kind == "rollout":
        engine._check(s["lib"].jc_rollout_device(s["model"]._h, s["x"].data_ptr(), s["meta"].data_ptr(),
                                                 case["ticks"], FLAGS, s["out"].data_ptr(), None,
                                                 s["stream"].cuda_stream))
        return s["out"]
    if kind == "batch":
        s["batch"].rollout(s["items"], device=True, stream=s["stream"].cuda_stream)
        return s["flat"]
    if kind == "serve":
        tasks = {"f": engine.TASK_FORWARD, "r": engine.TASK_REWIND, "c": engine.TASK_RECONSTRUCT}
        server, meta = s["server"], s["meta"].data_ptr()
        ids = []
        for (task, g, ticks), x in zip(s["jobs"], s["x"]):
            if task == "c":
                ids.append(server.submit_device(tasks[task], g, x[0].data_ptr(), meta, ticks, 0,
                                                known_ptr=x[1].data_ptr(), max_sweeps=SWEEPS, tol=0.0))
            else:
                ids.append(server.submit_device(tasks[task], g, x.data_ptr(), meta, ticks, FLAGS))
        for rid, out in zip(ids, s["out"]):
            server.wait_device(rid, out.data_ptr(), out.numel())
        return s["flat"]
    with torch.cuda.stream(s["stream"]):
        s["x"].copy_(s["x0"])
    engine._check(s["lib"].jc_sw_run_device(C.byref(s["p"]), s["x"].data_ptr(), case["count"], case["steps"],
                                            s["stream"].cuda_stream))
    return s["x"]


# ---- what a pass cannot do without --------------------------------------------------------


def _params(nx, ny, dim, layers):
    pos = nx * ny // 16 * dim
    block = 4 * dim * dim + 8 * dim * dim + 13 * dim
    return pos + 54 * dim + layers * block + 2 * dim + 9 * dim * dim + dim + 33 * dim + 9 * 35 * 32 + 9 * 32 * 3 + 99


def _cell_flops(dim, layers):
    token = 2 * 48 * dim + layers * (2 * 12 * dim * dim + 36 * dim) + 2 * 9 * dim * dim + 2 * 32 * dim
    return token / 16 + 2 * 9 * (35 * 32 + 32 * 3) + 32 * 6


def work(case):
    kind = case["kind"]
    if kind == "solver":
        n = case["count"] * case["nx"] * case["ny"]
        return {"bytes": 24 * n, "flops": 75 * n * case["steps"]}
    if kind in ("step", "rollout"):
        n, dim, layers = case["nx"] * case["ny"], case["dim"], case["layers"]
        ticks = case.get("ticks", 1)
        return {"bytes": 24 * n + (2 if case["bf16"] else 4) * _params(case["nx"], case["ny"], dim, layers),
                "flops": n * ticks * _cell_flops(dim, layers)}
    grids = _grids(case)
    flops, size = 0.0, (2 if case["bf16"] else 4) * sum(_params(nx, ny, 128, 4) for nx, ny in grids)
    for task, g, ticks in _jobs(case):
        n = grids[g][0] * grids[g][1]
        if task == "c":
            flops += SWEEPS * 2 * ticks * n * _cell_flops(128, 4)
            size += (ticks + 1) * n * 25
        else:
            flops += ticks * n * _cell_flops(128, 4)
            size += 24 * n
    return {"bytes": size, "flops": flops}


# ---- the same in float64 ----------------------------------------------------------------


class _Exact:
    """The reference's forward and projections on [B, 3, ny, nx] float64 states."""

    def __init__(self, nx, ny, dim, layers, seed):
        tensors, _, self.cfg = _checkpoint(nx, ny, dim, layers, seed)
        self.w = {k: torch.from_numpy(v).cuda().double() for k, v in tensors.items()}
        f = lambda v: float(np.float32(v))  # noqa: E731  the configuration is read as f32
        c = self.cfg
        self.mean, self.std = [f(v) for v in c.norm_mean], [f(v) for v in c.norm_std]
        self.depth, self.g, self.r_max = f(c.norm_depth), f(c.g), f(c.energy_r_max)
        self.meta = torch.from_numpy(_meta(c)).cuda().double()

    def _norm(self, x, name):
        m = x.mean(-1, keepdim=True)
        v = ((x - m) ** 2).mean(-1, keepdim=True)
        return (x - m) / torch.sqrt(v + float(np.float32(1e-5))) * self.w[name + ".gamma"] + self.w[name + ".beta"]

    def _lin(self, x, name):
        return x @ self.w[name + ".weight"] + self.w[name + ".bias"]

    @staticmethod
    def _gelu(x):
        return 0.5 * x * (1 + torch.erf(x / math.sqrt(2.0)))

    def _conv3(self, x, name):  # x [B, ny, nx, C], zero padding
        w = self.w[name + ".weight"]
        ny, nx = x.shape[1:3]
        p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
        y = self.w[name + ".bias"].expand(x.shape[0], ny, nx, -1).clone()
        for ky in range(3):
            for kx in range(3):
                y += p[:, ky:ky + ny, kx:kx + nx] @ w[:, :, ky, kx].T
        return y

    def _attention(self, n, name, ty, tx):
        b, heads = n.shape[0], self.cfg.heads
        q, k, v = (self._lin(n, name + p).reshape(b, ty, tx, heads, -1) for p in ("q", "k", "v"))
        pad = lambda t: torch.nn.functional.pad(t, (0, 0, 0, 0, 1, 1, 1, 1))  # noqa: E731
        k, v = pad(k), pad(v)
        inside = torch.nn.functional.pad(torch.ones(ty, tx, dtype=torch.bool, device="cuda"), (1, 1, 1, 1))
        at = [(dy, dx) for dy in range(3) for dx in range(3)]
        s = torch.stack([((q * k[:, dy:dy + ty, dx:dx + tx]).sum(-1) / math.sqrt(q.shape[-1])).masked_fill(
            ~inside[dy:dy + ty, dx:dx + tx, None], -math.inf) for dy, dx in at])
        s = torch.softmax(s, 0)
        o = sum(s[i][..., None] * v[:, dy:dy + ty, dx:dx + tx] for i, (dy, dx) in enumerate(at))
        return o.reshape(b, ty * tx, -1)

    @staticmethod
    def _up(z, dim):  # linear x4 along `dim`, the far neighbour clamped
        far = torch.cat([z.narrow(dim, 1, z.shape[dim] - 1), z.narrow(dim, z.shape[dim] - 1, 1)], dim)
        parts = [z * (1 - (i + 0.5) / 4) + far * ((i + 0.5) / 4) for i in range(4)]
        return torch.stack(parts, dim + 1).flatten(dim, dim + 1)

    def forward(self, x):
        c = self.cfg
        b, ty, tx = x.shape[0], c.ny // 4, c.nx // 4
        patches = x.reshape(b, 3, ty, 4, tx, 4).permute(0, 2, 4, 1, 3, 5).reshape(b, ty * tx, 48)
        h = self._lin(patches, "embed") + self.w["pos"] + self._lin(self.meta, "meta")
        for i in range(c.layers):
            p = "blocks.%d." % i
            h = h + self._lin(self._attention(self._norm(h, p + "norm1"), p, ty, tx), p + "proj")
            h = h + self._lin(self._gelu(self._lin(self._norm(h, p + "norm2"), p + "ff1")), p + "ff2")
        n = self._norm(h, "norm").reshape(b, ty, tx, -1)
        t = n + self._gelu(self._conv3(n, "head.token_mix"))
        z = t @ self.w["head.to_cells.weight"][:, :, 0, 0].T + self.w["head.to_cells.bias"]
        z = torch.cat([self._up(self._up(z, 1), 2), x.permute(0, 2, 3, 1)], -1)
        z = self._conv3(self._gelu(self._conv3(z, "head.conv1")), "head.conv2")
        return z.permute(0, 3, 1, 2)

    def _energy(self, x):
        h = x[:, 0] * self.std[0] + self.mean[0] + self.depth
        u, v = x[:, 1] * self.std[1] + self.mean[1], x[:, 2] * self.std[2] + self.mean[2]
        return (0.5 * self.g * h * h).sum((1, 2)), (0.5 * h * (u * u + v * v)).sum((1, 2)), u, v

    def rollout(self, x, ticks):
        mass = x[:, 0].mean((1, 2))
        e = sum(self._energy(x)[:2])
        for _ in range(ticks):
            x = x + self.forward(x)
            x[:, 0] += (mass - x[:, 0].mean((1, 2)))[:, None, None]
            pot, kin, u, v = self._energy(x)
            s = torch.sqrt((e * self.r_max - pot).clamp(min=0) / kin.clamp(min=1e-12)).clamp(0, 1)[:, None, None]
            x[:, 1] = (u * s - self.mean[1]) / self.std[1]
            x[:, 2] = (v * s - self.mean[2]) / self.std[2]
            e = sum(self._energy(x)[:2])
        return x


def _reconstruct(fwd, rev, vals, known):
    known = known.bool()[:, None]
    vals = vals.double()
    x = torch.where(known, vals, torch.zeros_like(vals))
    for _ in range(SWEEPS):
        f, r = x[:-1] + fwd.forward(x[:-1]), x[1:] + rev.forward(x[1:])
        new = torch.cat([r[:1], 0.5 * (f[:-1] + r[1:]), f[-1:]])
        x = torch.where(known, x, new)
    return x


def _solver(x, p, steps):
    h, u, v = x.unbind(1)
    r, i2, ii = p.dt / p.dx, 1 / (2 * p.dx), 1 / (p.dx * p.dx)
    for _ in range(steps):
        fx = 0.25 * (h[:, :, :-1] + h[:, :, 1:]) * (u[:, :, :-1] + u[:, :, 1:])
        fy = 0.25 * (h[:, :-1] + h[:, 1:]) * (v[:, :-1] + v[:, 1:])
        fx, fy = torch.nn.functional.pad(fx, (1, 1)), torch.nn.functional.pad(fy, (0, 0, 1, 1))
        h = h - r * (fx[:, :, 1:] - fx[:, :, :-1] + fy[:, 1:] - fy[:, :-1])

        def near(q, sx, sy):
            left, right = torch.cat([sx * q[:, :, :1], q[:, :, :-1]], 2), torch.cat([q[:, :, 1:], sx * q[:, :, -1:]], 2)
            down, up = torch.cat([sy * q[:, :1], q[:, :-1]], 1), torch.cat([q[:, 1:], sy * q[:, -1:]], 1)
            return left, right, down, up

        hl, hr, hd, hu = near(h, 1, 1)
        ul, ur, ud, uu = near(u, -1, 1)
        vl, vr, vd, vu = near(v, 1, -1)
        du = -u * (ur - ul) * i2 - v * (uu - ud) * i2 - p.g * (hr - hl) * i2 + p.nu * (ul + ur + ud + uu - 4 * u) * ii
        dv = -u * (vr - vl) * i2 - v * (vu - vd) * i2 - p.g * (hu - hd) * i2 + p.nu * (vl + vr + vd + vu - 4 * v) * ii
        u, v = u + p.dt * du, v + p.dt * dv
    return torch.stack([h, u, v], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "solver":
        cfg = _checkpoint(32, 32, 128, 4, FORWARD)[2]
        p = engine.JcSwParams(case["nx"], case["ny"], cfg.dx, cfg.dt, cfg.g, cfg.depth, cfg.nu)
        x = _solver_states(case, seed)
        return torch.cat([_solver(x[k:k + 16].double(), p, case["steps"]) for k in range(0, len(x), 16)])
    if kind in ("step", "rollout"):
        m = _Exact(case["nx"], case["ny"], case["dim"], case["layers"], FORWARD)
        x = _fields(m.cfg, 1, torch.Generator().manual_seed(seed)).double()
        return (x + m.forward(x))[0].cpu().numpy() if kind == "step" else m.rollout(x, case["ticks"])[0]
    grids, jobs, inputs = _grids(case), _jobs(case), _inputs(case, seed)
    made = functools.lru_cache(maxsize=None)(lambda g, way: _Exact(*grids[g], 128, 4, way))
    out = [None] * len(jobs)
    alike = {}  # jobs of one task, grid and horizon run together
    for k, (task, g, ticks) in enumerate(jobs):
        if task == "c":
            out[k] = _reconstruct(made(g, FORWARD), made(g, REVERSE), *inputs[k])
        else:
            alike.setdefault((task, g, ticks), []).append(k)
    for (task, g, ticks), ks in alike.items():
        m = made(g, FORWARD if task == "f" else REVERSE)
        for i in range(0, len(ks), 8):
            part = ks[i:i + 8]
            y = m.rollout(torch.stack([inputs[k] for k in part]).double(), ticks)
            for k, v in zip(part, y):
                out[k] = v
    return torch.cat([v.reshape(-1) for v in out])
