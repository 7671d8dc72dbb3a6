"""Performance cases: the work a program asks of this package, through its public entry points.

A case is a dict of plain values.  Its `kind` names the entry point:
  step    PBFSolver.step on records in device memory (options: exact math, resident state, SDF
          obstacles, mixed masses, table size), the simulation loop of a game or a solver study
  host    PBFSolver.step on a host array of records (pinned): a program whose particles live on
          the host between steps
  batch   BatchSolver.step: many independent scenes per step (parameter studies, training data)
  warm    PBFSolver.step with the learned lambda warm start attached
  train   LambdaNet.adam_step over minibatches, then the trained weights read back
  render  SplatRenderer.render: one frame of the records
  sort    akua_sort_pairs_noalloc: the stable pair sort without allocations

Fluid inputs are a block in motion: a slightly compressed lattice with jitter well beyond the
benchmark scenes' (the neighbourhoods of a developed flow, about 30 neighbours, not those of a
resting lattice), a smooth velocity field and noise, in a box it does not fill.  A step rewrites
its records, so a second pass on one state is the scene's next step.
"""
import ctypes
import math
import random

import numpy as np
import torch

import akuaengine_gb300 as ak
from akuaengine_gb300 import _abi
from akuaengine_gb300.render import Camera, SplatRenderer
from akuaengine_gb300.warm_start import LambdaNet, init_params

H = 0.1            # smoothing radius (PBFConfig's default)
SPACING = 0.05     # lattice spacing 0.5 h
COMPRESS = 0.98    # the flow's mean spacing over the lattice's
JITTER = 0.15      # of the spacing, uniform, per axis
DT = 0.0083
# float32 words of a 108-byte record: name -> (first word, words)
FIELDS = {"position": (0, 3), "velocity": (3, 3), "new_position": (6, 3), "new_velocity": (9, 3),
          "position_delta": (12, 3), "vorticity": (15, 3), "mass": (18, 1), "density": (19, 1),
          "lambda": (20, 1), "hash": (21, 1), "color": (22, 4), "size": (26, 1)}
# typical scales of the network's inputs and output on these scenes
NET_MEAN = [0.06, 0.95, 500.0, -6e-5, -1e-4, 5.0, 0.0, 2.0]
NET_INV_STD = [10.0, 8.0, 5e-3, 1e4, 5e3, 0.2, 0.2, 1.0]
NET_SCALE = 1e-4
BLEND = 0.1
LEARNING_RATE = 1e-3


# ---------------------------------------------------------------------------------------- cases
def listed():
    return [
        # a droplet or a unit test's scene: a step is its launches' latency
        {"name": "step_1k", "kind": "step", "n": 1000, "iterations": 4},
        # the reference's real-time dam break (30^3 particles)
        {"name": "step_27k", "kind": "step", "n": 27000, "iterations": 4},
        # a reproducibility study: exact math, two masses, an odd count
        {"name": "exact_100k", "kind": "step", "n": 100003, "iterations": 4, "exact_math": True,
         "mixed_mass": True},
        # an interactive scene with obstacles whose state stays on the device
        {"name": "resident_300k", "kind": "step", "n": 301119, "iterations": 3, "resident": True,
         "obstacles": True},
        # the benchmark's large dam break
        {"name": "step_1m", "kind": "step", "n": 1000000, "iterations": 4},
        # the double dam break with a 2^24-bucket table (buckets of several cells)
        {"name": "double_8m", "kind": "step", "n": 8000000, "iterations": 4, "blocks": 2,
         "table_size": 1 << 24},
        # 256 scenes of 2,000 to 64,000 particles, about 5 million in all
        {"name": "batch_256", "kind": "batch", "scenes": 256, "n_min": 2000, "n_max": 64000,
         "iterations": 4, "sizes_seed": 1},
        # the learned warm start: two iterations behind the network
        {"name": "warm_1m", "kind": "warm", "n": 1000000, "iterations": 2},
        # records on the host, copied in and out by every step
        {"name": "host_250k", "kind": "host", "n": 250047, "iterations": 4},
        # training the network: eight minibatches of the trainer's default size
        {"name": "train_8x64k", "kind": "train", "batch": 65536, "batches": 8},
        # one frame of the large scene
        {"name": "render_1m", "kind": "render", "n": 1000000, "width": 1280, "height": 720},
        # the allocation-free sort at its limit, on 27-bit cell hashes
        {"name": "sort_1m", "kind": "sort", "n": 1 << 20, "key_bits": 27},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "host", "batch", "warm", "train", "render",
                       "sort"])
    if kind in ("step", "host", "warm"):
        c = {"kind": kind, "n": _log(rng, 500, 1000000 if kind == "host" else 4000000),
             "iterations": rng.randint(1, 5)}
        if kind == "step":
            for flag, p in (("exact_math", 0.3), ("resident", 0.3), ("obstacles", 0.25),
                            ("mixed_mass", 0.25)):
                if rng.random() < p:
                    c[flag] = True
            if rng.random() < 0.25:
                c["blocks"] = 2
            if rng.random() < 0.25:
                c["table_size"] = max(64, c["n"] * rng.randint(1, 8))
        return c
    if kind == "batch":
        lo = _log(rng, 300, 3000)
        return {"kind": kind, "scenes": _log(rng, 2, 256), "n_min": lo,
                "n_max": lo + _log(rng, 100, 40000), "iterations": rng.randint(1, 5),
                "sizes_seed": rng.randrange(1 << 20)}
    if kind == "train":
        return {"kind": kind, "batch": _log(rng, 300, 200000), "batches": rng.randint(1, 8)}
    if kind == "render":
        return {"kind": kind, "n": _log(rng, 500, 4000000), "width": rng.randint(160, 1920),
                "height": rng.randint(120, 1080)}
    return {"kind": kind, "n": _log(rng, 100, 1 << 20), "key_bits": rng.randint(6, 32)}


# --------------------------------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _block_dims(n):
    side = max(1, int(round(n ** (1.0 / 3.0))))
    return -(-n // (side * side)), side, side


def _records(positions, gen, mixed_mass):
    """Records of a fluid at `positions` [n, 3]: velocities a smooth field plus noise."""
    n = positions.shape[0]
    buf = torch.zeros(n, 27, dtype=torch.float32, device="cuda")
    buf[:, 0:3] = positions
    phase = torch.rand(3, generator=gen, device="cuda") * 6.28
    noise = torch.randn(n, 3, generator=gen, device="cuda") * 0.1
    x = positions
    buf[:, 3] = 1.5 + 0.5 * torch.sin(2.0 * x[:, 1] + phase[0]) + noise[:, 0]
    buf[:, 4] = -1.0 + 0.5 * torch.sin(2.0 * x[:, 2] + phase[1]) + noise[:, 1]
    buf[:, 5] = 0.5 * torch.sin(2.0 * x[:, 0] + phase[2]) + noise[:, 2]
    buf[:, 18] = 1.0
    if mixed_mass:  # two fluids
        buf[:, 18] = torch.where(torch.rand(n, generator=gen, device="cuda") < 0.3, 0.8, 1.0)
    buf[:, 24] = 1.0  # blue, opaque
    buf[:, 25] = 1.0
    buf[:, 26] = 50.0
    return buf


def _fluid(n, seed, blocks=1, mixed_mass=False):
    """(records [n, 27], box_min, box_max): `blocks` blocks of particles, `n` in all."""
    gen = _generator(seed)
    per = [n // blocks + (1 if b < n % blocks else 0) for b in range(blocks)]
    dims = _block_dims(max(per))
    s = SPACING * COMPRESS
    width = dims[0] * SPACING
    high = (max(3.0 * blocks * width, 1.0), max(1.5 * dims[1] * SPACING, 0.6),
            max(1.5 * dims[2] * SPACING, 0.6))
    parts = []
    for b, m in enumerate(per):
        k = torch.arange(m, device="cuda")
        idx = torch.stack([k // (dims[1] * dims[2]), k // dims[2] % dims[1], k % dims[2]], 1)
        origin = torch.tensor([SPACING if b == 0 else high[0] - width, SPACING,
                               SPACING if b == 0 else high[2] - dims[2] * SPACING], device="cuda")
        parts.append(origin + idx.float() * s)
    x = torch.cat(parts)
    x = x + (torch.rand(n, 3, generator=gen, device="cuda") * 2 - 1) * (JITTER * SPACING)
    return _records(x, gen, mixed_mass), (0.0, 0.0, 0.0), tuple(round(v, 4) for v in high)


def _batch_scenes(case):
    """Sizes, gravities and boxes of a batch (fixed by the case, not by the inputs' seed)."""
    rng = random.Random(case["sizes_seed"])
    scenes = []
    for _ in range(case["scenes"]):
        n = _log(rng, case["n_min"], case["n_max"])
        aspect = [rng.uniform(0.5, 2.0) for _ in range(3)]
        c = (n / (aspect[0] * aspect[1] * aspect[2])) ** (1.0 / 3.0)
        ny, nz = max(2, round(aspect[1] * c)), max(2, round(aspect[2] * c))
        dims = (-(-n // (ny * nz)), ny, nz)
        box = tuple(round((d + 2) * SPACING * rng.uniform(2.0, 4.0), 4) for d in dims)
        scenes.append({"numParticles": n, "gravity": (0.0, -rng.uniform(5.0, 15.0), 0.0),
                       "box_min": (0.0, 0.0, 0.0), "box_max": box, "dims": dims})
    return scenes


def _batch_fluid(scenes, seed):
    gen = _generator(seed)
    sizes = torch.tensor([d["numParticles"] for d in scenes], device="cuda")
    total = int(sizes.sum())
    sid = torch.repeat_interleave(torch.arange(len(scenes), device="cuda"), sizes)
    k = torch.arange(total, device="cuda") - (torch.cumsum(sizes, 0) - sizes)[sid]
    dims = torch.tensor([d["dims"] for d in scenes], device="cuda")[sid]
    idx = torch.stack([k // (dims[:, 1] * dims[:, 2]), k // dims[:, 2] % dims[:, 1],
                       k % dims[:, 2]], 1)
    x = SPACING + idx.float() * (SPACING * COMPRESS)
    x = x + (torch.rand(total, 3, generator=gen, device="cuda") * 2 - 1) * (JITTER * SPACING)
    return _records(x, gen, False), sid


def _obstacles(box):
    """A ball, a rounded block and a post standing in the box."""
    c = [0.5 * v for v in box]
    r = 0.12 * min(box)
    return [{"type": "sphere", "a": (0.25 * box[0], 0.3 * box[1], c[2]), "radius": r},
            {"type": "box", "a": (c[0], r, c[2]), "b": (r, r, 0.5 * c[2]), "radius": 0.02},
            {"type": "capsule", "a": (0.4 * box[0], 0.0, 0.3 * box[2]),
             "b": (0.4 * box[0], 0.8 * box[1], 0.3 * box[2]), "radius": 0.5 * r}]


def _views(buf):
    """The fields of records [n, 27] as named views (hash: whole numbers)."""
    out = {k: buf[:, a:a + w] for k, (a, w) in FIELDS.items()}
    out["hash"] = buf.view(torch.int32)[:, 21]
    return out


def _config(case):
    return ak.PBFConfig(solverIterations=case["iterations"]), ak.LambdaCorrParams()


def _net(seed):
    net = LambdaNet(init_params(int(seed) % 1000))
    net.set_normalization(NET_MEAN, NET_INV_STD, NET_SCALE, BLEND)
    return net


def _training_data(case, seed):
    gen = _generator(seed)
    n = case["batch"] * case["batches"]
    mean = torch.tensor(NET_MEAN, device="cuda")
    x = mean + torch.randn(n, 8, generator=gen, device="cuda") / torch.tensor(NET_INV_STD,
                                                                            device="cuda")
    z = (x - mean) * torch.tensor(NET_INV_STD, device="cuda")
    y = NET_SCALE * (0.8 * z[:, 3] - 0.4 * torch.tanh(z[:, 0] * z[:, 5]) + 0.2 * z[:, 4]
                     + 0.1 * torch.randn(n, generator=gen, device="cuda"))
    return x.contiguous(), y.contiguous()


def _camera(box):
    """A view of the whole box from in front, as the reference's camera stands to its scene."""
    return Camera(position=(0.5 * box[0], 0.6 * box[1], 1.3 * box[0] + box[2]))


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("step", "warm"):
        buf, lo, hi = _fluid(case["n"], seed, case.get("blocks", 1), case.get("mixed_mass", False))
        cfg, corr = _config(case)
        options = ((ak.OPT_EXACT_MATH if case.get("exact_math") else 0)
                   | (ak.OPT_RESIDENT if case.get("resident") else 0))
        solver = ak.PBFSolver(case["n"], cfg, corr, options=options,
                              table_size=case.get("table_size"))
        if case.get("obstacles"):
            solver.set_sdf_shapes(_obstacles(hi))
        if kind == "warm":
            s["net"] = _net(seed)
            solver.set_warm_start(s["net"])
        s.update(solver=solver, buf=buf, lo=lo, hi=hi, out=_views(buf))
    elif kind == "host":
        buf, lo, hi = _fluid(case["n"], seed)
        pinned = torch.empty(case["n"], 27, dtype=torch.float32, pin_memory=True)
        pinned.copy_(buf)
        rec = pinned.numpy().view(ak.PARTICLE_DTYPE).reshape(-1)
        cfg, corr = _config(case)
        s.update(solver=ak.PBFSolver(case["n"], cfg, corr), rec=rec, pinned=pinned, lo=lo, hi=hi,
                 out=_views(pinned))
    elif kind == "batch":
        scenes = _batch_scenes(case)
        buf, _ = _batch_fluid(scenes, seed)
        cfg, corr = _config(case)
        s.update(solver=ak.BatchSolver(scenes, cfg, corr), buf=buf, out=_views(buf))
    elif kind == "train":
        x, y = _training_data(case, seed)
        s.update(net=_net(seed), x=x, y=y, batch=case["batch"])
    elif kind == "render":
        buf, _, hi = _fluid(case["n"], seed)
        s.update(renderer=SplatRenderer(case["width"], case["height"]), buf=buf,
                 camera=_camera(hi))
    else:
        gen = _generator(seed)
        bits, n = case["key_bits"], case["n"]
        keys = torch.randint(0, 1 << bits, (n,), generator=gen, device="cuda").to(torch.int32)
        s.update(lib=_abi.load_library(), n=n, bits=bits, keys=keys,
                 out={"keys": torch.empty_like(keys), "order": torch.empty_like(keys)})
    return s


def run(state):
    kind = state["kind"]
    if kind in ("step", "warm"):
        state["solver"].step(state["buf"], DT, state["lo"], state["hi"])
        return state["out"]
    if kind == "host":
        state["solver"].step(state["rec"], DT, state["lo"], state["hi"])
        return state["out"]
    if kind == "batch":
        state["solver"].step(state["buf"], DT)
        return state["out"]
    if kind == "train":
        b = state["batch"]
        for k in range(0, state["x"].shape[0], b):
            state["net"].adam_step(state["x"][k:k + b], state["y"][k:k + b], LEARNING_RATE)
        return state["net"].params()
    if kind == "render":
        return state["renderer"].render(state["buf"], state["camera"])
    out = state["out"]
    _abi.check(state["lib"].akua_sort_pairs_noalloc(
        ctypes.c_void_p(state["keys"].data_ptr()), None, ctypes.c_void_p(out["keys"].data_ptr()),
        ctypes.c_void_p(out["order"].data_ptr()), state["n"], state["bits"], None),
        "akua_sort_pairs_noalloc")
    return out


def work(case):
    kind = case["kind"]
    if kind in ("step", "warm", "host", "batch"):
        n = (sum(d["numParticles"] for d in _batch_scenes(case)) if kind == "batch"
             else case["n"])
        # per neighbour: distance test, density and its gradient sums, the position delta,
        # vorticity, confinement, XSPH; about 30 neighbours
        flops = 30 * (9 + case["iterations"] * (45 + 40) + 35 + 30 + 25)
        if kind == "warm":
            flops += 2 * (8 * 64 + 2 * 64 * 64 + 64)
        # records in and out; a resident step reads position, mass, velocity, colour and size
        return {"bytes": n * (168 if case.get("resident") else 216), "flops": n * flops}
    if kind == "train":
        n = case["batch"] * case["batches"]
        # forward, input gradients and weight gradients of the three hidden layers
        return {"bytes": 36 * n + 4 * 8961 * 6 * case["batches"],
                "flops": n * 2 * (2 * 8 * 64 + 3 * 2 * 64 * 64 + 3 * 64)}
    if kind == "render":
        pixels = case["width"] * case["height"]
        return {"bytes": 32 * case["n"] + 4 * pixels, "flops": 60 * case["n"] + 30 * pixels}
    return {"bytes": 12 * case["n"], "flops": 0}


# ------------------------------------------------------------------------- values in 64 bits
def _f32(t):
    return t.float().double()


def _cells(x32, cell):
    """floor(x / cell) in single precision, as whole numbers."""
    return torch.floor(x32.float() / torch.tensor(cell, dtype=torch.float32, device="cuda")).long()


def _hash(c, table):
    h = ((c[..., 0] * 73856093) & 0xFFFFFFFF) ^ ((c[..., 1] * 19349663) & 0xFFFFFFFF) \
        ^ ((c[..., 2] * 83492791) & 0xFFFFFFFF)
    return h % table


def _sdf(shapes, x):
    """[(signed distance, unit gradient)] of each obstacle at x."""
    out = []
    for d in shapes:
        a = torch.tensor(d["a"], dtype=torch.float32, device="cuda").double()
        r = float(np.float32(d["radius"]))
        if d["type"] == "box":
            p = x - a
            q = p.abs() - torch.tensor(d["b"], dtype=torch.float32, device="cuda").double()
            o = q.clamp_min(0.0)
            lo = o.norm(dim=1)
            qm, k = q.max(dim=1)
            inside = torch.zeros_like(x).scatter_(1, k[:, None], 1.0) * torch.where(p < 0, -1.0, 1.0)
            g = torch.where((lo > 0)[:, None], torch.copysign(o, p) / lo.clamp_min(1e-300)[:, None],
                            inside)
            out.append((lo + qm.clamp_max(0.0) - r, g))
            continue
        w = x - a
        if d["type"] == "capsule":
            u = torch.tensor(d["b"], dtype=torch.float32, device="cuda").double() - a
            t = ((w * u).sum(1) / (u * u).sum()).clamp(0.0, 1.0)
            w = w - t[:, None] * u
        l = w.norm(dim=1)
        out.append((l - r, w / l.clamp_min(1e-300)[:, None]))
    return out


def _network(params, f):
    """The network's estimate for features f, without its roundings to 16 bits."""
    p = torch.from_numpy(np.asarray(params)).double().cuda()
    at, parts = 0, []
    for shape in ((64, 8), (64,), (64, 64), (64,), (64, 64), (64,), (64,), (1,)):
        size = int(np.prod(shape))
        parts.append(p[at:at + size].view(shape))
        at += size
    w1, b1, w2, b2, w3, b3, w4, b4 = parts
    norm = lambda v: torch.tensor(v, dtype=torch.float32, device="cuda").double()  # noqa: E731
    a = (f - norm(NET_MEAN)) * norm(NET_INV_STD)
    for w, b in ((w1, b1), (w2, b2), (w3, b3)):
        a = torch.nn.functional.silu(a @ w.T + b)
    return (a @ w4 + b4) * float(np.float32(NET_SCALE))


def _exact_step(buf, iterations, gravity, lo, hi, table, offset, shapes=(), net=None):
    """One step of records [n, 27] in 64 bits; gravity, lo, hi are [n, 3] and table, offset [n].
    The cells are found in single precision: they fix which order the records come out in."""
    n = buf.shape[0]
    c32 = lambda v: float(np.float32(v))  # noqa: E731
    h, dt = c32(H), c32(DT)
    h2 = float(np.float32(H) * np.float32(H))
    pi = c32(3.14)
    kp, ks = 315.0 / (64.0 * pi * h ** 9), -45.0 / (pi * h ** 6)
    rho0, relax, vort_eps, visc = 7600.0, 600.0, c32(1e-5), c32(0.01)
    k_corr, dq2 = c32(1e-4), c32(0.03) ** 2
    poly6 = lambda r2: kp * (h2 - r2).clamp_min(0.0) ** 3  # noqa: E731
    wdq = kp * (h2 - dq2) ** 3
    x0, v0, m = buf[:, 0:3].double(), buf[:, 3:6].double(), buf[:, 18].double()
    v32 = _f32(v0 + gravity * dt)
    x32 = _f32(x0 + v32 * dt)
    cell = _cells(x32, H)
    key = offset + _hash(cell, table)
    order = torch.sort(key, stable=True).indices
    x0, v0, m, cell, key = x0[order], v0[order], m[order], cell[order], key[order]
    gravity, lo, hi, table, offset = gravity[order], lo[order], hi[order], table[order], offset[order]
    vs = v0 + gravity * dt
    xs = x0 + vs * dt
    # neighbour pairs: the 27 buckets around each particle, in chunks of particles
    step = torch.tensor([(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)],
                        device="cuda")
    pi_, pj_ = [], []
    for p0 in range(0, n, 100000):
        i = torch.arange(p0, min(n, p0 + 100000), device="cuda")
        hk = (offset[i][:, None] + _hash(cell[i][:, None, :] + step, table[i][:, None])).reshape(-1)
        first = torch.searchsorted(key, hk)
        count = torch.searchsorted(key, hk, right=True) - first
        owner = torch.repeat_interleave(i.repeat_interleave(27), count)
        start = torch.repeat_interleave(first - (torch.cumsum(count, 0) - count), count)
        j = start + torch.arange(owner.numel(), device="cuda")
        d = xs[owner] - xs[j]
        near = ((d * d).sum(1) < h2) & (j != owner)
        pi_.append(owner[near])
        pj_.append(j[near])
    I, J = torch.cat(pi_), torch.cat(pj_)
    del pi_, pj_
    chunks = [slice(a, a + 16000000) for a in range(0, I.numel(), 16000000)]

    def over_pairs(term, width, x):
        """sum over neighbours of term(i, j, x_i - x_j, r^2, gradient of the spiky kernel)."""
        acc = torch.zeros(n, width, dtype=torch.float64, device="cuda")
        for c in chunks:
            i, j = I[c], J[c]
            s = x[i] - x[j]
            r2 = (s * s).sum(1)
            r = r2.sqrt()
            g = (ks * (h - r) ** 2 / r.clamp_min(1e-30))
            g = torch.where((r > h) | (r < 1e-5), torch.zeros_like(g), g)[:, None] * s
            acc.index_add_(0, i, term(i, j, r2, g))
        return acc

    def density(i, j, r2, g):
        mj = m[j][:, None]
        return torch.cat([mj * poly6(r2)[:, None], mj * g, (mj * g / rho0).square().sum(1, True)], 1)

    x = xs
    rho = lam = delta = None
    lam_sum = None
    for it in range(iterations):
        acc = over_pairs(density, 5, x)
        rho = acc[:, 0] + m * kp * h2 ** 3
        grad = acc[:, 1:4] / rho0
        den = acc[:, 4] + grad.square().sum(1)
        lam = -(rho / rho0 - 1.0) / (den + relax)
        if net is not None and it == 0:
            counts = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(
                0, I, torch.ones(I.numel(), dtype=torch.float64, device="cuda"))
            along = (grad * gravity).sum(1) / gravity.norm(dim=1)
            f = torch.stack([rho / rho0 - 1.0, counts / 32.0, den, lam, torch.zeros_like(lam),
                             grad.norm(dim=1), along, vs.norm(dim=1)], 1)
            lam = lam + c32(BLEND) * (_network(net, f) - lam)

        def push(i, j, r2, g):
            scorr = -k_corr * (poly6(r2) / wdq) ** 4
            return ((lam[i] + lam[j] + scorr) * m[j])[:, None] * g / rho0

        delta = over_pairs(push, 3, x)
        x = x + delta
        low, high = lo + c32(0.025), hi - c32(0.025)
        x = x + 0.5 * (low - x).clamp_min(0.0) + 0.5 * (high - x).clamp_max(0.0)
        for s in range(len(shapes)):
            phi, g = _sdf(shapes[s:s + 1], x)[0]
            x = x + (0.5 * (c32(0.025) - phi).clamp_min(0.0))[:, None] * g
    v_new = (x - x0) / dt
    v = v_new.clone()
    keep = 1.0 - c32(0.95)
    walls = []
    for a in range(3):
        e = torch.zeros(1, 3, dtype=torch.float64, device="cuda")
        e[0, a] = 1.0
        walls += [(x[:, a] - lo[:, a], e), (hi[:, a] - x[:, a], -e)]
    for dist, g in walls + _sdf(shapes, x):
        appr = (v * g).sum(1, True)
        near = (dist < c32(0.025))[:, None]
        tangent = v - appr * g
        v = torch.where(near & (appr < 1e-5), keep * tangent, v)

    def curl(i, j, r2, g):
        return -m[j][:, None] * torch.linalg.cross(v[j] - v[i], g)

    om = over_pairs(curl, 3, x)
    wn = om.norm(dim=1)
    eta = over_pairs(lambda i, j, r2, g: (m[j] * (wn[i] - wn[j]))[:, None] * g, 3, x) / rho[:, None]
    el = eta.norm(dim=1, keepdim=True)
    side = torch.where(el < 1e-5, torch.zeros_like(eta), eta / el.clamp_min(1e-300))
    vc = v + dt * vort_eps * torch.linalg.cross(side, om)
    vol = m / rho
    smooth = over_pairs(lambda i, j, r2, g: (vol[j] * poly6(r2))[:, None] * (vc[j] - vc[i]), 3, x)
    v_out = vc + visc * smooth
    return {"position": x, "velocity": v_out, "new_position": x, "new_velocity": v_new,
            "position_delta": delta, "vorticity": om, "mass": m[:, None], "density": rho[:, None],
            "lambda": lam[:, None], "hash": None, "color": buf[order, 22:26].double(),
            "size": buf[order, 26:27].double()}


def _exact_training(case, seed):
    """The minibatches' Adam steps in 64 bits."""
    x, y = _training_data(case, seed)
    params = torch.from_numpy(init_params(int(seed) % 1000)).double().cuda().requires_grad_(True)
    norm = lambda v: torch.tensor(v, dtype=torch.float32, device="cuda").double()  # noqa: E731
    shapes = ((64, 8), (64,), (64, 64), (64,), (64, 64), (64,), (64,), (1,))
    m1 = torch.zeros_like(params)
    m2 = torch.zeros_like(params)
    b1, b2, lr, scale = (float(np.float32(v)) for v in (0.9, 0.999, LEARNING_RATE, NET_SCALE))
    for k in range(case["batches"]):
        part = slice(k * case["batch"], (k + 1) * case["batch"])
        at, w = 0, []
        for shape in shapes:
            size = int(np.prod(shape))
            w.append(params[at:at + size].view(shape))
            at += size
        a = (x[part].double() - norm(NET_MEAN)) * norm(NET_INV_STD)
        for q in range(3):
            a = torch.nn.functional.silu(a @ w[2 * q].T + w[2 * q + 1])
        loss = ((a @ w[6] + w[7]) - y[part].double() / scale).square().mean()
        g, = torch.autograd.grad(loss, params)
        m1 = b1 * m1 + (1 - b1) * g
        m2 = b2 * m2 + (1 - b2) * g * g
        step = (m1 / (1 - b1 ** (k + 1))) / ((m2 / (1 - b2 ** (k + 1))).sqrt() + 1e-8)
        params = (params - lr * step).detach().requires_grad_(True)
    return params.detach().cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_training(case, seed)
    if kind in ("render", "sort"):
        return None  # bytes and whole numbers
    with torch.no_grad():
        if kind == "batch":
            scenes = _batch_scenes(case)
            buf, sid = _batch_fluid(scenes, seed)
            of = lambda key: torch.tensor([d[key] for d in scenes],  # noqa: E731
                                          dtype=torch.float32, device="cuda").double()[sid]
            sizes = torch.tensor([d["numParticles"] for d in scenes], device="cuda") * 128
            return _exact_step(buf, case["iterations"], of("gravity"), of("box_min"),
                               of("box_max"), sizes[sid], (torch.cumsum(sizes, 0) - sizes)[sid])
        n = case["n"]
        buf, lo, hi = _fluid(n, seed, case.get("blocks", 1), case.get("mixed_mass", False))
        rows = lambda v: torch.tensor(v, dtype=torch.float32,  # noqa: E731
                                      device="cuda").double().expand(n, 3).contiguous()
        table = torch.full((n,), case.get("table_size") or 128 * n, device="cuda")
        return _exact_step(buf, case["iterations"], rows((0.0, -9.8, 0.0)), rows(lo), rows(hi),
                           table, torch.zeros_like(table),
                           _obstacles(hi) if case.get("obstacles") else (),
                           init_params(int(seed) % 1000) if kind == "warm" else None)
