"""The solver's measured workloads, through its public host API (`rfmm`).

Each case is one job a host program gives the solver: bodies in, solve or
steps, results out.  The inputs are made on the GPU from a seed with the
distributions of the repository's scene generators (uniform cube, Plummer
spheres with their equilibrium velocities, mixtures of Plummer spheres).
`exact` evaluates the same method in binary64 with plain torch: the discrete
decisions (which leaf a body lies in, which cell it samples) follow the
method's binary32 rule, everything else is 64 bits wide.
"""
import math
import os
import sys

import numpy as np
import torch

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(REPO, "fmm-rainbow_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(REPO, "fmm-rainbow_gb300"))

import rfmm  # noqa: E402

GRAVITY, DT = 1.0, 5e-4  # the measured workloads' (rfmm/workloads.py)


# ------------------------------------------------------------------- cases

def listed():
    return [
        # The smallest scene of the batched configuration, alone: one frame,
        # where launches and the upload's sort are everything.
        dict(name="step_4k", path="step", scene="uniform", n=4096, steps=1, source="device",
             float="exact", near="reference", control=0, softening=1e-3),
        # One force evaluation of the 65,536-body uniform configuration:
        # moments and fields are the result.
        dict(name="fields_64k", path="fields", scene="uniform", n=65536, noalloc=False, softening=1e-3),
        # A host application's job with the interactive vortex brush on: a
        # ragged body count from pinned host memory, 16 frames, back to the host.
        dict(name="host_250k", path="step", scene="clusters4", n=250001, steps=16, source="host",
             float="exact", near="reference", control=3, softening=1e-3),
        # The default preset and headline configuration.
        dict(name="plummer_1m", path="step", scene="plummer", n=1 << 20, steps=60, source="device",
             float="exact", near="reference", control=0, softening=1e-3),
        # The largest body count a plan admits.
        dict(name="clusters_5m", path="step", scene="clusters", n=5242880, steps=60, source="device",
             float="exact", near="reference", control=0, softening=5e-4),
        # The fast float variant at an odd size between those two.
        dict(name="fast_700k", path="step", scene="plummer", n=700001, steps=16, source="device",
             float="fast", near="reference", control=0, softening=1e-3),
        # Many scenes stepped together (the batched configuration).
        dict(name="batched_256", path="batch", scenes=256, n_min=4096, n_max=262144, steps=20, softening=1e-3),
        # A burst of requests of the served configuration's kind.
        dict(name="served_24", path="served", requests=24, n_min=16384, n_max=1 << 20, steps_max=60,
             softening=1e-3),
        # The accuracy mode: exact near-field pair sums, both float variants.
        dict(name="p2p_120k", path="step", scene="plummer", n=120001, steps=2, source="device",
             float="exact", near="p2p", control=0, softening=1e-3),
        dict(name="p2p_fast_600k", path="step", scene="clusters", n=600007, steps=1, source="device",
             float="fast", near="p2p", control=0, softening=1e-3),
        # One displayed frame of the default preset.
        dict(name="render_1m", path="render", scene="plummer", n=1 << 20, width=1920, height=1080),
        # An accuracy report: accelerations and potentials of every body,
        # conserved quantities, force error against the binary64 direct sum.
        dict(name="accuracy_262k", path="accuracy", scene="plummer", n=262144, targets=4096, softening=1e-3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["step", "step", "step", "p2p", "fields", "batch", "served", "render", "accuracy"])
    scene = rng.choice(["uniform", "plummer", "clusters4", "clusters"])
    soft = rng.choice([5e-4, 1e-3, 0.012])
    if path == "step":
        return dict(path="step", scene=scene, n=_log_int(rng, 2048, 5242880), steps=_log_int(rng, 1, 60),
                    source=rng.choice(["device", "device", "host"]), float=rng.choice(["exact", "exact", "fast"]),
                    near="reference", control=rng.choice([0, 0, 1, 2, 3]), softening=soft)
    if path == "p2p":
        return dict(path="step", scene=scene, n=_log_int(rng, 8192, 600000), steps=1, source="device",
                    float=rng.choice(["exact", "fast"]), near="p2p", control=0, softening=soft)
    if path == "fields":
        noalloc = rng.random() < 0.5
        return dict(path="fields", scene=scene, n=_log_int(rng, 2048, 131072 if noalloc else 4000000),
                    noalloc=noalloc, softening=soft)
    if path == "batch":
        return dict(path="batch", scenes=_log_int(rng, 2, 200), n_min=2048, n_max=_log_int(rng, 4096, 262144),
                    steps=_log_int(rng, 1, 20), softening=soft)
    if path == "served":
        return dict(path="served", requests=rng.randrange(2, 24), n_min=16384, n_max=_log_int(rng, 32768, 1 << 20),
                    steps_max=_log_int(rng, 4, 60), softening=soft)
    if path == "render":
        return dict(path="render", scene=scene, n=_log_int(rng, 8192, 2000000),
                    width=_log_int(rng, 320, 1920), height=_log_int(rng, 240, 1080))
    return dict(path="accuracy", scene=scene, n=_log_int(rng, 8192, 262144), targets=_log_int(rng, 128, 4096),
                softening=soft)


# ------------------------------------------------------------------ scenes

def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _unit(g, n):
    z = 2.0 * _rand(g, n) - 1.0
    phi = 2.0 * math.pi * _rand(g, n)
    s = torch.sqrt((1.0 - z * z).clamp_min(0.0))
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z], 1)


def _plummer(g, n, a, r_max, mass):
    """Offsets and equilibrium velocities of a truncated Plummer sphere."""
    m_max = r_max ** 3 / (r_max ** 2 + a ** 2) ** 1.5
    m = (m_max * _rand(g, n)).clamp_min(1e-12)
    r = a / torch.sqrt(m ** (-2.0 / 3.0) - 1.0)
    # Speed fraction q of the escape speed ~ q^2 (1 - q^2)^(7/2), by its
    # tabulated cumulative distribution.
    q = torch.linspace(0.0, 1.0, 4097, device="cuda", dtype=torch.float64)
    cdf = torch.cumsum(q * q * (1.0 - q * q) ** 3.5, 0)
    cdf = cdf / cdf[-1]
    u = _rand(g, n)
    k = torch.searchsorted(cdf, u).clamp(1, 4096)
    f = (u - cdf[k - 1]) / (cdf[k] - cdf[k - 1]).clamp_min(1e-300)
    speed = q[k - 1] + f.clamp(0.0, 1.0) * (q[k] - q[k - 1])
    v_esc = math.sqrt(2.0 * mass / a) * (1.0 + (r / a) ** 2) ** -0.25
    return r[:, None] * _unit(g, n), (speed * v_esc)[:, None] * _unit(g, n)


def _scene(kind, n, seed):
    """(n, 8) float32: x y z hue vx vy vz excitation (the Particle layout)."""
    g = _rng(seed)
    out = torch.zeros(n, 8, device="cuda")
    if kind == "uniform":
        out[:, 0:3] = _rand(g, n, 3).float()
    elif kind == "plummer":
        pos, vel = _plummer(g, n, 0.1, 0.5, 1.0)
        out[:, 0:3], out[:, 4:7] = (pos + 0.5).float(), vel.float()
    else:  # a shuffled mixture of k Plummer spheres
        k = 4 if kind == "clusters4" else 8
        order = torch.randperm(n, generator=g, device="cuda")
        for c in range(k):
            at = order[c * n // k: (c + 1) * n // k]
            a = 0.1 if kind == "clusters4" else 0.02 * 5.0 ** float(_rand(g, 1))
            centre, bulk = 0.2 + 0.6 * _rand(g, 1, 3), 0.1 * (_rand(g, 1, 3) - 0.5)
            pos, vel = _plummer(g, at.numel(), a, 5.0 * a, 1.0 / k)
            out[at, 0:3], out[at, 4:7] = (pos + centre).float(), (vel + bulk).float()
    # Hues away from the wrap at 1 (a display state; its drift per job is small).
    out[:, 3] = (0.05 + 0.9 * _rand(g, n)).float()
    return out


def _params(case, seed=0):
    """Solver parameters; the control brush sits at a seeded point."""
    kw = dict(gravity=GRAVITY, softening=case.get("softening", 1e-3), dt=DT)
    if case.get("control", 0):
        r = np.random.default_rng(seed)
        kw.update(control_point=[float(x) for x in r.uniform(0.3, 0.7, 3)] + [1.0],
                  control_axis_mode=[float(x) for x in r.uniform(0.2, 1.0, 3)] + [float(case["control"])])
    return rfmm.default_params(**kw)


def _batch_sizes(case, count, seed):
    r = np.random.default_rng(seed)
    return [int(x) for x in np.exp(r.uniform(math.log(case["n_min"]), math.log(case["n_max"]), count))]


# ----------------------------------------------------------------- prepare

def prepare(case, seed):
    path = case["path"]
    if path == "batch":
        # Sizes are the case's own, as a host knows them when it makes the batch.
        sizes = _batch_sizes(case, case["scenes"], 4)
        bodies = [_scene("uniform" if i % 2 == 0 else "plummer", n, seed * 1009 + i) for i, n in enumerate(sizes)]
        batch = rfmm.Batch(sizes, [_params(case) for _ in sizes])
        out = torch.empty(sum(sizes), 8, pin_memory=True)
        at = np.concatenate([[0], np.cumsum(sizes)])
        return dict(case=case, batch=batch, bodies=bodies, ptrs=[b.data_ptr() for b in bodies], out=out,
                    out_ptrs=[out.data_ptr() + 32 * int(a) for a in at[:-1]])
    if path == "served":
        sizes = _batch_sizes(case, case["requests"], 5)
        steps = np.random.default_rng(6).integers(1, case["steps_max"] + 1, len(sizes))
        bodies = []
        for i, n in enumerate(sizes):
            b = _scene(("uniform", "plummer", "clusters4")[i % 3], n, seed * 1009 + i).cpu().numpy()
            bodies.append(b.view(rfmm.PARTICLE_DTYPE).reshape(n))
        server = rfmm.Server(max_bodies=1 << 20, memory_budget_bytes=4 << 30, staging_bytes=1 << 29)
        return dict(case=case, server=server, bodies=bodies, steps=[int(s) for s in steps], params=_params(case))

    n = case["n"]
    state = dict(case=case, bodies=_scene(case["scene"], n, seed), params=_params(case, seed))
    if path == "fields" and case["noalloc"]:
        cells = rfmm.plan_unclamped(n)[1]
        state["moments"] = torch.empty(cells, 4, dtype=torch.int32, device="cuda")
        state["fields"] = torch.empty(cells, 12, device="cuda")
        return state
    s = state["solver"] = rfmm.Solver(n, state["params"])
    if path == "fields":
        state["moments"] = torch.empty(s.cells, 4, dtype=torch.int32, device="cuda")
        state["fields"] = torch.empty(s.cells, 12, device="cuda")
    elif path == "step":
        s.set_float_mode(rfmm.FLOAT_FAST if case["float"] == "fast" else rfmm.FLOAT_EXACT)
        s.set_near_mode(rfmm.NEAR_P2P if case["near"] == "p2p" else rfmm.NEAR_REFERENCE)
        if case["source"] == "host":
            state["bodies"] = state["bodies"].cpu().pin_memory()
            state["out"] = torch.empty(n, 8, pin_memory=True)
        else:
            state["out"] = torch.empty(n, 8, device="cuda")
    elif path == "render":
        s.upload_device(state["bodies"].data_ptr(), 32 * n)
        r = np.random.default_rng(seed)
        state["view"] = rfmm.default_render_params(width=case["width"], height=case["height"],
                                                   yaw=float(r.uniform(-1.0, 1.0)), pitch=float(r.uniform(-0.5, 0.5)))
        state["out"] = torch.empty(case["height"], case["width"], 4, dtype=torch.uint8, device="cuda")
    elif path == "accuracy":
        s.upload_device(state["bodies"].data_ptr(), 32 * n)
    torch.cuda.synchronize()
    return state


# --------------------------------------------------------------------- run

def run(state):
    case = state["case"]
    path = case["path"]
    if path == "step":
        s, bodies, out = state["solver"], state["bodies"], state["out"]
        host = case["source"] == "host"
        (s.upload_host_ptr if host else s.upload_device)(bodies.data_ptr(), 32 * case["n"])
        s.step(case["steps"])
        (s.download_host_ptr if host else s.download_device)(rfmm.BUF_PARTICLES, out.data_ptr(), 32 * case["n"])
        return out
    if path == "fields":
        m, f = state["moments"], state["fields"]
        if case["noalloc"]:
            rfmm.solve_fields_noalloc(state["bodies"].data_ptr(), case["n"], state["params"], m.data_ptr(),
                                      f.data_ptr(), torch.cuda.current_stream().cuda_stream)
        else:
            s = state["solver"]
            s.upload_device(state["bodies"].data_ptr(), 32 * case["n"])
            s.solve_fields()
            s.download_device(rfmm.BUF_MOMENTS, m.data_ptr(), 16 * s.cells)
            s.download_device(rfmm.BUF_FIELDS, f.data_ptr(), 48 * s.cells)
        return dict(moments=m, fields=f)
    if path == "batch":
        b = state["batch"]
        b.upload_device_all(state["ptrs"])
        b.commit()
        b.step(case["steps"])
        b.download_all_into(rfmm.BUF_PARTICLES, state["out_ptrs"])
        return state["out"]
    if path == "served":
        server = state["server"]
        ids = [server.submit(b, steps, state["params"]) for b, steps in zip(state["bodies"], state["steps"])]
        got = []
        for i in ids:
            server.wait(i)
            got.append(server.result(i).view(np.float32).reshape(-1, 8))
        return got
    if path == "render":
        state["solver"].render_device(state["view"], state["out"].data_ptr(), state["out"].numel())
        return state["out"]
    s = state["solver"]
    acc = s.accelerations()
    d = s.diagnostics()
    rms, worst = s.force_error(case["targets"], 1)
    return dict(acc=acc, conserved=[d["kinetic"], d["potential"], d["total"]] + d["momentum"] + d["angular_momentum"],
                force_rms=rms, force_max=worst)


# -------------------------------------------------------------------- work

def _depth(n):
    return rfmm.plan_unclamped(n)[0]


# Body pairs inside 3x3x3 leaf blocks over n^2, per planner depth 4, 5, 6.
_PAIRS = {"uniform": (0.14, 0.022, 0.003), "plummer": (0.84, 0.42, 0.113), "clusters4": (0.49, 0.16, 0.035),
          "clusters": (0.38, 0.20, 0.114)}


def work(case):
    """Bytes: every body read and written once per step (64 B), the results
    once.  Flops: about 200 per body step (the update's own operations), 20
    per exact pair, and in the accuracy report 20 per direct pair."""
    path = case["path"]
    if path == "step":
        n, steps = case["n"], case["steps"]
        pairs = _PAIRS[case["scene"]][_depth(n) - 4] * n * n if case["near"] == "p2p" else 0
        return dict(bytes=64.0 * n * steps, flops=steps * (200.0 * n + 20.0 * pairs))
    if path == "fields":
        cells = rfmm.plan_unclamped(case["n"])[1]
        return dict(bytes=32.0 * case["n"] + 64.0 * cells, flops=10.0 * case["n"])
    if path == "batch":
        n = sum(_batch_sizes(case, case["scenes"], 4))
        return dict(bytes=64.0 * n * case["steps"], flops=200.0 * n * case["steps"])
    if path == "served":
        sizes = _batch_sizes(case, case["requests"], 5)
        steps = np.random.default_rng(6).integers(1, case["steps_max"] + 1, len(sizes))
        n = float(np.dot(sizes, steps))
        return dict(bytes=64.0 * n, flops=200.0 * n)
    if path == "render":
        px = case["width"] * case["height"]
        return dict(bytes=32.0 * case["n"] + 4.0 * px, flops=100.0 * case["n"] + 100.0 * px)
    n = case["n"]
    return dict(bytes=3 * 32.0 * n + 16.0 * n, flops=20.0 * min(case["targets"], n) * n + 300.0 * n)


# ------------------------------------------------------------------- exact

_HALF = float(np.float32(1.6))
_CAP = 16


def _cells(pos, depth):
    """Leaf coordinates by the binary32 rule of the deposit."""
    p = pos.float()
    u = (p / 1.6).clamp(-0.99999, 0.99999) * 0.5 + 0.5
    return torch.floor(u * float(1 << depth)).long()


def _centre(c, level):
    return ((c.double() + 0.5) * 2.0 / (1 << level) - 1.0) * _HALF


def _pair(com, gm, target, eps):
    """The ten field terms of sources (..., S) on targets (..., 1), summed over S."""
    r = com - target[:, None, :]
    inv = (r.square().sum(-1) + eps * eps).rsqrt()
    i3 = inv * inv * inv
    tid = 3.0 * gm * i3 * inv * inv
    x, y, z = r.unbind(-1)
    dg = -gm * i3
    terms = (gm * x * i3, gm * y * i3, gm * z * i3, -gm * inv, dg + tid * x * x, tid * x * y, tid * x * z,
             dg + tid * y * y, tid * y * z, dg + tid * z * z)
    return torch.stack([t.sum(1) for t in terms], 1)


class _Solve:
    """One field solve in binary64: moments (integers) and fields per level."""

    def __init__(self, pos, depth, scale, n, soft, near=True):
        dev = pos.device
        self.depth, self.n, self.soft = depth, n, soft
        self.leaf = _cells(pos, depth)
        q = torch.round((pos.float() * scale)).clamp(-2147483648.0, 2147483520.0).long()
        dim = 1 << depth
        lin = self.leaf[:, 0] + dim * (self.leaf[:, 1] + dim * self.leaf[:, 2])
        m = torch.zeros(dim ** 3, 4, dtype=torch.int64, device=dev)
        m.index_add_(0, lin, torch.cat([torch.ones_like(q[:, :1]), q], 1))
        self.mom = [None] * (depth + 1)
        self.mom[depth] = m.view(dim, dim, dim, 4)
        for l in range(depth - 1, -1, -1):
            h = 1 << l
            self.mom[l] = self.mom[l + 1].view(h, 2, h, 2, h, 2, 4).sum((1, 3, 5))
        self.com, self.gm, self.field = [], [], []
        for l in range(depth + 1):
            cnt = self.mom[l][..., 0].double()
            self.com.append(self.mom[l][..., 1:].double() / (scale * cnt.clamp_min(1.0))[..., None])
            self.gm.append(GRAVITY * cnt / n)
            self.field.append(torch.zeros(*cnt.shape, 10, dtype=torch.float64, device=dev))
        off27 = torch.tensor([[x, y, z] for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)], device=dev)
        off8 = torch.tensor([[x, y, z] for z in (0, 1) for y in (0, 1) for x in (0, 1)], device=dev)
        off216 = (2 * off27[:, None, :] + off8[None]).reshape(-1, 3)
        for l in range(1, depth + 1):
            dim = 1 << l
            cnt = self.mom[l][..., 0]
            par = self.mom[l - 1][..., 0].repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)
            tz, ty, tx = torch.nonzero((cnt != 0) & (par > _CAP), as_tuple=True)
            for k in range(0, tx.numel(), 32768):
                t = torch.stack([tx, ty, tz], 1)[k: k + 32768]
                c = (t // 2) * 2
                s = c[:, None, :] + off216[None]
                ok = ((s >= 0) & (s < dim)).all(-1) & ((s - t[:, None, :]).abs() > 1).any(-1)
                f = self._sum(l, t, s, ok, float(np.float32(0.06)) * _HALF / dim)
                p = self.field[l - 1][t[:, 2] // 2, t[:, 1] // 2, t[:, 0] // 2]
                f += p
                d = _centre(t, l) - _centre(t // 2, l - 1)
                f[:, 0] += p[:, 4] * d[:, 0] + p[:, 5] * d[:, 1] + p[:, 6] * d[:, 2]
                f[:, 1] += p[:, 5] * d[:, 0] + p[:, 7] * d[:, 1] + p[:, 8] * d[:, 2]
                f[:, 2] += p[:, 6] * d[:, 0] + p[:, 8] * d[:, 1] + p[:, 9] * d[:, 2]
                f[:, 3] -= p[:, 0] * d[:, 0] + p[:, 1] * d[:, 1] + p[:, 2] * d[:, 2]
                self.field[l][t[:, 2], t[:, 1], t[:, 0]] = f
        if not near:
            return
        for l in range(1, depth + 1):  # adaptive leaves add their 26 neighbours
            dim = 1 << l
            cnt = self.mom[l][..., 0]
            par = self.mom[l - 1][..., 0].repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)
            tz, ty, tx = torch.nonzero((cnt != 0) & (par > _CAP) & ((cnt <= _CAP) | (l == depth)), as_tuple=True)
            for k in range(0, tx.numel(), 65536):
                t = torch.stack([tx, ty, tz], 1)[k: k + 65536]
                s = t[:, None, :] + off27[None]
                ok = ((s >= 0) & (s < dim)).all(-1)
                ok[:, 13] = False
                eps = max(soft, float(np.float32(0.72)) * _HALF / dim)
                self.field[l][t[:, 2], t[:, 1], t[:, 0]] += self._sum(l, t, s, ok, eps)

    def _sum(self, l, t, s, ok, eps):
        s = torch.where(ok[..., None], s, torch.zeros_like(s))
        at = (s[..., 2], s[..., 1], s[..., 0])
        return _pair(self.com[l][at], self.gm[l][at] * ok, _centre(t, l), eps)

    def flat(self):
        m = torch.cat([x.reshape(-1, 4) for x in self.mom])
        f = torch.cat([x.reshape(-1, 10) for x in self.field])
        return m.to(torch.int32), torch.cat([f, torch.zeros_like(f[:, :2])], 1)

    def sample(self):
        """Sample level of every body: the first with at most 16 bodies, else the leaf."""
        level = torch.full_like(self.leaf[:, 0], self.depth)
        for l in range(self.depth - 1, 0, -1):
            c = self.leaf >> (self.depth - l)
            level[self.mom[l][c[:, 2], c[:, 1], c[:, 0], 0] <= _CAP] = l
        return level

    def forces(self, pos, near=None):
        """Acceleration, potential and sample count of every body."""
        level = self.sample()
        acc = torch.zeros(pos.shape[0], 4, dtype=torch.float64, device=pos.device)
        count = torch.zeros(pos.shape[0], dtype=torch.int64, device=pos.device)
        for l in range(1, self.depth + 1):
            i = torch.nonzero(level == l).flatten()
            c = self.leaf[i] >> (self.depth - l)
            at = (c[:, 2], c[:, 1], c[:, 0])
            f, r = self.field[l][at], pos[i] - _centre(c, l)
            x, y, z = r.unbind(1)
            cnt = self.mom[l][at][:, 0]
            a = torch.stack([f[:, 0] + f[:, 4] * x + f[:, 5] * y + f[:, 6] * z,
                             f[:, 1] + f[:, 5] * x + f[:, 7] * y + f[:, 8] * z,
                             f[:, 2] + f[:, 6] * x + f[:, 8] * y + f[:, 9] * z,
                             f[:, 3] - (f[:, 0] * x + f[:, 1] * y + f[:, 2] * z)], 1)
            if near is None:
                d = self.com[l][at] - pos[i]
                eps = max(self.soft, float(np.float32(0.62)) * _HALF / (1 << l))
                inv = (d.square().sum(1) + eps * eps).rsqrt()
                gm = GRAVITY * (cnt - 1).double() / self.n
                a[:, :3] += (gm * inv ** 3)[:, None] * d
                a[:, 3] -= gm * inv
            acc[i], count[i] = a, cnt
        if near is not None:
            acc[:, :3] += GRAVITY / self.n * near
        return acc, count

    def pair_sums(self, pos):
        """Softened pair sums of every body over the 3x3x3 cells around its sample cell."""
        D, level = self.depth, self.sample()
        code = torch.zeros_like(level)
        for b in range(D):
            for ax in range(3):
                code |= ((self.leaf[:, ax] >> b) & 1) << (3 * b + ax)
        order = torch.argsort(code)
        code, p = code[order], pos[order]
        starts = torch.searchsorted(code, torch.arange(8 ** D + 1, device=pos.device)).cpu().numpy()
        level = level[order]
        head = (code >> (3 * (D - level))) + (level << 32)
        cells, runs = torch.unique_consecutive(head, return_counts=True)
        cells, runs = cells.cpu().numpy(), runs.cpu().numpy()
        out = torch.zeros_like(p)
        at = 0
        for cell, run in zip(cells, runs):
            l, m = int(cell >> 32), int(cell & 0xFFFFFFFF)
            c = [sum(((m >> (3 * b + ax)) & 1) << b for b in range(l)) for ax in range(3)]
            src = []
            for z in range(max(0, c[2] - 1), min(1 << l, c[2] + 2)):
                for y in range(max(0, c[1] - 1), min(1 << l, c[1] + 2)):
                    for x in range(max(0, c[0] - 1), min(1 << l, c[0] + 2)):
                        k = sum(((x >> b) & 1) << (3 * b) | ((y >> b) & 1) << (3 * b + 1) |
                                ((z >> b) & 1) << (3 * b + 2) for b in range(l)) << (3 * (D - l))
                        lo, hi = starts[k], starts[k + (1 << (3 * (D - l)))]
                        if hi > lo:
                            src.append((lo, hi))
            q = torch.cat([p[lo:hi] for lo, hi in src])
            step = max(1, 20_000_000 // q.shape[0])
            for k in range(at, at + int(run), step):
                d = q[None] - p[k: min(k + step, at + int(run)), None]
                w = (d.square().sum(2) + self.soft * self.soft).rsqrt() ** 3
                out[k: k + step][: d.shape[0]] = torch.einsum("ts,tsk->tk", w, d)
            at += int(run)
        back = torch.empty_like(out)
        back[order] = out
        return back


def _advance(s, acc, count, params):
    """Symplectic Euler with excitation, hue and the absorbing walls, in place on s (n, 8)."""
    dt = float(np.float32(params.dt) * np.float32(params.speed))
    pos, vel, hue, exc = s[:, 0:3].clone(), s[:, 4:7].clone(), s[:, 3].clone(), s[:, 7].clone()
    infl = torch.zeros_like(hue)
    acc = acc.clone()
    if params.control_point[3] > 0.5:
        delta = torch.tensor(list(params.control_point)[:3], dtype=torch.float64, device=s.device) - pos
        d2 = delta.square().sum(1)
        cr = max(float(params.control_radius), 0.02)
        infl = torch.exp(-2.0 * d2 / (cr * cr))
        amount = (params.control_strength * infl)[:, None]
        mode = params.control_axis_mode[3]
        if mode < 2.5:
            dirs = delta * (d2 + cr * cr * 0.018).rsqrt()[:, None]
            acc += dirs * amount if mode < 1.5 else -dirs * amount
        else:
            axis = torch.tensor(list(params.control_axis_mode)[:3], dtype=torch.float64, device=s.device)
            t = torch.linalg.cross((axis / axis.norm()).expand_as(delta), delta)
            tl = t.norm(dim=1, keepdim=True)
            acc += torch.where(tl > 1e-5, t / tl.clamp_min(1e-30) * amount, torch.zeros_like(t))
    radius, speed = pos.norm(dim=1).clamp_min(1e-4), vel.norm(dim=1).clamp_min(1e-4)
    radial = ((pos * vel).sum(1) / (radius * speed)).clamp(-1.0, 1.0)
    pulse = ((count.double() - _CAP) / 72.0).clamp(0.0, 1.0)
    strength = (acc.norm(dim=1) * (radius + 0.12) * 0.58).clamp(0.0, 1.0)
    want = (0.025 + radial.abs() ** 3 * 0.56 + pulse * 0.26 + strength * 0.13 + infl * 0.42).clamp(0.0, 1.0)
    t = torch.where(want > exc, dt * 10.0, dt * 1.05).clamp(0.0, 1.0)
    exc = exc * (1.0 - t) + want * t
    vel = vel + acc * dt
    pos = pos + vel * dt
    edge, band = _HALF * 0.985, 0.12 * _HALF
    over = pos.abs() - (edge - band)
    vel = torch.where(over > 0.0, vel * (1.0 - (over / band).clamp(0.0, 1.0) * 0.16), vel)
    vel = torch.where(pos.abs() > edge, vel * -0.55, vel)
    pos = pos.clamp(-edge, edge)
    st = ((exc - 0.30) / 0.40).clamp(0.0, 1.0)
    h = hue + dt * (1.0 - st * st * (3.0 - 2.0 * st)) * (0.012 + radial * 0.030 + exc * 0.036 + infl * 0.080)
    s[:, 0:3], s[:, 3], s[:, 4:7], s[:, 7] = pos, h - torch.floor(h), vel, exc


def _sampled(n, count, seed):
    """Body ids of the force-error sample (splitmix64 partial Fisher-Yates)."""
    mask, moved, ids, x = (1 << 64) - 1, {}, [], seed
    for i in range(count):
        x = (x + 0x9E3779B97F4A7C15) & mask
        z = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        z ^= z >> 31
        j = i + z % (n - i)
        a, b = moved.get(i, i), moved.get(j, j)
        ids.append(b)
        moved[i], moved[j] = b, a
    return ids


def exact(case, seed):
    path = case["path"]
    if path not in ("step", "fields", "accuracy"):
        return None  # pixels are bytes; hundreds of scene solves take too long here
    n = case["n"]
    depth, _, scale = rfmm.plan_unclamped(n)
    params = _params(case, seed)
    soft = float(np.float32(params.softening))
    s = _scene(case["scene"], n, seed).double()
    if path == "fields":
        m, f = _Solve(s[:, :3], depth, scale, n, soft).flat()
        return dict(moments=m, fields=f)
    if path == "step":
        p2p = case["near"] == "p2p"
        for _ in range(case["steps"]):
            pos = s[:, :3].clone()
            sol = _Solve(pos, depth, scale, n, soft, near=not p2p)
            acc, count = sol.forces(pos, sol.pair_sums(pos) if p2p else None)
            _advance(s, acc[:, :3], count, params)
        return s
    pos, vel = s[:, :3], s[:, 4:7]
    acc, _ = _Solve(pos, depth, scale, n, soft).forces(pos)
    kin, pot = float(0.5 * vel.square().sum() / n), float(0.5 * acc[:, 3].sum() / n)
    conserved = [kin, pot, kin + pot] + (vel.sum(0) / n).tolist() + (torch.linalg.cross(pos, vel).sum(0) / n).tolist()
    ids = torch.tensor(_sampled(n, min(case["targets"], n), 1), device=s.device)
    ref = []
    for t in ids.split(max(1, 20_000_000 // n)):
        d = pos[None] - pos[t, None]
        w = (d.square().sum(2) + soft * soft).rsqrt() ** 3
        ref.append(GRAVITY / n * torch.einsum("ts,tsk->tk", w, d))
    ref = torch.cat(ref)
    e2, r2 = (acc[ids, :3] - ref).square().sum(1), ref.square().sum(1)
    return dict(acc=acc, conserved=conserved, force_rms=float((e2.sum() / r2.sum()).sqrt()),
                force_max=float((e2 / r2).max().sqrt()))
