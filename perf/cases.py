"""Performance cases of the peridynamics step: what programs call, over the range of sizes they call it at.

Kinds of pass (``run``), each through the public binding (native.py, one Python call per C ABI call):

  step      a resident plate advanced from a host state to a host state, Context.step_host
  velocity  the one-call force + kick on page-locked host buffers, Context.compute_velocity
  device    the same on device buffers that the caller owns, pd_compute_velocity_noalloc
  batch     ragged plates: states in, Batch.step, states out
  assoc     the bond-associated model with the Mazars law updated before every step (the
            reference's main loop), Context.mazars_update + Context.step

``exact`` restates each in 64-bit torch on a plate's regular stencil (or padded neighbour lists), without the package.
"""
import importlib
import math
import random

import numpy as np
import torch

DX = 1e-3
MAT = {"E": 72e9, "nu": 0.33, "rho": 2440.0}
S_C = 5e-4
HORIZON = 3.015


def listed():
    return [
        # a caller with its own device pool and a small part, once per time step of its own loop: launch latency
        {"name": "device-call-30x31", "kind": "device", "nx": 30, "ny": 31, "penalty": False, "graded": False},
        # the largest plate that entry point takes (65,536 particles)
        {"name": "device-call-256x255", "kind": "device", "nx": 256, "ny": 255, "penalty": True, "graded": False},
        # the reference's own problem size and model (70 x 60 unit mesh, n1 = n2 = 10), its main loop for ten steps
        {"name": "reference-run-70x60", "kind": "assoc", "nx": 70, "ny": 60, "steps": 10, "n1": 10.0, "n2": 10.0,
         "mazars": True},
        # the 100-step FP64 plate of the validation runs
        {"name": "plate-fp64-100x100", "kind": "step", "precision": "fp64", "nx": 100, "ny": 100, "steps": 100,
         "crack": "centre", "graded": False, "breaking": True},
        # the FP64 plate at scale, advanced in chunks between looks at its state
        {"name": "plate-fp64-1000x1000", "kind": "step", "precision": "fp64", "nx": 1000, "ny": 1000, "steps": 10,
         "crack": "centre", "graded": False, "breaking": True},
        # the same plate coupled to a host code: the state crosses the link in every step
        {"name": "host-step-fp64-1000x1000", "kind": "step", "precision": "fp64", "nx": 1000, "ny": 1000, "steps": 1,
         "crack": "centre", "graded": False, "breaking": True},
        # the drop-in call on a middle-sized plate with cell volumes from a mesh file, the reference's plain model
        {"name": "velocity-call-317x251", "kind": "velocity", "nx": 317, "ny": 251, "penalty": False, "graded": True},
        # a short request at the small end of the served sizes, 2:1
        {"name": "plate-mixed-203x101", "kind": "step", "precision": "mixed", "nx": 203, "ny": 101, "steps": 50,
         "crack": "angled", "graded": False, "breaking": True},
        # the mixed form's main size
        {"name": "plate-mixed-1000x1000", "kind": "step", "precision": "mixed", "nx": 1000, "ny": 1000, "steps": 50,
         "crack": "centre", "graded": False, "breaking": True},
        # beyond the caches, uneven sides
        {"name": "plate-mixed-2048x1953", "kind": "step", "precision": "mixed", "nx": 2048, "ny": 1953, "steps": 20,
         "crack": "angled", "graded": False, "breaking": True},
        # ragged batches of 50 .. 400 particles a side, as in the batched workload and the serving loop
        {"name": "batch-mixed-16", "kind": "batch", "precision": "mixed", "plates": 16, "mix": 1, "steps": 100},
        {"name": "batch-fp64-9", "kind": "batch", "precision": "fp64", "plates": 9, "mix": 2, "steps": 20},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "step", "batch", "velocity", "device", "assoc"])
    if kind == "step":
        precision = rng.choice(["fp64", "mixed"])
        n = log(2000, 2000000)
        aspect = rng.choice([1.0, 2.0, rng.uniform(0.4, 2.5)])
        nx = max(24, int(math.sqrt(n * aspect)))
        ny = max(24, int(n / nx))
        most = (8e6 if precision == "fp64" else 4e7) / (nx * ny)
        return {"kind": "step", "precision": precision, "nx": nx, "ny": ny, "steps": max(1, min(log(1, 100), int(most))),
                "crack": rng.choice(["none", "centre", "angled"]), "graded": rng.random() < 0.3,
                "breaking": rng.random() < 0.8}
    if kind == "batch":
        precision = rng.choice(["fp64", "mixed"])
        return {"kind": "batch", "precision": precision, "plates": rng.randint(2, 9 if precision == "fp64" else 16),
                "mix": rng.randint(3, 10**6), "steps": rng.randint(4, 16 if precision == "fp64" else 80)}
    if kind == "velocity":
        return {"kind": "velocity", "nx": log(30, 900), "ny": log(30, 900), "penalty": rng.random() < 0.5,
                "graded": rng.random() < 0.5}
    if kind == "device":
        nx = log(12, 1024)
        ny = max(12, min(log(12, 1024), 65536 // nx))
        return {"kind": "device", "nx": nx, "ny": min(ny, 65536 // nx), "penalty": rng.random() < 0.5,
                "graded": rng.random() < 0.5}
    return {"kind": "assoc", "nx": log(20, 90), "ny": log(20, 90), "steps": rng.randint(1, 12),
            "n1": rng.choice([10.0, 4.5, 0.0]), "n2": rng.choice([10.0, 3.0, 2.5]), "mazars": rng.random() < 0.5}


# ---------------------------------------------------------------- inputs


def _plate(nx, ny, seed, crack="none", graded=False, material=None, load=1.0):
    """A jittered regular plate under tension: geometry, boundary groups and a state in mid-run."""
    r = np.random.default_rng([int(seed), nx, ny])
    n, w, h = nx * ny, (nx - 1) * DX, (ny - 1) * DX
    col, row = np.arange(n) % nx, np.arange(n) // nx
    base = np.stack([(col - nx // 2) * DX, (row - ny // 2) * DX], axis=1)
    x = base + (2.0 * r.random((n, 2)) - 1.0) * (0.01 * DX)
    vol = np.full(n, DX**3)
    if graded:
        vol *= 1.0 + 0.25 * (2.0 * r.random(n) - 1.0)
    mid = np.array([(-(nx // 2) + 0.5 * (nx - 1)) * DX, (-(ny // 2) + ny // 2 - 0.5) * DX])
    seg = np.zeros((0, 4))
    half = 0.25 * w
    if crack == "centre":
        seg = np.array([[mid[0] - half, mid[1], mid[0] + half, mid[1]]])
    elif crack == "angled":
        a = r.uniform(-math.pi / 6, math.pi / 6)
        c = mid + np.array([r.uniform(-0.1, 0.1) * w, r.uniform(-0.1, 0.1) * h])
        k = 0.2 * min(w, h)
        seg = np.array([[c[0] - k * math.cos(a), c[1] - k * math.sin(a), c[0] + k * math.cos(a), c[1] + k * math.sin(a)]])
    # a strain of 3e-4 with long waves, and hot spots above the critical stretch at the crack's ends
    u = np.stack([-1e-4 * base[:, 0], 3e-4 * base[:, 1]], axis=1)
    for _ in range(3):
        k, p = r.uniform(1.0, 4.0, 2) * math.pi / np.array([w, h]), r.uniform(0, 2 * math.pi)
        u += (r.uniform(-1, 1, 2) * 2e-5 / np.linalg.norm(k)) * np.sin(base @ k + p)[:, None]
    for s in seg:
        for e in (s[:2], s[2:]):
            q = (base - e) / (6 * DX)
            u[:, 1] += 3e-4 * 6 * DX * q[:, 1] * np.exp(-(q * q).sum(1))
    u += (2.0 * r.random((n, 2)) - 1.0) * (1e-5 * DX)
    v = np.stack([np.zeros(n), 2.0 * load * base[:, 1] / max(h, DX)], axis=1) + (2.0 * r.random((n, 2)) - 1.0) * 0.01
    f = 1e8 * np.stack([np.sin(base[:, 0] * 40 / w), np.cos(base[:, 1] * 30 / h)], axis=1) * r.uniform(0.5, 1.0)
    group = np.zeros(n, dtype=np.uint8)
    group[row >= ny - 3] = 1
    group[row < 3] = 2
    m = dict(MAT if material is None else material)
    c11 = m["E"] / (1.0 - m["nu"] ** 2)
    cutoff = 1.01 * DX * HORIZON
    return {"nx": nx, "ny": ny, "n": n, "x": x, "vol": vol, "seg": seg, "u": u, "v": v, "f": f, "group": group,
            "gval": np.array([[0.0, load], [0.0, -load]]), "cutoff": cutoff, "dt": 0.8 * DX / math.sqrt(m["E"] / m["rho"]),
            "k_hg": 0.25 * c11 / (float(vol.mean()) * cutoff * cutoff), **m}


def _members(case, seed):
    r = random.Random(case["mix"])
    out = []
    for k in range(case["plates"]):
        m = {"E": r.uniform(50e9, 100e9), "nu": r.uniform(0.2, 0.35), "rho": 2440.0}
        side = r.randint(50, 400)
        out.append(_plate(side, side, seed * 1000 + k, "angled", k % 3 == 2, m, r.uniform(0.5, 2.0)))
    return out


def _problem(case, seed):
    if case["kind"] == "step":
        return _plate(case["nx"], case["ny"], seed, case["crack"], case["graded"])
    return _plate(case["nx"], case["ny"], seed, "none", case["graded"])


def _assoc(case, seed):
    """The reference's mesh rule (unit cells) at nx x ny, its GPU main's material, a strained state."""
    nx, ny = case["nx"], case["ny"]
    r = np.random.default_rng([int(seed), nx, ny, 5])
    col, row = np.arange(nx * ny) % nx, np.arange(nx * ny) // nx
    x = np.stack([col - 0.5 * (nx - 1), row - 0.5 * (ny - 1)], axis=1).astype(np.float64)
    u = np.stack([-2e-5 * x[:, 0], 9e-5 * x[:, 1]], axis=1)
    for _ in range(4):
        k, p = r.uniform(1.0, 5.0, 2) * math.pi / np.array([nx, ny]), r.uniform(0, 2 * math.pi)
        u += (r.uniform(-1, 1, 2) * 3e-5 / np.linalg.norm(k)) * np.sin(x @ k + p)[:, None]
    v = np.stack([np.zeros(nx * ny), 10.0 * x[:, 1] / ny], axis=1)
    group = np.zeros(nx * ny, dtype=np.uint8)
    group[row == ny - 1] = 1
    group[row == 0] = 2
    return {"nx": nx, "ny": ny, "n": nx * ny, "x": x, "vol": np.ones(nx * ny), "u": u, "v": v, "f": np.zeros_like(u),
            "group": group, "gval": np.array([[0.0, 5.0], [0.0, -5.0]]), "cutoff": 1.01 * 3.0, "E": 3.5e4, "nu": 0.2,
            "rho": 2.5e-6, "dt": 1e-9, "wlen": 3.0, "kappa0": 3.0 / 3.5e4}


# ---------------------------------------------------------------- the package's side


def _package():
    return importlib.import_module("2d_pd_gpu_gb300")


def _params(nat, p, precision, s_c, k_hg, fail, **kw):
    return nat.default_params(precision=precision, device=0, E=p["E"], nu=p["nu"], rho=p["rho"], dt=p["dt"], s_c=s_c,
                              k_hg=k_hg, damage_fail=fail, **kw)


def _context(nat, p, precision, s_c, k_hg, fail, **kw):
    c = nat.Context(_params(nat, p, precision, s_c, k_hg, fail, **kw))
    c.set_particles(p["x"], p["vol"])
    c.build_families(p["cutoff"], p.get("seg"))
    c.set_bc([nat.PD_BC_VELOCITY] * 2, p["gval"], p["group"])
    return c


class _Held(np.ndarray):
    """A view of a page-locked buffer that keeps the buffer (whose finaliser frees it)."""


def _pinned(nat, *arrays):
    out = []
    for a in arrays:
        b = nat.PinnedArray(a.shape)
        b.array[...] = a
        h = b.array.view(_Held)
        h.owner = b
        out.append(h)
    return out


def prepare(case, seed):
    nat = _package().native
    kind = case["kind"]
    if kind == "batch":
        prec = nat.PD_MIXED if case["precision"] == "mixed" else nat.PD_FP64
        ms = _members(case, seed)
        b = nat.Batch(prec)
        ctx = [_context(nat, p, prec, S_C, p["k_hg"], 0.5) for p in ms]
        for c in ctx:
            b.add(c)
        return {"case": case, "nat": nat, "batch": b, "ctx": ctx, "in": [_pinned(nat, p["u"], p["v"], p["f"]) for p in ms],
                "out": [_pinned(nat, p["u"], p["v"], p["f"]) for p in ms]}
    if kind == "assoc":
        p = _assoc(case, seed)
        c = _context(nat, p, nat.PD_FP64, 0.0, 0.0, 1.0, n1=case["n1"], n2=case["n2"], weight_len=p["wlen"])
        return {"case": case, "nat": nat, "ctx": c, "u": p["u"], "v": p["v"], "f": p["f"],
                "law": nat.mazars_default_params(kappa0=p["kappa0"])}
    p = _problem(case, seed)
    if kind == "device":
        k_hg = p["k_hg"] if case["penalty"] else 0.0
        idx, ok = _lists(p)
        dev = {k: torch.from_numpy(np.ascontiguousarray(p[k])).cuda() for k in ("x", "vol", "u", "v")}
        deg = ok.sum(1)
        rp = torch.zeros(p["n"] + 1, dtype=torch.int64, device="cuda")
        rp[1:] = deg.cumsum(0)
        return {"case": case, "nat": nat, "rp": rp, "col": idx[ok].to(torch.int32).contiguous(), **dev,
                "acce": torch.zeros_like(dev["u"]), "netf": torch.zeros_like(dev["u"]), "n": p["n"],
                "params": _params(nat, p, nat.PD_FP64, 0.0, k_hg, 1.0)}
    if kind == "velocity":
        c = _context(nat, p, nat.PD_FP64, 0.0, p["k_hg"] if case["penalty"] else 0.0, 1.0)
        return {"case": case, "nat": nat, "ctx": c, "buf": _pinned(nat, p["u"], p["v"], np.zeros_like(p["u"]), p["f"])}
    prec = nat.PD_MIXED if case["precision"] == "mixed" else nat.PD_FP64
    c = _context(nat, p, prec, S_C if case["breaking"] else 0.0, p["k_hg"], 0.5)
    return {"case": case, "nat": nat, "ctx": c, "in": _pinned(nat, p["u"], p["v"], p["f"]),
            "out": _pinned(nat, p["u"], p["v"], p["f"])}


def run(s):
    case, nat = s["case"], s["nat"]
    kind = case["kind"]
    if kind == "step":
        i, o, c = s["in"], s["out"], s["ctx"]
        c.step_host(case["steps"], *i, *o)
        r = list(o)
        if c.n <= 50000:
            r.append(c.damage())  # a small plate's fracture state is looked at with its motion
        return r
    if kind == "velocity":
        b = s["buf"]
        s["ctx"].compute_velocity(*b)
        return b[1:]
    if kind == "device":
        rc = nat.lib().pd_compute_velocity_noalloc(
            s["n"], s["x"].data_ptr(), s["vol"].data_ptr(), s["rp"].data_ptr(), s["col"].data_ptr(), s["u"].data_ptr(),
            s["v"].data_ptr(), s["acce"].data_ptr(), s["netf"].data_ptr(), s["params"],
            torch.cuda.current_stream().cuda_stream, None, 0)
        if rc != nat.PD_OK:
            raise nat.PdError(rc, "pd_compute_velocity_noalloc")
        return [s["v"], s["acce"], s["netf"]]
    if kind == "batch":
        for c, i in zip(s["ctx"], s["in"]):
            c.set_state(*i)
        s["batch"].step(case["steps"])
        for c, o in zip(s["ctx"], s["out"]):
            c._ck(nat.lib().pd_get_state(c.handle, *(nat.ptr(a) for a in o)))
        return s["out"]
    c = s["ctx"]
    c.set_state(s["u"], s["v"], s["f"])
    if not case["mazars"]:
        c.step(case["steps"])
        return list(c.state())
    c.mazars_init(s["law"])
    for _ in range(case["steps"]):
        c.mazars_update()
        c.step(1)
    return list(c.state()) + list(c.mazars())


def work(case):
    """State in and out once, and per step the state, the geometry and one 4-byte id per bond once."""
    if case["kind"] == "batch":
        r, n = random.Random(case["mix"]), 0
        for _ in range(case["plates"]):
            r.uniform(0, 1), r.uniform(0, 1)
            n += r.randint(50, 400) ** 2
            r.uniform(0, 1)
    else:
        n = case["nx"] * case["ny"]
    bonds, steps = 28 * n, case.get("steps", 1)
    state = 80 if case.get("precision") == "mixed" else 96
    per_step = n * (state + 24) + 4 * bonds
    flops = 29 * bonds + 110 * n
    if case["kind"] in ("velocity", "device"):
        return {"bytes": n * (48 + 48 + 24) + 4 * bonds, "flops": flops + 8 * bonds}
    if case["kind"] == "assoc":
        pairs = 28 * bonds
        one = 16 * pairs + 30 * bonds
        return {"bytes": steps * (n * 120 + 4 * bonds + (32 * bonds if case["mazars"] else 0)) + 96 * n,
                "flops": steps * (one + (8 * pairs + 60 * bonds if case["mazars"] else 0))}
    return {"bytes": steps * per_step + 96 * n, "flops": steps * flops}


# ---------------------------------------------------------------- the 64-bit restatement


def _grid(p):
    """Positions and volumes on the padded grid, the stencil's offsets and which of them are bonds."""
    nx, ny, P = p["nx"], p["ny"], 4
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = {k: torch.as_tensor(p[k], dtype=torch.float64, device=dev).reshape(ny, nx, -1) for k in ("x", "vol", "u", "v", "f")}

    def pad(a):
        out = torch.zeros((ny + 2 * P, nx + 2 * P, a.shape[2]), dtype=a.dtype, device=dev)
        out[P:P + ny, P:P + nx] = a
        return out

    def near(a, offs):
        q = pad(a)
        return torch.stack([q[P + j:P + j + ny, P + i:P + i + nx] for i, j in offs])

    inside = torch.ones((ny, nx, 1), dtype=torch.float64, device=dev)
    offs = sorted(((i, j) for i in range(-P, P + 1) for j in range(-P, P + 1) if (i or j) and i * i + j * j < 12),
                  key=lambda o: (o[1], o[0]))
    xi = near(t["x"], offs) - t["x"]
    ok = (near(inside, offs)[..., 0] > 0) & (torch.sqrt((xi * xi).sum(-1)) < p["cutoff"])
    for s in p.get("seg", ()):  # proper crossings of the segment
        a, b = torch.tensor(s[:2], device=dev), torch.tensor(s[2:], device=dev)
        q = t["x"] + xi

        def side(o, d, c):
            return (d[..., 0] - o[..., 0]) * (c[..., 1] - o[..., 1]) - (d[..., 1] - o[..., 1]) * (c[..., 0] - o[..., 0])

        own = t["x"].expand_as(q)
        d1, d2 = side(a, b, own), side(a, b, q)
        d3, d4 = side(own, q, a.expand_as(q)), side(own, q, b.expand_as(q))
        ok &= ~((d1 * d2 < 0) & (d3 * d4 < 0))
    return t, offs, xi, ok, near


def _lists(p):
    """Padded neighbour lists (ids ascending) and which entries are bonds."""
    t, offs, _, ok, _ = _grid(p)
    n, nx = p["n"], p["nx"]
    ids = torch.arange(n, device=ok.device).reshape(p["ny"], nx)
    idx = torch.stack([ids + j * nx + i for i, j in offs]).reshape(len(offs), n).T.contiguous()
    return idx, ok.reshape(len(offs), n).T.contiguous()


class _Exact:
    """The plain model on a grid in 64 bits: stretch test, K, F - I, stress, penalty, force."""

    def __init__(self, p, s_c, k_hg, fail):
        self.p, self.s_c, self.k, self.fail = p, s_c, k_hg, fail
        self.t, self.offs, self.xi, self.alive, self.near = _grid(p)
        self.family = self.alive.sum(0).to(torch.float64)
        self.vj = self.near(self.t["vol"], self.offs)
        pre = p["E"] / (1 - p["nu"] ** 2)
        self.c = (pre, p["nu"] * pre, (1 - p["nu"]) * pre)
        self.group = torch.as_tensor(p["group"].reshape(p["ny"], p["nx"]), device=self.xi.device)
        self._shape()

    def _shape(self):
        live = self.alive[..., None].to(torch.float64)
        t = self.vj * live * self.xi
        K = torch.einsum("oyxa,oyxb->yxab", t, self.xi)
        det = K[..., 0, 0] * K[..., 1, 1] - K[..., 0, 1] ** 2
        self.damage = 1.0 - live[..., 0].sum(0) / self.family.clamp(min=1)
        good = (det > 1e-10 * K[..., 0, 0] * K[..., 1, 1]) & ~(self.damage > self.fail)
        inv = torch.stack([K[..., 1, 1], -K[..., 0, 1], -K[..., 1, 0], K[..., 0, 0]], -1).reshape(K.shape)
        self.inv = torch.where(good[..., None, None], inv / torch.where(good, det, 1.0)[..., None, None], 0.0)
        self.m = t.sum(0) * good[..., None]
        self.t_xi = t

    def force(self, u):
        d = self.near(u, self.offs) - u
        if self.s_c > 0:
            x2 = (self.xi * self.xi).sum(-1)
            gone = self.alive & ((d * (2 * self.xi + d)).sum(-1) > ((1 + self.s_c) ** 2 - 1) * x2)
            if bool(gone.any()):
                self.alive = self.alive & ~gone
                self._shape()
        live = self.alive[..., None].to(torch.float64)
        G = torch.einsum("oyxa,oyxb->yxab", d, self.t_xi) @ self.inv
        e11, e22, e12 = G[..., 0, 0], G[..., 1, 1], 0.5 * (G[..., 0, 1] + G[..., 1, 0])
        c11, c12, c33 = self.c
        sig = torch.stack([c11 * e11 + c12 * e22, c33 * e12, c33 * e12, c12 * e11 + c11 * e22], -1).reshape(G.shape)
        S = sig @ self.inv - self.k * G * (self.inv.abs().sum((-1, -2)) > 0)[..., None, None]
        W = S * self.t["vol"][..., None]
        f = (S @ self.m[..., None])[..., 0]
        Wj = self.near(W.reshape(*W.shape[:2], 4), self.offs).reshape(len(self.offs), *W.shape)
        f = f + ((Wj @ self.xi[..., None])[..., 0] * live).sum(0)
        return f + 2 * self.k * (self.vj * live * d).sum(0)

    def steps(self, n):
        p, (u, v, f) = self.p, (self.t[k].clone() for k in ("u", "v", "f"))
        dt, rho = p["dt"], p["rho"]
        for _ in range(n):
            for g, val in enumerate(p["gval"]):
                v[self.group == g + 1] = torch.as_tensor(val, device=v.device)
            u = u + v * dt + 0.5 * (f / rho) * dt * dt
            new = self.force(u)
            v = v + 0.5 * (f + new) / rho * dt
            f = new
        return [a.reshape(-1, 2).cpu() for a in (u, v, f)]


def _exact_assoc(case, p):
    idx, ok = _lists({**p, "f": p["f"], "seg": ()})
    dev, n = idx.device, p["n"]
    idx = torch.where(ok, idx, torch.arange(n, device=dev)[:, None])
    T = {k: torch.as_tensor(p[k], dtype=torch.float64, device=dev) for k in ("x", "vol", "u", "v", "f")}
    live = ok.to(torch.float64)
    xi = T["x"][idx] - T["x"][:, None]
    L = torch.where(ok, torch.sqrt((xi * xi).sum(-1)), 1.0)
    V = T["vol"][idx] * live
    cos = (torch.einsum("nba,nka->nbk", xi, xi) / (L[:, :, None] * L[:, None, :])).clamp(-1.0, 1.0)
    w = torch.exp(-case["n1"] * (L[:, :, None] - L[:, None, :]).abs() / p["wlen"]) * (0.5 + 0.5 * cos) ** case["n2"]
    w = w * live[:, :, None] * live[:, None, :]
    t = V[..., None] * xi
    K = torch.einsum("nbk,nkp,nkq->nbpq", w, t, xi)
    det = K[..., 0, 0] * K[..., 1, 1] - K[..., 0, 1] ** 2
    good = ok & (det > 1e-10 * K[..., 0, 0] * K[..., 1, 1])
    inv = torch.stack([K[..., 1, 1], -K[..., 0, 1], -K[..., 1, 0], K[..., 0, 0]], -1).reshape(K.shape)
    inv = torch.where(good[..., None, None], inv / torch.where(good, det, 1.0)[..., None, None], 0.0)
    back = torch.zeros_like(idx)  # the slot of the reverse bond
    for k in range(idx.shape[1]):
        hit = (idx[idx[:, k]] == torch.arange(n, device=dev)[:, None]) & ok[idx[:, k]]
        back[:, k] = hit.to(torch.int64).argmax(1)
    pre = p["E"] / (1 - p["nu"] ** 2)
    c11, c12, c33 = pre, p["nu"] * pre, (1 - p["nu"]) * pre
    fam = ok.sum(1).to(torch.float64)
    thr = torch.full(idx.shape, p["kappa0"], dtype=torch.float64, device=dev)
    bd = torch.zeros_like(thr)
    group = torch.as_tensor(p["group"], device=dev)
    u, v, f = T["u"], T["v"].clone(), T["f"]

    def strain(u):
        d = u[idx] - u[:, None]
        G = torch.einsum("nbk,nkp,nkq->nbpq", w, d * V[..., None], xi) @ inv
        return G[..., 0, 0], G[..., 1, 1], 0.5 * (G[..., 0, 1] + G[..., 1, 0])

    for _ in range(case["steps"]):
        if case["mazars"]:
            a, b, c = strain(u)
            rad = torch.sqrt((0.5 * (a - b)) ** 2 + c * c)
            l0, l1 = 0.5 * (a + b) - rad, 0.5 * (a + b) + rad
            eq = torch.sqrt(l0.clamp(min=0) ** 2 + l1.clamp(min=0) ** 2)
            up = ok & (eq > thr)
            q = torch.where(up, eq, 1.0)  # (the tensile share is 1, the compressive one 0, whatever the signs)
            bd = torch.where(up, 1.0 - thr * (1 - 0.87) / q - 0.87 / torch.exp(20000.0 * (q - thr)), bd)
            thr = torch.where(up, eq, thr)
        for g, val in enumerate(p["gval"]):
            v[group == g + 1] = torch.as_tensor(val, device=dev)
        u = u + v * p["dt"] + 0.5 * (f / p["rho"]) * p["dt"] ** 2
        e11, e22, e12 = strain(u)
        sig = torch.stack([c11 * e11 + c12 * e22, c33 * e12, c33 * e12, c12 * e11 + c11 * e22], -1).reshape(K.shape)
        M = torch.einsum("njb,nbpq->njpq", w, sig @ inv * V[..., None, None]) / V.sum(1)[:, None, None, None]
        Tij = (M @ xi[..., None])[..., 0]
        new = ((Tij - Tij[idx, back]) * V[..., None]).sum(1)
        v = v + 0.5 * (f + new) / p["rho"] * p["dt"]
        f = new
    out = [u, v, f]
    if case["mazars"]:
        out += [thr[ok], bd[ok], (bd * live / fam[:, None]).sum(1)]
    return [a.cpu() for a in out]


def exact(case, seed):
    kind = case["kind"]
    if kind == "assoc":
        return _exact_assoc(case, _assoc(case, seed))
    if kind == "batch":
        return [_Exact(p, S_C, p["k_hg"], 0.5).steps(case["steps"]) for p in _members(case, seed)]
    p = _problem(case, seed)
    if kind == "step":
        e = _Exact(p, S_C if case["breaking"] else 0.0, p["k_hg"], 0.5)
        r = e.steps(case["steps"])
        return r + [e.damage.reshape(-1).cpu()] if p["n"] <= 50000 else r
    e = _Exact(p, 0.0, p["k_hg"] if case["penalty"] else 0.0, 1.0)
    f = e.force(e.t["u"])
    a = f / p["rho"]
    v = e.t["v"] + 0.5 * a * p["dt"]
    return [x.reshape(-1, 2).cpu() for x in (v, a, f)]
