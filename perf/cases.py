"""Timed workloads of the solver: what a program does with it, at the sizes it meets.

listed() gives fixed cases, draw(rng) more of the same ranges.  prepare() makes
a case's inputs on the GPU from a seed, run() is one pass through the public
entry points (zsph_b200.Solver and the C entry points of zsph_b200.lib),
work() what the pass cannot do without, and exact() the pass in 64 bits, in
plain torch.

The particle states are dam breaks in motion: the lattice column of
zsph_b200.cases.dam_break with positions moved off the lattice, a velocity
field, compressed densities, sorted by cell as every state but a run's first
is, then displaced by less than a half step, so that the next search meets the
few per cent of cell changes that a running case has.  "mixed" states carry
the particles of a cell in arbitrary order, as a flow does once it has mixed;
the others in the lattice's.
"""
import functools
import math

import numpy as np
import torch

import zsph_b200 as z
from zsph_b200 import cases as zc

DEV = "cuda"


def listed():
    return [
        # the smallest runs: a coarse scene, one step per call, where launches and latency count
        {"name": "step_20k", "kind": "step", "api": "step", "dx": 0.04, "mixed": False},
        # the plain dam break of the benchmark's first configuration, through the step loop
        {"name": "run_105k", "kind": "step", "api": "run", "dx": 0.02, "mixed": True},
        # the dam break at scale: the largest state of the repository's configurations
        {"name": "run_4m", "kind": "step", "api": "run", "dx": 0.005, "mixed": False},
        # the neighbour search alone at that size (a caller with equations of its own)
        {"name": "search_4m", "kind": "search", "dx": 0.005, "mixed": True},
        # the two equation passes on a sorted state, as a caller with its own integrator uses them
        {"name": "pairs_445k", "kind": "pairs", "dx": 0.0115, "mixed": True},
        # the reference driver's twelve separate calls per step
        {"name": "dropin_105k", "kind": "dropin", "dx": 0.02, "mixed": True},
        # many small scenes of uneven size in one handle
        {"name": "batch_24", "kind": "batch", "scenes": 24, "scene_seed": 7},
        # precision form with a floating body
        {"name": "body_362k", "kind": "body", "dx": 0.02},
        # the simple-SPH equations (the reference's other target)
        {"name": "simple_105k", "kind": "simple", "dx": 0.02, "mixed": True},
        # the learned form's list-reuse corrector in place of the second search
        {"name": "reuse_270k", "kind": "reuse", "dx": 0.014, "mixed": False},
        # the corrector network: inference over the rows of a large case
        {"name": "mlp_forward_1m", "kind": "mlp_forward", "rows": 1000003},
        # the corrector network: one pass over a training set of 8 batches, weights read at its end
        {"name": "mlp_epoch_8", "kind": "mlp_epoch", "batches": 8, "batch_tiles": 148},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "search", "pairs", "pairs", "dropin", "batch", "body", "simple",
                       "reuse", "mlp_forward", "mlp_epoch"])
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(3, 40), "scene_seed": rng.randrange(10000)}
    if kind == "body":
        return {"kind": kind, "dx": round(_log(rng, 0.02, 0.045), 5)}
    if kind == "mlp_forward":
        return {"kind": kind, "rows": int(_log(rng, 1, 1500000))}
    if kind == "mlp_epoch":
        return {"kind": kind, "batches": rng.randint(2, 12), "batch_tiles": rng.randint(1, 400)}
    c = {"kind": kind, "dx": round(_log(rng, 0.0058, 0.05), 5), "mixed": rng.random() < 0.5,
         "wx": round(rng.uniform(0.3, 0.8), 3), "wy": round(rng.uniform(0.3, 0.62), 3),
         "wz": round(rng.uniform(0.4, 1.2), 3), "lx": round(rng.uniform(0.9, 1.7), 3)}
    if kind == "step":
        c["api"] = rng.choice(["step", "run"])
        if rng.random() < 0.2:
            c["gf"] = 2  # the case file's grid_size_factor 2: cells of h, a 5x5 stencil
    return c


# ---- states ------------------------------------------------------------------

def _dam(case):
    wx, wy, wz, lx = (case.get(k, d) for k, d in (("wx", 0.6), ("wy", 0.6), ("wz", 1.2), ("lx", 1.6)))
    phys = {"grid_size_factor": 2.0} if case.get("gf", 1) == 2 else {}
    dx = case["dx"]
    up = lambda v: math.ceil(v / dx - 1e-6) * dx  # whole lattice layers
    return zc.dam_break(dx, water=(up(wx), up(wy), up(wz)), tank=(up(lx), up(wy), up(max(wz, 0.6))), **phys)


@functools.lru_cache(maxsize=4)
def _lattice(key):
    """The lattice case and its arrays on the GPU (no seed enters)."""
    c = _dam(dict(key))
    s = c.state
    return c, {k: torch.from_numpy(getattr(s, k)).to(DEV) for k in ("pos", "vel", "rhop", "type")}


def _geometry(case):
    return _lattice(tuple(sorted((k, v) for k, v in case.items() if k in ("dx", "wx", "wy", "wz", "lx", "gf"))))


def _cell(gp, pos):
    """Cell keys in the solver's FP32 arithmetic (hash.cu:12-15)."""
    q = []
    for a, lo in enumerate((gp.grid_xmin, gp.grid_ymin, gp.grid_zmin)):
        lo_t = torch.tensor(lo, dtype=torch.float32, device=pos.device)
        gs_t = torch.tensor(gp.grid_size, dtype=torch.float32, device=pos.device)
        q.append(torch.floor((pos[:, a] - lo_t) / gs_t).long())
    return q[2] * (gp.grid_xdim * gp.grid_ydim) + q[1] * gp.grid_xdim + q[0]


def _in_motion(gp, dx, base, seed, mixed):
    """A running case's state from the lattice arrays: see the module's comment."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    rnd = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=torch.float32)
    n = base["pos"].shape[0]
    fluid = (base["type"] == 1)
    f = fluid[:, None].float()
    pos = base["pos"] + f * (rnd(n, 3) - 0.5) * (0.25 * dx)
    amp = rnd(3) + 0.5
    swirl = torch.stack([amp[0] * torch.sin(3.0 * pos[:, 2]), amp[1] * torch.sin(4.0 * pos[:, 0]) * 0.3,
                         -amp[2] * torch.cos(3.0 * pos[:, 0]) * 0.5], 1)
    vel = f * (0.4 * swirl + 0.1 * (rnd(n, 3) - 0.5))
    rho = base["rhop"][:, 0] + fluid.float() * rnd(n)
    cs2, rho0 = float(gp.cs2), float(gp.rho0)
    rhop = torch.where(fluid[:, None], torch.stack([rho, cs2 * (rho - rho0)], 1), base["rhop"])
    order = torch.randperm(n, generator=g, device=DEV) if mixed else torch.arange(n, device=DEV)
    perm = order[torch.sort(_cell(gp, pos)[order], stable=True).indices]
    take = lambda a: a[perm].contiguous()
    typ = take(base["type"])
    pos = take(pos) + (typ == 1)[:, None].float() * (rnd(n, 3) - 0.5) * (0.03 * dx)
    vel, rhop = take(vel), take(rhop)
    table = (perm - torch.arange(n, device=DEV)).to(torch.int32)
    return {"pos": pos, "vel": vel, "rhop": rhop, "type": typ, "table": table, "tmp_pos": pos.clone(),
            "tmp_vel": vel.clone(), "tmp_rhop": rhop.clone()}


def _inputs(case, seed):
    c, base = _geometry(case)
    _, gp = z.params_from_json(c.json)
    return gp, _in_motion(gp, case["dx"], base, seed, case.get("mixed", False))


class _Mem:
    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner  # the tensors made from this keep the solver's memory
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(sol, ptr, shape, typestr="<f4"):
    """A device array of the solver as a tensor (no copy)."""
    return torch.as_tensor(_Mem(sol, ptr, tuple(shape), typestr), device=DEV)


_PTC = {"pos": (3, "<f4"), "vel": (3, "<f4"), "rhop": (2, "<f4"), "tmp_pos": (3, "<f4"), "tmp_vel": (3, "<f4"),
        "tmp_rhop": (2, "<f4"), "type": (1, "<i4"), "table": (1, "<i4")}


def _ptc(sol, which, names):
    b = sol.old if which == "old" else sol.new
    return {k: _view(sol, getattr(b, k), (sol.n, _PTC[k][0]) if _PTC[k][0] > 1 else (sol.n,), _PTC[k][1]) for k in names}


def _tmp(sol, names):
    shapes = {"acc_drhodt": ((sol.n, 4), "<f4"), "dofv_grandrho": ((sol.n, 4), "<f4"), "dofv": ((sol.n,), "<f4"),
              "index": ((sol.n,), "<i4"), "hash": ((sol.n,), "<i4"), "grid_start": ((sol.G,), "<i4"),
              "grid_end": ((sol.G,), "<i4")}
    return {k: _view(sol, getattr(sol.tmp, k), *shapes[k]) for k in names}


def _load(sol, st, which="old"):
    for k, v in _ptc(sol, which, list(_PTC)).items():
        v.copy_(st[k])


def _scenes(case):
    return zc.batch_scenes(case["scenes"], seed=case["scene_seed"])[0]


def _batch_inputs(case, seed):
    out = []
    for k, c in enumerate(_scenes(case)):
        _, gp = z.params_from_json(c.json)
        base = {a: torch.from_numpy(getattr(c.state, a)).to(DEV) for a in ("pos", "vel", "rhop", "type")}
        out.append((gp, _in_motion(gp, float(c.json.dx), base, seed * 1000 + k, k % 2 == 1)))
    return out


def _net(seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(-1, 1, z.MLP_NPARAM).astype(np.float32)
    p[:4096] *= 0.3          # W1
    p[4096:4224] *= 0.05     # b1
    p[4224:20608] *= 0.15    # W2
    p[20608:20736] *= 0.05   # b2
    p[20736:21248] *= 0.15   # W3
    return p


def _rows(n, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn(n, 32, generator=g, device=DEV)


def _train_set(case, seed):
    n = case["batches"] * case["batch_tiles"] * z.MLP_TILE
    x = _rows(n, seed)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 1)
    y = torch.stack([torch.tanh(x[:, 0] + x[:, 5]), x[:, 1] * x[:, 2], torch.sin(x[:, 3]), x[:, 4]], 1)
    y = (y + 0.1 * torch.randn(n, 4, generator=g, device=DEV)).contiguous()
    w = (torch.rand(n, generator=g, device=DEV) < 0.8).float()
    ids = torch.randperm(n // z.MLP_TILE, generator=g, device=DEV).to(torch.int32)
    rng = np.random.default_rng(seed + 2)
    m1 = (rng.normal(size=z.MLP_NPARAM) * 1e-2).astype(np.float32)
    m2 = (1e-3 * (0.5 + rng.uniform(size=z.MLP_NPARAM))).astype(np.float32)
    return x, y, w, ids, m1, m2


def _pack(x):
    tiles = torch.empty((x.shape[0] + z.MLP_TILE - 1) // z.MLP_TILE, 4096, dtype=torch.int16, device=DEV)
    z.check(z.lib.zsph_mlp_pack(x.data_ptr(), x.shape[0], None, None, tiles.data_ptr(), None))
    torch.cuda.synchronize()
    return tiles


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp_forward":
        net = z.Mlp(seed=1)
        net.params = _net(seed)
        n = case["rows"]
        return {"case": case, "net": net, "tiles": _pack(_rows(n, seed)), "n": n,
                "out": torch.zeros(n, 4, device=DEV)}
    if kind == "mlp_epoch":
        net = z.Mlp(seed=1)
        net.params = _net(seed)
        x, y, w, ids, m1, m2 = _train_set(case, seed)
        net.set_moments(m1, m2, 200)
        inv = [1.0 / max(float(w.view(-1, z.MLP_TILE)[b.long()].sum()), 1.0) for b in ids.split(case["batch_tiles"])]
        return {"case": case, "net": net, "tiles": _pack(x), "y": y, "w": w, "ids": ids, "inv": inv,
                "partial": torch.zeros(512, z.MLP_NPARTIAL, device=DEV)}
    if kind == "batch":
        sol = z.Solver.from_batch(_scenes(case))
        parts = [st for _, st in _batch_inputs(case, seed)]
        _load(sol, {k: torch.cat([p[k] for p in parts]) for k in _PTC})
    elif kind == "body":
        c = zc.floating_body(case["dx"])
        rng = np.random.default_rng(seed)
        fl = c.state.type == 1
        pos64 = c.pos64 + fl[:, None] * rng.uniform(-0.1, 0.1, (c.n, 3)) * case["dx"]
        c.state.pos = pos64.astype(np.float32)
        c.state.vel = (fl[:, None] * rng.uniform(-0.1, 0.1, (c.n, 3))).astype(np.float32)
        sol = z.Solver.from_case(c)
        sol.set_precision(True, pos64)
        sol.attach_body(c.body["first"], c.body["count"], c.body["mass"])
    else:
        gp, st = _inputs(case, seed)
        cp, _ = z.params_from_json(_geometry(case)[0].json)
        sol = z.Solver(gp, cp.grid_num)
        if kind == "simple":
            sol.set_equations(z.EQ_SIMPLE)
        _load(sol, st)
        if kind == "pairs":
            sol.neighbor_search("old", "new")
    torch.cuda.synchronize()
    if kind == "search":
        out = {**_ptc(sol, "new", list(_PTC)), **_tmp(sol, ("index", "hash", "grid_start", "grid_end"))}
    elif kind == "pairs":
        out = {**_ptc(sol, "new", ("rhop",)), **_tmp(sol, ("acc_drhodt", "dofv_grandrho"))}
    else:
        out = {**_ptc(sol, "old", ("pos", "vel", "rhop", "type", "table")),
               **_tmp(sol, ("acc_drhodt", "index", "hash"))}
    return {"case": case, "sol": sol, "out": out}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mlp_forward":
        z.check(z.lib.zsph_mlp_forward(state["net"].h, state["tiles"].data_ptr(), state["n"],
                                       state["out"].data_ptr(), None))
        return state["out"]
    if kind == "mlp_epoch":
        net, bt = state["net"], case["batch_tiles"]
        nparts = z.ctypes.c_int(0)
        for b in range(case["batches"]):
            z.check(z.lib.zsph_mlp_grad(net.h, state["tiles"].data_ptr(), state["y"].data_ptr(),
                                        state["w"].data_ptr(), state["ids"].data_ptr() + 4 * b * bt, bt,
                                        state["inv"][b], state["partial"].data_ptr(), z.ctypes.byref(nparts), None))
            z.check(z.lib.zsph_mlp_adam(net.h, state["partial"].data_ptr(), nparts.value, 1e-3, 0.9, 0.999, 1e-8,
                                        None))
        return net.params
    sol = state["sol"]
    if kind == "search":
        sol.neighbor_search("old", "new")
    elif kind == "pairs":
        sol.boundary("new")
        sol.governing("new")
    elif kind == "dropin":
        for src, dst, integrate in (("old", "new", sol.prediction), ("new", "old", sol.correction)):
            sol.hash(src)
            sol.sort_index()
            sol.sort_data(src, dst)
            sol.boundary(dst)
            sol.governing(dst)
            integrate(dst)
    elif kind == "reuse":
        sol.run_learned(None, 1, judge_every=0, corrector=z.CORR_REUSE_FRESH)
    elif kind == "step" and case["api"] == "step":
        sol.step()
    else:
        sol.run(1)
    return state["out"]


def _particles(case):
    kind = case["kind"]
    if kind == "batch":
        return [c.n for c in _scenes(case)]
    if kind == "body":
        dx = case["dx"]
        tx, ty, tz, layers = (int(round(v / dx)) for v in (4.0, 1.0, 1.0, 3 * dx))
        cube = int(round(0.2 / dx)) ** 3
        return [tx * ty * int(round(0.5 / dx)) + cube + (tx + 6) * (ty + 6) * (tz + layers) - tx * ty * tz]
    return [_geometry(case)[0].n]


def work(case):
    kind = case["kind"]
    if kind == "mlp_forward":
        # bf16 features in, four floats out; 2 * (32*128 + 128*128 + 128*4) operations a row
        return {"bytes": case["rows"] * (64 + 16) + 4 * z.MLP_NPARAM, "flops": case["rows"] * 41984}
    if kind == "mlp_epoch":
        rows = case["batches"] * case["batch_tiles"] * z.MLP_TILE
        return {"bytes": rows * (64 + 16 + 4) + 28 * z.MLP_NPARAM, "flops": 3 * rows * 41984}
    n = sum(_particles(case))
    if kind == "search":  # the state read and written, index and key written, cell bounds
        return {"bytes": n * (72 + 72 + 8), "flops": n * 9}
    if kind == "pairs":   # pos, vel, rhop, type and key read; two float4 results
        return {"bytes": n * (12 + 12 + 8 + 4 + 4 + 32), "flops": n * (50 * 54 + 76 * 68)}
    # a step: the state in and out once, accelerations, keys and index; per sub-step some
    # 50 boundary pairs of 54 and 76 governing pairs of 68 operations a particle
    pairs = 50 * 20 + 76 * 50 if kind == "simple" else 50 * 54 + 76 * 68
    return {"bytes": n * (72 + 72 + 16 + 8), "flops": 2 * n * pairs}


# ---- the same passes in 64 bits, in plain torch --------------------------------

class _Fp64:
    """delta-SPH / simple-SPH passes on a sorted state (delta_ns.cu, simple_ns.cu)."""

    CHUNK = 120000

    def __init__(self, gp):
        self.gp = gp
        self.c = {k: float(getattr(gp, k)) for k in ("half_dt", "h", "g", "m", "rho0", "adh", "h2", "eta2", "cs2",
                                                     "alpha", "delta_h_cs", "h_cs_rho_m")}
        self.gf = int(gp.grid_factor)

    def search(self, st):
        key = _cell(self.gp, st["pos"].float())
        key, perm = torch.sort(key, stable=True)
        new = {k: v[perm] for k, v in st.items()}
        n = key.numel()
        G = self.gp.grid_xdim * self.gp.grid_ydim * self.gp.grid_zdim
        lb = torch.searchsorted(key, torch.arange(G + 1, device=key.device))
        self.key, self.gs, self.ge = key, lb[:-1].clamp(max=n - 1), lb[1:].clamp(max=n - 1)
        self.G = G
        return new, perm

    def pairs(self, pos, lo, hi):
        """(i, j, boundary row) of the interacting pairs of particles lo..hi-1, in visit order."""
        X, XY, gf = self.gp.grid_xdim, self.gp.grid_xdim * self.gp.grid_ydim, self.gf
        i = torch.arange(lo, hi, device=DEV)
        c = self.key[lo:hi]
        S, E, B = [], [], []
        for dz in range(-gf, gf + 1):
            for dy in range(-gf, gf + 1):
                cell = c + dz * XY + dy * X
                ok = (cell - gf >= 0) & (cell + gf <= self.G - 1)
                S.append(self.gs[(cell - gf).clamp(0, self.G - 1)])
                E.append(torch.where(ok, self.ge[(cell + gf).clamp(0, self.G - 1)], S[-1]))
                B.append(dy < gf)
        S, E = torch.stack(S, 1), torch.stack(E, 1)
        B = torch.tensor(B, device=DEV)
        cnt = (E - S).clamp(min=0).reshape(-1)
        flat = torch.repeat_interleave(torch.arange(cnt.numel(), device=DEV), cnt)
        first = torch.cumsum(cnt, 0) - cnt
        j = S.reshape(-1)[flat] + torch.arange(flat.numel(), device=DEV) - first[flat]
        ii = i[torch.div(flat, B.numel(), rounding_mode="floor")]
        r2 = (pos[ii] - pos[j]).square().sum(1)
        keep = (r2.sqrt() / self.c["h"] <= 2.0) & (ii != j)
        return ii[keep], j[keep], B[flat[keep] % B.numel()]

    def _each(self, n):
        return [(a, min(a + self.CHUNK, n)) for a in range(0, n, self.CHUNK)]

    @staticmethod
    def _sum(n, lo, idx, v):
        return torch.zeros((n,) + v.shape[1:], dtype=torch.float64, device=DEV).index_add_(0, idx - lo, v)

    def walls(self, st, rhop):
        c, pos, fluid = self.c, st["pos"], st["type"] == 1
        new = rhop.clone()
        for lo, hi in self._each(pos.shape[0]):
            i, j, b = self.pairs(pos, lo, hi)
            k = b & ~fluid[i] & fluid[j]
            i, j = i[k], j[k]
            d = pos[i] - pos[j]
            q = d.square().sum(1).sqrt() / c["h"]
            w = (1 - q / 2) ** 4 * (2 * q + 1) * c["adh"]
            p = self._sum(hi - lo, lo, i, (rhop[j, 1] - rhop[j, 0] * (0.0 - c["g"]) * d[:, 2]) * w)
            ws = self._sum(hi - lo, lo, i, w)
            p = torch.where(ws.abs() > 1e-8, p / torch.where(ws == 0, 1.0, ws), 0.0).clamp(min=0.0)
            wall = ~fluid[lo:hi]
            new[lo:hi][wall] = torch.stack([p / c["cs2"] + c["rho0"], p], 1)[wall]
        return new

    def boundary(self, st, rhop_new):
        """grad(rho) renormalised and div(v): (n, 4); for simple equations (n,) div(v)."""
        c, pos, vel, fluid = self.c, st["pos"], st["vel"], st["type"] == 1
        out = torch.zeros(pos.shape[0], 4, dtype=torch.float64, device=DEV)
        for lo, hi in self._each(pos.shape[0]):
            i, j, b = self.pairs(pos, lo, hi)
            i, j = i[b], j[b]
            d = pos[i] - pos[j]
            q = d.square().sum(1).sqrt() / c["h"]
            rj = rhop_new[j, 0]
            t = -5 * c["adh"] / c["h2"] * (1 - q / 2) ** 3 * c["m"] / rj
            L = self._sum(hi - lo, lo, i, -(d[:, :, None] * d[:, None, :]) * t[:, None, None])
            s = self._sum(hi - lo, lo, i, d * (t * (rj - st["rhop"][i, 0]))[:, None])
            ff = (fluid[i] & fluid[j]).double()
            dv = self._sum(hi - lo, lo, i, -t * ff * ((vel[i] - vel[j]) * d).sum(1))
            xx, xy, xz, yy, yz, zz = L[:, 0, 0], L[:, 0, 1], L[:, 0, 2], L[:, 1, 1], L[:, 1, 2], L[:, 2, 2]
            det = (xx * yy * zz + xy * yz * xz + xz * xy * yz - xz * yy * xz - xx * yz * yz - xy * xy * zz)
            big = det.abs() > 1.8e-8
            idet = 1 / torch.where(big, det, 1.0)
            M = torch.stack([yy * zz - yz * yz, xz * yz - xy * zz, xy * yz - yy * xz,
                             xz * yz - xy * zz, xx * zz - xz * xz, xy * xz - xx * yz,
                             xy * yz - xz * yy, xz * xy - xx * yz, xx * yy - xy * xy], 1) * idet[:, None]
            M = torch.where(big[:, None, None], M.view(-1, 3, 3), torch.eye(3, dtype=torch.float64, device=DEV))
            out[lo:hi, :3] = (M @ s[:, :, None])[:, :, 0]
            out[lo:hi, 3] = dv
        return out

    def governing(self, st, rhop, dg):
        c, pos, vel, fluid = self.c, st["pos"], st["vel"], st["type"] == 1
        acc = torch.zeros(pos.shape[0], 4, dtype=torch.float64, device=DEV)
        for lo, hi in self._each(pos.shape[0]):
            n = hi - lo
            i, j, _ = self.pairs(pos, lo, hi)
            d = pos[i] - pos[j]
            r2 = d.square().sum(1)
            q = r2.sqrt() / c["h"]
            fr = -5 * c["adh"] / c["h2"] * (1 - q / 2) ** 3
            r0, r1 = rhop[i, 0], rhop[j, 0]
            dvdx = ((vel[i] - vel[j]) * d).sum(1)
            frm = fr * c["m"] / r1
            add = dg[j, 0] * d[:, 0] + (dg[i, 1] + dg[j, 1]) * d[:, 1] + (dg[i, 2] + dg[j, 2]) * d[:, 2]
            cnt = torch.bincount(i - lo, minlength=n)
            start = torch.cumsum(cnt, 0) - cnt
            g, gk = dg[lo:hi, 0].clone(), torch.zeros_like(add)
            for k in range(int(cnt.max()) if cnt.numel() else 0):  # delta_ns.cu:244-245 in visit order
                m = (cnt > k).nonzero()[:, 0]
                e = start[m] + k
                g[m] = g[m] * d[e, 0] + add[e]
                gk[e] = g[m]
            ff = (fluid[i] & fluid[j]).double()
            eta = r2 + c["eta2"]
            drho = r0 * dvdx * frm + ff * c["delta_h_cs"] * frm * ((r0 - r1) * 2 * r2 / eta - gk)
            vt = -(rhop[i, 1] + rhop[j, 1]) * frm / r0
            vt = vt + ff * c["h_cs_rho_m"] * fr * (dg[i, 3] + dg[j, 3] + c["alpha"] * dvdx / eta) / (r0 * r1)
            acc[lo:hi] = self._sum(n, lo, i, torch.cat([vt[:, None] * d, drho[:, None]], 1))
        acc[:, 2] += c["g"]
        return acc

    def simple(self, st, rhop):
        c, pos, vel, fluid = self.c, st["pos"], st["vel"], st["type"] == 1
        dv = torch.zeros(pos.shape[0], dtype=torch.float64, device=DEV)
        acc = torch.zeros(pos.shape[0], 4, dtype=torch.float64, device=DEV)
        for step in (0, 1):
            for lo, hi in self._each(pos.shape[0]):
                i, j, b = self.pairs(pos, lo, hi)
                if step == 0:
                    k = b & fluid[i] & fluid[j]
                    i, j = i[k], j[k]
                d = pos[i] - pos[j]
                r2 = d.square().sum(1)
                fr = -5 * c["adh"] / c["h2"] * (1 - r2.sqrt() / c["h"] / 2) ** 3
                dvdx = ((vel[i] - vel[j]) * d).sum(1)
                r0, r1 = rhop[i, 0], rhop[j, 0]
                if step == 0:
                    dv[lo:hi] = self._sum(hi - lo, lo, i, -fr * dvdx * c["m"] / r1)
                    continue
                eta = r2 + c["eta2"]
                drho = (r0 * dvdx * fr + (r0 - r1) * r2 * fr * c["delta_h_cs"] / eta) * c["m"] / r1
                vt = -(rhop[i, 1] + rhop[j, 1]) * c["m"] * fr / (r0 * r1)
                ff = (fluid[i] & fluid[j]).double()
                vt = vt + ff * c["h_cs_rho_m"] * fr * (dv[i] + dv[j] + c["alpha"] * dvdx / eta) / (r0 * r1)
                acc[lo:hi] = self._sum(hi - lo, lo, i, torch.cat([vt[:, None] * d, drho[:, None]], 1))
        acc[:, 2] += c["g"]
        return acc

    def integrate(self, st, rhop, acc, mode):
        hd, f = self.c["half_dt"], (st["type"] == 1)[:, None]
        new = dict(st)
        new["rhop"] = rhop
        if mode == 1:
            new["tmp_pos"], new["tmp_vel"], new["tmp_rhop"] = (torch.where(f, a, b) for a, b in (
                (st["pos"], st["tmp_pos"]), (st["vel"], st["tmp_vel"]), (rhop, st["tmp_rhop"])))
            pos, vel, rho = st["pos"] + st["vel"] * hd, st["vel"] + acc[:, :3] * hd, rhop[:, 0] + acc[:, 3] * hd
            pos = pos.float().double()  # the FP32 value that the next search hashes
        else:
            pos, vel, rho = (st["tmp_pos"] + st["vel"] * hd * 2, st["tmp_vel"] + acc[:, :3] * hd * 2,
                             st["tmp_rhop"][:, 0] + acc[:, 3] * hd * 2)
        rho = rho.clamp(min=self.c["rho0"])
        new["pos"], new["vel"] = torch.where(f, pos, st["pos"]), torch.where(f, vel, st["vel"])
        new["rhop"] = torch.where(f, torch.stack([rho, self.c["cs2"] * (rho - self.c["rho0"])], 1), rhop)
        return new

    def step(self, st, simple=False):
        for mode in (1, 2):
            st, _ = self.search(st)
            rhop = self.walls(st, st["rhop"])
            acc = self.simple(st, rhop) if simple else self.governing(st, rhop, self.boundary(st, rhop))
            st = self.integrate(st, rhop, acc, mode)
        return {"pos": st["pos"], "vel": st["vel"], "rhop": st["rhop"], "acc_drhodt": acc}


def _double(st):
    return {k: v.double() if v.is_floating_point() else v for k, v in st.items() if k != "table"}


def _mlp64(p, x):
    W1, b1, W2 = p[:4096].view(128, 32), p[4096:4224], p[4224:20608].view(128, 128)
    b2, W3, b3 = p[20608:20736], p[20736:21248].view(4, 128), p[21248:]
    silu = torch.nn.functional.silu
    return silu(silu(x @ W1.T + b1) @ W2.T + b2) @ W3.T + b3


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp_forward":
        p = torch.from_numpy(_net(seed)).to(DEV).double()
        return torch.cat([_mlp64(p, x.double()) for x in _rows(case["rows"], seed).split(100000)])
    if kind == "mlp_epoch":
        x, y, w, ids, m1, m2 = _train_set(case, seed)
        p, m1, m2 = (torch.from_numpy(a).to(DEV).double() for a in (_net(seed), m1, m2))
        T = z.MLP_TILE
        for k, b in enumerate(ids.split(case["batch_tiles"])):
            rows = (b.long()[:, None] * T + torch.arange(T, device=DEV)).reshape(-1)
            q = p.clone().requires_grad_(True)
            ws = max(float(w[rows].sum()), 1.0)
            loss = ((_mlp64(q, x[rows].double()) - y[rows].double()).square().sum(1) * w[rows].double()).sum() / ws
            g, = torch.autograd.grad(loss, q)
            t = 201 + k
            m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
            p = p - 1e-3 * (m1 / (1 - 0.9 ** t)) / ((m2 / (1 - 0.999 ** t)).sqrt() + 1e-8)
        return p
    if kind in ("body", "reuse"):  # couplings and approximations that only the framework defines
        return None
    if kind == "batch":
        parts = [_Fp64(gp).step(_double(st)) for gp, st in _batch_inputs(case, seed)]
        out = {k: torch.cat([p[k] for p in parts]) for k in parts[0]}
    else:
        gp, st = _inputs(case, seed)
        f, st = _Fp64(gp), _double(st)
        if kind == "search":
            new, _ = f.search(st)
            return {k: v if k not in ("type",) else None for k, v in new.items()}
        if kind == "pairs":
            new, _ = f.search(st)
            rhop = f.walls(new, new["rhop"])
            dg = f.boundary(new, rhop)
            return {"rhop": rhop, "acc_drhodt": f.governing(new, rhop, dg), "dofv_grandrho": dg}
        out = f.step(st, simple=kind == "simple")
    return out
