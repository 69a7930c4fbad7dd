"""Performance cases of the SNAC step: what programs that use this library spend their time on.

A case is one call pattern on one model:

  steps     n steps between two dumps: SnacContext.step(n), then the state into page-locked host arrays
  hooks     the loop-level hooks one by one, n steps, as a StGermain plugin host drives them, then the state
  host      one step of a state that the host keeps (SnacContext.step_host)
  ensemble  n batched steps of many small models (SnacBatch.step), then every model's state
  adjoint   misfit of the top surface after n steps and its gradients (snac_b200.adjoint)

The models are the workloads of snac_b200/workloads.py at their own and at odd sizes: elastic, Mohr-Coulomb
plastic and visco-plastic with temperature; dynamic, wave and constant dt; one phase and a phase per element;
regular and deformed meshes.  Inputs come from the seed: node positions or cohesion, the temperature anomaly,
initial velocities and the misfit's targets.

exact() evaluates the same formulas on whole arrays in torch, in 64 bits, without the library.
"""
import numpy as np
import torch
import torch.utils.checkpoint

from snac_b200 import workloads as W
from snac_b200.abi import State
from snac_b200.adjoint import adjoint
from snac_b200.batch import SnacBatch
from snac_b200.context import SnacContext


def _case(name, do, physics, nx, ny, nz, n, dt="dynamic", phases=1, yields=False, deformed=False):
    c = {"do": do, "physics": physics, "nx": nx, "ny": ny, "nz": nz, "n": n, "dt": dt, "phases": phases,
         "yields": yields, "deformed": deformed}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a first small run, a parameter study on one small box: launches and latency
        _case("steps_elastic_16x8x16", "steps", "elastic", 16, 8, 16, 20),
        # the size of the reference's own regression box, with its constant dt
        _case("steps_elastic_constant_12x10x10", "steps", "elastic", 12, 10, 10, 20, dt="constant", deformed=True),
        # the benchmark model
        _case("steps_plastic_64x32x64", "steps", "plastic", 64, 32, 64, 50),
        # a regional model in mid-life: two phases, a deformed mesh, yielding and softening tets, sizes that fill no tile
        _case("steps_plastic_phases_37x21x43", "steps", "plastic", 37, 21, 43, 20, phases=2, yields=True, deformed=True),
        # the largest model of the benchmark
        _case("steps_viscoplastic_128x64x128", "steps", "viscoplastic", 128, 64, 128, 20),
        # the same physics at an odd, ordinary size
        _case("steps_viscoplastic_47x23x39", "steps", "viscoplastic", 47, 23, 39, 20, deformed=True),
        # a parameter sweep over uneven small models, half of them plastic, half visco-plastic
        _case("ensemble_24_models", "ensemble", "mixed", 48, 24, 48, 16),
        # SNAC itself calling the hooks of its plugin
        _case("hooks_plastic_24x12x24", "hooks", "plastic", 24, 12, 24, 5),
        # a host that owns the state between steps: benchmark size, and an odd one with temperature
        _case("host_plastic_64x32x64", "host", "plastic", 64, 32, 64, 1),
        _case("host_viscoplastic_45x21x37", "host", "viscoplastic", 45, 21, 37, 1, deformed=True),
        # one iteration of an inversion, and a small one for a gradient check
        _case("adjoint_viscoplastic_32x16x32", "adjoint", "viscoplastic", 32, 16, 32, 60, dt="constant", deformed=True),
        _case("adjoint_viscoplastic_10x6x8", "adjoint", "viscoplastic", 10, 6, 8, 24, dt="constant", deformed=True),
    ]


def _mesh(rng, least, most):
    """Sides of a box of about least to most hexes, even over the logarithm, about half as high as wide."""
    e = least * (most / least) ** rng.random()
    x = (2.0 * e) ** (1.0 / 3.0)
    nx, nz = (max(3, round(x * rng.uniform(0.75, 1.3))) for _ in range(2))
    return nx, max(2, round(e / (nx * nz))), nz


def draw(rng):
    do = rng.choice(["steps"] * 5 + ["ensemble", "hooks", "host", "host", "adjoint"])
    deformed = rng.random() < 0.6
    if do == "ensemble":
        return _case(None, do, "mixed", rng.randint(24, 48), rng.randint(12, 24), rng.randint(24, 48), rng.randint(4, 16))
    if do == "adjoint":
        return _case(None, do, "viscoplastic", *_mesh(rng, 300, 17e3), rng.randint(8, 60), dt="constant", deformed=True)
    physics = rng.choice(["elastic", "plastic", "plastic", "viscoplastic", "viscoplastic"])
    dt = "dynamic" if physics == "viscoplastic" else rng.choice(["dynamic", "dynamic", "dynamic", "wave", "constant"])
    phases = 2 if physics != "elastic" and rng.random() < 0.35 else 1
    yields = physics == "plastic" and dt == "dynamic" and rng.random() < 0.4
    size = _mesh(rng, 1e3, {"steps": 6e5, "hooks": 6e4, "host": 3e5}[do])
    n = {"steps": rng.randint(5, 20), "hooks": rng.randint(1, 5), "host": 1}[do]
    return _case(None, do, physics, *size, n, dt, phases, yields, deformed)


# ---- the models -------------------------------------------------------------------------------------------

def _config(c, seed):
    """The model of a single-model case."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    if c["do"] == "adjoint":
        cfg = W.c5_adjoint(nx, ny, nz, seed=seed, extent=(3.1e3 * nx, 1.25e3 * ny, 3.1e3 * nz))
        cfg.element_cohesion_scale = 1.0 + W.smooth_field(nx, ny, nz, seed, 0.05)
        cfg.element_friction_scale = 1.0 + W.smooth_field(nx, ny, nz, seed + 1, 0.05)
        cfg.element_visc_scale = 1.0 + W.smooth_field(nx, ny, nz, seed + 2, 0.05)
    elif c["physics"] == "elastic":
        cfg = W.c1_elastic(nx, ny, nz)
    elif c["physics"] == "plastic":
        cfg = W.c2_plastic(nx, ny, nz, seed=seed, extent=(3.1e3 * nx, 1.25e3 * ny, 3.1e3 * nz))
    else:
        cfg = W.c3_viscoplastic(nx, ny, nz, seed=seed, extent=(3.1e3 * nx, 1.6e3 * ny, 3.1e3 * nz), sigma=5.0e3)
    if c["yields"]:  # weak rock under extension, no overburden: tets yield within a few steps
        cfg.gravity, cfg.hydrostatic_ic = 0.0, False
        cfg.materials = [W.mc_phase(c0=2.0e5, c1=2.0e4, eps1=0.001)]
    if c["phases"] == 2:
        m = dict(cfg.materials[0])
        m.update({k: 1.5 * m[k] for k in m if k.startswith("cohesion")}, density=2900.0, mu=2.5e10)
        cfg.materials = [cfg.materials[0], m]
        cfg.element_material = (rng.random(cfg.n_elements) < 0.5).astype(np.int32)
        cfg.element_cohesion_scale = None
    if c["dt"] != "dynamic" and c["do"] != "adjoint":
        cfg.dtType = c["dt"]
        cfg.timeStep = 2.0e7 if c["dt"] == "constant" else 0.0
    if c["deformed"]:  # every node off its place by up to 3 % of a cell
        x, jit = [], []
        for q, k in enumerate((nx, ny, nz)):
            x.append(cfg.min[q] + (cfg.max[q] - cfg.min[q]) * np.arange(k + 1) / k)
            jit.append(0.03 * (cfg.max[q] - cfg.min[q]) / k)
        Z, Y, X = np.meshgrid(x[2], x[1], x[0], indexing="ij")
        cfg.node_coords = (np.stack([X, Y, Z], -1).reshape(-1, 3) + np.array(jit) * rng.uniform(-1, 1, (cfg.n_nodes, 3))).reshape(-1)
    cfg.init_velocity = 1.0e-11 * rng.uniform(-1, 1, cfg.n_nodes * 3)
    return cfg


def _ensemble(c, seed):
    """24 models whose sizes come from the case and whose rocks come from the seed."""
    layout = c["nx"] + 100 * c["ny"] + 10000 * c["nz"]
    cfgs = W.c4_ensemble(24, seed=layout, xz=(8, min(c["nx"], c["nz"])), y=(4, c["ny"]))
    rng = np.random.default_rng(seed)
    for cfg in cfgs:
        f = rng.uniform(0.9, 1.1)
        cfg.materials[0].update({k: v * f for k, v in cfg.materials[0].items() if k.startswith("cohesion") or k == "refvisc"})
        cfg.init_velocity = 1.0e-11 * rng.uniform(-1, 1, cfg.n_nodes * 3)
    return cfgs


_SHAPES = {"coord": ("n", 3), "velocity": ("n", 3), "stress": ("e", 10, 6), "plastic_strain": ("e", 10),
           "viscosity": ("e", 10), "temperature": ("n",), "force": ("n", 3), "inertial_mass": ("n",)}


def _fields(cfg, do):
    f = ["coord", "velocity", "stress"]
    if cfg.plugin != "SnacElastic":
        f.append("plastic_strain")
    if cfg.temperature:
        f += ["viscosity", "temperature"]
    return f if do == "host" else f + ["force", "inertial_mass"]


def _host_states(cfgs, do):
    """Page-locked states, one per model, as slices of one array per field; and those arrays by field."""
    big, states = {}, [dict.fromkeys(_SHAPES) for _ in cfgs]
    for f, (per, *tail) in _SHAPES.items():
        n = [(c.n_nodes if per == "n" else c.n_elements) if f in _fields(c, do) else 0 for c in cfgs]
        if not any(n):
            continue
        big[f] = torch.zeros((sum(n), *tail), dtype=torch.float64, pin_memory=True).numpy()
        at = 0
        for s, k in zip(states, n):
            s[f] = big[f][at:at + k] if k else None
            at += k
    out = []
    for s in states:
        s = State(**s)
        s.plastic_strain_tensor = None
        out.append(s)
    return out, big


def prepare(case, seed):
    if case["do"] == "ensemble":
        cfgs = _ensemble(case, seed)
        b = SnacBatch(cfgs)
        b.time_step_zero()
        out, big = _host_states(cfgs, "ensemble")
        return {"do": "ensemble", "batch": b, "out": out, "big": big, "n": case["n"]}
    cfg = _config(case, seed)
    ctx = SnacContext(cfg)
    ctx.time_step_zero()
    s = {"do": case["do"], "ctx": ctx, "n": case["n"]}
    if case["do"] == "adjoint":
        (s["entry"],), s["big"] = _host_states([cfg], "host")
        ctx.state(s["entry"])
        s["targets"] = _targets(cfg, seed)
        return s
    (s["out"],), s["big"] = _host_states([cfg], case["do"])
    if case["do"] == "host":
        ctx.step(2)
        (s["in"],), s["big_in"] = _host_states([cfg], "host")
        ctx.state(s["in"])
        s["fields"] = _fields(cfg, "host")
    return s


def _targets(cfg, seed):
    rng = np.random.default_rng(seed)
    nt = (cfg.nx + 1) * (cfg.nz + 1)
    return 1.0e-10 * rng.uniform(-1, 1, nt), 50.0 * rng.uniform(-1, 1, nt)


def run(s):
    if s["do"] == "steps":
        s["ctx"].step(s["n"])
        s["ctx"].state(s["out"])
    elif s["do"] == "hooks":
        for _ in range(s["n"]):
            s["ctx"].solve()
        s["ctx"].state(s["out"])
    elif s["do"] == "host":
        s["ctx"].step_host(s["in"], s["out"], s["fields"], s["fields"])
    elif s["do"] == "ensemble":
        s["batch"].step(s["n"])
        for m, o in zip(s["batch"].models, s["out"]):
            m.state(o)
    else:  # every iteration of an inversion starts from the same entry state
        s["ctx"].set_state(s["entry"], ["coord", "velocity", "stress", "plastic_strain", "temperature"])
        r = adjoint(s["ctx"], s["n"], *s["targets"], w_v=1.0e22, w_h=1.0, state=True)
        return {"loss": r.loss, **r.grad}
    return s["big"]


# what one hex-step needs: its persistent state read once and written once, and the operations of its ten
# tets' formulas (geometry, strain rate, rotation, update, force terms), each divide or root counted as one
_FLOPS_PER_TET = {"elastic": 430, "plastic": 480, "viscoplastic": 640, "mixed": 560}


def work(case):
    do, physics = case["do"], case["physics"]
    if do == "ensemble":
        cfgs = _ensemble(case, 1)
    else:
        cfgs = [None]
    total = {"bytes": 0.0, "flops": 0.0}
    for cfg in cfgs:
        nx, ny, nz = (cfg.nx, cfg.ny, cfg.nz) if cfg else (case["nx"], case["ny"], case["nz"])
        kind = physics if cfg is None else "viscoplastic" if cfg.temperature else "plastic"
        ne, nn = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
        state = 480 * ne + 48 * nn + (80 * ne if kind != "elastic" else 0) + (80 * ne + 8 * nn if kind == "viscoplastic" else 0)
        step = 2 * state
        flops = 10 * ne * _FLOPS_PER_TET[kind] + nn * (200 + (100 if kind == "viscoplastic" else 0))
        if do == "adjoint":  # the steps, then their reverse: the state and its adjoint, about three times the operations
            total["bytes"] += case["n"] * 3 * step
            total["flops"] += case["n"] * 4 * flops
        else:
            total["bytes"] += case["n"] * step + (0 if do == "host" else state + 32 * nn)
            total["flops"] += case["n"] * flops
    return total


# ---- the same formulas on whole arrays --------------------------------------------------------------------

_TET = [[7, 2, 3, 0], [0, 5, 4, 7], [2, 5, 1, 0], [5, 2, 6, 7], [2, 5, 0, 7],
        [3, 4, 7, 6], [4, 3, 0, 1], [6, 1, 2, 3], [1, 6, 5, 4], [1, 3, 6, 4]]
_FACE = [[0, 1, 2], [1, 3, 2], [0, 2, 3], [3, 1, 0]]
_CORNER = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
_WALL_FACES = [[(0, 2), (1, 2), (5, 0), (6, 0)], [(2, 0), (3, 0), (7, 0), (8, 0)],
               [(0, 1), (2, 2), (6, 1), (7, 1)], [(1, 1), (3, 2), (5, 1), (8, 1)]]
_F32 = lambda x: float(np.float32(x))  # noqa: E731


def _sym(s):
    """[..., 6] (xx, yy, zz, xy, xz, yz) as matrices."""
    return torch.stack([s[..., 0], s[..., 3], s[..., 4], s[..., 3], s[..., 1], s[..., 5], s[..., 4], s[..., 5],
                        s[..., 2]], -1).reshape(*s.shape[:-1], 3, 3)


class _Plain:
    """One model.  Stress is [hex, tet, 6]; x, v are [node, 3]; scales may require gradients."""

    def __init__(self, cfg):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.cfg, self.dev = cfg, dev
        nx, ny, nz = cfg.nx, cfg.ny, cfg.nz
        self.t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        k, j, i = torch.meshgrid(torch.arange(nz), torch.arange(ny), torch.arange(nx), indexing="ij")
        self.i, self.k = i.reshape(-1).to(dev), k.reshape(-1).to(dev)
        node = lambda a, b, c: a + b * (nx + 1) + c * (nx + 1) * (ny + 1)  # noqa: E731
        hexes = torch.stack([node(i + d[0], j + d[1], k + d[2]).reshape(-1) for d in _CORNER], -1)
        self.tets = hexes[:, torch.tensor(_TET)].to(dev)  # [hex, tet, corner]
        nk, nj, ni = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
        ijk = [a.reshape(-1) for a in (ni, nj, nk)]
        self.top = self.t(np.flatnonzero(ijk[1] == ny))
        ne, nn = cfg.n_elements, cfg.n_nodes
        if cfg.node_coords is not None:
            x = cfg.node_coords.reshape(nn, 3)
        else:
            x = np.stack([cfg.min[q] + (cfg.max[q] - cfg.min[q]) * (ijk[q] / (nx, ny, nz)[q]) for q in range(3)], -1)
        self.x = self.t(x)
        walls = {"left": ijk[0] == 0, "right": ijk[0] == nx, "bottom": ijk[1] == 0, "top": ijk[1] == ny,
                 "back": ijk[2] == 0, "front": ijk[2] == nz}
        fix, val = np.zeros((nn, 3), bool), np.zeros((nn, 3))
        for bc in cfg.velocityBCs:
            for q, key in enumerate(("vx", "vy", "vz")):
                if key in bc:
                    fix[walls[bc["wall"]], q], val[walls[bc["wall"]], q] = True, bc[key]
        self.fix, self.val = self.t(fix), self.t(val)
        v = np.zeros((nn, 3)) if cfg.init_velocity is None else cfg.init_velocity.reshape(nn, 3)
        self.v = torch.where(self.fix, self.val, self.t(v))
        self.T = None
        if cfg.temperature:
            tf, tv = np.zeros(nn, bool), np.zeros(nn)
            for bc in cfg.temperatureBCs:
                tf[walls[bc["wall"]]], tv[walls[bc["wall"]]] = True, bc["T"]
            self.tfix, self.tval = self.t(tf), self.t(tv)
            self.T = torch.where(self.tfix, self.tval, self.t(cfg.init_temperature))
        ph = np.zeros(ne, np.int64) if cfg.element_material is None else cfg.element_material.astype(np.int64)
        self.m = lambda key: self.t(np.array([m[key] for m in cfg.materials])[ph][:, None])  # [hex, 1]
        self.rho, self.lam, self.mu = self.m("density"), self.m("lambda"), self.m("mu")
        one = lambda a: self.t(np.ones((ne, 1)) if a is None else np.asarray(a).reshape(ne, 1))  # noqa: E731
        self.scale = {"cohesion": one(cfg.element_cohesion_scale), "friction": one(cfg.element_friction_scale),
                      "viscosity": one(cfg.element_visc_scale)}
        self.s = torch.zeros(ne, 10, 6, dtype=torch.float64, device=dev)
        if cfg.hydrostatic_ic:
            self.s[..., :3] = self.t(self._lithostatic(x, ph))[:, None, None]
        self.eps = torch.zeros(ne, 10, dtype=torch.float64, device=dev)
        self.dt = float(cfg.timeStep)
        if cfg.temperature:
            self.visc = self.m("vis_min").expand(ne, 10).clone()
            most = min(0.9 * m["vis_min"] / m["mu"] for m in cfg.materials)
            if cfg.dtType != "constant":
                self.dt = min(self.dt, most)
        g = self._geometry(self.x)
        self.s = self._rotate(self.s, self.v, g)
        self._sync(g)

    def _lithostatic(self, x, ph):
        cfg = self.cfg
        nx, ny, nz = cfg.nx, cfg.ny, cfg.nz
        y = x[:, 1].reshape(nz + 1, ny + 1, nx + 1)
        rho = np.array([m["density"] for m in cfg.materials])[ph].reshape(nz, ny, nx)
        up, lo = y[:, 1:], y[:, :-1]
        mean4 = lambda a: 0.25 * (a[:-1, :, :-1] + a[:-1, :, 1:] + a[1:, :, :-1] + a[1:, :, 1:])  # noqa: E731
        d = rho * cfg.gravity * (mean4(up) - mean4(lo))
        above = np.flip(np.cumsum(np.flip(d, 1), 1), 1) - d
        return -(above + 0.5 * d).reshape(-1)

    def _geometry(self, x):
        c = x[self.tets]
        d = [c[..., q, :] - c[..., 0, :] for q in (1, 2, 3)]
        V = (torch.linalg.cross(d[0], d[1]) * d[2]).sum(-1).abs() / 6.0
        w = [0.5 * torch.linalg.cross(c[..., f[1], :] - c[..., f[0], :], c[..., f[2], :] - c[..., f[0], :]) for f in _FACE]
        return V, w  # volume; area vector of each face (node q goes with face q + 1)

    def _sums(self, v, w):
        """S[..., a, b] = sum over nodes of v_a w_b."""
        c = v[self.tets]
        return sum(c[..., q, :, None] * w[(q + 1) % 4][..., None, :] for q in range(4))

    def _rotate(self, s, v, g):
        V, w = g
        S = self._sums(v, w)
        r01, r02, r12 = (-(S[..., a, b] - S[..., b, a]) / (6.0 * V) for a, b in ((0, 1), (0, 2), (1, 2)))
        dt = self.dt
        xx, yy, zz, xy, xz, yz = s.unbind(-1)
        xx = xx + (2 * r01 * xy + 2 * r02 * xz) * dt
        yy = yy + (-2 * r01 * xy + 2 * r12 * yz) * dt
        zz = zz + (-2 * r02 * xz - 2 * r12 * yz) * dt
        xy = xy + r01 * (yy - xx) * dt + (r02 * yz + r12 * xz) * dt
        xz = xz + r02 * (zz - xx) * dt + (r01 * yz - r12 * xy) * dt
        yz = yz + r12 * (zz - yy) * dt + (-r01 * xz - r02 * xy) * dt
        return torch.stack([xx, yy, zz, xy, xz, yz], -1)

    def _sync(self, g):
        cfg = self.cfg
        if cfg.dtType == "constant":
            return
        V, w = g
        least = min(float((V / f.norm(dim=-1)).min()) for f in w)
        if cfg.dtType == "wave":
            self.dt = 0.5 * least / float(((self.lam + 2 * self.mu) / self.rho).sqrt().max())
            return
        vmax = max(float(self.v[self.fix.any(1)].norm(dim=1).max()), 3.0e-11)
        self.dt = least * _F32(0.45) * cfg.strain_inert / vmax
        self.sos = least * 0.5 / self.dt

    def _heat(self, g):
        V, w = g
        T = self.T[self.tets]
        n = torch.stack([f / f.norm(dim=-1, keepdim=True) for f in w], -2)  # [hex, tet, face, 3]
        grad = sum(T[..., q, None] * w[(q + 1) % 4] for q in range(4)) / (3.0 * V[..., None])
        q = self.m("thermal_conduct")[..., None] * grad
        nx, nz = self.cfg.nx, self.cfg.nz
        normal, wall = torch.zeros_like(grad[:, 0]), torch.zeros_like(self.i, dtype=torch.bool)
        for side, faces in zip((self.i == 0, self.i == nx - 1, self.k == 0, self.k == nz - 1), _WALL_FACES):
            mean = 0.25 * sum(n[:, t, f] for t, f in faces)
            normal, wall = torch.where(side[:, None], mean, normal), wall | side
        normal = normal[:, None]
        q = torch.where(wall[:, None, None], q + (grad * normal).sum(-1, keepdim=True) * normal, q)
        energy, lump = torch.zeros_like(self.T), torch.zeros_like(self.T)
        cap = self.m("heatCapacity") * self.rho * V * 0.125
        for c in range(4):
            energy.index_add_(0, self.tets[..., c].reshape(-1), ((q * w[(c + 1) % 4]).sum(-1) / 6.0).reshape(-1))
            lump.index_add_(0, self.tets[..., c].reshape(-1), cap.reshape(-1))
        T = self.T - energy * self.dt / lump
        self.T = torch.where(self.tfix, self.tval, T)

    def _averaged(self, s, V):
        tr = (s[..., 0] + s[..., 1] + s[..., 2]) / 3.0
        add = (tr * V).sum(1, keepdim=True) / V.sum(1, keepdim=True) - tr
        return torch.cat([s[..., :3] + add[..., None], s[..., 3:]], -1)

    def _viscous(self, s, e):
        tr_e, p = e[..., :3].sum(-1, keepdim=True), s[..., :3].sum(-1, keepdim=True) / 3.0
        ed, sd = e[..., :3] - tr_e / 3.0, s[..., :3] - p
        Q = ed[..., 1] * ed[..., 2] + ed[..., 2] * ed[..., 0] + ed[..., 0] * ed[..., 1]
        J = Q.abs().sqrt() / self.dt
        J = torch.where(J == 0, self.m("refsrate").expand_as(J), J)
        T = self.T[self.tets].mean(-1)
        eta = self.m("refvisc") * self.scale["viscosity"] * (J / self.m("refsrate")) ** (1.0 / self.m("srexponent") - 1.0) * torch.exp(
            self.m("activationE") / 8.31448 * (1.0 / (T + 273.15) - 1.0 / (self.m("reftemp") + 273.15)))
        eta = torch.minimum(torch.maximum(eta, self.m("vis_min")), self.m("vis_max"))
        self.visc = eta
        tmp = (self.mu / (2.0 * eta) * self.dt)[..., None]
        mu2 = (2.0 * self.mu)[..., None]
        bulk = (self.lam + 2.0 * self.mu / 3.0)[..., None]
        sd = (sd * (1 - tmp) + mu2 * ed) / (1 + tmp)
        shear = (s[..., 3:] * (1 - tmp) + mu2 * e[..., 3:]) / (1 + tmp)
        return torch.cat([sd + p + bulk * tr_e, shear], -1)

    def _table(self, key, scale):
        """The piecewise-linear table at the plastic strain, and its slope."""
        nseg = self.cfg.materials[0]["nsegments"]
        val, slope = 0.0, 0.0
        for a in range(nseg):
            e0, e1 = self.m("plstrain%d" % a), self.m("plstrain%d" % (a + 1))
            f0, f1 = scale * self.m("%s%d" % (key, a)), scale * self.m("%s%d" % (key, a + 1))
            inside, past = (self.eps >= e0) & (self.eps <= e1), self.eps > e1
            k = (f1 - f0) / (e1 - e0)
            val = torch.where(inside, f0 + k * (self.eps - e0), torch.where(past, f1, val))
            slope = torch.where(inside, k, torch.where(past, torch.zeros_like(k), slope))
        return val, slope

    def _return_map(self, s):
        co, hard = self._table("cohesion", self.scale["cohesion"])
        fr, _ = self._table("frictionAngle", self.scale["friction"])
        di, _ = self._table("dilationAngle", 1.0)
        rad = np.pi / 180.0
        anphi = (1 + torch.sin(fr * rad)) / (1 - torch.sin(fr * rad))
        anpsi = (1 + torch.sin(di * rad)) / (1 - torch.sin(di * rad))
        cut = torch.minimum(co / torch.tan(fr * rad), self.m("ten_off"))
        with torch.no_grad():  # tets whose principal stresses (Gershgorin's bounds) may reach a yield surface
            r = torch.stack([s[..., 3].abs() + s[..., 4].abs(), s[..., 3].abs() + s[..., 5].abs(), s[..., 4].abs() + s[..., 5].abs()], -1)
            hi, lo = (s[..., :3] + r).amax(-1), (s[..., :3] - r).amin(-1)
            tol = 1e-9 * (s[..., :3].abs().sum(-1) + 2 * r.sum(-1)) * (1 + anphi)
            at = ~((hi - cut < -tol) & (lo - hi * anphi + 2 * co * anphi.sqrt() > tol))
        if not bool(at.any()):
            return s
        pick = lambda a: a.expand_as(at)[at]  # noqa: E731
        co, hard, anphi, anpsi, cut = (pick(a) for a in (co, hard, anphi, anpsi, cut))
        a1, a2 = pick(self.lam + 2 * self.mu), pick(self.lam)
        M = _sym(s[at])
        p, vec = [torch.cat(a) for a in zip(*(torch.linalg.eigh(b) for b in M.split(1 << 19)))]  # ascending
        fs, ft = p[:, 0] - p[:, 2] * anphi + 2 * co * anphi.sqrt(), p[:, 2] - cut
        yielding = (fs < 0) | (ft > 0)
        aP = (1 + anphi * anphi).sqrt() + anphi
        shear = p[:, 2] - cut + aP * (p[:, 0] - (cut * anphi - 2 * co * anphi.sqrt())) < 0
        al = fs / (a1 - a2 * anpsi + a1 * anphi * anpsi - a2 * anphi + 2 * anphi.sqrt() * hard)
        al_t = ft / a1
        zero = torch.zeros_like(al)
        ps = p - torch.stack([al * (a1 - a2 * anpsi), al * a2 * (1 - anpsi), al * (a2 - a1 * anpsi)], -1)
        pt = p - torch.stack([al_t * a2, al_t * a2, al_t * a1], -1)
        q = torch.where(shear[:, None], ps, pt)
        dep = torch.where(shear[:, None], torch.stack([al, zero, -al * anpsi], -1), torch.stack([zero, zero, al_t], -1))
        dm = dep.sum(-1) / 3.0
        grown = (0.5 * (((dep - dm[:, None]) ** 2).sum(-1) + dm * dm)).sqrt()
        R = vec @ (q[:, :, None] * vec.transpose(1, 2))
        new = torch.stack([R[:, 0, 0], R[:, 1, 1], R[:, 2, 2], R[:, 0, 1], R[:, 0, 2], R[:, 1, 2]], -1)
        where = at.nonzero(as_tuple=True)
        where = tuple(a[yielding] for a in where)
        self.eps = self.eps.index_put(where, grown[yielding], accumulate=True)
        return s.index_put(where, new[yielding])

    def step(self):
        cfg, dt = self.cfg, self.dt
        g = V, w = self._geometry(self.x)
        if cfg.temperature and any(m["thermal_conduct"] for m in cfg.materials):
            self._heat(g)
        S = self._sums(self.v, w)
        sr = torch.stack([-S[..., a, a] / (3 * V) for a in range(3)] + [-(S[..., a, b] + S[..., b, a]) / (6 * V) for a, b in ((0, 1), (0, 2), (1, 2))], -1)
        del S
        e = self._averaged(sr, V) * dt
        if cfg.temperature:
            s = self._viscous(self.s, e)
        else:
            tr = (self.lam * e[..., :3].sum(-1))[..., None]
            s = self.s + (2 * self.mu)[..., None] * e + torch.cat([tr.expand(*e.shape[:-1], 3), torch.zeros_like(e[..., 3:])], -1)
        if cfg.plugin != "SnacElastic":
            s = self._return_map(s)
        s = self._averaged(s, V)
        F, mass = torch.zeros_like(self.x), torch.zeros_like(self.x[:, 0])
        M = _sym(s)
        for c in range(4):
            f = w[(c + 1) % 4]
            t = (M @ f[..., None])[..., 0] / 6.0
            t[..., 1] -= cfg.gravity * self.rho * V / 8.0
            if cfg.dtType == "constant":
                im = (self.lam + 2 * self.mu) * (f * f).amax(-1) / (9 * V) * (dt * dt)
            elif cfg.dtType == "wave":
                im = 0.25 * self.rho * V
            else:
                im = 0.25 * (self.lam + 2 * self.mu) / self.sos ** 2 * V
            at = self.tets[..., c].reshape(-1)
            F = F.index_add(0, at, t.reshape(-1, 3))
            mass = mass.index_add(0, at, im.reshape(-1))
        F = F - cfg.demf * torch.sign(self.v) * F.abs()
        self.v = torch.where(self.fix, self.val, self.v + dt * F / mass[:, None])
        self.x = self.x + dt * self.v
        self.F, self.mass, self.s = F, mass, s
        g = self._geometry(self.x)
        self.s = self._rotate(self.s, self.v, g)
        self._sync(g)

    def state(self, do):
        out = {"coord": self.x, "velocity": self.v, "stress": self.s}
        if self.cfg.plugin != "SnacElastic":
            out["plastic_strain"] = self.eps
        if self.cfg.temperature:
            out.update(viscosity=self.visc, temperature=self.T)
        if do != "host":
            out.update(force=self.F, inertial_mass=self.mass)
        return out


def _exact_adjoint(case, seed):
    cfg = _config(case, seed)
    vy, y = _targets(cfg, seed)
    m = _Plain(cfg)
    entry = {"cohesion": m.scale["cohesion"], "friction": m.scale["friction"], "viscosity": m.scale["viscosity"],
             "coordinates": m.x, "velocity": m.v, "stress": m.s, "plastic_strain": m.eps}
    leaf = {k: a.clone().requires_grad_(True) for k, a in entry.items()}
    m.scale = {k: leaf[k] for k in ("cohesion", "friction", "viscosity")}
    m.x, m.v, m.s, m.eps = (leaf[k] for k in ("coordinates", "velocity", "stress", "plastic_strain"))

    def one(x, v, s, eps, *scales):
        m.scale = dict(zip(("cohesion", "friction", "viscosity"), scales))
        m.x, m.v, m.s, m.eps = x, v, s, eps
        m.step()
        return m.x, m.v, m.s, m.eps

    st = (m.x, m.v, m.s, m.eps)
    scales = tuple(leaf[k] for k in ("cohesion", "friction", "viscosity"))
    for _ in range(case["n"]):
        st = torch.utils.checkpoint.checkpoint(one, *st, *scales, use_reentrant=False)
    x, v = st[0], st[1]
    loss = 1.0e22 * ((v[m.top, 1] - m.t(vy)) ** 2).sum() + ((x[m.top, 1] - m.t(y)) ** 2).sum()
    grads = torch.autograd.grad(loss, list(leaf.values()), allow_unused=True)
    out = {"loss": float(loss)}
    for (k, a), gr in zip(leaf.items(), grads):
        gr = torch.zeros_like(a) if gr is None else gr
        out[k] = gr.reshape(-1) if k in ("cohesion", "friction", "viscosity", "plastic_strain") else gr.reshape(-1, a.shape[-1])
    return out


def exact(case, seed):
    if case["do"] == "adjoint":
        return _exact_adjoint(case, seed)
    with torch.no_grad():
        cfgs = _ensemble(case, seed) if case["do"] == "ensemble" else [_config(case, seed)]
        states = []
        for cfg in cfgs:
            m = _Plain(cfg)
            for _ in range(case["n"] + (2 if case["do"] == "host" else 0)):
                m.step()
            states.append(m.state(case["do"]))
        return {f: torch.cat([s[f] for s in states if f in s]) for f in _SHAPES if any(f in s for s in states)}
