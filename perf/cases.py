"""Performance cases of the peridynamics engine, through its public entry points.

A case is one call, or one short run of steps, of the work that users have the
engine do:

  force     one bond-force evaluation between torch code (operator by operator
            use, as the reference's host launchers are used)
  verlet    explicit velocity-Verlet steps of a 2-D bond-based plate
  adr       quasi-static ADR steps of a 2-D bond-based plate with moving rows
  state2d   explicit steps of a 2-D state-based plate with moving rows
  slab      explicit steps of the notched 3-D slab under the rigid impactor,
            bond-based or state-based
  batch     ADR steps of many uneven plates in one context
  setup     family, corrections, pre-crack and force layout of a new specimen,
            up to its first force evaluation
  gradient  forward and backward pass of the warm start's network
  predict   one prediction of the learned warm start

Sizes, materials, loads and time steps are those of ``pd_gpu1_gb300.presets``
and of the reference's drivers.  ``exact`` evaluates the same model in plain
torch in 64 bits, with the extension of a bond formed from the displacement
difference, (2 xi.eta + eta.eta) / (L + L0), so that it has no cancellation.
"""
import ctypes as C
import math

import numpy as np
import torch

from pd_gpu1_gb300 import presets
from pd_gpu1_gb300._abi import PD_MODE_DYNAMIC, PD_MODE_STATIC, PD_MODEL_BOND, PD_MODEL_STATE, PDCylinder
from pd_gpu1_gb300._lib import check, lib
from pd_gpu1_gb300.engine import Batch, Engine, coord_kw, derive_params
from pd_gpu1_gb300.warm import N_PARAMS, WEIGHTS, Net, init_params, record_history

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
HORIZON = 3.015  # horizon over lattice spacing, as the reference fixes it
WARM_INC = 5e-7  # boundary displacement per load increment of the warm-start plate


def listed():
    return [
        # the smallest call: a force evaluation of the 100 x 100 tensile plate
        dict(name="force_10k", kind="force", nx=100, ny=100),
        # the reference's tensile driver: its 100 x 100 plate, a stretch of its 1000 ADR steps
        dict(name="adr_10k", kind="adr", nx=100, ny=100, dx=5e-4, steps=20),
        # a parameter study's crack-branching plate, odd sizes, bonds breaking, damage at the end
        dict(name="verlet_69k", kind="verlet", nx=413, ny=167, steps=40, crack=False),
        # the crack-branching benchmark at full size
        dict(name="verlet_1600k", kind="verlet", nx=2000, ny=800, steps=20, crack=True),
        # an increment of the quasi-static crack-growth plate at full size
        dict(name="adr_1000k", kind="adr", nx=1000, ny=1000, dx=1e-4, steps=12),
        # the reference's crack-grow driver: 500 x 500 state-based plate
        dict(name="state2d_253k", kind="state2d", nx=500, ny=500, steps=20),
        # the impact slab with each material model
        dict(name="slab_state_181k", kind="slab", state=True, scale=1.0, steps=10),
        dict(name="slab_bond_181k", kind="slab", state=False, scale=1.0, steps=10),
        # a batch of uneven plates (a quarter of the 256-plate benchmark)
        dict(name="batch_64", kind="batch", count=64, low=50, high=300, steps=12),
        # a new 500 x 500 bond-based specimen, up to its first force
        dict(name="setup_250k", kind="setup", nx=500, ny=500),
        # a training batch of the warm start's network
        dict(name="gradient_16k", kind="gradient", rows=16384),
        # the prediction of one increment on the full-size plate
        dict(name="predict_1000k", kind="predict", nx=1000, ny=1000, smooth=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["force", "adr", "verlet", "state2d", "slab", "batch", "setup", "gradient", "predict"])
    if kind == "gradient":
        return dict(kind=kind, rows=_log(rng, 1000, 65536))
    if kind == "slab":
        return dict(kind=kind, state=rng.random() < 0.5, scale=round(rng.uniform(0.3, 1.0), 3),
                    steps=rng.randint(4, 10))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 64), low=rng.randint(20, 80), high=rng.randint(100, 300),
                    steps=rng.randint(5, 12))
    top = {"force": 1600, "adr": 1000, "verlet": 1400, "state2d": 700, "setup": 700, "predict": 1000}[kind]
    nx, ny = _log(rng, 40, top), _log(rng, 40, top)
    if kind in ("force", "setup"):
        return dict(kind=kind, nx=nx, ny=ny)
    if kind == "predict":
        return dict(kind=kind, nx=nx, ny=ny, smooth=rng.randint(0, 16))
    if kind == "adr":
        return dict(kind=kind, nx=nx, ny=ny, dx=rng.choice([1e-4, 2.5e-4, 5e-4]), steps=rng.randint(5, 12))
    steps = rng.randint(8, 20)
    if kind == "verlet":
        return dict(kind=kind, nx=nx, ny=ny, steps=steps, crack=rng.random() < 0.5)
    return dict(kind=kind, nx=nx, ny=ny, steps=steps)


# ---- materials -------------------------------------------------------------------
def _material(c):
    """dx, dt, E, nu, rho, s0 and the row speed of a case's specimen."""
    k = c["kind"]
    if k in ("verlet", "setup"):  # presets.build_crack_branching
        dx, E = 5e-5, 72.0e9
        return dict(dx=dx, dt=1.0e-8, E=E, nu=1.0 / 3.0, rho=2440.0, s0=presets.s0_2d(3.8, E, HORIZON * dx), load=0.0)
    if k == "state2d":  # presets.build_crack_grow
        return dict(dx=1e-4, dt=1.3367e-8, E=192.0e9, nu=0.3, rho=7850.0, s0=0.04472, load=20.0)
    if k == "slab":  # presets.build_kalthoff_winkler
        dx, E, nu = 1e-3, 190.0e9, 0.25
        return dict(dx=dx, dt=1.0e-7, E=E, nu=nu, rho=8000.0, s0=presets.s0_3d(22170.0, E, nu, HORIZON * dx), load=0.0)
    dx = c.get("dx", 1e-4 if k == "predict" else 5e-4)  # presets.build_plate_tensile / build_warm_start_plate
    s0 = presets.s0_2d(2.65e3, 192.0e9, HORIZON * 1e-4) if k == "predict" else 0.04472
    return dict(dx=dx, dt=1.0, E=192.0e9, nu=1.0 / 3.0, rho=8000.0, s0=s0, load=2.7e-8)


def _crack(c):
    """(length, x, y, angle) of a plate's pre-crack, None without one."""
    m = _material(c)
    L = c["nx"] * m["dx"]
    if c["kind"] == "setup" or (c["kind"] == "verlet" and c["crack"]):
        return L / 2.0, -L / 4.0, 0.0, 0.0  # from the left edge to the middle
    if c["kind"] == "state2d":
        return L / 5.0, 0.0, 0.0, 0.0  # centred
    if c["kind"] == "predict":
        return L / 5.0, -L / 2.0 + L / 10.0, 0.0, 0.0  # edge crack
    return None


def _rows(c):
    """Whether the plate has the three moving rows above and below."""
    return c["kind"] in ("adr", "state2d", "predict", "force")


def _params(c):
    m = _material(c)
    state = c["kind"] == "state2d"
    mode = PD_MODE_STATIC if c["kind"] in ("adr", "force", "predict") else PD_MODE_DYNAMIC
    dx, nx, ny = m["dx"], c["nx"], c["ny"]
    p = derive_params(2, PD_MODEL_STATE if state else PD_MODEL_BOND, mode, m["dt"], 1000, dx, 0.0, dx, nx * dx, ny * dx,
                      0.0, m["E"], m["nu"], m["rho"], m["s0"])
    p.nx, p.ny, p.N_int = nx, ny, nx * ny
    p.N = p.N_int + (6 * nx if _rows(c) else 0)
    return p


# ---- inputs ----------------------------------------------------------------------
def _smooth(rng, coords, size, strain, base):
    """A smooth displacement component field per coordinate: a uniform strain
    (base) and six waves between the specimen's size and an eighth of it."""
    out = []
    for a in range(len(coords)):
        u = float(rng.uniform(0.5, 1.0)) * base[a] * coords[a]
        for _ in range(6):
            k = [2.0 * math.pi / size * float(rng.uniform(-8.0, 8.0)) for _ in coords]
            arg = float(rng.uniform(0.0, 2.0 * math.pi)) + sum(ki * x for ki, x in zip(k, coords))
            norm = max(math.sqrt(sum(ki * ki for ki in k)), 2.0 * math.pi / size)
            u = u + strain * float(rng.uniform(-1.0, 1.0)) / (3.0 * norm) * torch.cos(arg)
        out.append(u)
    return out


def _fields(c, seed, coords, rows=None):
    """Initial displacement and velocity (lists per component) of a run; rows:
    a mask of the prescribed nodes of an ADR run."""
    rng = np.random.default_rng(seed)
    size = max(float(x.max() - x.min()) for x in coords)
    dim = len(coords)
    k = c["kind"]
    if k in ("verlet", "setup"):
        # tension across the crack line; without a pre-crack the waves take some bonds past s0 = 7e-4
        free = k == "verlet" and not c["crack"]
        u = _smooth(rng, coords, size, 6e-4 if free else 5e-5, (0.0, 4e-4 if free else 8e-5))
        v = _smooth(rng, coords, size, 0.0 if k == "setup" else 40.0, (0.0, 0.0))
    elif k == "state2d":
        u = _smooth(rng, coords, size, 3e-4, (0.0, 1e-3))
        v = _smooth(rng, coords, size, 60.0, (0.0, 400.0))
    elif k == "slab":
        u = _smooth(rng, coords, size, 2e-4, (0.0,) * dim)
        v = _smooth(rng, coords, size, 20.0, (0.0,) * dim)
    else:
        u = _smooth(rng, coords, size, 1e-4, (0.0, 5e-4))
        v = [torch.zeros_like(x) for x in coords]
        if k in ("adr", "batch"):
            # from rest, the prescribed rows displaced: the damping coefficient is
            # a sum of quotients by the velocities, and from an arbitrary field it
            # turns a change in the last bits of the forces into another path
            # within a few steps
            u = [torch.where(rows, x, torch.zeros_like(x)) for x in u]
    return u, v


def _history(c, seed, coords):
    """Displacement after and before the last increment, of a proportional loading with a
    small departure (what pd_warm_record sees along a real chain)."""
    rng = np.random.default_rng(seed + 1)
    u, _ = _fields(c, seed, coords)
    d = _smooth(rng, coords, max(float(x.max() - x.min()) for x in coords), 2e-9, (0.0, 0.0))
    return u, [a * (19.0 / 20.0) + b for a, b in zip(u, d)]


def _batch_table(c):
    return presets.batch_specimens(c["count"], 20240607, 5e-4, side=(c["low"], c["high"]))


def _prescribed(x, n_int):
    return torch.arange(x.numel(), device=x.device) >= n_int


def _net_inputs(rows, seed):
    """Feature rows and targets of a training batch (warm.py's scales)."""
    g = torch.Generator().manual_seed(seed)
    x = torch.zeros(rows, 16, dtype=torch.bfloat16)
    x[:, 0:2] = (torch.rand(rows, 2, generator=g) * 2.0 - 1.0).bfloat16()
    x[:, 2] = (1.0 / torch.randint(1, 60, (rows,), generator=g)).bfloat16()
    x[:, 3] = (torch.rand(rows, generator=g) < 0.01).bfloat16() * 0.4
    x[:, 4] = (torch.rand(rows, generator=g) < 0.03).bfloat16()
    x[:, 5:7] = (torch.randn(rows, 2, generator=g) * 0.7).bfloat16()
    x[:, 7] = (torch.rand(rows, generator=g) < 0.005).bfloat16() * 0.1
    t = torch.randn(rows, 2, generator=g) * 0.1
    p = init_params(seed)
    p[-258:-2] = np.random.default_rng(seed).standard_normal(256).astype(np.float32) * 0.1  # a trained output layer
    return x.to(DEVICE), t.to(DEVICE), p


# ---- prepare and run ----------------------------------------------------------------
def _views(eng, names):
    """The engine's own fields; each view keeps the engine, whose memory it shows."""
    out = {}
    for n in names:
        out[n] = eng.device_view(n)
        out[n].engine = eng
    return out


def prepare(case, seed):
    k = case["kind"]
    if k == "gradient":
        x, t, p = _net_inputs(case["rows"], seed)
        return dict(case=case, net=Net(case["rows"], p), x=x, t=t, grad=np.zeros(N_PARAMS, dtype=np.float32))
    if k == "batch":
        return _prepare_batch(case, seed)
    if k == "slab":
        return _prepare_slab(case, seed)
    p = _params(case)
    eng = Engine(p)
    _coords(eng, case)
    coords = [eng.device_view("X"), eng.device_view("Y")]
    u, v = _fields(case, seed, coords, _prescribed(coords[0], p.N_int))
    s = dict(case=case, eng=eng, u=u, v=v, load=_material(case)["load"])
    if k == "setup":
        return s
    _specimen(eng, case)
    if k == "verlet" and case["crack"]:
        # the traction of the benchmark on the top and bottom rows
        eng.set("BY", presets.traction_field(p, 12.0e6))
    if k == "predict":
        u, up = _history(case, seed, coords)
        s["net"] = Net.load(WEIGHTS, max_rows=65536)
        s["du"] = torch.zeros(4 * p.N_int, dtype=F64, device="cuda")
        _put(eng, ["UX", "UY"], u)
        eng.damage()
        before = torch.cat([a[: p.N_int] for a in up])
        record_history(eng, 19 * WARM_INC, WARM_INC, before, 0.98 * eng.device_view("DMG", p.N_int))
        eng.sync()
    return s


def _coords(eng, c):
    if _rows(c):
        eng.coord_plate_crack()
    else:
        eng.coord_plate()


def _specimen(eng, c):
    """Family to force layout of a plate, in the order of presets' set-ups."""
    eng.find_neighbor_gpu()
    if c["kind"] != "state2d":
        eng.surface_correct_gpu()
    eng.initial_state()
    if _crack(c):
        eng.set_crack_2d(*_crack(c))
    if c["kind"] == "state2d":
        eng.initial_weight()
    eng.prepare()


def _cylinder(c):
    m, s = _material(c), c["scale"]
    cyl = PDCylinder()
    cyl.rad, cyl.mass, cyl.height, cyl.v = 0.025 * s, 1.57, 0.05 * s, -32.0
    # closer than presets' 0.1 dx, so that the slab is hit in the first steps
    cyl.x, cyl.y, cyl.z = 0.0, 0.1 * s / 2.0 + cyl.height / 2.0 + 0.005 * m["dx"], 0.0
    cyl.vel[1] = cyl.v
    return cyl


def _prepare_slab(case, seed):
    model = PD_MODEL_STATE if case["state"] else PD_MODEL_BOND
    p, setup, _ = presets.build_kalthoff_winkler(scale=case["scale"], model=model, derive=derive_params,
                                                 coord_fn=coord_kw)
    eng = Engine(p)
    setup(eng)
    u, v = _fields(case, seed, [eng.device_view(n) for n in "XYZ"])
    return dict(case=case, eng=eng, u=u, v=v, load=0.0, cyl=_cylinder(case))


def _prepare_batch(case, seed):
    base = derive_params(2, PD_MODEL_BOND, PD_MODE_STATIC, 1.0, 1000, 5e-4, 0.0, 5e-4, 0.05, 0.05, 0.0, 192.0e9,
                         1.0 / 3.0, 8000.0, 0.04472)
    eng = Batch(base, _batch_table(case))
    coords = [eng.device_view("X"), eng.device_view("Y")]
    u, v = _fields(case, seed, coords, _prescribed(coords[0], eng.p.N_int))
    return dict(case=case, eng=eng, u=u, v=v, load=2.7e-8)


def _put(eng, names, values):
    for n, x in zip(names, values):
        eng.device_view(n).copy_(x)


def _zero(eng, names):
    for n in names:
        eng.device_view(n).zero_()


def run(state):
    c, k = state["case"], state["case"]["kind"]
    if k == "gradient":
        loss = C.c_float()
        check(lib().pd_mlp_grad(state["net"].h, state["x"].data_ptr(), state["t"].data_ptr(), c["rows"],
                                state["grad"].ctypes.data, C.byref(loss), None), None, "pd_mlp_grad")
        return dict(grad=state["grad"], loss=np.float32(loss.value))
    eng = state["eng"]
    if k == "predict":
        check(lib().pd_warm_predict(eng.ctx, state["net"].h, 20 * WARM_INC, WARM_INC, c["smooth"],
                                    state["du"].data_ptr(), eng.stream), eng.ctx, "pd_warm_predict")
        return dict(du=state["du"])
    if k == "setup":
        _specimen(eng, c)
        _put(eng, ["UX", "UY"], state["u"])
        eng.bond_force_gpu()
        # copies: the next specimen's family takes new bond arrays
        out = {n: eng.device_view(n).clone() for n in ("NN", "NL", "IDIST", "FAC", "SCR", "FAIL")}
        return dict(out, **_views(eng, ["FX", "FY"]))
    if k == "force":
        _put(eng, ["UX", "UY"], state["u"])
        eng.bond_force_gpu()
        return _views(eng, ["FX", "FY"])
    if k in ("adr", "batch"):
        _put(eng, ["UX", "UY"], state["u"])
        _zero(eng, ["VHX", "VHY", "FOX", "FOY"])
        eng.run_adr(0, c["steps"], state["load"])
        return _views(eng, ["UX", "UY", "VX", "VY", "FX", "FY"])
    if k == "verlet" and not c["crack"]:
        eng.initial_state()  # a new load case on the same specimen: every bond intact again
    if k == "slab":
        _put(eng, ["UX", "UY", "UZ", "VX", "VY", "VZ"], state["u"] + state["v"])
        _zero(eng, ["AX", "AY", "AZ"])
        eng.cylinder_init(state["cyl"])
        eng.run_explicit(c["steps"])
        cyl = eng.cylinder()
        out = _views(eng, ["UX", "UY", "UZ", "VX", "VY", "VZ", "FX", "FY", "FZ"])
        return dict(out, cylinder=np.array([*cyl.vel, *cyl.disp]))
    _put(eng, ["UX", "UY", "VX", "VY"], state["u"] + state["v"])
    _zero(eng, ["AX", "AY"])
    eng.run_explicit(c["steps"], load=state["load"], dmg_every=c["steps"])
    return _views(eng, ["UX", "UY", "VX", "VY", "FX", "FY", "DMG"])


# ---- work --------------------------------------------------------------------------
def _slab_shape(c):
    d = _material(c)["dx"]
    s = c["scale"]
    return [int((L - d / 2.0) / d + 1) for L in (0.2 * s, 0.1 * s, 0.009)]


def _size(c):
    """(nodes, directed bonds) of a case, the bonds counted as in the interior."""
    if c["kind"] == "slab":
        nx, ny, nz = _slab_shape(c)
        n = (nx + 1) * (ny + 1) * nz
        return n, 104 * n
    if c["kind"] == "batch":
        n = sum(s["nx"] * (s["ny"] + 6) for s in _batch_table(c))
        return n, 28 * n
    n = c["nx"] * (c["ny"] + (6 if _rows(c) else 0))
    return n, 28 * n


def work(case):
    k = case["kind"]
    if k == "gradient":
        m = case["rows"]
        return {"bytes": m * (32 + 8) + 4 * N_PARAMS * 2, "flops": 6 * m * (8 * 128 + 2 * 128 * 128 + 2 * 128)}
    n, b = _size(case)
    if k == "predict":
        # features and candidates per node; per smoothing pass both components of every neighbour
        sm = case["smooth"]
        return {"bytes": n * (7 * 8 + 4 * 8) + sm * (n * 32 + b * 4.125),
                "flops": 2 * n * (8 * 128 + 2 * 128 * 128 + 2 * 128) + sm * 2 * b}
    if k == "setup":
        # coordinates read, the bond arrays written: id, length, volume and surface factors, flag
        return {"bytes": n * 16 + b * (4 + 8 + 8 + 8 + 4), "flops": 60 * b}
    # per step and bond: neighbour id, coefficient and flag; per node the state read and written
    d3 = k == "slab"
    state = k == "state2d" or (d3 and case["state"])
    steps = case.get("steps", 1)
    per_bond = 16.125 if state else 12.125
    per_node = (72 if d3 else 48) + (40 if state else 0)
    return {"bytes": steps * (b * per_bond + n * per_node), "flops": steps * b * ((60 if state else 30) + 10 * d3)}


# ---- the model in 64 bits ------------------------------------------------------------
class Lattice:
    """Nodes on an integer grid with their families: neighbour ids nb[k][i]
    (i itself where offset k has no node), a mask has[k][i], reference vectors."""

    def __init__(self, cells, coords, dx):
        # cells: integer grid position per node and axis
        self.x, self.n, self.dim, self.dx = coords, len(cells[0]), len(cells), dx
        r = int(HORIZON)
        lo = [int(c.min()) - r for c in cells]
        shape = [int(c.max()) + r + 1 - l for c, l in zip(cells, lo)]
        grid = torch.full(shape, -1, dtype=torch.int64, device=DEVICE)
        me = torch.arange(self.n, device=DEVICE)
        at = [c - l for c, l in zip(cells, lo)]
        grid[tuple(at)] = me
        span = [torch.arange(-r, r + 1)] * self.dim
        offsets = torch.cartesian_prod(*span)
        offsets = offsets[((offsets**2).sum(1) > 0) & ((offsets**2).sum(1) < HORIZON**2)]
        self.nb, self.has = [], []
        for o in offsets.tolist():
            j = grid[tuple(a + b for a, b in zip(at, o))]
            self.has.append(j >= 0)
            self.nb.append(torch.where(j >= 0, j, me))

    def bonds(self):
        return range(len(self.nb))

    def xi(self, k):
        return [x[self.nb[k]] - x for x in self.x]

    def length(self, k):
        L = torch.sqrt(sum(d * d for d in self.xi(k)))
        return torch.where(self.has[k], L, torch.ones_like(L))

    def fac(self, k):
        L, d, h = self.length(k), HORIZON * self.dx, self.dx / 2.0
        f = torch.where(L <= d - h, torch.ones_like(L), torch.where(L <= d + h, (d + h - L) / self.dx, 0.0 * L))
        return f * self.has[k]

    def stretch(self, k, u):
        """(d per component, L, e = L - L0) of the bonds at displacement u."""
        xi, L0 = self.xi(k), self.length(k)
        eta = [a[self.nb[k]] - a for a in u]
        d = [a + b for a, b in zip(xi, eta)]
        L = torch.where(self.has[k], torch.sqrt(sum(a * a for a in d)), torch.ones_like(L0))
        e = sum(b * (2.0 * a + b) for a, b in zip(xi, eta)) / (L + L0)
        return d, L, e


def _plate_lattice(nx, ny, dx, rows):
    """Plate nodes row by row, then (rows) three rows above and three below."""
    i = torch.arange(nx, device=DEVICE)
    js = list(range(ny)) + ([ny, ny + 1, ny + 2, -1, -2, -3] if rows else [])
    j = torch.tensor(js, device=DEVICE).repeat_interleave(nx)
    i = i.repeat(len(js))
    x = (-nx / 2.0 + 0.5 + i.to(F64)) * dx
    y = (-ny / 2.0 + 0.5 + j.to(F64)) * dx
    return Lattice([i, j], [x, y], dx)


def _slab_lattice(c):
    m, rad = _material(c), 0.025 * c["scale"]
    dx = m["dx"]
    nx, ny, nz = _slab_shape(c)
    nx, ny = nx + 1, ny + 1
    k, j, i = torch.meshgrid(*(torch.arange(n, device=DEVICE) for n in (nz, ny, nx)), indexing="ij")
    i, j, k = i.reshape(-1), j.reshape(-1), k.reshape(-1)
    x = (-(nx - 1) / 2.0 + i.to(F64)) * dx
    y = (-(ny - 1) / 2.0 + j.to(F64)) * dx
    z = (-nz / 2.0 + 0.5 + k.to(F64)) * dx
    strip = ((x > -rad - 1.1 * dx) & (x < -rad + 0.1 * dx)) | ((x > rad - 0.1 * dx) & (x < rad + 1.1 * dx))
    keep = ~strip | (y < -1.0e-10)
    lat = Lattice([i[keep], j[keep], k[keep]], [x[keep], y[keep], z[keep]], dx)
    cut = []
    for b in lat.bonds():
        xc, yc = lat.x[0][lat.nb[b]], lat.x[1][lat.nb[b]]
        xi, yi = lat.x[0], lat.x[1]
        upper = (yc >= -1.0e-10) | (yi >= -1.0e-10)
        over = ((xc > -rad) & (xi < -rad)) | ((xi > -rad) & (xc < -rad))
        over |= ((xc > rad) & (xi < rad)) | ((xi > rad) & (xc < rad))
        cut.append(over & upper)
    return lat, cut


def _segment_cut(lat, free, crack):
    """Bonds of the free nodes that cross a crack segment."""
    length, lx, ly, theta = crack
    t = math.tan(theta)
    x, y = lat.x[0], lat.x[1]
    side = t * (x - lx) + (ly - y)
    off = side / math.sqrt(1.0 + t * t)
    along = torch.sqrt(((x - lx) ** 2 + (y - ly) ** 2 - off * off).clamp_min(0.0))
    near = along < length / 2.0
    return [near & near[lat.nb[k]] & (side * side[lat.nb[k]] <= 0.0) & free for k in lat.bonds()]


def _energy_factor(lat, k, a, bc, vol):
    """Strain energy density of the bonds under the test field u_a = 0.001 x_a."""
    u = [torch.zeros_like(x) for x in lat.x]
    u[a] = 0.001 * lat.x[a]
    _, _, e = lat.stretch(k, u)
    return torch.where(lat.has[k], 0.25 * bc * e * e / lat.length(k) * vol * lat.fac(k), torch.zeros_like(e))


def _surface(lat, bc, vol, sed):
    """Surface correction factor of every bond."""
    fn = []
    for a in range(lat.dim):
        fn.append(sed / sum(_energy_factor(lat, k, a, bc, vol) for k in lat.bonds()))
    out = []
    for k in lat.bonds():
        xi = [d.abs() for d in lat.xi(k)]
        sc = [(f + f[lat.nb[k]]) / 2.0 for f in fn]
        flat = torch.sqrt(xi[0] ** 2 + xi[1] ** 2)
        on_axis = flat < 1.0e-10
        flat = torch.where(on_axis, torch.ones_like(flat), flat)
        q = (xi[0] / flat / sc[0]) ** 2 + (xi[1] / flat / sc[1]) ** 2
        if lat.dim == 3:
            q = q + (xi[2] / lat.length(k) / sc[2]) ** 2
        s = 1.0 / torch.sqrt(q)
        out.append(torch.where(on_axis, sc[-1], s))
    return out


def _pmb(c, lat, E=None, s0=None):
    """Bond constants of a bond-based specimen: k of f = k e d / L, and s0."""
    m = _material(c)
    E = m["E"] if E is None else E
    d, dx, nu = HORIZON * m["dx"], m["dx"], m["nu"]
    vol = dx**3
    if lat.dim == 2:
        bc, sed = 6.0 * E / (math.pi * dx * d**3 * (1.0 - nu)), 0.5 * E / (1.0 - nu * nu) * 1e-6
    else:
        bc, sed = 6.0 * E / (math.pi * d**4 * (1.0 - 2.0 * nu)), 0.6 * E * 1e-6
    scr = _surface(lat, bc, vol, sed)
    k = [vol * lat.fac(b) * bc * scr[b] / lat.length(b) for b in lat.bonds()]
    mass = 0.25 * m["dt"] ** 2 * (math.pi * d * d * dx) * bc / dx * 5.0
    return dict(k=k, scr=scr, mass=mass, s0=m["s0"] if s0 is None else s0)


def _pmb_force(lat, P, alive, u, guard=None):
    """Force on every node; bonds past s0 break after contributing."""
    f = [torch.zeros_like(x) for x in lat.x]
    for b in lat.bonds():
        d, L, e = lat.stretch(b, u)
        t = torch.where(alive[b], P["k"][b] * e / L, torch.zeros_like(e))
        for a in range(lat.dim):
            f[a] += t * d[a]
        brk = e / lat.length(b) > P["s0"]
        alive[b] &= ~(brk if guard is None else brk & guard & guard[lat.nb[b]])
    return f


def _lps(c, lat):
    m = _material(c)
    E, nu, d = m["E"], m["nu"], HORIZON * m["dx"]
    vol, G = m["dx"] ** 3, 0.5 * E / (1.0 + nu)
    if lat.dim == 2:
        K, q = 0.5 * E / (1.0 - nu), (2.0 * nu - 1.0) / (nu - 1.0)
        a, b, th = q * (2.0 * K - 32.0 * G / 9.0), 8.0 * G, 2.0 * q
    else:
        K = E / (3.0 * (1.0 - 2.0 * nu))
        a, b, th = 3.0 * K - 5.0 * G, 15.0 * G, 3.0
    w = [torch.exp(-((lat.length(k) / d) ** 2)) * lat.fac(k) * vol for k in lat.bonds()]
    wm = sum(w[k] * lat.length(k) ** 2 for k in lat.bonds())
    return dict(w=w, m=wm, a=a, b=b, th=th, s0=m["s0"])


def _lps_force(lat, P, alive, u, guard=None):
    th = torch.zeros_like(lat.x[0])
    for k in lat.bonds():
        # the 2-D dilatation counts broken bonds too, the 3-D one does not
        on = lat.has[k] if lat.dim == 2 else alive[k]
        th += torch.where(on, P["th"] * P["w"][k] * lat.length(k) * lat.stretch(k, u)[2], torch.zeros_like(th))
    th = th / P["m"] / P["m"]
    f = [torch.zeros_like(x) for x in lat.x]
    im = 1.0 / P["m"]
    for k in lat.bonds():
        d, L, e = lat.stretch(k, u)
        j, L0 = lat.nb[k], lat.length(k)
        t = P["w"][k] * (P["a"] * L0 * (th + th[j]) + P["b"] * e * (im + im[j])) / L
        t = torch.where(alive[k], t, torch.zeros_like(t))
        for a in range(lat.dim):
            f[a] += t * d[a]
        brk = e / L0 > P["s0"]
        alive[k] &= ~(brk if guard is None else brk & guard & guard[j])
    return f


def _rows_move(u, n_int, nx, step):
    u[1][n_int:n_int + 3 * nx] += step
    u[1][n_int + 3 * nx:n_int + 6 * nx] -= step


def _adr(lat, force, u, mass, steps, move, free, groups=None, count=1):
    """ADR steps (kernel_cnn, cal_cn, kernel_integrate of the reference), one
    damping coefficient per group of nodes."""
    dt = 1.0
    vh, fo = [torch.zeros_like(x) for x in u], [torch.zeros_like(x) for x in u]
    v, f = [torch.zeros_like(x) for x in u], None
    g = torch.zeros(lat.n, dtype=torch.int64, device=DEVICE) if groups is None else groups
    move(u)
    for t in range(steps):
        f = [torch.where(free, x, torch.zeros_like(x)) for x in force(u)]
        num, den = torch.zeros_like(u[0]), torch.zeros_like(u[0])
        for a in range(len(u)):
            s = torch.where(vh[a] != 0.0, vh[a], torch.ones_like(vh[a]))
            num += torch.where(vh[a] != 0.0, -u[a] * u[a] * (f[a] / mass - fo[a] / mass) / (dt * s), 0.0 * s)
            den += u[a] * u[a]
        num = torch.zeros(count, dtype=F64, device=DEVICE).index_add_(0, g[free], num[free])
        den = torch.zeros(count, dtype=F64, device=DEVICE).index_add_(0, g[free], den[free])
        r = torch.where(den != 0.0, num / den, torch.zeros_like(num)).clamp_min(0.0)
        cn = 2.0 * torch.sqrt(r)
        cn = torch.where(cn > 2.0, torch.full_like(cn, 1.9), cn)[g]
        for a in range(len(u)):
            if t == 0:
                new = dt / mass * f[a] / 2.0
            else:
                new = ((2.0 - cn * dt) * vh[a] + 2.0 * dt / mass * f[a]) / (2.0 + cn * dt)
            new = torch.where(free, new, torch.zeros_like(new))
            v[a] = torch.where(free, 0.5 * (vh[a] + new), v[a])
            u[a] = u[a] + new * dt
            vh[a], fo[a] = new, f[a]
        if t + 1 < steps:
            move(u)
    return dict(UX=u[0], UY=u[1], VX=v[0], VY=v[1], FX=f[0], FY=f[1])


def _contact(c, lat, m, u, v, cyl):
    """Nodes inside the impactor moved to its surface; the reaction on it."""
    rad, half = cyl["rad"], cyl["height"] / 2.0
    p = [lat.x[a] + u[a] - cyl["pos"][a] - cyl["disp"][a] for a in range(3)]
    r = torch.sqrt(p[0] ** 2 + p[2] ** 2)
    hit = (r <= rad) & (p[1].abs() <= half)
    side = rad - r <= half - p[1].abs()
    to = [torch.where(side, p[0] / r * rad, p[0]), torch.where(side, p[1], torch.sign(p[1]) * half),
          torch.where(side, p[2] / r * rad, p[2])]
    force = []
    for a in range(3):
        new = torch.where(hit, cyl["pos"][a] + cyl["disp"][a] + to[a] - lat.x[a], u[a])
        vn = torch.where(hit, (new - u[a]) / m["dt"], v[a])
        force.append(torch.where(hit, -m["rho"] * (vn - v[a]) / m["dt"] * m["dx"] ** 3, torch.zeros_like(vn)).sum())
        u[a], v[a] = new, vn
    return force


def _verlet(c, lat, force, u, v, body, free, move=None, cyl=None):
    m = _material(c)
    dt = m["dt"]
    a = [torch.zeros_like(x) for x in u]

    def half():
        if move is not None:
            move(u)
        for k in range(lat.dim):
            v[k] = v[k] + torch.where(free, dt / 2.0 * a[k], 0.0 * a[k])
            u[k] = u[k] + torch.where(free, v[k] * dt, 0.0 * v[k])
        if cyl is not None:
            for k in range(3):
                cyl["vel"][k] = cyl["vel"][k] + dt / 2.0 * cyl["acc"][k]
                cyl["disp"][k] = cyl["disp"][k] + cyl["vel"][k] * dt

    half()
    for t in range(c["steps"]):
        f = [torch.where(free, x, torch.zeros_like(x)) for x in force(u)]
        if cyl is not None:
            reaction = _contact(c, lat, m, u, v, cyl)
        for k in range(lat.dim):
            a[k] = (f[k] + body[k]) / m["rho"]
            v[k] = v[k] + torch.where(free, dt / 2.0 * a[k], 0.0 * a[k])
        if cyl is not None:
            for k in range(3):
                cyl["acc"][k] = reaction[k] / cyl["mass"]
                cyl["vel"][k] = cyl["vel"][k] + dt / 2.0 * cyl["acc"][k]
        if t + 1 < c["steps"]:
            half()
    out = {}
    for name, field in (("U", u), ("V", v), ("F", f)):
        out.update({name + ax: x for ax, x in zip("XYZ", field)})
    return out


def _damage(lat, alive):
    every = sum(lat.fac(k) for k in lat.bonds())
    return 1.0 - sum(lat.fac(k) * alive[k] for k in lat.bonds()) / every


def _exact_net(p, x):
    """Layer inputs and outputs of the network in 64 bits (weights as the BF16
    operands the tensor cores take)."""
    w, at = [], 0
    for o, i in ((128, 8), (128, 128), (128, 128), (2, 128)):
        W = torch.from_numpy(p[at:at + o * i].reshape(o, i)).to(DEVICE).bfloat16().to(F64)
        b = torch.from_numpy(p[at + o * i:at + o * i + o]).to(DEVICE).to(F64)
        w.append((W.requires_grad_(), b.requires_grad_()))
        at += o * i + o
    h = x[:, :8].to(F64)
    for k, (W, b) in enumerate(w):
        z = h @ W.T + b
        h = torch.nn.functional.gelu(z) if k < 3 else z
    return h, w


def exact(case, seed):
    k = case["kind"]
    if k == "gradient":
        x, t, p = _net_inputs(case["rows"], seed)
        y, w = _exact_net(p, x)
        loss = ((y - t.to(F64)) ** 2).sum() / (2.0 * case["rows"])
        loss.backward()
        g = torch.cat([q.grad.reshape(-1) for layer in w for q in layer])
        return dict(grad=g, loss=loss.detach())
    if k == "batch":
        return _exact_batch(case, seed)
    m = _material(case)
    if k == "slab":
        lat, cut = _slab_lattice(case)
    else:
        lat = _plate_lattice(case["nx"], case["ny"], m["dx"], _rows(case))
    n_int = lat.n if k == "slab" else case["nx"] * case["ny"]
    free = torch.arange(lat.n, device=DEVICE) < n_int
    if k != "slab":
        cut = _segment_cut(lat, free, _crack(case)) if _crack(case) else [torch.zeros_like(free)] * len(lat.nb)
    alive = [h & ~q for h, q in zip(lat.has, cut)]
    u, v = _fields(case, seed, lat.x, ~free)
    zero = [torch.zeros_like(x) for x in lat.x]
    if k == "predict":
        return _exact_predict(case, seed, lat, alive, n_int)
    state = k == "state2d" or (k == "slab" and case["state"])
    P = _lps(case, lat) if state else _pmb(case, lat)
    guard = lat.x[1] >= -0.04 if k == "slab" else None
    law = _lps_force if state else _pmb_force

    def force(w):
        return law(lat, P, alive, w, guard)

    if k in ("force", "setup"):
        f = [torch.where(free, x, torch.zeros_like(x)) for x in force(u)]
        out = dict(FX=f[0], FY=f[1])
        if k == "setup":
            out.update(_csr(lat, P["scr"]), NN=None, NL=None, FAIL=None)
        return out

    def move(w):
        if m["load"]:
            _rows_move(w, n_int, case["nx"], m["load"] * m["dt"])

    if k == "adr":
        return _adr(lat, force, u, P["mass"], case["steps"], move, free)
    if k == "slab":
        q = _cylinder(case)
        cyl = dict(rad=q.rad, mass=q.mass, height=q.height, pos=[q.x, q.y, q.z], vel=[0.0, q.v, 0.0],
                   disp=[0.0] * 3, acc=[0.0] * 3)
        out = _verlet(case, lat, force, u, v, zero, free, cyl=cyl)
        out["cylinder"] = np.array([float(a) for a in [*cyl["vel"], *cyl["disp"]]])
        return out
    if k == "verlet" and case["crack"]:
        nx = case["nx"]
        zero[1][:nx] -= 12.0e6 / m["dx"]
        zero[1][(case["ny"] - 1) * nx:case["ny"] * nx] += 12.0e6 / m["dx"]
    out = _verlet(case, lat, force, u, v, zero, free, move if _rows(case) else None)
    out["DMG"] = torch.where(free, _damage(lat, alive), torch.zeros_like(u[0]))
    return out


def _csr(lat, scr):
    """Bond arrays in the family's order: rows by node, ascending neighbours."""
    nb = torch.stack([torch.where(h, j, torch.full_like(j, 1 << 40)) for h, j in zip(lat.has, lat.nb)], 1)
    nb, order = nb.sort(1)
    mask = nb < (1 << 40)
    out = {}
    for name, vals in (("IDIST", [lat.length(k) for k in lat.bonds()]), ("FAC", [lat.fac(k) for k in lat.bonds()]),
                       ("SCR", scr)):
        out[name] = torch.stack(vals, 1).gather(1, order)[mask]
    return out


def _exact_batch(case, seed):
    """All specimens as one graph: interiors from multiples of 32, then the
    moving rows of every specimen."""
    specs = _batch_table(case)
    dx = 5e-4
    starts, bstarts, n_int, n_bnd = [], [], 0, 0
    for s in specs:
        starts.append(n_int)
        bstarts.append(n_bnd)
        n_int += (s["nx"] * s["ny"] + 31) // 32 * 32
        n_bnd += 6 * s["nx"]
    n = n_int + n_bnd
    x = [torch.zeros(n, dtype=F64, device=DEVICE) for _ in range(2)]
    rows, lats = [], []
    for q, s in enumerate(specs):
        lat = _plate_lattice(s["nx"], s["ny"], dx, True)
        own = s["nx"] * s["ny"]
        r = torch.cat([starts[q] + torch.arange(own, device=DEVICE),
                       n_int + bstarts[q] + torch.arange(6 * s["nx"], device=DEVICE)])
        for a in range(2):
            x[a][r] = lat.x[a]
        rows.append(r)
        lats.append(lat)
    u, _ = _fields(case, seed, x, _prescribed(x[0], n_int))
    out = {f: torch.zeros(n, dtype=F64, device=DEVICE) for f in ("UX", "UY", "VX", "VY", "FX", "FY")}
    out["UX"], out["UY"] = u[0].clone(), u[1].clone()
    # one graph over the specimens' nodes, in their own order
    big = Lattice.__new__(Lattice)
    big.n, big.dim, big.dx = sum(l.n for l in lats), 2, dx
    big.x = [torch.cat([l.x[a] for l in lats]) for a in range(2)]
    base = np.cumsum([0] + [l.n for l in lats])
    big.nb = [torch.cat([l.nb[k] + int(b) for l, b in zip(lats, base)]) for k in lats[0].bonds()]
    big.has = [torch.cat([l.has[k] for l in lats]) for k in lats[0].bonds()]
    at = torch.cat(rows)
    free = at < n_int
    of = torch.cat([torch.full((l.n,), q, dtype=torch.int64, device=DEVICE) for q, l in enumerate(lats)])
    E = torch.tensor([s["emod"] for s in specs], dtype=F64, device=DEVICE)[of]
    s0 = torch.tensor([s["critical_s"] for s in specs], dtype=F64, device=DEVICE)[of]
    P = _pmb(dict(kind="adr", dx=dx), big, E, s0)
    alive = [h.clone() for h in big.has]
    for q, (l, s) in enumerate(zip(lats, specs)):
        if s["crack_len"] > 0.0:
            own = torch.arange(l.n, device=DEVICE) < s["nx"] * s["ny"]
            for k, cut in enumerate(_segment_cut(l, own, (s["crack_len"], 0.0, 0.0, s["crack_theta"]))):
                alive[k][int(base[q]):int(base[q + 1])] &= ~cut
    up = torch.cat([torch.cat([torch.zeros(s["nx"] * s["ny"]), torch.ones(3 * s["nx"]), -torch.ones(3 * s["nx"])])
                    for s in specs]).to(DEVICE).to(F64)

    def move(w):
        w[1] = w[1] + up * 2.7e-8

    r = _adr(big, lambda w: _pmb_force(big, P, alive, w), [a[at] for a in u], P["mass"], case["steps"], move, free,
             of, len(specs))
    for f in out:
        out[f][at] = r[f]
    return out


def _exact_predict(case, seed, lat, alive, n):
    u, up = _history(case, seed, lat.x)
    U, Up, inc = 20 * WARM_INC, 19 * WARM_INC, WARM_INC
    dmg = _damage(lat, alive)[:n]
    u, up = [a[:n] for a in u], [a[:n] for a in up]
    hist = [((a - b) - b * (inc / Up)) / Up for a, b in zip(u, up)]
    edge = lat.x[1][:n].abs() > case["ny"] * lat.dx / 2.0 - HORIZON * lat.dx
    one = torch.ones_like(u[0])
    feats = [u[0] / U, u[1] / U, one * (inc / U), dmg, edge.to(F64), hist[0] * 65536.0, hist[1] * 65536.0,
             dmg - 0.98 * dmg]
    x = torch.stack(feats, 1).bfloat16()
    p = np.fromfile(WEIGHTS, dtype=np.float32)
    net = torch.cat([_exact_net(p, q)[0].detach() for q in x.split(1 << 18)])
    corr = [U * net[:, a] / 65536.0 for a in range(2)]
    cnt = 1.0 + sum(a[:n].to(F64) for a in alive)
    for _ in range(case["smooth"]):
        out = []
        for q in corr:
            full = torch.zeros(lat.n, dtype=F64, device=DEVICE)  # prescribed rows count as zero
            full[:n] = q
            out.append((q + sum(full[lat.nb[k][:n]] * alive[k][:n] for k in lat.bonds())) / cnt)
        corr = out
    skip = [a * (inc / U) for a in u]
    du = [s + U * h + q for s, h, q in zip(skip, hist, corr)]
    return dict(du=torch.cat(du + skip))
